"""Embedding and norms of prompts with rows enough for the many-rows instance (592 and more), at widths that fill its threads, that
end inside a thread's columns and that take several, and just below that number of rows, against the plain float64 evaluation."""
import pytest

from tests import lm_models as lm
from tests.test_lm_gpu import both, driver, run, tokens_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [512, 516, 2100])
@both
def test_many_rows(cuda, tmp_path, width, f32):
    m = lm.Model(tmp_path, lm.config(width, 64, [lm.retention(2, 8, 8, [0.9, 0.97])], [None]), width)
    tok = tokens_for(m, 600)
    want, bar = m.plain(tok)[0], m.bar(tok, f32)
    d = driver(m, f32, max_seq=640)
    for slot, cuts in ((0, [600]), (1, [592, 8])):
        err = lm.rel_error(run(d, slot, tok, cuts), want)
        assert err.max() < bar, (cuts, int(err.argmax()), err.max(), bar)
    d.close()
