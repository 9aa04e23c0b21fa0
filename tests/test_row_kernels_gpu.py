"""Embedding and norms of prompts with rows enough for the instance that does four threads' work in one, at widths that fill its
threads and that end inside a thread's columns, and at a width that has no such instance, against the plain float64 evaluation;
and the bits of a row, which do not depend on how many rows there are."""
import numpy as np
import pytest

from tests import lm_models as lm
from tests.test_lm_gpu import both, driver, run, tokens_for

pytestmark = pytest.mark.gpu


def model(tmp_path, width):
    return lm.Model(tmp_path, lm.config(width, 64, [lm.retention(2, 8, 8, [0.9, 0.97])], [None]), width)


@pytest.mark.parametrize("width,rows", [(512, 600), (512, 1800), (516, 600), (1000, 960), (2048, 600), (2100, 600)])
@both
def test_many_rows(cuda, tmp_path, width, rows, f32):
    m = model(tmp_path, width)
    tok = tokens_for(m, rows)
    want, bar = m.plain(tok)[0], m.bar(tok, f32)
    d = driver(m, f32, max_seq=rows, max_portion=rows)
    for slot, cuts in ((0, [rows]), (1, [rows - 8, 8])):
        err = lm.rel_error(run(d, slot, tok, cuts), want)
        assert err.max() < bar, (cuts, int(err.argmax()), err.max(), bar)
    d.close()


# in 32-bit mode every other kernel computes a row alike in any portion
@pytest.mark.parametrize("width,rows", [(2048, 640), (1000, 960)])
def test_a_row_has_the_same_bits_in_any_portion(cuda, tmp_path, width, rows):
    m = model(tmp_path, width)
    tok = tokens_for(m, rows)
    d = driver(m, True, max_seq=rows, max_portion=rows)
    assert np.array_equal(run(d, 0, tok, [rows]), run(d, 1, tok, [320]))
    d.close()
