"""The gated group norm behind mamba2 and retention at every form of group: several heads, half a head, more columns than a warp
keeps in registers, padded heads (both: a block per group), against the plain float64 evaluation; and the same bits from a warp and
from a block per group."""
import numpy as np
import pytest

from tests import lm_models as lm
from tests.test_lm_gpu import both, driver, run, tokens_for

pytestmark = pytest.mark.gpu


# heads, head size, groups -> columns of a group: 2048 (beyond the 1024 of a warp), 1024, 512, 520, 32 (half a head), 60 (padded heads:
# 3 of 20), 24 (one head each)
@pytest.mark.parametrize("heads,vdim,groups", [(32, 64, 1), (32, 64, 2), (32, 64, 4), (13, 40, 1), (8, 64, 16), (6, 20, 2), (5, 24, 5)])
@both
def test_groups(cuda, tmp_path, heads, vdim, groups, f32):
    m = lm.Model(tmp_path, lm.config(48, 64, [lm.mamba2(heads, vdim, 16, 1, 2, groups)], [None]), heads + groups)
    tok = tokens_for(m, 70)
    want, bar = m.plain(tok)[0], m.bar(tok, f32)
    d = driver(m, f32)
    for slot, cuts in ((0, [70]), (1, [66, 1])):
        err = lm.rel_error(run(d, slot, tok, cuts), want)
        assert err.max() < bar, (cuts, int(err.argmax()), err.max(), bar)
    d.close()


# columns of a group 512, 1024, 520: rows whose groups are many enough for a warp each, and portions of 64 whose groups take a block
# each.  In 32-bit mode every other kernel computes a row alike in portions of whole chunks.
@pytest.mark.parametrize("heads,vdim,groups,rows", [(32, 64, 4, 192), (32, 64, 2, 384), (13, 40, 1, 640)])
@both
def test_a_warp_and_a_block_per_group(cuda, tmp_path, heads, vdim, groups, rows, f32):
    m = lm.Model(tmp_path, lm.config(48, 64, [lm.mamba2(heads, vdim, 16, 1, 2, groups)], [None]), heads + groups)
    tok = tokens_for(m, rows)
    want, bar = m.plain(tok)[0], m.bar(tok, f32)
    d = driver(m, f32, max_seq=rows, max_portion=rows)
    out = [run(d, 0, tok, [rows]), run(d, 1, tok, [64])]
    for y in out:
        err = lm.rel_error(y, want)
        assert err.max() < bar, (int(err.argmax()), err.max(), bar)
    if f32:
        assert np.array_equal(*out)
    d.close()
