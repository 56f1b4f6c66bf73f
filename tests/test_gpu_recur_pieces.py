"""Prompts through the chunk scan (csrc/recurrence_chunk.cu) by the width of a CTA's state columns: few heads take 16 (delta rule) or 32
(state space), many heads 32 or 64; keys within and beyond 128, value sizes that are and are not whole pieces, and a second pass that
starts from the state of the first.

Bar: that of the design's own tests for either activation type."""
import numpy as np
import pytest

import fomalix_models as M
from oracle import fomalix as F
from test_gpu_fomalix import DTYPES, TOL, make  # noqa: F401

pytestmark = pytest.mark.gpu

MIXERS = {
    "delta_narrow": M.delta(heads=4, kv_heads=2, dim=128, vdim=72), "delta_narrow_wide_keys": M.delta(heads=2, kv_heads=1, dim=160, vdim=48),
    "delta_wide": M.delta(heads=40, kv_heads=20, dim=32, vdim=64), "delta_wide_wide_keys": M.delta(heads=76, kv_heads=2, dim=144, vdim=32),
    "space_narrow": M.mamba(heads=6, groups=2, state=64, vdim=80, norm_groups=1), "space_wide": M.mamba(heads=80, groups=2, state=32, vdim=64, norm_groups=1),
    "space_narrow_wide_keys": M.mamba(heads=4, groups=1, state=200, vdim=33, norm_groups=1), "space_wide_wide_keys": M.mamba(heads=76, groups=1, state=144, vdim=32, norm_groups=1)}


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("name", list(MIXERS))
def test_prompt_in_two_passes(make, name, dtype):  # noqa: F811
    cfg = M.config([(MIXERS[name], None)], width=64)
    w = M.random_weights(cfg, 3)
    m = make(cfg, w, dtype, prefill_rows=140, max_seq=256)
    t = M.tokens(cfg, 210, 5)
    got = np.concatenate([m.forward(t[:133], list(range(133))), m.forward(t[133:], list(range(77)))])
    assert M.error(got, F.forward(cfg, w, t)) < TOL[dtype]
