"""The expanded form of latent attention (csrc/latent_attn.cu, prompt passes of LATENT_EXPAND_ROWS rows and more) against the oracle, with
one token that stands out: windows from one key to more than the prompt, at and next to the edges of the 64-key tiles, passes that wrap
the cache, that end inside a tile of 128 rows, and that follow passes of the other form.

Bar: that of the design's bfloat16 tests (0.12 of the logits' root mean square); rows that cannot see the token equal those of the
prompt without it bit for bit."""
import numpy as np
import pytest

import tivazen_models as M
from oracle import tivazen as T
from test_gpu_tivazen import TOL, make  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window,kv_rank,heads", [(1, 64, 2), (63, 64, 3), (64, 128, 1), (65, 64, 2), (200, 192, 2), (700, 64, 3), (700, 64, 16)])
def test_windows_and_cuts(make, window, kv_rank, heads):  # noqa: F811
    a = dict(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=kv_rank, scale=0.08)
    cfg = M.config([(M.attn(window=window, **a), M.dense(40)), (M.attn(window=min(window, 90), kv_from=0, **a), None)], width=64)
    w = M.plant_marker(cfg, M.random_weights(cfg, window))
    m = make(cfg, w, "bfloat16", prefill_rows=260, max_seq=600)
    n, at = 590, 210
    t = M.tokens(cfg, n)
    s = list(t)
    s[at] = M.MARK
    ref = T.forward(cfg, w, s)
    reach = at + (window - 1) + (min(window, 90) - 1)          # through both layers
    for cut in ([n], [200, 200, 190], [7, 193, 30, 260, 100]):
        out = []
        for seq in (t, s):
            m.reset()
            rows, p = [], 0
            for k in cut:
                rows.append(m.forward(seq[p:p + k], list(range(k))))
                p += k
            out.append(np.concatenate(rows))
        plain, marked = out
        assert M.error(marked, ref) < TOL["bfloat16"], cut
        assert np.array_equal(plain[:at], marked[:at]) and np.array_equal(plain[reach + 1:], marked[reach + 1:]), cut
