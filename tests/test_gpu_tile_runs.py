"""Contexts whose chunks are shorter than a group of four tiles (32, 64, 96 and 128 positions), so that a group holds the end of one chunk
and the start of the next, against the oracle: every position of a chunk's first tile inside a group, runs that end with a whole
and with a ragged tile, 1 to 8 tokens (16 query rows to a softmax warp: 6, 12, 18, 30, 48 rows). Tolerance: the path's 2e-3
(gpu_util.check_flips)."""
import pytest

import kv_oracle as ko
import kvdata
from gpu_util import attend_both, check_flips, fill_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spec,win", [("", 0), ("K*=5r,V*=6", 640)])
@pytest.mark.parametrize("L,T", [(1, 1), (33, 2), (129, 3), (160, 5), (640, 8), (641, 1), (705, 8), (833, 3), (1280, 2), (1281, 1), (1377, 5),
                                 (1664, 8), (1889, 3), (1920, 8), (1921, 1), (2177, 2), (2559, 5), (2560, 8)])
def test_groups_across_chunk_bounds(mk, torch_cuda, monkeypatch, spec, win, L, T):
    monkeypatch.setenv("MK_KV_ATTN", "tc")
    n = L - T
    if n < 0 or mk.cap_T(n, T) < T:
        T = 1
        n = L - T
    eng, orc = mk.Engine(1, L + 16, spec, win), ko.Cache(1, L + 16, spec, win)
    fill_both(torch_cuda, eng, orc, 0, 0, L, seed=L)
    Q = kvdata.q_rows(L, 0, n, T)
    O, Oref = attend_both(torch_cuda, eng, orc, 0, n, Q)
    check_flips(O, Oref, orc, 0, n, Q, (spec, L, T))
    eng.close()
