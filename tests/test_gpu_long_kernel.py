"""The kernel for long contexts (attn_ts_kernel) where it can go wrong: every compiled-in format pair, one and two sets of softmax warps with rows (6 ..
48 query rows, 24 and 30 on either side of the sets' bound), runs whose last tile holds 1, 31 or 32 positions or that end with a lone tile,
tiles of the q8_0 ring beside low-bit ones, spread over the SMs and item by item. Against the oracle with the path's 2e-3 (gpu_util)."""
import numpy as np
import pytest

import kv_oracle as ko
import kvdata
from gpu_util import TOL, attend_both, check_flips, fill_both

pytestmark = pytest.mark.gpu

SPECS = ["K*=5r,V*=6", "K*=5r,V*=5", "K*=6,V*=5"]


@pytest.fixture(autouse=True)
def tensor_core_kernel(monkeypatch):
    monkeypatch.setenv("MK_KV_ATTN", "tc")


@pytest.mark.parametrize("spec", SPECS)
@pytest.mark.parametrize("L,T", [(2561, 1), (2592, 4), (2719, 5), (2721, 2), (3208, 8), (4511, 3)])
def test_item_by_item(mk, torch_cuda, spec, L, T):
    """8 layers in one launch: 3 to 4 items a CTA, of chunks of 160 to 256 positions"""
    torch, layers, n = torch_cuda, 8, L - T
    eng, orc = mk.Engine(layers, n + 64, spec, 640), ko.Cache(layers, n + 64, spec, 640)
    for l in range(layers):
        fill_both(torch, eng, orc if l in (0, layers - 1) else None, l, 0, n, seed=70 + l)
    new = [kvdata.kv_rows(7, l, n, T) for l in range(layers)]
    K, V = (np.stack([r[w] for r in new]) for w in range(2))
    Q = np.stack([kvdata.q_rows(7, l, n, T) for l in range(layers)])
    O = torch.full((layers, T, 24, 256), float("nan"), dtype=torch.float32, device="cuda")
    eng.step_layers(n, *(torch.from_numpy(x).cuda() for x in (K, V, Q)), O)
    eng.sync()
    assert torch.isfinite(O).all()
    for l in (0, layers - 1):
        orc.append(l, n, K[l], V[l])
        check_flips(O[l].cpu().numpy(), orc.attend(l, n, Q[l]), orc, l, n, Q[l], (spec, L, T, l))
    eng.close()


@pytest.mark.parametrize("spec,L,T", [(SPECS[0], 23681, 1), (SPECS[1], 23712, 4), (SPECS[2], 24001, 5), (SPECS[0], 24319, 8)])
def test_spread(mk, torch_cuda, spec, L, T):
    """one layer: the first lengths of six groups a CTA and the last of their 640"""
    n = L - T
    eng, orc = mk.Engine(1, L + 16, spec, 2048), ko.Cache(1, L + 16, spec, 2048)
    fill_both(torch_cuda, eng, orc, 0, 0, L, seed=L, chunk=8192)
    O, Oref = attend_both(torch_cuda, eng, orc, 0, n, kvdata.q_rows(L, 0, n, T))
    assert np.isfinite(O).all() and np.abs(O - Oref).max() <= TOL
    eng.close()


def test_expired_wait_of_the_spread_instance(mk, torch_cuda):
    """zero rounds: the launch ends with an error, the next one with the default limits gives the same bits as before"""
    torch, n, T = torch_cuda, 24000, 8
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    rows = lambda m, h: torch.randn((m, h, 256), generator=g, device="cuda").half()
    K, V, Q = rows(n + T, 4), rows(n + T, 4), rows(T, 24)
    eng = mk.Engine(1, n + 64, SPECS[0], 2048)

    def call():
        eng.append(0, 0, K, V)
        O = torch.zeros((T, 24, 256), dtype=torch.float32, device="cuda")
        eng.attend(0, n, Q, O)
        eng.sync()
        return O

    good = call()
    for limits in (None, (20, 20, 20), (20, 100, 100)):
        gave_up = False
        try:
            eng.wait_limits(*limits) if limits else eng.wait_limits_expire_now()
            O = call()
        except mk.EngineError as e:
            assert "gave up waiting" in str(e)
            gave_up = True
        finally:
            eng.wait_limits()
        assert gave_up or limits
        assert torch.equal(call() if gave_up else O, good)
    eng.close()
