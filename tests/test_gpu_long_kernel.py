"""The kernel for long runs of 5-bit keys (attn_ts_kernel: 16 groups and more a CTA, item by item) where it can go wrong: either compiled-in
value format, one and two sets of softmax warps with rows (6, 24, 30 and 48 query rows: 24 is a set's bound), a last chunk of 1, 31 and 32 positions beside the whole
ones, a last group of one and of three tiles, tiles of the q8_0 ring beside low-bit ones, more items than CTAs and fewer, a position range. Against the oracle
with the path's 2e-3 (gpu_util.TOL)."""
import numpy as np
import pytest

import kv_oracle as ko
import kvdata
from gpu_util import TOL, fill_both

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def tensor_core_kernel(monkeypatch):
    monkeypatch.setenv("MK_KV_ATTN", "tc")


def new_rows(layers, n, T):
    new = [kvdata.kv_rows(7, l, n, T) for l in range(layers)]
    return np.stack([r[0] for r in new]), np.stack([r[1] for r in new]), np.stack([kvdata.q_rows(7, l, n, T) for l in range(layers)])


# (chunks of 1,024 positions up to 20,480, of 1,056 up to 21,120; 80 or 76 items a layer)
@pytest.mark.parametrize("spec,layers,L,T", [("K*=5r,V*=6", 2, 19841, 1), ("K*=5r,V*=5", 4, 20063, 4), ("K*=5r,V*=6", 4, 20448, 5), ("K*=5r,V*=5", 2, 20481, 1),
                                             ("K*=5r,V*=6", 6, 20577, 8), ("K*=5r,V*=6", 2, 21087, 3)])
def test_layers(mk, torch_cuda, spec, layers, L, T):
    torch, n = torch_cuda, L - T
    eng, orc = mk.Engine(layers, n + 64, spec, 2048), ko.Cache(layers, n + 64, spec, 2048)
    for l in range(layers):
        fill_both(torch, eng, orc if l in (0, layers - 1) else None, l, 0, n, seed=70 + l, chunk=8192)
    K, V, Q = new_rows(layers, n, T)
    O = torch.full((layers, T, 24, 256), float("nan"), dtype=torch.float32, device="cuda")
    eng.step_layers(n, *(torch.from_numpy(x).cuda() for x in (K, V, Q)), O)
    eng.sync()
    assert torch.isfinite(O).all()
    for l in (0, layers - 1):
        orc.append(l, n, K[l], V[l])
        assert np.abs(O[l].cpu().numpy() - orc.attend(l, n, Q[l])).max() <= TOL, (spec, L, T, l)
    eng.close()


@pytest.mark.parametrize("T", [1, 5, 8])
def test_no_allocation_entry(mk, torch_cuda, T):
    """80 items of 16 groups, a CTA each"""
    spec, n = "K*=5r,V*=6", 40400
    eng, orc = mk.Engine(1, n + 64, spec, 2048), ko.Cache(1, n + 64, spec, 2048)
    fill_both(torch_cuda, eng, orc, 0, 0, n + T, seed=5, chunk=8192)
    Q = kvdata.q_rows(9, 0, n, T)
    O = torch_cuda.zeros((T, 24, 256), dtype=torch_cuda.float32, device="cuda")
    eng.attend_static(0, n, torch_cuda.from_numpy(Q).cuda(), O)
    eng.sync()
    assert np.abs(O.cpu().numpy() - orc.attend(0, n, Q)).max() <= TOL
    eng.close()


def test_expired_waits(mk, torch_cuda):
    """zero rounds: the launch ends with an error; short limits: it may. The next one with the default limits gives the same bits as before."""
    torch, layers, n, T = torch_cuda, 4, 20000, 8
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    rows = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    K, V, Kt, Vt, Q = rows(n, 4, 256), rows(n, 4, 256), rows(layers, T, 4, 256), rows(layers, T, 4, 256), rows(layers, T, 24, 256)
    eng = mk.Engine(layers, n + 64, "K*=5r,V*=6", 2048)

    def call(limits):
        for l in range(layers):
            eng.append(l, 0, K, V)
        eng.sync()
        O = torch.zeros((layers, T, 24, 256), dtype=torch.float32, device="cuda")
        try:
            if limits is not None:
                eng.wait_limits(*limits) if limits else eng.wait_limits_expire_now()
            eng.step_layers(n, Kt, Vt, Q, O)
            eng.sync()
        except mk.EngineError as e:
            assert "gave up waiting" in str(e)
            return None
        finally:
            eng.wait_limits()
        return O

    good = call(None)
    for limits in ((), (20, 2, 2), (20, 20, 20), (20, 100, 100), (100, 100, 100)):
        O = call(limits)
        assert O is None or limits
        assert torch.equal(call(None) if O is None else O, good)
    eng.close()
