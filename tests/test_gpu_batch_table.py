"""step_batch with as many jobs as travel with the append launch (32), one fewer and one more (uploaded), and a single one: every sequence's
output is what a call of its own gives (same kernel, same partition: 1e-5), its rows are the same bytes."""
import numpy as np
import pytest

import kvdata

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("njobs", [1, 31, 32, 33, 40])
def test_batch_equals_single_calls(mk, torch_cuda, monkeypatch, njobs):
    monkeypatch.setenv("MK_KV_ATTN", "tc")
    torch = torch_cuda
    spec, win = "K*=5r,V*=6", 640
    ns = [(37 * j * j + 5 * j) % 1500 for j in range(njobs)]
    Ts = [min(1 + j % 8, mk.cap_T(n, 8)) for j, n in enumerate(ns)]
    engs = [mk.Engine(1, 64, spec, win) for _ in range(2)]
    for e in engs:
        e.slots_open(njobs, 1600)
        e.reserve_batch(njobs)
        for j, n in enumerate(ns):
            if n:
                K, V = kvdata.kv_rows(200 + j, 0, 0, n)
                e.append(0, 0, torch.from_numpy(K).cuda(), torch.from_numpy(V).cuda(), seq=j)
                e.sync()
    K, V = (torch.from_numpy(np.concatenate([kvdata.kv_rows(300 + j, 0, n, T)[w] for j, (n, T) in enumerate(zip(ns, Ts))])).cuda() for w in (0, 1))
    Q = torch.from_numpy(np.concatenate([kvdata.q_rows(300 + j, 0, n, T) for j, (n, T) in enumerate(zip(ns, Ts))])).cuda()
    O = [torch.full((sum(Ts), 24, 256), float("nan"), dtype=torch.float32, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(2):  # (a second call writes the table again)
        engs[0].step_batch(list(range(njobs)), 0, ns, Ts, K, V, Q, O[0])
    row = 0
    for j, (n, T) in enumerate(zip(ns, Ts)):
        engs[1].step(0, n, K[row:row + T], V[row:row + T], Q[row:row + T], O[1][row:row + T], seq=j)
        row += T
    for e in engs:
        e.sync()
    assert torch.isfinite(O[0]).all()
    assert float((O[0] - O[1]).abs().max()) <= 1e-5 * float(O[1].abs().max())
    for j, (n, T) in enumerate(zip(ns, Ts)):
        for w in range(2):
            for p in (n, n + T - 1):
                (a, sa), (b, sb) = (e.read_row(0, w, j % 4, p, seq=j) for e in engs)
                assert np.array_equal(a, b) and np.array_equal(sa, sb)
    for e in engs:
        e.close()
