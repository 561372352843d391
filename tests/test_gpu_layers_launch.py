"""A decode step's layers in one attention launch (the tensor-core kernel's batch mode) against the oracle, at the partition's edges:
one chunk, short last chunks, chunks of 1, 2 and 3 groups of 128 positions, the first length past each, mixed formats per layer; and
the same for a position range whose cuts fall inside chunks. Tolerance: the path's 2e-3 (gpu_util.check_flips)."""
import subprocess

import numpy as np
import pytest

import kv_oracle as ko
import kvdata
import test_plan_cpu
from gpu_util import check_flips, fill_both

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def tensor_core_kernel(monkeypatch):
    monkeypatch.setenv("MK_KV_ATTN", "tc")  # (the mma.sync kernel has no such mode)


def rows(layers, seed, n, T):
    K = np.stack([kvdata.kv_rows(seed, l, n, T)[0] for l in range(layers)])
    V = np.stack([kvdata.kv_rows(seed, l, n, T)[1] for l in range(layers)])
    return K, V, np.stack([kvdata.q_rows(seed, l, n, T) for l in range(layers)])


@pytest.mark.parametrize("spec,win,n,T,layers", [
    ("", 0, 0, 1, 2), ("", 0, 31, 2, 3), ("K*=5r,V*=6", 2048, 640, 8, 2), ("K*=6,V*=5", 640, 2552, 8, 5), ("K*=5r,V*=5", 2048, 2560, 5, 3),
    ("K*=5r,V*=6", 2048, 5119, 1, 2), ("K*=5r,V*=6,K1=8,V0=4r,*2=7", 640, 5127, 4, 6), ("K*=5r,V*=6", 2048, 7003, 3, 16)])
def test_layers_in_one_launch_match_oracle(mk, torch_cuda, spec, win, n, T, layers):
    torch = torch_cuda
    spill = win == 640  # (rows then go to their main format when they leave the window: launches of their own)
    eng, orc = mk.Engine(layers, n + 64, spec, win, spill=spill), ko.Cache(layers, n + 64, spec, win)
    for l in range(layers):
        if n:
            fill_both(torch, eng, orc, l, 0, n, seed=40 + l)
    eng.sync()
    K, V, Q = rows(layers, 5, n, T)
    O = torch.full((layers, T, 24, 256), float("nan"), dtype=torch.float32, device="cuda")
    before = eng.launches()
    eng.step_layers(n, *(torch.from_numpy(x).cuda() for x in (K, V, Q)), O)
    assert spill or eng.launches() - before == 3  # append, attention, merge
    eng.sync()
    for l in range(layers):
        orc.append(l, n, K[l], V[l])
        if l in (0, 1, layers - 1):
            check_flips(O[l].cpu().numpy(), orc.attend(l, n, Q[l]), orc, l, n, Q[l], (spec, n, T, l))
    eng.close()


def test_ranges_in_one_launch_match_oracle(mk, torch_cuda):
    """8 layers of a 9,003-position sequence cut at 32-position boundaries inside chunks: three ranges, merged"""
    torch = torch_cuda
    spec, win, n, T, layers, cuts = "K*=5r,V*=6", 2048, 9003, 5, 8, [0, 1056, 6432, 9056]
    orc = ko.Cache(layers, n + 64, spec, win)
    engs = [mk.Engine(layers, b - a + 64, spec, win) for a, b in zip(cuts, cuts[1:])]
    for a, eng in zip(cuts, engs):
        eng.set_base(a)
    for l in range(layers):
        Kl, Vl = kvdata.kv_rows(60 + l, l, 0, n)
        orc.append(l, 0, Kl, Vl)
        for a, b, eng in zip(cuts, cuts[1:], engs):
            b = min(b, n)
            eng.append(l, a, torch.from_numpy(Kl[a:b]).cuda(), torch.from_numpy(Vl[a:b]).cuda())
    K, V, Q = rows(layers, 6, n, T)
    Kd, Vd, Qd = (torch.from_numpy(x).cuda() for x in (K, V, Q))
    parts = torch.zeros((3, layers, 4, 48, 256), dtype=torch.float32, device="cuda")
    mls = torch.zeros((3, layers, 4, 48, 2), dtype=torch.float32, device="cuda")
    for r, (a, b, eng) in enumerate(zip(cuts, cuts[1:], engs)):
        before = eng.launches()
        eng.step_layers_partial(n, Kd, Vd, Qd, a, b, a, b, parts[r], mls[r])
        assert eng.launches() - before == 3
        eng.sync()
    O = torch.empty((layers, T, 24, 256), dtype=torch.float32, device="cuda")
    engs[0].combine_layers(T, 3, parts, mls, O)
    engs[0].sync()
    for l in range(layers):
        orc.append(l, n, K[l], V[l])
        if l in (0, layers - 1):
            assert np.abs(O[l].cpu().numpy() - orc.attend(l, n, Q[l])).max() <= 2e-3
    for eng in engs:
        eng.close()


@pytest.mark.parametrize("n", [31, 32, 33, 638, 1022, 1023, 1024, 1025, 1727, 1728, 1729, 2175, 2176])
def test_chunks_that_end_beside_the_new_tokens(mk, torch_cuda, n):
    """chunks of 32, 64, 96 and 128 positions whose last position is the first new token, the one before it or a later one: what a row
    must not see there differs by token in the first and last case only. Every entry that runs such chunks."""
    torch = torch_cuda
    spec, win, T = "K*=5r,V*=6", 2048, min(8, ko.att_cap_T(n, 8))
    eng, orc = mk.Engine(2, n + 64, spec, win), ko.Cache(2, n + 64, spec, win)
    for l in range(2):
        fill_both(torch, eng, orc, l, 0, n, seed=70 + l)
    K, V, Q = rows(2, 7, n, T)
    Qd = torch.from_numpy(Q).cuda()
    O = torch.full((3, 2, T, 24, 256), float("nan"), dtype=torch.float32, device="cuda")
    eng.step_layers(n, torch.from_numpy(K).cuda(), torch.from_numpy(V).cuda(), Qd, O[0])
    for l in range(2):
        eng.attend(l, n, Qd[l], O[1, l])
        eng.attend_static(l, n, Qd[l], O[2, l])
    eng.sync()
    assert torch.equal(O[0], O[1])  # up to 2,560 positions the one launch gives the per-layer calls' bits
    for l in range(2):
        orc.append(l, n, K[l], V[l])
        Oref = orc.attend(l, n, Q[l])
        for e in range(3):
            check_flips(O[e, l].cpu().numpy(), Oref, orc, l, n, Q[l], (n, T, l, e))
    eng.close()


def test_scratch_of_the_one_launch_step_is_taken_where_it_can_run(mk, torch_cuda, monkeypatch):
    """partials for all layers at once (80 slots of 48 x 258 floats a layer) only in an engine whose steps can be one launch"""
    torch = torch_cuda
    held = {}
    for kernel, layers in (("fast", 16), ("tc", 1), ("tc", 16)):
        monkeypatch.setenv("MK_KV_ATTN", kernel)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        eng = mk.Engine(layers, 64)
        held[kernel, layers] = before - torch.cuda.mem_get_info()[0]
        eng.close()
    partials, rows = 16 * 80 * 48 * 258 * 4, 32 << 20
    assert held["tc", 16] >= partials - (4 << 20) and held["fast", 16] < rows and held["tc", 1] < rows, held


@pytest.mark.parametrize("n,layers", [(1000, 1), (3000, 8)])
def test_tracing_changes_neither_launches_nor_results(mk, torch_cuda, monkeypatch, n, layers):
    torch = torch_cuda
    K, V, Q = (torch.from_numpy(x).cuda() for x in rows(layers, 8, n, 3))
    got = []
    for traced in (False, True):
        if traced:
            monkeypatch.setenv("MK_KV_PROFILE", "1")
        eng = mk.Engine(layers, n + 64, "K*=5r,V*=6", 2048)
        for l in range(layers):
            fill_both(torch, eng, None, l, 0, n, seed=90 + l)
        O = torch.zeros((layers, 3, 24, 256), dtype=torch.float32, device="cuda")
        before = eng.launches()
        eng.step_layers(n, K, V, Q, O)
        eng.sync()
        got.append((eng.launches() - before, O.cpu().numpy(), eng.profile() is not None))
        eng.close()
    assert got[0][0] == got[1][0] == 3 and np.array_equal(got[0][1], got[1][1]) and (got[0][2], got[1][2]) == (False, True)


@pytest.mark.parametrize("o_stride", [0, 24 * 256, 24 * 256 + 64])
def test_layers_whose_outputs_overlap_keep_their_order(mk, torch_cuda, o_stride):
    """an output stride of less than a layer's rows: layer after layer, the last writer's values stay"""
    torch = torch_cuda
    n, T, layers = 1500, 2, 3
    eng = mk.Engine(layers, n + 64, "K*=5r,V*=6", 2048)
    for l in range(layers):
        fill_both(torch, eng, None, l, 0, n, seed=95 + l)
    K, V, Q = (torch.from_numpy(x).cuda() for x in rows(layers, 9, n, T))
    want = torch.zeros((layers - 1) * o_stride + T * 24 * 256, dtype=torch.float32, device="cuda")
    one = torch.zeros((T, 24, 256), dtype=torch.float32, device="cuda")
    for l in range(layers):
        eng.step(l, n, K[l], V[l], Q[l], one)
        eng.sync()
        want[l * o_stride:l * o_stride + T * 24 * 256] = one.view(-1)
    for _ in range(5):
        got = torch.zeros_like(want)
        eng.step_layers(n, K, V, Q, got.as_strided((layers, T, 24, 256), (o_stride, 24 * 256, 256, 1)))
        eng.sync()
        assert torch.equal(got, want)
    eng.close()


def test_long_ranges_are_cut_into_even_items(mk, torch_cuda, tmp_path):
    """16 layers of a 45,000-position sequence on two ranges, cut into even pieces (the first range ends inside a chunk, the second holds the
    window and the new rows). Against the oracle with the chunks, whose P is rounded against other maxima, the path's 2e-3; the oracle with
    the same pieces must be at least four times nearer (there P differs only where the last bits of a score turn its rounding, a
    few values in a thousand against all)."""
    torch = torch_cuda
    plan = test_plan_cpu.build(tmp_path)
    spec, win, n, T, layers, cuts = "K*=5r,V*=6", 2048, 45003, 3, 16, [0, 23008, 45056]
    used = (0, layers - 1)  # (the layers with rows of their own; the others share layer 0's)
    orc = ko.Cache(2, n + 64, spec, win)
    engs = [mk.Engine(layers, b - a + 64, spec, win) for a, b in zip(cuts, cuts[1:])]
    for a, eng in zip(cuts, engs):
        eng.set_base(a)
    for i, l in enumerate(used):
        Kl, Vl = kvdata.kv_rows(80 + i, 0, 0, n)
        orc.append(i, 0, Kl, Vl)
        for a, b, eng in zip(cuts, cuts[1:], engs):
            b = min(b, n)
            for m in range(layers) if i == 0 else [l]:
                eng.append(m, a, torch.from_numpy(Kl[a:b]).cuda(), torch.from_numpy(Vl[a:b]).cuda())
            eng.sync()
    K, V, Q = rows(layers, 6, n, T)
    Kd, Vd, Qd = (torch.from_numpy(x).cuda() for x in (K, V, Q))
    parts = torch.zeros((2, layers, 4, 48, 256), dtype=torch.float32, device="cuda")
    mls = torch.zeros((2, layers, 4, 48, 2), dtype=torch.float32, device="cuda")
    for r, (a, b, eng) in enumerate(zip(cuts, cuts[1:], engs)):
        before = eng.launches()
        eng.step_layers_partial(n, Kd, Vd, Qd, a, b, a, b, parts[r], mls[r])
        assert eng.launches() - before == 3
        eng.sync()
    O = torch.empty((layers, T, 24, 256), dtype=torch.float32, device="cuda")
    engs[0].combine_layers(T, 2, parts, mls, O)
    engs[0].sync()
    bounds = []
    for a, b in zip(cuts, cuts[1:]):
        p = int(subprocess.run([plan] + [str(x) for x in (n, T, a, b, layers)], capture_output=True, text=True, check=True).stdout)
        assert p < ko.attn_dims(n + T)[1]
        bounds += [a] + list(range((a // p + 1) * p, min(b, n + T), p))
    for i, l in enumerate(used):
        orc.append(i, n, K[l], V[l])
        got, chunks, pieces = O[l].cpu().numpy(), orc.attend(i, n, Q[l]), orc.attend_pieces(i, n, Q[l], bounds[1:])
        assert np.abs(got - chunks).max() <= 2e-3
        assert np.linalg.norm(got - pieces) <= np.linalg.norm(got - chunks) / 4
    for eng in engs:
        eng.close()


@pytest.mark.parametrize("n,lo,hi", [(230009, 196608, 262144), (262136, 98304, 131072), (262136, 120000, 130016)])
def test_pieces_of_a_range_are_those_of_every_call(mk, torch_cuda, n, lo, hi):
    """A range's partial must not depend on how many layers or tokens share the call: 16 layers in the one launch, 2 layers and 1 layer in the
    spread mode, 8 tokens and 1, over the same rows, 1e-5 (a P rounded against another maximum moves the output by 2e-5 .. 4e-5); and
    the layers of a call, given the same rows, the same bits. The context's end, with the new rows, an inner range and one that lies in a single chunk."""
    torch = torch_cuda
    layers, T, end = 16, 8, min(hi, n)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    scale = torch.rand((4, 256), generator=g, device="cuda") * 1.5 + 0.5
    rows = lambda m, h=4: torch.randn((m, h, 256), generator=g, device="cuda")
    eng = mk.Engine(layers, hi - lo + 64, "K*=5r,V*=6", 2048)
    eng.set_base(lo)
    for a in range(lo, end, 16384):
        m = min(16384, end - a)
        K, V = ((rows(m) * scale).half() for _ in range(2))
        for l in range(layers):
            eng.append(l, a, K, V)
    K, V = ((rows(T) * scale).half().expand(layers, T, 4, 256).contiguous() for _ in range(2))
    Q = rows(T, 24).half().expand(layers, T, 24, 256).contiguous()

    def call(nlayers, tokens):
        part = torch.zeros((nlayers, 4, 48, 256), dtype=torch.float32, device="cuda")
        ml = torch.zeros((nlayers, 4, 48, 2), dtype=torch.float32, device="cuda")
        O = torch.zeros((nlayers, tokens, 24, 256), dtype=torch.float32, device="cuda")
        eng.step_layers_partial(n, *(x[:nlayers, :tokens].contiguous() for x in (K, V, Q)), lo, hi, lo, hi, part, ml)
        eng.combine_layers(tokens, 1, part, ml, O)
        eng.sync()
        return O

    want = call(layers, T)
    for l in range(1, layers):
        assert torch.equal(want[l], want[0]), l
    for nlayers, tokens in ((2, T), (1, T), (layers, 1), (2, 1), (1, 1)):
        got = call(nlayers, tokens)
        rel = float((got[0] - want[0, :tokens]).norm() / want[0, :tokens].norm())
        assert rel <= 1e-5, (nlayers, tokens, rel)
    eng.close()


@pytest.mark.parametrize("n", [3004, 3580, 4157, 4733, 5112, 5121])
def test_tokens_of_a_call_do_not_change_its_mode(mk, torch_cuda, n):
    """one layer just below and at the lengths where the number of a chunk's groups or of the launch's items changes: a 1-token and an 8-token
    call take the same launches, and the first token's output is the same up to the order of fp32 sums"""
    torch = torch_cuda
    eng = mk.Engine(1, n + 64, "K*=5r,V*=6", 2048)
    fill_both(torch, eng, None, 0, 0, n + 8, seed=33)
    Q = torch.from_numpy(kvdata.q_rows(33, 0, n, 8)).cuda()
    O = torch.zeros((2, 8, 24, 256), dtype=torch.float32, device="cuda")
    counts = []
    for i, T in enumerate((1, 8)):
        before = eng.launches()
        eng.attend(0, n, Q[:T], O[i, :T])
        counts.append(eng.launches() - before)
    eng.sync()
    assert counts[0] == counts[1] == (3 if n < 5120 else 2)  # staging, attention and, behind the batch launch, the merge
    assert float((O[0, 0] - O[1, 0]).abs().max()) <= 1e-6 * float(O[1, 0].abs().max())
    eng.close()


def test_pieces_are_those_of_the_other_kernel(mk, torch_cuda, monkeypatch):
    """the mma.sync kernel runs a range's pieces too: its result over the last range of 45,000 positions is the tensor-core kernel's, 1e-5"""
    torch = torch_cuda
    n, T, layers, lo, hi = 45003, 3, 2, 23008, 45056
    got = []
    for kernel in ("tc", "fast"):
        monkeypatch.setenv("MK_KV_ATTN", kernel)
        eng = mk.Engine(layers, hi - lo + 64, "K*=5r,V*=6", 2048)
        eng.set_base(lo)
        Kl, Vl = (torch.from_numpy(x).cuda() for x in kvdata.kv_rows(85, 0, lo, n - lo))
        for l in range(layers):
            eng.append(l, lo, Kl, Vl)
        K, V, Q = (torch.from_numpy(x).cuda() for x in rows(layers, 6, n, T))
        part = torch.zeros((layers, 4, 48, 256), dtype=torch.float32, device="cuda")
        ml = torch.zeros((layers, 4, 48, 2), dtype=torch.float32, device="cuda")
        O = torch.zeros((layers, T, 24, 256), dtype=torch.float32, device="cuda")
        eng.step_layers_partial(n, K, V, Q, lo, hi, lo, hi, part, ml)
        eng.combine_layers(T, 1, part, ml, O)
        eng.sync()
        got.append(O)
        eng.close()
    rel = float((got[0] - got[1]).norm() / got[0].norm())
    assert rel <= 1e-5, rel
