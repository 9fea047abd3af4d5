"""Kernel variants at the sizes where their dispatch or their tiles change over: remainders, the smallest and largest of each
range, ties.  Integer-valued or index results are compared bit for bit, sums against float64."""
import concurrent.futures

import numpy as np
import pytest
import torch

import expertscattergather_b200 as egs
from expertscattergather_b200 import _lib, ops, workloads
from expertscattergather_b200.workloads import Workload
from expertscattergather_b200.step import train_step
from gpu_util import STEP_KEYS, gpu_step
from oracle import egs_oracle as orc

pytestmark = pytest.mark.gpu


# keys per thread and warps per expert change at T = 256, 1024, 2048, 4096, 8192, 16384 (beyond: the shared-memory kernel);
# E around the eight experts of a CTA; few (batch, expert) pairs: fewer experts per CTA
@pytest.mark.parametrize("B,T,E,K", [(1, 1, 1, 1), (2, 256, 9, 256), (40, 257, 33, 31), (3, 1024, 8, 1000), (20, 1025, 65, 3),
                                     (20, 2049, 70, 1024), (2, 4097, 12, 77), (1, 8193, 5, 1024), (1, 16385, 3, 200)])
@pytest.mark.parametrize("ties", [False, True])
def test_route_topk_edges(cuda_device, B, T, E, K, ties):
    g = torch.Generator().manual_seed(T + E)
    scores = torch.randint(-3, 4, (B, T, E), generator=g).float() if ties else torch.randn(B, T, E, generator=g)
    Ind = ops.route_topk(scores.to(cuda_device), K).cpu()
    order = torch.sort(scores.permute(0, 2, 1), dim=-1, descending=True, stable=True).indices      # ties: lower token first
    assert torch.equal(Ind, order[..., :K])


@pytest.mark.parametrize("B,T,E,K", [(3, 1, 2, 5), (2, 1023, 7, 9), (5, 1025, 300, 20), (1, 20000, 11, 13), (1, 30000, 4, 9)])
@pytest.mark.parametrize("one_row", [False, True])
def test_index_csr_edges(cuda_device, B, T, E, K, one_row):
    g = torch.Generator().manual_seed(T)
    Ind = torch.randint(0, T, (B, E, K), generator=g)
    if one_row:
        Ind[:, : E // 2] = T - 1            # half of all slots in one row
    Ind[B - 1, E - 1, K - 1] = T            # out of range: left out
    csr = ops.build_index_csr(Ind.to(cuda_device), T)
    flat = Ind + torch.arange(B).view(-1, 1, 1) * T
    valid = (Ind < T).reshape(-1)
    rows, slots = flat.reshape(-1)[valid], torch.arange(Ind.numel())[valid]
    counts = torch.bincount(rows, minlength=B * T)
    assert torch.equal(csr.counts.cpu().long(), counts)
    assert torch.equal(csr.offsets.cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]))
    assert torch.equal(csr.entries.cpu().long()[: slots.numel()], slots[torch.sort(rows, stable=True).indices])
    assert csr.summary() == {"max_per_row": int(counts.max()), "rows_touched": int((counts > 0).sum()), "out_of_range": True,
                             "valid_slots": int(valid.sum())}


# generic kernels: tile widths of 32, 64, 96 and 128 columns, remainders in rows (B*K around 64), features and contraction steps
@pytest.mark.parametrize("B,T,E,K,I,J", [(1, 3, 1, 1, 1, 1), (7, 40, 2, 9, 31, 33), (5, 33, 3, 13, 65, 95), (9, 70, 2, 29, 127, 97),
                                         (3, 50, 2, 21, 161, 5), (2, 20, 1, 150, 33, 257)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_generic_kernels_edges(cuda_device, B, T, E, K, I, J, dtype):
    w = Workload("gen", B, T, E, K, I, J, dtype, "replace", 77)
    ins = workloads.make_inputs(w, integer_valued=True)
    ref = orc.np_step(ins["X"], ins["Wg"], ins["Ws"], ins["Ind"], ins["G"])
    got = gpu_step(ins, cuda_device, "generic")
    for k in STEP_KEYS:         # small integers: exact in float32; 16-bit results are the float32 sums rounded once
        if dtype == torch.float32:
            assert np.array_equal(got[k].double().numpy(), ref[k]), k
        elif k in ("Y", "dY"):
            assert torch.equal(got[k], torch.from_numpy(ref[k]).to(dtype)), k


# generic kernels at widths whose narrowest tiles would exceed a grid's y
@pytest.mark.parametrize("N", [32 * 65535, 32 * 65536 + 32])
def test_generic_kernels_take_wide_outputs(cuda_device, N):
    x, W, Ind = torch.tensor([[[3.0], [2.0]]]), torch.arange(N).view(1, 1, N).float() % 7, torch.ones(1, 1, 1, dtype=torch.int64)
    x, W, Ind = x.to(cuda_device), W.to(cuda_device), Ind.to(cuda_device)
    assert torch.equal(ops.gather_gemm(x, W, Ind, path="generic"), 2 * W.view(1, 1, 1, N))
    assert torch.equal(ops.gemm_scatter(x[:, :1].view(1, 1, 1, 1), W, Ind, 2, path="generic")[0], torch.cat([0 * W[0], 3 * W[0]]))
    assert torch.equal(ops.dweight(x, W.view(1, 1, 1, N), Ind, path="generic"), 2 * W)


@pytest.mark.parametrize("B,T,E,K,N", [(1, 5, 1, 1, 1), (3, 40, 4, 50, 24), (16, 64, 2, 100, 72), (70, 33, 3, 30, 33)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("gathered", [False, True])
def test_expert_row_sum(cuda_device, B, T, E, K, N, dtype, gathered):
    g = torch.Generator().manual_seed(N)
    Ind = torch.randint(0, T, (B, E, K), generator=g)
    src = torch.randint(-4, 5, (B, T, N) if gathered else (B, E, K, N), generator=g).to(dtype)
    out = torch.full((E, N), float("nan"), dtype=dtype, device=cuda_device)
    d_src, d_ind = src.to(cuda_device), Ind.to(cuda_device)
    rc = _lib.load().egs_expert_row_sum(d_src.data_ptr(), d_ind.data_ptr() if gathered else None, out.data_ptr(), B, T, E, K, N,
                                        ops.dtype_to_type_id(dtype), _lib.I64, None, torch.cuda.current_stream().cuda_stream)
    assert rc == _lib.OK
    rows = torch.gather(src.double(), 1, Ind.reshape(B, -1, 1).expand(-1, -1, N)).reshape(B, E, K, N) if gathered else src.double()
    assert torch.equal(out.cpu(), rows.sum((0, 2)).to(dtype))       # integers: exact in float32, rounded once


# long sums: no worse than 64-bit truth rounded a few times (2^-24 each), with rows read 16 bytes a lane (N = 8) and one column a lane
@pytest.mark.parametrize("N", [8, 5])
def test_expert_row_sum_of_many_rows(cuda_device, N):
    B, E, K = 512, 1, 4096
    m = egs.ExpertGather(E, 1, N, bias=True).to(cuda_device)
    dY = torch.randn(B, E, K, N, generator=torch.Generator(device=cuda_device).manual_seed(2), device=cuda_device)
    Y = m(torch.zeros(B, 1, 1, device=cuda_device), torch.zeros(B, E, K, dtype=torch.int64, device=cuda_device))
    Y.backward(dY)
    ref = dY.double().sum((0, 2)).view(-1)
    # eight-row trees lose 2^-24 of partial sums of a few units, 2^18 of them at random: 2^-24 * 3 * 2^9; the sums themselves are ~2^10.5
    assert ((m.bias.grad.double().view(-1) - ref).abs().max() <= 2.0 ** -24 * (3 * 2 ** 9 + 4 * ref.abs().max())).item()
    dY[0, 0, 7, 1], dY[3, 0, 9, 2], dY[4, 0, 2, 2] = float("inf"), float("inf"), float("-inf")
    m.bias.grad = None
    m(torch.zeros(B, 1, 1, device=cuda_device), torch.zeros(B, E, K, dtype=torch.int64, device=cuda_device)).backward(dY)
    got = m.bias.grad.view(-1)
    assert got[1] == float("inf") and got[2].isnan() and got[0].isfinite()


def test_expert_row_sum_takes_wide_rows(cuda_device):
    N = 8 * 65536 + 9                                              # more blocks of columns than a grid's y holds
    m = egs.ExpertGather(1, 1, N, bias=True).to(cuda_device)
    m(torch.ones(1, 2, 1, device=cuda_device), torch.zeros(1, 1, 3, dtype=torch.int64, device=cuda_device)).sum().backward()
    assert torch.equal(m.bias.grad, torch.full_like(m.bias, 3.0))


# strict float32 kernels: tile widths 32 / 64 / 96 / 128 with partial last tiles, contractions around one step (32), one chunk
# (512) and several, rows around one block of 128, one and several row ranges of D (1024 rows each)
@pytest.mark.parametrize("B,T,E,K,I,J", [(1, 4, 1, 1, 4, 4), (3, 60, 2, 43, 36, 28), (5, 90, 3, 51, 516, 68), (4, 200, 2, 65, 1028, 136),
                                         (2, 300, 1, 128, 2048, 200), (9, 400, 2, 230, 544, 96), (2, 50, 70, 9, 260, 140)])
def test_strict_float32_edges(cuda_device, B, T, E, K, I, J):
    w = Workload("strict", B, T, E, K, I, J, torch.float32, "replace", 78)
    exact = workloads.make_inputs(w, integer_valued=True)           # every product and sum is exact: bit for bit
    exact["Ind"][B - 1, E - 1, K - 1] = T                           # out of range: skipped
    ref = orc.np_step(exact["X"], exact["Wg"], exact["Ws"], exact["Ind"].clamp(0, T - 1), exact["G"])
    ops.reset_status()
    d = {k: v.to(cuda_device) for k, v in exact.items()}
    Y = ops.gather_gemm(d["X"], d["Wg"], d["Ind"], path="tensor")
    dY = ops.gather_gemm(d["G"], d["Ws"], d["Ind"], w_layout="nc", path="tensor")
    ref["Y"][B - 1, E - 1, K - 1] = 0
    ref["dY"][B - 1, E - 1, K - 1] = 0
    assert np.array_equal(Y.cpu().double().numpy(), ref["Y"]) and np.array_equal(dY.cpu().double().numpy(), ref["dY"])
    safe = exact["Ind"].clamp(0, T - 1)                             # the masked slot's row of Y is zero: it adds nothing
    Yc, dYc = Y.cpu(), dY.cpu()
    Out = ops.gemm_scatter(Y, d["Ws"], d["Ind"], T, path="tensor")
    dX = ops.gemm_scatter(dY, d["Wg"], d["Ind"], T, w_layout="nc", path="tensor")
    assert np.array_equal(Out.cpu().double().numpy(), orc.np_scatter(Yc, exact["Ws"], safe, T))
    assert np.array_equal(dX.cpu().double().numpy(), orc.np_scatter(dYc, exact["Wg"].transpose(1, 2).contiguous(), safe, T))
    dWg = ops.dweight(d["X"], dY, d["Ind"], path="tensor")
    dWs = ops.dweight(d["G"], Y, d["Ind"], out_layout="direct_rows", path="tensor")
    assert np.array_equal(dWg.cpu().double().numpy(), orc.np_dweight(exact["X"], dYc, safe))
    assert np.array_equal(dWs.cpu().double().numpy(), orc.np_dweight(exact["G"], Yc, safe).transpose(0, 2, 1))
    with pytest.raises(RuntimeError, match="outside"):
        ops.check_status()
    real = workloads.make_inputs(w)                                 # and the float32 bar of the parity tests on real values
    truth = orc.np_step(real["X"], real["Wg"], real["Ws"], real["Ind"], real["G"])
    got = gpu_step(real, cuda_device, "tensor")
    for k in STEP_KEYS:
        assert orc.rel_err(got[k], truth[k]) <= 1e-5, k


# strict float32: tiles of 32 to 128 columns and their remainders, one step, fewer steps than split groups and many, row ranges of D, slot
# rows as boxes (K = 1, 16, 32, 128) and gathered (K = 7, 43, 101), more units than SMs.  Small integers are exact as TF32 products; `big`: one
# operand is multiples of 5461 up to 14 bits, whose lo parts are not zero (those of both together would meet in the product that is left
# out), and every sum stays an integer below 2^24.
@pytest.mark.parametrize("B,T,E,K,I,J", [(1, 8, 1, 1, 4, 4), (3, 60, 2, 43, 36, 96), (5, 90, 3, 32, 132, 68), (9, 33, 2, 7, 100, 160),
                                         (2, 300, 3, 128, 260, 32), (5, 300, 40, 101, 64, 516), (40, 64, 33, 16, 228, 200), (130, 20, 2, 16, 64, 136)])
@pytest.mark.parametrize("big", ["none", "rows", "columns"])
def test_strict_kernels_edges(cuda_device, B, T, E, K, I, J, big):
    ins = workloads.make_inputs(Workload("strict", B, T, E, K, I, J, torch.float32, "replace", 31), integer_valued=True)
    ins["Ind"][B - 1, E - 1, K - 1] = T           # out of range: left out
    known = (ins["Ind"] < T).unsqueeze(-1)
    slots = ins["Ind"].clamp(max=T - 1).reshape(B, E * K, 1)
    rows = lambda A: torch.gather(A.double(), 1, slots.expand(-1, -1, A.shape[-1])).reshape(B, E, K, -1) * known
    a, b = 5461 if big == "rows" else 1, 5461 if big == "columns" else 1
    Y = torch.randint(-3, 4, (B, E, K, J), generator=torch.Generator().manual_seed(1)).float()
    X, Wg, Ws = ins["X"] * a, ins["Wg"] * b, ins["Ws"] * b
    dev, run = lambda t: t.contiguous().to(cuda_device), dict(path="tensor", precision="strict")

    def same(got, want):
        assert want.abs().max() < 2 ** 24 and torch.equal(got.double().cpu(), want)

    contributions = torch.einsum("bekj,eji->beki", Y.double() * a, Ws.double()) * known
    Out = torch.zeros(B, T, I, dtype=torch.float64).scatter_add_(1, slots.expand(-1, -1, I), contributions.reshape(B, E * K, I))
    P = torch.einsum("bekf,bekg->efg", rows(X), Y.double() * b)
    Ind = dev(ins["Ind"])
    same(ops.gather_gemm(dev(X), dev(Wg), Ind, **run), torch.einsum("beki,eij->bekj", rows(X), Wg.double()))
    same(ops.gather_gemm(dev(X), dev(Ws), Ind, w_layout="nc", **run), torch.einsum("beki,eji->bekj", rows(X), Ws.double()))
    same(ops.gemm_scatter(dev(Y * a), dev(Ws), Ind, T, **run), Out)
    same(ops.gemm_scatter(dev(Y * a), dev(Ws.transpose(1, 2)), Ind, T, w_layout="nc", **run), Out)
    same(ops.dweight(dev(X), dev(Y * b), Ind, **run), P)
    same(ops.dweight(dev(X), dev(Y * b), Ind, out_layout="direct_rows", **run), P.transpose(1, 2))
    ops.reset_status()


# contractions beyond 512 on the tensor cores: no further from float64 than the float32 sums of the generic kernels
@pytest.mark.parametrize("C", [516, 1024, 2048])
@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("op", ["G", "S"])
def test_strict_float32_long_contractions_are_as_good_as_ffma(cuda_device, C, positive, op):
    B, T, E, K, N = 3, 400, 2, 100, 136
    g = torch.Generator(device=cuda_device).manual_seed(C)
    normal = lambda *s: torch.randn(s, generator=g, device=cuda_device).abs_() if positive else torch.randn(s, generator=g, device=cuda_device)
    W, Ind = normal(E, C, N), torch.randperm(T, generator=g, device=cuda_device)[: E * K].view(1, E, K).expand(B, E, K).contiguous()
    A = normal(B, T, C) if op == "G" else normal(B, E, K, C)
    rows = torch.gather(A, 1, Ind.reshape(B, -1, 1).expand(-1, -1, C)).view(B, E, K, C) if op == "G" else A
    ref = torch.einsum("bekc,ecn->bekn", rows.double(), W.double())

    def err(path):
        if op == "G":
            got = ops.gather_gemm(A, W, Ind, path=path)
        else:                                     # distinct tokens: one contribution a row
            got = torch.gather(ops.gemm_scatter(A, W, Ind, T, path=path), 1, Ind.reshape(B, -1, 1).expand(-1, -1, N)).view(B, E, K, N)
        return ((got.double() - ref).norm() / ref.norm()).item()

    assert ops.describe_plan(op, B, T, E, K, C, N, torch.float32)["tensor_path"] == 1
    assert err("auto") <= err("generic")


# ... and the same infinities and NaNs
@pytest.mark.parametrize("w_layout", ["cn", "nc"])
def test_strict_float32_long_contractions_keep_infinities(cuda_device, w_layout):
    B, T, E, K, C, N = 2, 60, 3, 50, 520, 140
    g = torch.Generator().manual_seed(6)
    X, W = torch.randint(-3, 4, (B, T, C), generator=g).float(), torch.randint(1, 4, (E, C, N), generator=g).float()
    Y = torch.randint(-3, 4, (B, E, K, C), generator=g).float()
    Ind = torch.randint(0, T, (B, E, K), generator=g)
    Ind[0, 1, 3] = T                              # out of range: a row of zeros
    for A in (X.view(-1, C), Y.view(-1, C)):
        A[3, 7], A[9, 519], A[9, 2], A[17, 300] = float("inf"), float("inf"), float("-inf"), float("nan")
    W[2, 33, 5], W[1, 0, 139], W[0, 4, 64] = float("-inf"), float("nan"), 0.0
    Wd = (W if w_layout == "cn" else W.transpose(1, 2)).contiguous().to(cuda_device)
    Xd, Yd, Id = X.to(cuda_device), Y.to(cuda_device), Ind.to(cuda_device)
    for f in (lambda path: ops.gather_gemm(Xd, Wd, Id, w_layout=w_layout, path=path),
              lambda path: ops.gemm_scatter(Yd, Wd, Id, T, w_layout=w_layout, path=path)):
        got, want = f("tensor"), f("generic")
        assert got.isinf().any() and got.isnan().any() and torch.equal(got.nan_to_num(nan=12345.0), want.nan_to_num(nan=12345.0))
        assert torch.equal(got.isnan(), want.isnan())
    ops.reset_status()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs a device that is not the current one")
def test_train_step_on_another_device_than_the_current():
    w = Workload("other", 4, 64, 4, 16, 64, 32, torch.float32, "distinct", 9)
    ins = workloads.make_inputs(w, integer_valued=True)
    ref = orc.np_step(ins["X"], ins["Wg"], ins["Ws"], ins["Ind"], ins["G"])
    with torch.cuda.device(0):
        got = gpu_step(ins, torch.device("cuda", 1))
    for k in STEP_KEYS:
        assert np.array_equal(got[k].double().numpy(), ref[k]), k


# 16-bit kernels: one CTA or a pair per tile, slot rows as boxes (K = 1, 16, 64, 128) or gathered (K = 43, 101), one row or one column
# block in the last tile, row ranges of D that are split and that are not
DENSE16_EDGES = [(1, 8, 1, 1, 8, 8), (3, 60, 2, 43, 72, 40), (5, 90, 3, 64, 264, 136), (33, 70, 5, 16, 520, 264),
                 (5, 300, 2, 128, 1000, 200), (9, 777, 24, 101, 1000, 200), (20, 200, 24, 64, 520, 512), (40, 64, 2, 128, 72, 40),
                 (8, 100, 40, 50, 40, 256)]

PAIR_SHAPES = [(20, 200, 24, 64, 520, 512), (24, 600, 40, 72, 1280, 320)]          # compared on the device: see the repeated launches


def _dense16_plans(B, T, E, K, I, J):
    plan = lambda op, c, n, **kw: ops.describe_plan(op, B, T, E, K, c, n, torch.float16, **kw)
    return {"G": plan("G", I, J), "dY": plan("G", I, J, w_layout="nc"), "S": plan("S", J, I), "dX": plan("S", J, I, w_layout="nc"),
            "D": plan("D", I, J)}


def test_dense16_edges_reach_every_form(cuda_device):
    plans = [_dense16_plans(*shape) for shape in DENSE16_EDGES + PAIR_SHAPES]
    for op in ("G", "dY", "S", "dX", "D"):
        assert {p[op]["pair"] for p in plans} == {0, 1}, op
    assert {(p["D"]["splits"] > 1) for p in plans} == {False, True} and {p["D"]["swap"] for p in plans} == {0, 1}
    for op in ("S", "D"):         # slot rows as boxes and gathered, on one CTA and in a pair
        assert {(p[op]["pair"], p[op]["slot_boxes"]) for p in plans} == {(0, 0), (0, 1), (1, 0), (1, 1)}, op


@pytest.mark.parametrize("B,T,E,K,I,J", DENSE16_EDGES)
@pytest.mark.parametrize("bias", [False, True])
def test_dense16_edges(cuda_device, B, T, E, K, I, J, bias):
    g = torch.Generator().manual_seed(I + J)
    dt = torch.float16                                              # integers to 2048 are exact, and no sum here comes near that
    small = lambda *shape: torch.randint(-1, 2, shape, generator=g).to(dt)
    X, G, Y, dY = small(B, T, I), small(B, T, I), small(B, E, K, J), small(B, E, K, J)
    Wg, Ws, bg, bs = small(E, I, J), small(E, J, I), small(E, 1, J), small(E, 1, I)
    # one slot after another through all the tokens: every row meets about E * K / T contributions
    Ind = (torch.arange(B * E * K).view(B, E, K) * 7 + torch.arange(B).view(B, 1, 1)) % T
    d = {k: v.to(cuda_device) for k, v in dict(X=X, G=G, Y=Y, dY=dY, Wg=Wg, Ws=Ws, bg=bg, bs=bs, Ind=Ind).items()}

    def same(got, want):
        assert np.abs(want).max() <= 2048 and np.array_equal(got.cpu().double().numpy(), want)

    rows = orc.np_gather(X, Wg, Ind) + (bg[:, 0].double().numpy()[None, :, None, :] if bias else 0)
    same(ops.gather_gemm(d["X"], d["Wg"], d["Ind"], bias=d["bg"] if bias else None, path="tensor"), rows)
    same(ops.gather_gemm(d["G"], d["Ws"], d["Ind"], w_layout="nc", path="tensor"), orc.np_gather(G, Ws.transpose(1, 2).contiguous(), Ind))
    sums = orc.np_scatter(Y, Ws, Ind, T)
    if bias:
        for e in range(E):
            for b in range(B):
                np.add.at(sums[b], Ind[b, e].numpy(), bs[e, 0].double().numpy())
    same(ops.gemm_scatter(d["Y"], d["Ws"], d["Ind"], T, bias=d["bs"] if bias else None, path="tensor"), sums)
    same(ops.gemm_scatter(d["dY"], d["Wg"], d["Ind"], T, w_layout="nc", path="tensor"), orc.np_scatter(dY, Wg.transpose(1, 2).contiguous(), Ind, T))
    same(ops.dweight(d["X"], d["dY"], d["Ind"], path="tensor"), orc.np_dweight(X, dY, Ind))
    same(ops.dweight(d["G"], d["Y"], d["Ind"], out_layout="direct_rows", path="tensor"), orc.np_dweight(G, Y, Ind).transpose(0, 2, 1))


# 16-bit weight gradients: one accumulator sums at most 8192 rows.  Values of one sign: its truncating additions (16 products each)
# all err the same way, by at most a unit in the last place of the result, and fp16 rounding has no bias over 10^7 elements
@pytest.mark.parametrize("B,T,E,K,I,J", [(200, 64, 18, 177, 1984, 288)])
def test_dense16_dweight_sums_long_contractions_in_ranges(cuda_device, B, T, E, K, I, J):
    assert ops.describe_plan("D", B, T, E, K, I, J, torch.float16)["rows_per_split"] <= 8192
    g = torch.Generator(device=cuda_device).manual_seed(5)
    X, Y = (torch.rand(s, generator=g, device=cuda_device).mul_(0.05).half() for s in ((B, T, I), (B, E, K, J)))
    Ind = torch.randint(0, T, (B, E, K), generator=g, device=cuda_device)
    got = ops.dweight(X, Y, Ind).double()
    bias = []
    for e in range(E):
        rows = X[torch.arange(B, device=cuda_device)[:, None], Ind[:, e]].reshape(B * K, I).double()
        ref = rows.T @ Y[:, e].reshape(B * K, J).double()
        bias.append(((got[e] - ref) / ref).mean())
    assert torch.stack(bias).mean().abs().item() <= 8192 / 16 * 2.0 ** -23


# G and D at sizes of one to four waves, on pairs and on single CTAs; columns that come as boxes of whole segments and of partial ones, weights of
# both layouts.  Small integers: exact in float32, then rounded once.
@pytest.mark.parametrize("B,T,E,K,I,J", [(6, 100, 38, 101, 456, 192), (15, 100, 11, 32, 1032, 432), (11, 100, 52, 50, 400, 224), (7, 100, 56, 64, 704, 232),
                                         (11, 100, 15, 64, 912, 640), (11, 100, 33, 50, 424, 248), (9, 100, 48, 45, 816, 256), (20, 90, 40, 64, 512, 512)])
def test_dense16_last_wave_in_half_tiles(cuda_device, B, T, E, K, I, J):
    plans = [ops.describe_plan(op, B, T, E, K, I, J, torch.bfloat16, w_layout=w) for op, w in (("G", "cn"), ("G", "nc"), ("D", "cn"))]
    assert any(p["pair"] and p["tile_n"] >= 128 for p in plans), plans
    g = torch.Generator().manual_seed(I)
    X, Y = (torch.randint(-2, 3, s, generator=g).to(torch.bfloat16) for s in ((B, T, I), (B, E, K, J)))
    W = torch.randint(-1, 2, (E, I, J), generator=g).to(torch.bfloat16)
    Ind = torch.randint(0, T, (B, E, K), generator=g)
    d = lambda t: t.to(cuda_device)
    ref = torch.from_numpy(orc.np_gather(X, W, Ind)).to(torch.bfloat16)
    assert torch.equal(ops.gather_gemm(d(X), d(W), d(Ind)).cpu(), ref)
    assert torch.equal(ops.gather_gemm(d(X), d(W.transpose(1, 2).contiguous()), d(Ind), w_layout="nc").cpu(), ref)
    ref = torch.from_numpy(orc.np_dweight(X, Y, Ind)).to(torch.bfloat16)
    assert torch.equal(ops.dweight(d(X), d(Y), d(Ind)).cpu(), ref)
    assert torch.equal(ops.dweight(d(X), d(Y), d(Ind), out_layout="direct_rows").cpu(), ref.transpose(1, 2))
    ops.check_status()


# G on single CTAs: of the widths that need as many waves the narrowest; a wider one where it saves a wave; pairs where copies hold steps up
@pytest.mark.parametrize("B,T,E,K,C,N,pair,tile_n", [(37, 388, 133, 8, 1432, 280, 0, 144), (15, 350, 85, 19, 504, 264, 0, 144), (1, 1021, 238, 69, 1240, 280, 0, 144), (2, 5283, 78, 13, 1840, 264, 0, 96),
                                                     (5, 676, 56, 138, 152, 200, 0, 208), (1, 3265, 195, 75, 72, 128, 0, 128), (32, 1024, 256, 16, 512, 128, 1, 128)])
@pytest.mark.parametrize("w_layout", ["cn", "nc"])
def test_dense16_gather_tiles(cuda_device, B, T, E, K, C, N, pair, tile_n, w_layout):
    plan = ops.describe_plan("G", B, T, E, K, C, N, torch.bfloat16, w_layout=w_layout)
    assert (plan["pair"], plan["tile_n"]) == (pair, tile_n)


# G on pairs whose last wave is half empty or more: its tiles are cut in two, into halves of 128 and 96, 96 and 96 or 64, 128 and 128 columns (fewer
# in a row's last tile), boxes of whole segments and of partial ones.  Small integers: exact in float32, then rounded once.
@pytest.mark.parametrize("B,E,K,I,J,first", [(27, 10, 70, 648, 152, 96), (23, 11, 76, 392, 320, 96), (20, 10, 94, 584, 192, 96), (20, 9, 73, 592, 360, 96), (19, 10, 97, 400, 216, 128),
                                             (25, 9, 52, 424, 424, 128), (31, 10, 41, 400, 448, 128), (23, 10, 52, 392, 464, 128), (32, 9, 75, 400, 256, 128), (16, 11, 65, 416, 512, 128)])
@pytest.mark.parametrize("dtype,bias", [(torch.bfloat16, False), (torch.float16, True)])
def test_dense16_gather_in_half_tiles(cuda_device, B, E, K, I, J, first, dtype, bias):
    T = 100
    g = torch.Generator().manual_seed(I)
    X, W = torch.randint(-2, 3, (B, T, I), generator=g).to(dtype), torch.randint(-1, 2, (E, I, J), generator=g).to(dtype)
    Ind = torch.randint(0, T, (B, E, K), generator=g)
    b = torch.randint(-5, 6, (E, J), generator=g).to(dtype) if bias else None
    ref = orc.np_gather(X, W, Ind) + (b.double().numpy()[None, :, None] if bias else 0.0)
    d = lambda t: None if t is None else t.to(cuda_device)
    for w_layout in ("cn", "nc"):
        units, first_columns = ops.describe_half_tiles(B, T, E, K, I, J, dtype, w_layout=w_layout)
        assert units > 0 and first_columns == first
        got = ops.gather_gemm(d(X), d(W if w_layout == "cn" else W.transpose(1, 2).contiguous()), d(Ind), w_layout=w_layout, bias=d(b))
        assert torch.equal(got.cpu(), torch.from_numpy(ref).to(dtype))
    ops.check_status()


# weight gradients on pairs whose slot rows are gathered too, with an odd and an even number of stages (two groups of warps share the ring's
# slots), widths whose last tile is narrow, ranges that end within a batch of ids.  Small integers: exact in float32, then rounded once.
@pytest.mark.parametrize("B,T,E,K,FG,FD,stages", [(9, 300, 24, 101, 1000, 200, 5), (39, 80, 13, 21, 1936, 344, 5), (20, 90, 74, 45, 512, 520, 5), (15, 200, 74, 64, 512, 512, 6)])
@pytest.mark.parametrize("out_layout", ["gathered_rows", "direct_rows"])
def test_dense16_dweight_groups_share_the_ring(cuda_device, B, T, E, K, FG, FD, stages, out_layout):
    plan = ops.describe_plan("D", B, T, E, K, FG, FD, torch.bfloat16)
    assert plan["pair"] == 1 and plan["splits"] == 1 and plan["stages"] == stages, plan
    g = torch.Generator().manual_seed(FG)
    X = torch.randint(-2, 3, (B, T, FG), generator=g).to(torch.bfloat16)
    Y = torch.randint(-2, 3, (B, E, K, FD), generator=g).to(torch.bfloat16)
    Ind = torch.randint(0, T, (B, E, K), generator=g)
    ref = torch.from_numpy(orc.np_dweight(X, Y, Ind))
    if out_layout == "direct_rows":
        ref = ref.transpose(1, 2)
    d = [t.to(cuda_device) for t in (X, Y, Ind)]
    for _ in range(10):
        got = ops.dweight(*d, out_layout=out_layout)
    ops.check_status()
    assert torch.equal(got.cpu(), ref.to(torch.bfloat16))


# ... all of many results, launched back to back
@pytest.mark.parametrize("B,T,E,K,FG,FD", [(39, 80, 13, 21, 1936, 344), (15, 200, 74, 64, 512, 512)])
def test_dense16_dweight_groups_share_the_ring_every_time(cuda_device, B, T, E, K, FG, FD):
    assert ops.describe_plan("D", B, T, E, K, FG, FD, torch.bfloat16)["pair"] == 1
    g = torch.Generator().manual_seed(FD)
    X = torch.randint(-2, 3, (B, T, FG), generator=g).to(torch.bfloat16)
    Y = torch.randint(-2, 3, (B, E, K, FD), generator=g).to(torch.bfloat16)
    Ind = torch.randint(0, T, (B, E, K), generator=g)
    ref = torch.from_numpy(orc.np_dweight(X, Y, Ind)).to(torch.bfloat16).to(cuda_device)
    d = [t.to(cuda_device) for t in (X, Y, Ind)]
    got = [ops.dweight(*d) for _ in range(10)]
    ops.check_status()
    for x in got:
        assert torch.equal(x, ref)


# the first CUDA call of a thread: boxes are described to the driver before anything else has made a context current there
@pytest.mark.parametrize("op", ["G", "S", "D"])
def test_dense16_first_call_of_a_thread(cuda_device, op):
    B, T, E, K, I, J = 8, 128, 8, 16, 256, 64
    X, Y = torch.ones(B, T, I, device=cuda_device).half(), torch.ones(B, E, K, J, device=cuda_device).half()
    Wg, Ws = torch.ones(E, I, J, device=cuda_device).half(), torch.ones(E, J, I, device=cuda_device).half()
    Ind = (torch.arange(B * E * K, device=cuda_device) % T).view(B, E, K)
    run = {"G": lambda: ops.gather_gemm(X, Wg, Ind), "S": lambda: ops.gemm_scatter(Y, Ws, Ind, T), "D": lambda: ops.dweight(X, Y, Ind)}[op]
    torch.cuda.synchronize()
    with concurrent.futures.ThreadPoolExecutor(max_workers=1) as pool:
        got = pool.submit(run).result(timeout=120)
    assert (got == {"G": I, "S": J * E * K // T, "D": B * K}[op]).all().item()


# pairs of SMs: the leader multiplies what both CTAs have staged.  The same launches over and over, under copies on another stream
# that disturb their timing, give the same bits (integer values: every sum is exact in any order), with slot rows that come as boxes
# (K = 64) and that are gathered (K = 72)
@pytest.mark.parametrize("B,T,E,K,I,J", PAIR_SHAPES)
def test_dense16_pairs_repeat_their_bits(cuda_device, B, T, E, K, I, J):
    for plan in _dense16_plans(B, T, E, K, I, J).values():
        assert plan["pair"] and plan["slot_boxes"] in (0, int(K == 64)), plan
    g = torch.Generator(device=cuda_device).manual_seed(J)
    dt = torch.float16
    small = lambda *shape: torch.randint(-1, 2, shape, generator=g, device=cuda_device).to(dt)
    X, Y, Wg, Ws = small(B, T, I), small(B, E, K, J), small(E, I, J), small(E, J, I)
    Ind = (torch.arange(B * E * K, device=cuda_device).view(B, E, K) * 7) % T
    runs = {"G": lambda: ops.gather_gemm(X, Wg, Ind), "dY": lambda: ops.gather_gemm(X, Ws, Ind, w_layout="nc"),
            "S": lambda: ops.gemm_scatter(Y, Ws, Ind, T), "dX": lambda: ops.gemm_scatter(Y, Wg, Ind, T, w_layout="nc"),
            "D": lambda: ops.dweight(X, Y, Ind), "D direct": lambda: ops.dweight(X, Y, Ind, out_layout="direct_rows")}
    rows = torch.gather(X.float(), 1, Ind.reshape(B, -1, 1).expand(-1, -1, I)).reshape(B, E, K, I)
    outs = torch.einsum("bekj,eji->beki", Y.float(), Ws.float())
    want = {"G": torch.einsum("beki,eij->bekj", rows, Wg.float()), "D": torch.einsum("beki,bekj->eij", rows, Y.float()),
            "S": torch.zeros(B, T, I, device=cuda_device).scatter_add_(1, Ind.reshape(B, -1, 1).expand(-1, -1, I), outs.reshape(B, -1, I))}
    first = {k: f() for k, f in runs.items()}
    for k, w in want.items():
        assert w.abs().max() <= 2048 and torch.equal(first[k].float(), w), k
    assert torch.equal(first["D direct"], first["D"].transpose(1, 2))
    other, noise = torch.cuda.Stream(), torch.empty(1 << 25, device=cuda_device)
    for i in range(40):
        with torch.cuda.stream(other):
            noise[: 1 << (16 + i % 10)].add_(1.0)
        for k, f in runs.items():
            assert torch.equal(f(), first[k]), (k, i)
    torch.cuda.synchronize()
    ops.check_status()


# 16-bit scatter with hot token rows in some batch elements only; tiles of 128 expert rows here span elements with and without (K = 48)
@pytest.mark.parametrize("C,N", [(40, 72), (256, 1032), (520, 64)])
@pytest.mark.parametrize("pair", [False, True])
def test_scatter16_mixes_both_kinds_of_batch_elements(cuda_device, C, N, pair):
    if pair and (C % 16 or C > 256):
        pytest.skip("shape the pair kernel does not take")
    B, T, E, K = 9, 130, 40, 48
    g = torch.Generator().manual_seed(C)
    Ind = torch.randint(0, T, (B, E, K), generator=g)              # about 15 per row
    Ind[2, :, 0] = 7                                               # 40 more on one row of batch elements 2 and 5
    Ind[5, :, 1] = 129
    most = torch.stack([torch.bincount(Ind[b].reshape(-1), minlength=T).max() for b in range(B)])
    assert (most[[2, 5]] > 32).all() and (most <= 32).sum() >= 5
    Y = torch.randint(-2, 3, (B, E, K, C), generator=g).to(torch.bfloat16)
    W = torch.randint(-1, 2, (E, C, N), generator=g).to(torch.bfloat16)
    if pair:
        X = torch.randint(-1, 2, (B, T, 32), generator=g).to(torch.bfloat16)
        W1 = torch.randint(-1, 2, (E, 32, C), generator=g).to(torch.bfloat16)
        Mid, Out = ops.gather_scatter_pair(X.to(cuda_device), W1.to(cuda_device), W.to(cuda_device), Ind.to(cuda_device))
        Y = Mid.cpu()
    else:
        Out = ops.gemm_scatter(Y.to(cuda_device), W.to(cuda_device), Ind.to(cuda_device), T)
    ref = orc.np_scatter(Y, W, Ind, T)
    err = np.abs(Out.cpu().double().numpy() - ref).max((1, 2)) / np.abs(ref).max()
    assert err.max() <= 3e-2, err
    # sums in float32 rows are rounded once: half a unit in the last of bf16's eight bits
    for b in (2, 5):
        exact = torch.from_numpy(ref[b]).to(torch.bfloat16).double().numpy()
        assert np.abs(Out[b].cpu().double().numpy() - exact).max() <= 2.0 ** -8 * np.abs(ref[b]).max()


# ... and one hot token row anywhere makes every row of the call a float32 sum that is rounded once: bf16 has eight significant bits,
# so half a unit in the last place is at most 2^-8 of the value (the float32 sums themselves are good to 1e-5 of the largest)
@pytest.mark.parametrize("B", [1, 2, 30, 700])        # counted by the zeroing kernel itself (1, 2), by a CTA an element, by fewer CTAs
@pytest.mark.parametrize("pair", [False, True])
def test_scatter16_one_hot_row_rounds_all_rows_once(cuda_device, B, pair):
    T, E, K, C, N = 40, 12, 24, 32, 64
    g = torch.Generator().manual_seed(B)
    Ind = (torch.arange(B * E * K).view(B, E, K) * 7) % T          # 7 or 8 per row
    Ind[B - 1, :, :4] = 3                                          # 40 more on one row of the last batch element
    Y, W = torch.randn(B, E, K, C, generator=g).bfloat16(), torch.randn(E, C, N, generator=g).bfloat16()
    d_ind = Ind.to(cuda_device)
    if pair:
        X, W1 = torch.randn(B, T, 32, generator=g).bfloat16(), torch.randn(E, 32, C, generator=g).bfloat16()
        Mid, Out = ops.gather_scatter_pair(X.to(cuda_device), W1.to(cuda_device), W.to(cuda_device), d_ind)
        Y = Mid.cpu()
    else:
        Out = ops.gemm_scatter(Y.to(cuda_device), W.to(cuda_device), d_ind, T)
    ref = orc.np_scatter(Y, W, Ind, T)
    assert (np.abs(Out.cpu().double().numpy() - ref) <= 2.0 ** -8 * np.abs(ref) + 1e-5 * np.abs(ref).max()).all()


# small outputs of float32 rows are rounded by the scatter's last CTA, those of more than 64 Ki elements by a launch of their own.  Small
# integers: every sum is exact in float32, so the result is the exact one, rounded once.
@pytest.mark.parametrize("B,T,E,K,C,N", [(1, 1, 1, 40, 8, 8), (1, 1, 40, 1, 32, 2064), (2, 512, 5, 16, 64, 64), (2, 513, 5, 16, 64, 64), (7, 24, 140, 2, 40, 376)])
@pytest.mark.parametrize("form", ["plain", "out"])
def test_scatter16_rounds_small_outputs(cuda_device, B, T, E, K, C, N, form):
    g = torch.Generator().manual_seed(N)
    Ind = torch.randint(0, T, (B, E, K), generator=g)
    Ind.view(-1)[:40] = 0                                          # a hot row in the first batch element
    Y = torch.randint(-7, 8, (B, E, K, C), generator=g).to(torch.bfloat16)
    W = torch.randint(-7, 8, (E, C, N), generator=g).to(torch.bfloat16)
    out = torch.randint(-64, 65, (B, T, N), generator=g).to(torch.bfloat16) if form == "out" else None
    ref = orc.np_scatter(Y, W, Ind, T) + (0.0 if out is None else out.double().numpy())
    got = ops.gemm_scatter(Y.to(cuda_device), W.to(cuda_device), Ind.to(cuda_device), T, out=None if out is None else out.to(cuda_device))
    assert torch.equal(got.cpu(), torch.from_numpy(ref).to(torch.bfloat16))


# ... column tile by column tile in the scatter kernel, where no token row gets more than half of the limit's contributions in the mean and the
# tiles have a counter each: launches of a call with a counting preparation.  CTAs of one unit and of several, one tile and many.
@pytest.mark.parametrize("B,T,E,K,C,N,launches", [(1, 5, 2, 40, 8, 8, 2), (1, 5, 3, 27, 8, 8, 3), (1, 64, 64, 16, 128, 256, 2), (1, 64, 41, 25, 64, 256, 3), (1, 512, 5, 16, 64, 128, 2),
                                                  (1, 513, 5, 16, 64, 128, 3), (1, 2048, 512, 64, 64, 32, 2), (1, 8, 2, 64, 32, 992, 2), (1, 8, 2, 64, 32, 1008, 3), (3, 100, 60, 8, 64, 200, 2)])
@pytest.mark.parametrize("hot", [True, False])
def test_scatter16_rounds_column_tiles(cuda_device, B, T, E, K, C, N, launches, hot):
    g = torch.Generator().manual_seed(N)
    Ind = torch.randint(0, T, (B, E, K), generator=g)
    if hot:
        Ind[B - 1].view(-1)[:40] = T - 1
    Y = torch.randint(-7, 8, (B, E, K, C), generator=g).to(torch.bfloat16)
    W = torch.randint(-7, 8, (E, C, N), generator=g).to(torch.bfloat16)
    ref = torch.from_numpy(orc.np_scatter(Y, W, Ind, T)).to(torch.bfloat16)
    d = [t.to(cuda_device) for t in (Y, W, Ind)]
    n = ops.launch_count()
    got = ops.gemm_scatter(*d, T)
    assert ops.launch_count() - n == launches
    if hot:
        assert torch.equal(got.cpu(), ref)
    ops.check_status()


# what large buffers are zeroed and rounded by goes in stretches with a CTA each: sizes just beyond where that begins, last stretches that are not
# whole.  The allocator hands out blocks that hold NaN.
def _leave_nan_blocks(dev, *byte_counts):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    blocks = [torch.full((n,), -1, dtype=torch.uint8, device=dev) for n in byte_counts]
    torch.cuda.synchronize()
    del blocks


def test_fills_in_stretches(cuda_device):
    for n in ((32 << 20) + 16, (32 << 20) + 3 * 16384 + 7 * 16 + 5):
        x = torch.full((n + 64,), 255, dtype=torch.uint8, device=cuda_device)
        ops.fill_zero(x[:n])
        assert not x[:n].any().item() and (x[n:] == 255).all().item()


@pytest.mark.parametrize("dtype,N", [(torch.float32, 808), (torch.bfloat16, 1608), (torch.float16, 1608)])
@pytest.mark.parametrize("hot", [False, True])
def test_scatter_into_zeros_in_stretches(cuda_device, dtype, N, hot):
    B, T, E, K, C = 3, 17479, 4, 64, 64
    n = B * T * N * (4 if dtype == torch.float32 else 2)
    assert n > 160 << 20
    Ind, Y, W, _, _ = _sparse_scatter(cuda_device, B, T, E, K, N, C)
    if hot:
        Ind[1, :, :10] = T - 1
    Out = _scatter_sum(Ind, torch.einsum("bekc,ecn->bekn", Y, W), torch.zeros(B, T, N, device=cuda_device))
    _leave_nan_blocks(cuda_device, n, 2 * n + (1 << 20))
    got = ops.gemm_scatter(Y.to(dtype), W.to(dtype), Ind, T)
    assert torch.equal(got, Out.to(dtype))
    ops.check_status()


def test_dweight_rounds_ranges_in_stretches(cuda_device):
    B, T, E, K, FG, FD = 129, 70, 8, 64, 1064, 1000
    assert 4 * E * FG * FD > 32 << 20 and ops.describe_plan("D", B, T, E, K, FG, FD, torch.bfloat16)["splits"] > 1
    g = torch.Generator(device=cuda_device).manual_seed(9)
    X, Y = (torch.randint(-2, 3, s, generator=g, device=cuda_device).float() for s in ((B, T, FG), (B, E, K, FD)))
    Ind = torch.randint(0, T, (B, E, K), generator=g, device=cuda_device)
    ref = torch.stack([torch.cat([X[b, Ind[b, e]] for b in range(B)]).T @ Y[:, e].reshape(B * K, FD) for e in range(E)])      # (sums below 2^24: exact)
    _leave_nan_blocks(cuda_device, 2 * E * FG * FD, 4 * E * FG * FD + (1 << 20))
    got = ops.dweight(X.bfloat16(), Y.bfloat16(), Ind)
    assert torch.equal(got, ref.bfloat16())
    ops.check_status()


# kernels become resident under the end of the ones before them: operators issued back to back, with nothing of torch between them, have to
# give what they give one by one.  Each reads what the one before it has just written, or writes what it has just read: every family of
# kernels, with and without prepared indices, more than one wave of tiles, the helper stream's fork and join.  A column of the weights has one
# entry of +-1, so that all values are small integers: the same bits in any order, also in 16 bits.
@pytest.mark.parametrize("B,T,E,K,I,J", [(6, 128, 8, 32, 128, 64), (5, 33, 3, 13, 65, 95), (40, 300, 9, 40, 256, 128), (64, 256, 32, 16, 128, 64),
                                         (32, 512, 32, 32, 768, 192), (9, 200, 12, 43, 520, 72), (30, 90, 7, 20, 129, 121)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_operators_back_to_back(cuda_device, B, T, E, K, I, J, dtype):
    g = torch.Generator(device=cuda_device).manual_seed(I)
    ints = lambda *s: torch.randint(-1, 2, s, generator=g, device=cuda_device).to(dtype)
    one = lambda n, m: torch.zeros(E, n, m, device=cuda_device, dtype=dtype).scatter_(1, torch.randint(0, n, (E, 1, m), generator=g, device=cuda_device),
                                                                                      ints(E, 1, m))
    Xs, G, Wg, Ws = [ints(B, T, I) for _ in range(4)], ints(B, T, I), one(I, J), one(J, I)
    scores = torch.rand(B, T, E, generator=g, device=cuda_device)
    Ind = torch.rand(B, E, T, generator=g, device=cuda_device).topk(K, -1).indices
    bias = ints(E, J)

    def one_pass(X, sync):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        out = []
        def keep(t):
            wait()
            out.append(t)
            return t
        Y = keep(ops.gather_gemm(X, Wg, Ind))
        Out = keep(ops.gemm_scatter(Y, Ws, Ind, T))                                    # reads Y; counts ids by itself
        Y2 = keep(ops.gather_gemm(Out, Wg, Ind, bias=bias))                            # gathers what was just added
        dW = keep(ops.dweight(Out, Y2, Ind))
        dWd = keep(ops.dweight(X, Y2, Ind, out_layout="direct_rows"))
        ops.fill_zero(Y)                                                               # overwrites what the scatter has read
        wait()
        ind = keep(ops.route_topk(scores, K, index_dtype=torch.int32))
        csr = ops.build_index_csr(ind, T)
        keep(csr.entries)
        Y3 = keep(ops.gather_gemm(X, Wg, ind))
        O3 = keep(ops.gemm_scatter(Y3, Ws, ind, T, csr=csr))
        ops.gemm_scatter(Y3, Ws, ind, T, out=O3)                                       # adds to what was just added to
        wait()
        step = train_step(X, Wg, Ws, Ind, G)
        wait()
        return [Y, Out, Y2, dW, dWd, ind, csr.entries, Y3, O3] + [step[k] for k in STEP_KEYS]
    alone = [one_pass(X, True) for X in Xs]
    together = [one_pass(X, False) for X in Xs]
    for X in Xs * 2:                              # results dropped: torch hands their memory to the next operators
        last = one_pass(X, False)
    ops.check_status()
    for x, y in zip(alone + [alone[-1]], together + [last]):
        assert max(t.abs().max().item() for t in x[:3] + x[7:9]) <= 256
        for i, (p, q) in enumerate(zip(x, y)):
            assert torch.equal(p, q), i


# 16-bit scatters on pairs whose rows stay for `kept` column tiles: whole waves of row blocks and a rest, a last tile of few columns, rows as
# boxes and gathered, as many contraction steps as stages, more (eight read-out warps, the last bytes of shared memory), and too many to
# stay.  Every row of Y has eight entries of +-1, so a token row's sum stays below 256: exact in 16 bits in any order.
def _sparse_scatter(dev, B, T, E, K, N, C):
    g = torch.Generator(device=dev).manual_seed(N)
    ints = lambda *s: torch.randint(-1, 2, s, generator=g, device=dev)
    Ind = torch.rand(B, E, T, generator=g, device=dev).topk(K, -1).indices
    Y = torch.zeros(B, E, K, C, device=dev).scatter_(-1, torch.rand(B, E, K, C, generator=g, device=dev).topk(8, -1).indices, ints(B, E, K, 8).float())
    return Ind, Y, ints(E, C, N).float(), ints(E, N).float(), ints(B, T, N).float()


def _scatter_sum(Ind, rows, out):
    B, E, K, N = rows.shape
    return out.scatter_add_(1, Ind.reshape(B, E * K, 1).expand(-1, -1, N), rows.reshape(B, E * K, N))


@pytest.mark.parametrize("B,T,E,K,N,C,kept,full", [(16, 700, 60, 64, 768, 256, 1, 3), (16, 700, 60, 64, 1032, 192, 2, 3), (20, 500, 50, 96, 760, 256, 2, 5),
                                                   (13, 600, 160, 59, 504, 136, 1, 6), (6, 900, 40, 128, 1032, 512, 2, 1), (6, 900, 40, 128, 520, 640, 0, 0),
                                                   (16, 300, 60, 64, 1032, 136, 2, 3), (8, 300, 64, 32, 1000, 320, 4, 0), (16, 300, 16, 59, 1032, 512, 5, 0),
                                                   (48, 300, 8, 59, 1032, 512, 2, 1)])
@pytest.mark.parametrize("w_layout", ["cn", "nc"])
def test_scatter_rows_that_stay(cuda_device, B, T, E, K, N, C, kept, full, w_layout):
    Ind, Y, W, _, _ = _sparse_scatter(cuda_device, B, T, E, K, N, C)
    assert ops.describe_kept_rows(B, T, E, K, C, N, torch.bfloat16, w_layout=w_layout) == (kept, full)
    assert ops.describe_plan("S", B, T, E, K, C, N, torch.bfloat16, w_layout=w_layout)["pair"] == 1
    Out = _scatter_sum(Ind, torch.einsum("bekc,ecn->bekn", Y, W), torch.zeros(B, T, N, device=cuda_device))
    got = ops.gemm_scatter(Y.bfloat16(), (W if w_layout == "cn" else W.transpose(1, 2).contiguous()).bfloat16(), Ind, T, w_layout=w_layout)
    assert torch.equal(got.float(), Out)
    ops.check_status()


# ... gathered rows, which the gathering warps load with a row block's first column tile only: even and odd numbers of stages, row blocks of
# fewer and of more steps than stages, and all of several results back to back
@pytest.mark.parametrize("B,E,K,N,C,w_layout,stages", [(4, 50, 37, 512, 512, "cn", 4), (9, 37, 37, 512, 392, "nc", 5), (4, 31, 36, 992, 416, "nc", 5), (7, 50, 57, 616, 144, "cn", 6),
                                                       (9, 52, 43, 624, 176, "nc", 7)])
def test_gathered_scatter_rows_that_stay(cuda_device, B, E, K, N, C, w_layout, stages):
    T = 300
    Ind, Y, W, _, _ = _sparse_scatter(cuda_device, B, T, E, K, N, C)
    plan = ops.describe_plan("S", B, T, E, K, C, N, torch.bfloat16, w_layout=w_layout)
    assert ops.describe_kept_rows(B, T, E, K, C, N, torch.bfloat16, w_layout=w_layout)[0] > 1 and (plan["pair"], plan["slot_boxes"], plan["stages"]) == (1, 0, stages)
    Out = _scatter_sum(Ind, torch.einsum("bekc,ecn->bekn", Y, W), torch.zeros(B, T, N, device=cuda_device)).bfloat16()
    args = Y.bfloat16(), (W if w_layout == "cn" else W.transpose(1, 2).contiguous()).bfloat16(), Ind, T
    got = [ops.gemm_scatter(*args, w_layout=w_layout) for _ in range(10)]
    ops.check_status()
    for x in got:
        assert torch.equal(x, Out)


# ... and the other forms of the operator: a bias, an output that is added to, a hot token row (float32 rows), both 16-bit types
@pytest.mark.parametrize("B,T,E,K,N,C", [(16, 700, 60, 64, 768, 256), (20, 500, 50, 96, 760, 256), (8, 300, 64, 32, 1000, 320)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["bias", "out", "hot", "bias out hot"])
def test_scatter_rows_that_stay_in_every_form(cuda_device, B, T, E, K, N, C, dtype, form):
    Ind, Y, W, bias, out = _sparse_scatter(cuda_device, B, T, E, K, N, C)
    assert ops.describe_kept_rows(B, T, E, K, C, N, dtype)[0] > 0
    if "hot" in form:
        Ind[:, :, 0] = 3                          # 50 contributions and more: the call sums in float32 and rounds once
    rows = torch.einsum("bekc,ecn->bekn", Y, W) + (bias[None, :, None] if "bias" in form else 0)
    Out = _scatter_sum(Ind, rows, out.clone() if "out" in form else torch.zeros_like(out))
    got = ops.gemm_scatter(Y.to(dtype), W.to(dtype), Ind, T, bias=bias.to(dtype) if "bias" in form else None, out=out.to(dtype) if "out" in form else None)
    assert torch.equal(got, Out.to(dtype))
    ops.check_status()


# generic weight gradients of rows that are no multiples of 16 bytes: tiles of 32 to 128 gathered features with remainders, up to 32 direct
# features and more, grids of few CTAs and of many, one row, remainders of the 16-row steps, the 256-row tables and the row ranges.  Small
# integers: float32 sums are exact in any order, and a 16-bit result is rounded once.
@pytest.mark.parametrize("B,T,E,K,FG,FD", [(1, 5, 1, 1, 1, 33), (3, 40, 2, 5, 31, 65), (2, 60, 5, 17, 33, 101), (7, 50, 3, 37, 65, 35), (1, 300, 2, 257, 97, 129),
                                           (16, 300, 40, 16, 129, 67), (5, 90, 150, 9, 63, 35), (40, 70, 30, 33, 101, 103), (9, 64, 300, 3, 3, 77),
                                           (30, 400, 12, 90, 127, 47), (6, 30, 4, 13, 15, 31)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("out_layout", ["gathered_rows", "direct_rows"])
def test_generic_dweight_edges(cuda_device, B, T, E, K, FG, FD, dtype, out_layout):
    g = torch.Generator(device=cuda_device).manual_seed(FG + FD)
    X, Y = (torch.randint(-2, 3, s, generator=g, device=cuda_device).to(dtype) for s in ((B, T, FG), (B, E, K, FD)))
    Ind = torch.randint(0, T, (B, E, K), generator=g, device=cuda_device)
    Ind[B - 1, E - 1, K - 1] = T                  # out of range: left out
    known = (Ind < T).unsqueeze(-1)
    rows = torch.gather(X.double(), 1, Ind.clamp(max=T - 1).reshape(B, E * K, 1).expand(-1, -1, FG)).reshape(B, E, K, FG) * known
    P = torch.einsum("bekf,bekg->efg" if out_layout == "gathered_rows" else "bekf,bekg->egf", rows, Y.double())
    assert torch.equal(ops.dweight(X, Y, Ind, out_layout=out_layout, path="generic"), P.to(dtype))
    ops.reset_status()


# operands that begin 16 bytes into their storage (the least the tensor-core kernels and their boxes take) or at any element (generic kernels)
@pytest.mark.parametrize("offset_bytes", [16, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_operands_at_offsets(cuda_device, dtype, offset_bytes):
    B, T, E, K, I, J = 6, 90, 3, 32, 136, 72
    g = torch.Generator(device=cuda_device).manual_seed(2)
    n = offset_bytes // dtype.itemsize

    def at_offset(t):
        whole = torch.empty(t.numel() + n, dtype=t.dtype, device=cuda_device)
        return whole[n:].copy_(t.reshape(-1)).view(t.shape)
    small = lambda *s: torch.randint(-1, 2, s, generator=g, device=cuda_device).to(dtype)
    X, Y, Wg, Ws = small(B, T, I), small(B, E, K, J), small(E, I, J), small(E, J, I)
    Ind = (torch.arange(B * E * K, device=cuda_device).view(B, E, K) * 7) % T
    Xo, Yo, Wgo, Wso, Indo = (at_offset(t) for t in (X, Y, Wg, Ws, Ind.int()))
    assert {t.data_ptr() % 32 for t in (Xo, Yo, Wgo, Wso)} == {offset_bytes}
    assert torch.equal(ops.gather_gemm(Xo, Wgo, Indo), ops.gather_gemm(X, Wg, Ind))
    assert torch.equal(ops.gather_gemm(Xo, Wso, Indo, w_layout="nc"), ops.gather_gemm(X, Ws, Ind, w_layout="nc"))
    assert torch.equal(ops.gemm_scatter(Yo, Wso, Indo, T), ops.gemm_scatter(Y, Ws, Ind, T))
    assert torch.equal(ops.gemm_scatter(Yo, Wgo, Indo, T, w_layout="nc"), ops.gemm_scatter(Y, Wg, Ind, T, w_layout="nc"))
    assert torch.equal(ops.dweight(Xo, Yo, Indo), ops.dweight(X, Y, Ind))
    ops.check_status()


# generic row kernel: one to four times 32 columns a CTA with remainders; 65 to 96 columns have two forms, for one contraction step (up to 32
# elements) and for more
@pytest.mark.parametrize("C,N", [(1, 67), (31, 96), (32, 81), (33, 67), (65, 257), (101, 89), (97, 33), (33, 127), (5, 31)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("w_layout", ["cn", "nc"])
def test_generic_rowgemm_edges(cuda_device, C, N, dtype, w_layout):
    B, T, E, K = 3, 70, 4, 43
    g = torch.Generator(device=cuda_device).manual_seed(C + N)
    small = lambda *s: torch.randint(-1, 2, s, generator=g, device=cuda_device).to(dtype)
    X, Y, W = small(B, T, C), small(B, E, K, C), small(E, C, N)
    Wl = W if w_layout == "cn" else W.transpose(1, 2).contiguous()
    Ind = torch.randint(0, T, (B, E, K), generator=g, device=cuda_device)
    Ind[B - 1, E - 1, K - 1] = T                  # out of range: a row of zeros, and left out
    known, slots = (Ind < T).unsqueeze(-1), Ind.clamp(max=T - 1).reshape(B, E * K, 1)
    rows = torch.gather(X.double(), 1, slots.expand(-1, -1, C)).reshape(B, E, K, C) * known
    assert torch.equal(ops.gather_gemm(X, Wl, Ind, w_layout=w_layout, path="generic"), torch.einsum("bekc,ecn->bekn", rows, W.double()).to(dtype))
    products = torch.einsum("bekc,ecn->bekn", Y.double(), W.double()) * known
    Out = torch.zeros(B, T, N, dtype=torch.float64, device=cuda_device).scatter_add_(1, slots.expand(-1, -1, N), products.reshape(B, E * K, N))
    assert torch.equal(ops.gemm_scatter(Y, Wl, Ind, T, w_layout=w_layout, path="generic"), Out.to(dtype))
    ops.reset_status()
