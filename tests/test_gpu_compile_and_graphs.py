"""The modules under torch.compile (the dispatcher ops carry fake implementations so that a compiled graph can trace through
them, as the reference's do, egs/triton_kernels.py:527-567) and under CUDA-graph capture (forward + backward, helper
streams included), both against the CPU oracle."""
import subprocess
import sys

import pytest
import torch

import expertscattergather_b200 as egs
from expertscattergather_b200 import ops, workloads
from expertscattergather_b200.workloads import Workload
from gpu_util import tol_for
from oracle import egs_oracle as orc

pytestmark = pytest.mark.gpu


def _modules(w, ins, dev):
    g = egs.ExpertGather(w.E, w.I, w.J).to(dev).to(w.dtype)
    s = egs.ExpertScatter(w.E, w.J, w.I).to(dev).to(w.dtype)
    with torch.no_grad():
        g.W.copy_(ins["Wg"]); s.W.copy_(ins["Ws"])
    return g, s


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_modules_compile_with_fullgraph(cuda_device, dtype):
    """torch.compile(fullgraph=True) over gather -> scatter -> loss: tracing must get through the autograd Functions and the
    four dispatcher ops without a graph break (backend aot_eager: the traced forward and backward graphs run through the
    ops' real implementations; no code generation is involved)."""
    w = Workload("cmp", 4, 64, 6, 16, 64, 32, dtype, "distinct", 51)
    ins = workloads.make_inputs(w)
    ref = orc.torch_step(ins["X"], ins["Wg"], ins["Ws"], ins["Ind"], ins["G"])
    g, s = _modules(w, ins, cuda_device)

    def block(x, ind, grad):
        return (s(g(x, ind), ind, w.T).float() * grad.float()).sum()

    compiled = torch.compile(block, fullgraph=True, backend="aot_eager")
    X = ins["X"].to(cuda_device).requires_grad_(True)
    ops.reset_status()
    loss = compiled(X, ins["Ind"].to(cuda_device), ins["G"].to(cuda_device))
    loss.backward()
    torch.cuda.synchronize()
    ops.check_status()
    tol = tol_for(dtype, "strict")
    assert orc.rel_err(X.grad.cpu(), ref["dX"]) <= tol
    assert orc.rel_err(g.W.grad.cpu(), ref["dWg"]) <= tol
    assert orc.rel_err(s.W.grad.cpu(), ref["dWs"]) <= tol
    ref_loss = float((ref["Out"].double() * ins["G"].double()).sum())
    assert abs(float(loss.detach()) - ref_loss) <= tol * max(1.0, float((ref["Out"].double() * ins["G"].double()).abs().sum()))


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("block", [False, True])
def test_bias_modules_and_the_block_compile(cuda_device, bias, block):
    """Compiled calls run the Python functions (with graph breaks): the same gradients as the eager calls."""
    w = Workload("cb", 4, 64, 6, 16, 64, 32, torch.float32, "distinct", 52)
    ins = {k: v.to(cuda_device) for k, v in workloads.make_inputs(w).items()}
    torch.manual_seed(3)
    m = egs.ExpertGatherScatter(w.E, w.I, w.J, bias=bias).to(cuda_device)
    f = m if block else lambda x, ind: m.scatter(m.gather(x, ind), ind, w.T)

    def grads(f):
        m.zero_grad()
        x = ins["X"].clone().requires_grad_(True)
        out = f(x, ins["Ind"])
        out.backward(ins["G"])
        return [out.detach(), x.grad] + [p.grad for p in m.parameters()]

    for a, b in zip(grads(torch.compile(f, backend="aot_eager")), grads(f)):
        assert orc.rel_err(a.cpu(), b.cpu()) <= 1e-5


def test_the_functions_overlap_weight_gradients_like_the_modules(cuda_device):
    """A direct caller of the Functions launches what the modules launch: no ones-contraction, no torch reduction."""
    w = Workload("direct", 8, 256, 8, 64, 256, 128, torch.bfloat16, "distinct", 54)
    ins = {k: v.to(cuda_device) for k, v in workloads.make_inputs(w).items()}
    bg = torch.zeros(w.E, 1, w.J, device=cuda_device, dtype=w.dtype, requires_grad=True)
    bs = torch.zeros(w.E, 1, w.I, device=cuda_device, dtype=w.dtype, requires_grad=True)
    Wg, Ws, X = (ins[k].clone().requires_grad_(True) for k in ("Wg", "Ws", "X"))
    host = ops._host()

    def run(gather, scatter):
        out = scatter(gather())
        n = ops.launch_count()
        got = torch.autograd.grad(out, (X, Wg, bg, Ws, bs), ins["G"])
        torch.cuda.synchronize()
        return ops.launch_count() - n, got

    n_fn, fn = run(lambda: egs.kernels.ExpertGatherBiasFunction.apply(X, Wg, bg, ins["Ind"]),
                   lambda Y: egs.kernels.ExpertScatterBiasFunction.apply(Y, Ws, bs, ins["Ind"], w.T))
    n_native, native = run(lambda: host.gather_autograd(X, Wg, bg, ins["Ind"]), lambda Y: host.scatter_autograd(Y, Ws, bs, ins["Ind"], w.T))
    assert n_fn == n_native
    for a, b in zip(fn, native):
        assert a.shape == b.shape and orc.rel_err(a.cpu(), b.cpu()) <= 1e-2


@pytest.mark.filterwarnings("ignore:.*an autograd kernel was not registered")
def test_backward_with_create_graph_returns_a_graph(cuda_device):
    """The dispatcher ops have no second derivative of their own: torch warns and goes on, for the modules as for the Functions."""
    g, s = egs.ExpertGather(4, 64, 32).to(cuda_device), egs.ExpertScatter(4, 32, 64).to(cuda_device)
    x = torch.randn(2, 40, 64, device=cuda_device, requires_grad=True)
    ind = torch.randint(0, 40, (2, 4, 8), device=cuda_device)
    gx, = torch.autograd.grad(s(g(x, ind), ind, 40).pow(2).sum(), x, create_graph=True)
    assert gx.requires_grad
    gx.pow(2).sum().backward()


def test_the_first_call_of_a_process_may_be_captured(cuda_device):
    code = """
import torch
from expertscattergather_b200 import ops
X, W = torch.ones(2, 8, 32, device="cuda"), torch.ones(2, 32, 16, device="cuda")
Ind = torch.zeros(2, 2, 4, dtype=torch.int64, device="cuda")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    Y = ops.gather_gemm(X, W, Ind)
for _ in range(2):
    X.add_(1.0)
    graph.replay()
    assert (Y == 32 * X[0, 0, 0]).all().item()
ops.check_status()
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("block", [False, True])
def test_jit_traces_run_on_new_inputs(cuda_device, bias, block):
    if block:
        m = egs.ExpertGatherScatter(4, 64, 32, bias=bias).to(cuda_device)
    else:
        class Pair(torch.nn.Module):
            def __init__(self):
                super().__init__()
                self.g, self.s = egs.ExpertGather(4, 64, 32, bias=bias), egs.ExpertScatter(4, 32, 64, bias=bias)

            def forward(self, x, ind):
                return self.s(self.g(x, ind), ind, 40)
        m = Pair().to(cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(1)
    new = lambda: (torch.randn(2, 40, 64, generator=g, device=cuda_device), torch.randint(0, 40, (2, 4, 8), generator=g, device=cuda_device))
    traced = torch.jit.trace(m, new(), check_trace=False)
    x, ind = new()
    assert orc.rel_err(traced(x, ind).detach().cpu(), m(x, ind).detach().cpu()) <= 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_modules_forward_and_backward_in_a_cuda_graph(cuda_device, dtype):
    """Forward + backward of the modules captured once and replayed on new input values: the helper streams the backward
    pass uses (weight gradients beside dX / dY) fork from and join the capturing stream, so the whole step lands in the graph."""
    w = Workload("cg", 6, 128, 8, 32, 128, 64, dtype, "distinct", 53)
    ins = workloads.make_inputs(w)
    g, s = _modules(w, ins, cuda_device)
    x_static = torch.zeros_like(ins["X"], device=cuda_device).requires_grad_(True)
    ind = ins["Ind"].to(cuda_device)
    grad = ins["G"].to(cuda_device)

    def step():
        g.W.grad = None; s.W.grad = None; x_static.grad = None
        out = s(g(x_static, ind), ind, w.T)
        (out.float() * grad.float()).sum().backward()
        return out

    side = torch.cuda.Stream(cuda_device)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    grads = (x_static.grad, g.W.grad, s.W.grad)
    tol = tol_for(dtype, "strict")
    for trial in range(2):                           # two different inputs through the same graph
        Xv = ins["X"] if trial == 0 else torch.roll(ins["X"], 1, 0)
        ref = orc.torch_step(Xv, ins["Wg"], ins["Ws"], ins["Ind"], ins["G"])
        with torch.no_grad():
            x_static.copy_(Xv.to(cuda_device))
        graph.replay()
        torch.cuda.synchronize()
        ops.check_status()
        assert orc.rel_err(out.detach().cpu(), ref["Out"]) <= tol
        assert orc.rel_err(grads[0].cpu(), ref["dX"]) <= tol
        assert orc.rel_err(grads[1].cpu(), ref["dWg"]) <= tol
        assert orc.rel_err(grads[2].cpu(), ref["dWs"]) <= tol


def test_block_backward_from_saved_tensors_that_are_not_contiguous(cuda_device):
    """What saved-tensor hooks hand back may lie otherwise in memory: the helper stream reads a copy that is made before it is forked.  Small integers and
    weights with one entry a row: sums in 16 bits are exact in any order."""
    B, T, E, K, I, J = 4, 128, 16, 64, 256, 128
    g = torch.Generator().manual_seed(8)
    ints = lambda *s: torch.randint(-1, 2, s, generator=g).to(torch.bfloat16).to(cuda_device)
    m = egs.ExpertGatherScatter(E, I, J).to(cuda_device).to(torch.bfloat16)
    X, G, Ind = ints(B, T, I), ints(B, T, I), torch.rand(B, E, T, generator=g).topk(K, -1).indices.to(cuda_device)
    one = (torch.arange(I)[:, None] % J == torch.arange(J)[None]).to(cuda_device)
    with torch.no_grad():
        m.gather.W.copy_(ints(E, I, J) * one)
        m.scatter.W.copy_(ints(E, J, I) * one.T)

    def grads():
        m.zero_grad()
        x = X.clone().requires_grad_(True)
        m(x, Ind).backward(G)
        return [x.grad] + [p.grad for p in m.parameters()]

    plain = grads()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.transpose(-1, -2).contiguous().transpose(-1, -2)):
        moved = [grads() for _ in range(5)]
    ops.check_status()
    assert all(t.any().item() for t in plain)
    for got in moved:
        for a, b in zip(got, plain):
            assert torch.equal(a, b)
