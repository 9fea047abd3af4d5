"""Performance cases of the expert gather / scatter path: what users of this package run, at the sizes they run it.

Three kinds of pass:
  train   gather -> scatter -> backward from a given gradient of the output: through the two modules ("modules"), through
          the block module ("block") or through the explicit step ("step")
  serve   route_topk -> gather -> scatter without gradients: through the block module ("block") or through the tensor-level
          operators with a prepared CSR ("ops")
Sizes: B batch elements of T tokens, E experts with K routed tokens each, model width I, expert width J.
"""
import math

import torch

import expertscattergather_b200 as egs
from expertscattergather_b200 import ops
from expertscattergather_b200.step import train_step

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}
INDEX_DTYPES = {"int64": torch.int64, "int32": torch.int32, "int16": torch.int16}

# A drawn case stays at or below these: routed multiply-adds (12 or 4 N*I*J operations), routed slots, bytes of one
# [B,T,I] tensor, entries of one [B,E,T] table of scores.
MAX_FLOPS = {"float32": 1.2e11, "bfloat16": 6.6e12, "float16": 6.6e12}
MAX_SLOTS = 1 << 21
MAX_TOKEN_BYTES = 1.1e9
MAX_SCORES = 1 << 26


def _case(kind, dtype, B, T, E, K, I, J, api, index="distinct", index_dtype="int64", bias=False, name=None):
    c = {"kind": kind, "dtype": dtype, "B": B, "T": T, "E": E, "K": K, "I": I, "J": J, "api": api, "index": index,
         "index_dtype": index_dtype, "bias": bias}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one short prompt through a small block: a handful of launches, latency is all there is
        _case("serve", "bfloat16", 1, 64, 8, 8, 512, 128, "block", name="serve-tiny-bf16"),
        # a unit-test or debugging sized training step in the modules' default type
        _case("train", "float32", 2, 64, 4, 16, 128, 64, "modules", name="train-tiny-f32"),
        # the sizes of the modules' own randomised tests: every dimension odd, int16 ids drawn with replacement
        _case("train", "float32", 53, 71, 45, 23, 83, 29, "modules", index="replace", index_dtype="int16", name="train-odd-f32"),
        # benchmark configuration: B=64, T=256, E=32, float32
        _case("train", "float32", 64, 256, 32, 32, 128, 64, "modules", name="train-B64-T256-f32"),
        # benchmark configuration: long sequences of which the experts take few tokens, float32
        _case("train", "float32", 16, 16384, 32, 32, 128, 64, "block", name="train-T16384-f32"),
        # float32 training at an ordinary model width
        _case("train", "float32", 16, 1024, 32, 64, 1024, 256, "modules", name="train-wide-f32"),
        # benchmark configuration: many small experts, Zipf-distributed routing (hot tokens collide), bf16
        _case("train", "bfloat16", 32, 1024, 256, 16, 512, 128, "modules", index="zipf", name="train-E256-zipf-bf16"),
        # benchmark configuration: wide experts, bf16, the explicit step
        _case("train", "bfloat16", 8, 2048, 64, 128, 2048, 512, "step", name="train-I2048-bf16"),
        # benchmark configuration: the largest single-GPU one, bf16
        _case("train", "bfloat16", 512, 1024, 64, 64, 1024, 256, "modules", name="train-B512-bf16"),
        # a serving batch of long prompts, fp16, index preparation shared through a CSR
        _case("serve", "float16", 32, 2048, 64, 128, 1024, 256, "ops", index_dtype="int32", name="serve-B32-T2048-fp16"),
        # training with biases on both modules
        _case("train", "bfloat16", 32, 512, 32, 64, 768, 192, "modules", bias=True, name="train-bias-bf16"),
        # ragged sizes: no dimension a multiple of a tile
        _case("train", "float16", 9, 777, 24, 101, 1000, 200, "block", index="replace", index_dtype="int32",
              name="train-ragged-fp16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    shape = rng.random()
    if shape < 0.15:      # the randomised tests' sizes: six dimensions from [1, 128)
        B, T, E, K, I, J = (rng.randint(1, 127) for _ in range(6))
        return _case("train", "float32", B, T, E, K, I, J, "modules", index="replace", index_dtype="int16")
    kind = "train" if shape < 0.75 else "serve"
    dtype = rng.choice(["float32", "bfloat16", "bfloat16", "float16"])
    es = 4 if dtype == "float32" else 2
    while True:
        B, T, E = _log(rng, 1, 512), _log(rng, 64, 16384), _log(rng, 4, 256)
        K, I, J = _log(rng, 4, 256), 8 * _log(rng, 8, 256), 8 * _log(rng, 4, 64)
        slots = B * E * K
        if (K <= T and slots <= MAX_SLOTS and 12.0 * slots * I * J <= MAX_FLOPS[dtype] and B * T * I * es <= MAX_TOKEN_BYTES
                and B * E * T <= MAX_SCORES):
            break
    index_dtype = rng.choice(["int64", "int64", "int32", "int16"])
    if kind == "serve":
        return _case(kind, dtype, B, T, E, K, I, J, rng.choice(["block", "ops"]), index_dtype=index_dtype)
    api = rng.choice(["modules", "block", "step"])
    bias = api == "modules" and rng.random() < 0.25
    return _case(kind, dtype, B, T, E, K, I, J, api, rng.choice(["distinct", "replace", "zipf"]), index_dtype, bias)


def _indices(case, gen):
    B, T, E, K = case["B"], case["T"], case["E"], case["K"]
    if case["index"] == "replace":
        ind = torch.randint(0, T, (B, E, K), generator=gen, device="cuda")
    else:
        ind = torch.empty((B, E, K), dtype=torch.int64, device="cuda")
        step = max(1, (1 << 24) // (E * T))
        for b in range(0, B, step):
            n = min(step, B - b)
            if case["index"] == "zipf":       # popularity rank^-1.1 over a random order of the tokens of each batch element
                rank = torch.rand((n, 1, T), generator=gen, device="cuda").argsort(-1) + 1
                keys = -1.1 * rank.float().log()
            else:
                keys = torch.zeros((n, 1, 1), device="cuda")
            u = torch.rand((n, E, T), generator=gen, device="cuda").clamp_(1e-7, 1 - 1e-7)
            ind[b:b + n] = (keys - (-u.log()).log()).topk(K, -1).indices
    return ind.to(INDEX_DTYPES[case["index_dtype"]])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    B, T, E, K, I, J = (case[k] for k in ("B", "T", "E", "K", "I", "J"))

    def normal(*shape, scale=1.0):
        return torch.randn(shape, generator=gen, device="cuda", dtype=dt).mul_(scale)

    s = {"case": case}
    with torch.device("cuda"):
        if case["api"] == "block":
            s["block"] = egs.ExpertGatherScatter(E, I, J).to(dt)
            s["gather"], s["scatter"] = s["block"].gather, s["block"].scatter
        else:
            s["gather"] = egs.ExpertGather(E, I, J, bias=case["bias"]).to(dt)
            s["scatter"] = egs.ExpertScatter(E, J, I, bias=case["bias"]).to(dt)
    with torch.no_grad():
        s["gather"].W.copy_(normal(E, I, J, scale=I ** -0.5))
        s["scatter"].W.copy_(normal(E, J, I, scale=J ** -0.5))
        if case["bias"]:
            s["gather"].bias.copy_(normal(E, 1, J, scale=I ** -0.5))
            s["scatter"].bias.copy_(normal(E, 1, I, scale=J ** -0.5))
    s["X"] = normal(B, T, I)
    if case["kind"] == "serve":
        s["scores"] = torch.randn((B, T, E), generator=gen, device="cuda")
        return s
    s["Ind"] = _indices(case, gen)
    s["G"] = normal(B, T, I)
    if case["api"] != "step":
        s["X"].requires_grad_()
    s["leaves"] = [s["X"]] + [p for m in (s["gather"], s["scatter"]) for p in m.parameters()]
    return s


def _serve(s):
    case = s["case"]
    with torch.no_grad():
        Ind = ops.route_topk(s["scores"], case["K"], index_dtype=INDEX_DTYPES[case["index_dtype"]])
        if case["api"] == "block":
            return {"Ind": Ind, "Out": s["block"](s["X"], Ind)}
        csr = ops.build_index_csr(Ind, case["T"])
        Y = ops.gather_gemm(s["X"], s["gather"].W, Ind)
        Out = ops.gemm_scatter(Y, s["scatter"].W, Ind, case["T"], csr=csr)
        return {"Ind": Ind, "offsets": csr.offsets, "entries": csr.entries, "Y": Y, "Out": Out}


def run(s):
    case = s["case"]
    if case["kind"] == "serve":
        return _serve(s)
    if case["api"] == "step":
        return train_step(s["X"], s["gather"].W.detach(), s["scatter"].W.detach(), s["Ind"], s["G"])
    for p in s["leaves"]:
        p.grad = None
    if case["api"] == "block":
        Out = s["block"](s["X"], s["Ind"])
    else:
        Out = s["scatter"](s["gather"](s["X"], s["Ind"]), s["Ind"], case["T"])
    Out.backward(s["G"])
    return [Out.detach()] + [p.grad for p in s["leaves"]]


def work(case):
    B, T, E, K, I, J = (case[k] for k in ("B", "T", "E", "K", "I", "J"))
    es = 4 if case["dtype"] == "float32" else 2
    slots = B * E * K
    rows = B * T * (1.0 - (1.0 - min(K, T) / T) ** E)      # token rows that some expert takes, for uniform draws
    tokens, weights, ids = B * T * I * es, 2 * E * I * J * es, slots * int(case["index_dtype"][3:]) // 8
    mid = slots * J * es if case["api"] != "block" else 0  # the middle tensor is an output of its own there
    bias = E * (I + J) * es if case["bias"] else 0
    if case["kind"] == "serve":
        csr = 4 * (B * T + slots) if case["api"] == "ops" else 0
        return {"bytes": 4 * B * T * E + ids + csr + rows * I * es + weights + mid + tokens, "flops": 4.0 * slots * I * J}
    # X and the gradient of the output are read where a row is taken; the output and dX are written whole
    return {"bytes": ids + 2 * rows * I * es + 2 * tokens + 2 * weights + (2 if case["api"] == "step" else 1) * mid + 2 * bias,
            "flops": 12.0 * slots * I * J}


def tolerance(case):
    # float32 products and sums; 16-bit results are rounded once per contribution that meets in a token row
    return {"rel": {"float32": 1e-5, "bfloat16": 1e-2, "float16": 2e-3}[case["dtype"]]}
