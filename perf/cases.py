"""What the MoE layer is asked to do in use, as sized cases for timing.

Every case goes through a public entry point of the package the way a user's program calls it:

  block    `MoeBlock.forward`            routing, experts, combine and shared expert of one layer
  layer    `MoeBlock.layer_forward`      the same inside a transformer layer: norm before, residual after
  host     `MoeBlock.forward_host`       a decode call on pinned host buffers, result read on the host
  seam     `MoeBlock.experts_forward`    the caller has routed already (the `ExpertFfn` seam)
  ops      `MoeBlock.forward_unfused`    the op-by-op runner a host engine drives through `ops.*`
  lm_head  `ops.mul_mv`                  the quantized vocabulary projection of a decode step

The layer shape is the benchmark's (hidden 3072, 256 experts of width 1024, top-10, Q4_K gate / up, Q6_K down,
one shared expert) unless the case says otherwise; weights, router and hidden states are synthetic with the
benchmark's distributions.
"""
import torch

from maxuna_b200 import ops
from maxuna_b200.gguf import Q6_K, ExpertStack
from maxuna_b200.moe import MoeBlock

BASE = {"hidden": 3072, "ff": 1024, "experts": 256, "top_k": 10}
# from this many tokens on the entry points leave the mat-vec kernel (21- or 15-bit activations) for the grouped
# GEMM (f16 operands); used only to state the tolerance
GEMM_FROM = 65


def listed():
    return [
        # one sequence being decoded: latency of a single call
        dict(BASE, name="block_1", kind="block", t=1, bias="uniform", routing=False),
        # a few sequences, activations and results in host memory (an engine whose residual stream is on the host)
        dict(BASE, name="host_4", kind="host", t=4, bias="uniform"),
        # a small odd batch whose routing the engine did itself
        dict(BASE, name="seam_7", kind="seam", t=7, bias="uniform", shared=True),
        # an ordinary decode batch, with the routing decision logged
        dict(BASE, name="block_16", kind="block", t=16, bias="uniform", routing=True),
        # a large decode batch inside a transformer layer
        dict(BASE, name="layer_64", kind="layer", t=64, bias="uniform"),
        # a short prompt on a smaller layer: ragged token count, other widths
        dict(hidden=2048, ff=768, experts=128, top_k=8, name="block_130_small", kind="block", t=130, bias="uniform", routing=False),
        # a prompt chunk inside a transformer layer
        dict(BASE, name="layer_2048", kind="layer", t=2048, bias="uniform"),
        # a prompt with skewed expert popularity
        dict(BASE, name="block_4096_zipf", kind="block", t=4096, bias="zipf", routing=False),
        # the largest prefill batch
        dict(BASE, name="block_16384", kind="block", t=16384, bias="zipf", routing=False),
        # the vocabulary projection of one decoded token
        dict(name="lm_head_1", kind="lm_head", t=1, n_out=100352, hidden=3072),
        # the op-by-op runner, decode (mat-vec ops) and prompt chunk (grouped-GEMM ops)
        dict(BASE, name="ops_3", kind="ops", t=3, bias="uniform"),
        dict(BASE, name="ops_512", kind="ops", t=512, bias="uniform"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["block"] * 6 + ["layer"] * 4 + ["host"] * 2 + ["seam"] * 2 + ["ops"] * 3 + ["lm_head"] * 2)
    if kind == "lm_head":
        n_out = _log_int(rng, 16384, 131072)
        return {"kind": kind, "t": rng.randint(1, 4), "n_out": n_out if rng.random() < 0.5 else n_out // 64 * 64,
                "hidden": rng.choice([2048, 3072])}
    shape = dict(BASE)
    if rng.random() < 0.25:
        shape = {"hidden": rng.choice([2048, 4096]), "ff": rng.choice([512, 768]), "experts": rng.choice([64, 128]),
                 "top_k": rng.choice([6, 8])}
    most = {"block": 16384, "layer": 4096, "host": 64, "seam": 256, "ops": 1024}[kind]
    case = dict(shape, kind=kind, t=_log_int(rng, 1, most), bias=rng.choice(["uniform", "zipf"]))
    if kind == "block":
        case["routing"] = rng.random() < 0.5
    if kind == "seam":
        case["shared"] = rng.random() < 0.5
    return case


def _zipf_bias(n_expert, gen):
    """Selection bias that skews how many tokens an expert gets: Zipf(1.1) over a shuffle of the experts."""
    z = 1.0 / torch.arange(1, n_expert + 1, dtype=torch.float32, device="cuda") ** 1.1
    bias = torch.empty(n_expert, device="cuda")
    bias[torch.randperm(n_expert, generator=gen, device="cuda")] = z * 0.3 - 0.1
    return bias


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    t, hidden = case["t"], case["hidden"]
    x = torch.randn(t, hidden, generator=gen, device="cuda")
    state = {"case": case, "x": x}
    if case["kind"] == "lm_head":
        state["w"] = ExpertStack.random(Q6_K, 1, case["n_out"], hidden, seed=seed, chunk_experts=1)
        return state
    bias = _zipf_bias(case["experts"], gen) if case["bias"] == "zipf" else None
    blk = state["blk"] = MoeBlock.random(hidden, case["ff"], case["experts"], case["top_k"], seed=seed, bias=bias)
    if case["kind"] == "layer":
        state["norm"] = 0.5 + torch.rand(hidden, generator=gen, device="cuda")
    if case["kind"] == "seam":
        state["ids"], state["w"] = blk.route(x)
    if case["kind"] == "host":
        state["x"] = x.cpu().pin_memory()
        state["out"] = torch.empty(t, hidden).pin_memory()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "block":
        return state["blk"].forward(state["x"], return_routing=case["routing"])
    if kind == "layer":
        return state["blk"].layer_forward(state["x"], state["norm"])
    if kind == "host":
        return state["blk"].forward_host(state["x"], state["out"])
    if kind == "seam":
        return state["blk"].experts_forward(state["x"], state["ids"], state["w"], add_shared=case["shared"])
    if kind == "ops":
        return state["blk"].forward_unfused(state["x"])
    w = state["w"]
    return ops.mul_mv(w.buffer, w.dtype, w.n_out, w.k, state["x"])


def work(case):
    """Each weight that the routing reaches once (distinct experts in expectation, for an even routing), the
    activations in and the result out once; two operations per weight and token."""
    t, h = case["t"], case["hidden"]
    if case["kind"] == "lm_head":
        n = case["n_out"]
        return {"bytes": n * (h // 256) * 210 + 4 * t * (h + n), "flops": 2 * t * n * h}
    f, e, k = case["ff"], case["experts"], case["top_k"]
    shared = 1 if case.get("shared", True) else 0
    routes = case["kind"] != "seam"
    distinct = e * (1.0 - (1.0 - k / e) ** t) + shared
    expert_bytes = 2 * f * (h // 256) * 144 + h * (f // 256) * 210
    return {"bytes": distinct * expert_bytes + (4 * e * h if routes else 0) + 8 * t * h,
            "flops": t * (k + shared) * 6 * h * f + (2 * t * e * h if routes else 0)}


def tolerance(case):
    """Relative error between two correct evaluations at the entry point's own precision; expert ids are exact."""
    if case["kind"] == "lm_head" or (case["kind"] == "ops" and case["t"] < GEMM_FROM):
        return {"rel": 1e-5}      # 32-bit sums, activations of at least 21 bits
    if case["t"] >= GEMM_FROM:
        return {"rel": 2e-3}      # both operands of three chained products rounded to f16
    if case["t"] <= 8:
        return {"rel": 1e-5}      # activations carried at 21 bits, exact integer products
    return {"rel": 3e-4}          # activations carried at 15 bits
