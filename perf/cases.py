"""Performance cases: what a user's program has this framework do on one GPU, through its public entry points.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare` makes what a program has in hand
before the call, `run` is one pass, `exact` the same result in 64 bits from plain torch.  Kinds of case:

* ``gemm``      ``ops.fused_gemm.gemm``: a linear layer's product, with and without the fused tanh-GELU
* ``mlp``       ``models.tp_mlp.TensorParallelMLP``: forward and backward of a tensor-parallel MLP block
* ``moe``       a mixture-of-experts layer given its routing: dispatch, two grouped GEMMs over the experts, combine
* ``exchange``  dispatch and combine alone, the experts replaced by a copy of the received rows
* ``dispatch``  the fp8 dispatch alone; the rows are read back by slot number, as their order inside an expert's
                segment is not fixed
* ``combine``   the weighted combine alone
* ``coll``      the stream-ordered collectives on symmetric tensors (a team of one: the local data path and the launch)
"""
from __future__ import annotations

import math

import torch

import nvshmem_b200.core as nv
from nvshmem_b200.models.tp_mlp import TensorParallelMLP
from nvshmem_b200.ops import fused_gemm as fg
from nvshmem_b200.ops.moe import MoeDispatchCombine

BF16 = torch.bfloat16
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16, "i32": torch.int32, "u8": torch.uint8}


def listed():
    return [
        # the smallest linear layer the GEMM takes: latency of one call
        {"name": "gemm_smallest", "kind": "gemm", "M": 128, "N": 512, "K": 512, "act": ""},
        # decode: one block of 128 tokens against the up projection (with GELU) of one of two ranks of the bench's MLP
        {"name": "gemm_decode_gelu", "kind": "gemm", "M": 128, "N": 3584, "K": 8192, "act": "gelu_tanh"},
        # an odd number of row blocks, column blocks and K steps
        {"name": "gemm_ragged", "kind": "gemm", "M": 1152, "N": 2816, "K": 1984, "act": ""},
        # the benchmark's GEMM (row-parallel product of 8192 tokens)
        {"name": "gemm_prefill", "kind": "gemm", "M": 8192, "N": 8192, "K": 3584, "act": ""},
        # a training step of the benchmark's MLP block: forward, gradients of the input and of both weights
        {"name": "mlp_train", "kind": "mlp", "tokens": 4096, "hidden": 8192, "ffn": 3584},
        # one rank's experts (32 of 256) of a large MoE layer, prefill: 4096 tokens, top-8
        {"name": "moe_layer_prefill", "kind": "moe", "T": 4096, "H": 7168, "F": 2048, "E": 32, "K": 8},
        # the same layer in decode: 61 tokens, every expert gets a few rows and the weights are read once
        {"name": "moe_layer_decode", "kind": "moe", "T": 61, "H": 7168, "F": 2048, "E": 32, "K": 8},
        # the exchange alone in decode: latency of the two kernels
        {"name": "exchange_decode", "kind": "exchange", "T": 64, "H": 7168, "E": 256, "K": 8},
        # fp8 dispatch of a prefill batch, top-8 of 256 experts
        {"name": "dispatch_fp8", "kind": "dispatch", "T": 4096, "H": 7168, "E": 256, "K": 8},
        # combine of a prefill batch
        {"name": "combine_prefill", "kind": "combine", "T": 4096, "H": 7168, "E": 256, "K": 8},
        # a small all-reduce, as of a loss or a norm
        {"name": "reduce_small", "kind": "coll", "coll": "reduce", "dtype": "f32", "n": 2051},
        # an all-reduce of a gradient bucket
        {"name": "reduce_large", "kind": "coll", "coll": "reduce", "dtype": "bf16", "n": 1 << 27},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mult(rng, lo, hi, step):
    return min(hi, max(lo, round(_log(rng, lo, hi) / step) * step))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "mlp", "moe", "moe", "exchange", "dispatch", "combine", "coll", "coll"])
    if kind == "gemm":
        return {"kind": kind, "M": _mult(rng, 128, 8192, 128), "N": _mult(rng, 256, 8192, 256), "K": _mult(rng, 64, 8192, 64), "act": rng.choice(["", "gelu_tanh"])}
    if kind == "mlp":
        return {"kind": kind, "tokens": _mult(rng, 128, 4096, 128), "hidden": _mult(rng, 512, 8192, 256), "ffn": _mult(rng, 256, 3584, 256)}
    if kind == "moe":
        return {"kind": kind, "T": _log(rng, 1, 4096), "H": _mult(rng, 512, 7168, 256), "F": _mult(rng, 256, 2048, 128), "E": rng.choice([8, 16, 32]), "K": rng.randint(1, 8)}
    if kind in ("exchange", "dispatch", "combine"):
        return {"kind": kind, "T": _log(rng, 1, 4096), "H": _mult(rng, 256, 7168, 128), "E": rng.choice([16, 32, 64, 128, 256]), "K": rng.randint(1, 10)}
    dtype = rng.choice(["f32", "bf16", "f16", "i32", "u8"])
    size = torch.empty((), dtype=DTYPES[dtype]).element_size()
    return {"kind": "coll", "coll": rng.choice(["reduce", "reducescatter", "fcollect", "alltoall", "broadcast"]), "dtype": dtype, "n": _log(rng, 64, (1 << 28) // size)}


# ------------------------------------------------------------------ inputs
def _init():
    if not torch.cuda.is_available():
        raise RuntimeError("the cases need a GPU")
    torch.cuda.set_device(0)
    nv.init(device=0, uid=nv.get_unique_id(), rank=0, nranks=1)  # the first call initialises, later ones return


def _randn(gen, *shape, scale=1.0):
    return torch.randn(*shape, device="cuda", generator=gen, dtype=torch.float32).mul_(scale).to(BF16)


def _weights(gen, groups, *shape, scale=0.02):
    w = torch.empty(groups, *shape, device="cuda", dtype=BF16)
    for g in range(groups):
        w[g] = _randn(gen, *shape, scale=scale)
    return w


def _routing(gen, T, E, K):
    """top-K of E experts and their weights, from the softmax of normal logits."""
    w, idx = torch.randn(T, E, device="cuda", generator=gen).softmax(-1).topk(K, dim=-1)
    return idx.to(torch.int32).contiguous(), w.float().contiguous()


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k = case["kind"]
    if k == "gemm":
        return {"x": _randn(gen, case["M"], case["K"]), "w": _randn(gen, case["N"], case["K"], scale=0.02)}
    if k == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        return {"x": _randn(gen, t, h), "dy": _randn(gen, t, h, scale=0.1), "w_up": _randn(gen, f, h, scale=0.02), "w_down": _randn(gen, h, f, scale=0.02)}
    if k in ("moe", "exchange", "dispatch", "combine"):
        d = {"x": _randn(gen, case["T"], case["H"])}
        d["idx"], d["weight"] = _routing(gen, case["T"], case["E"], case["K"])
        if k == "moe":
            d["w_in"] = _weights(gen, case["E"], 2 * case["F"], case["H"])    # gate rows, then up rows
            d["w_out"] = _weights(gen, case["E"], case["H"], case["F"])
        return d
    dtype = DTYPES[case["dtype"]]
    if dtype.is_floating_point:
        return {"src": torch.randn(case["n"], device="cuda", generator=gen).to(dtype)}
    return {"src": torch.randint(0, 100, (case["n"],), device="cuda", generator=gen).to(dtype)}


class _Symmetric:
    """Source and destination of a collective in symmetric memory, given back with the state."""

    def __init__(self, src):
        self.src = nv.tensor(tuple(src.shape), src.dtype)
        self.dst = nv.tensor(tuple(src.shape), src.dtype, zero=True)
        self.src.copy_(src)

    def __del__(self):
        for t in (self.src, self.dst):
            nv.free_tensor(t)


def prepare(case, seed):
    _init()
    s, k = {"case": case, **_inputs(case, seed)}, case["kind"]
    if k == "gemm":
        s["act"] = case["act"] or None
    elif k == "mlp":
        mlp = TensorParallelMLP(hidden=case["hidden"], ffn=case["ffn"], tokens=case["tokens"])
        with torch.no_grad():
            mlp.up.weight.copy_(s.pop("w_up"))
            mlp.down.weight.copy_(s.pop("w_down"))
        s["mlp"] = mlp
        s["x"].requires_grad_(True)
    elif k in ("moe", "exchange", "dispatch", "combine"):
        s["moe"] = MoeDispatchCombine(case["T"], case["H"], case["K"], case["E"], payload="fp8" if k == "dispatch" else "bf16")
        if k == "moe":
            s["w_in"] = torch.stack([fg.interleave_gate_up(w) for w in s["w_in"]])
            s["act"] = torch.empty(case["T"] * case["K"], case["F"], dtype=BF16, device="cuda")
        if k == "combine":
            recv, _ = s["moe"].dispatch(s["x"], s["idx"])
            s["moe"].expert_out.copy_(recv)
    else:
        s["sym"] = _Symmetric(s.pop("src"))
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    k = s["case"]["kind"]
    if k == "gemm":
        return fg.gemm(s["x"], s["w"], act=s["act"])
    if k == "mlp":
        y = s["mlp"](s["x"])
        dx, dup, ddown = torch.autograd.grad(y, [s["x"], s["mlp"].up.weight, s["mlp"].down.weight], s["dy"])
        return {"y": y, "dx": dx, "d_up": dup, "d_down": ddown}
    if k == "moe":
        moe = s["moe"]
        recv, offsets = moe.dispatch(s["x"], s["idx"])
        fg.grouped_gemm(recv, s["w_in"], offsets, out=s["act"], act="swiglu")
        fg.grouped_gemm(s["act"], s["w_out"], offsets, out=moe.expert_out)
        return {"out": moe.combine(s["idx"], s["weight"]), "offsets": offsets}
    if k == "exchange":
        moe = s["moe"]
        recv, offsets = moe.dispatch(s["x"], s["idx"])
        moe.expert_out.copy_(recv)
        return {"out": moe.combine(s["idx"], s["weight"]), "offsets": offsets}
    if k == "dispatch":
        moe = s["moe"]
        _, offsets = moe.dispatch(s["x"], s["idx"])
        rows = moe.slot_map.view(-1)
        return {"bytes": moe.recv_raw.index_select(0, rows), "scale": moe.recv_scale.index_select(0, rows), "offsets": offsets}
    if k == "combine":
        return s["moe"].combine(s["idx"], s["weight"])
    sym = s["sym"]
    nv.collective_on_buffer(s["case"]["coll"], nv.Teams.TEAM_WORLD, sym.dst, sym.src, op="sum")
    return sym.dst


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    k = case["kind"]
    if k == "gemm":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 2 * (M * K + N * K + M * N), "flops": 2 * M * N * K}
    if k == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        # inputs x, dy and two weights; outputs y, dx and two weight gradients; six products
        return {"bytes": 2 * (4 * t * h + 4 * h * f), "flops": 12 * t * h * f}
    T, H, E, K = (case[n] for n in ("T", "H", "E", "K")) if k != "coll" else (0, 0, 0, 0)
    routing = T * K * 8
    if k == "moe":
        F = case["F"]
        # distinct experts that T * K choices reach on average: only their weights have to be read
        reached = E * (1.0 - (1.0 - K / E) ** T)
        return {"bytes": 2 * 2 * T * H + routing + 2 * reached * 3 * F * H, "flops": 6 * T * K * F * H}
    if k == "exchange":
        return {"bytes": 2 * (T * H + 4 * T * K * H + T * H) + routing, "flops": 2 * T * K * H}
    if k == "dispatch":
        row = H + H // 32
        return {"bytes": 2 * T * H + 3 * T * K * row + routing // 2, "flops": 2 * T * H}
    if k == "combine":
        return {"bytes": 2 * T * K * H + 2 * T * H + routing, "flops": 2 * T * K * H}
    return {"bytes": 2 * case["n"] * torch.empty((), dtype=DTYPES[case["dtype"]]).element_size(), "flops": 0}


def tolerance(case):
    k = case["kind"]
    if k in ("coll", "dispatch"):
        return "exact"      # bytes are moved; the fp8 codes and scales are those of one documented quantisation
    if k == "gemm":
        return {"rel": 4e-3, "max": 0.03}   # one rounding to bf16 of sums that may be taken in another order
    if k in ("exchange", "combine"):
        return {"rel": 4e-3, "max": 0.03}
    return {"rel": 1e-2, "max": 0.1}        # intermediate results are rounded to bf16 as well


# ------------------------------------------------------------------ the same in 64 bits
def _gelu(h):
    return 0.5 * h * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (h + 0.044715 * h ** 3)))


def exact(case, seed):
    _init()
    k, d = case["kind"], _inputs(case, seed)
    if k == "gemm":
        y = d["x"].double() @ d["w"].double().t()
        return _gelu(y) if case["act"] else y
    if k == "mlp":
        x, w1, w2 = (d[n].double().requires_grad_(True) for n in ("x", "w_up", "w_down"))
        y = _gelu(x @ w1.t()) @ w2.t()
        dx, d1, d2 = torch.autograd.grad(y, [x, w1, w2], d["dy"].double())
        return {"y": y.detach(), "dx": dx, "d_up": d1, "d_down": d2}
    if k == "coll":
        return d["src"].double() if d["src"].is_floating_point() else None
    T, H, E, K = (case[n] for n in ("T", "H", "E", "K"))
    idx, weight, x = d["idx"].long(), d["weight"].double(), d["x"].double()
    if k == "dispatch":
        amax = x.view(T, H // 128, 128).abs().amax(-1).clamp(min=1e-10)
        scale = (amax / 448.0).unsqueeze(1).expand(T, K, H // 128).reshape(T * K, H // 128)
        return {"bytes": None, "scale": scale, "offsets": None}
    if k in ("exchange", "combine"):
        out = x * weight.sum(-1, keepdim=True)
        return {"out": out, "offsets": None} if k == "exchange" else out
    out = torch.zeros(T, H, dtype=torch.float64, device="cuda")
    for e in range(E):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        if tok.numel():
            h = x[tok] @ d["w_in"][e].double().t()
            h = torch.nn.functional.silu(h[:, :case["F"]]) * h[:, case["F"]:]
            out.index_add_(0, tok, (h @ d["w_out"][e].double().t()) * weight[tok, slot].unsqueeze(-1))
    return {"out": out, "offsets": None}
