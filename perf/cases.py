"""What a user of this library has it do, as cases that can be timed on one GPU.

A case is one call (or one short chain of calls) through the public entry
points, at the sizes one rank of a tensor-parallel program sees: row-parallel
linear layers with all-reduce or reduce-scatter and RMSNorm, gathered and
dispatched GEMMs, the reference-compatible layer with its reordering RMSNorm,
RMSNorm alone, and a decoder block.  Decode is the low end (the smallest tile
height, 128 tokens), prefill the rest; both 16-bit types appear.

The tile configuration (``algo``) of a case is the first that the library's own
model proposes for the shape (``gather_algo_candidates``) and that divides it,
which is what a program without a tuning file takes.
"""
from __future__ import annotations

import math

import torch

import flashoverlap_b200  # noqa: F401  (loads the native library)
from flashoverlap_b200 import ops
from flashoverlap_b200.models import FusedRowParallelLinear, OverlapRowParallelLayer, ReorderRMSNorm
from flashoverlap_b200.models.decoder_block import TPDecoderBlock
from flashoverlap_b200.tune.model import gather_algo_candidates
from flashoverlap_b200.utils.config import ALGO_TILES

EPS = 1e-5
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
# hidden, ffn, heads, kv heads of the decoder block
BLOCK = (4096, 14336, 32, 8)
# the most multiply-adds a case may have (the largest listed one)
MOST = 8192 * 8192 * 28672


def _algo(m: int, n: int) -> int:
    for algo in gather_algo_candidates(m, n):
        if m % ALGO_TILES[algo][0] == 0:
            return algo
    raise ValueError(f"no tile configuration divides {m} x {n}")


def _linear(kind: str, m: int, n: int, k: int, dtype: str, norm: bool, name: str = "") -> dict:
    c = {"kind": kind, "m": m, "n": n, "k": k, "dtype": dtype, "norm": norm, "algo": _algo(m, n)}
    return dict(c, name=name) if name else c


def listed() -> list:
    return [
        # the norm of a decode step: a few dozen tokens, launch latency only; a width that is no power of two
        {"name": "rmsnorm-decode", "kind": "rmsnorm", "m": 37, "n": 8000, "dtype": "fp16"},
        # the norm between the layers of a long prefill
        {"name": "rmsnorm-prefill", "kind": "rmsnorm", "m": 16384, "n": 4096, "dtype": "bf16"},
        # a decode step's attention out-projection, hidden 8192 split over 8 ranks
        _linear("all_reduce", 128, 8192, 1024, "fp16", True, "allreduce-norm-decode"),
        # the same projection in prefill: one rank's share, and the whole of it on one GPU
        _linear("all_reduce", 4096, 8192, 1024, "fp16", True, "allreduce-norm-prefill-tp8"),
        _linear("all_reduce", 4096, 8192, 8192, "fp16", True, "allreduce-norm-prefill-tp1"),
        # the MLP down-projection with sequence parallelism: one rank of 8, and all of it (the largest case)
        _linear("reduce_scatter", 8192, 8192, 3584, "bf16", True, "reducescatter-norm-tp8"),
        _linear("reduce_scatter", 8192, 8192, 28672, "bf16", True, "reducescatter-norm-tp1"),
        # a decode step's QKV projection: reads its weights once, the tokens are few
        _linear("all_gather", 128, 10240, 8192, "bf16", False, "allgather-gemm-decode"),
        # tokens dispatched to an expert: as many rows as the router sends, not a multiple of any tile
        {"name": "all2all-gemm-ragged", "kind": "all_to_all", "m": 3333, "n": 2048, "k": 4096, "dtype": "fp16",
         "norm": False, "algo": 8},
        # a plain projection at sizes that fill no wave and no K step evenly
        _linear("gemm", 1152, 5120, 1720, "bf16", False, "gemm-odd"),
        # the reference-compatible layer with its tile-reordered output, followed by the norm that undoes the order
        {"name": "overlap-layer-reorder-norm", "kind": "overlap", "m": 2048, "n": 8192, "k": 1024, "dtype": "fp16",
         "norm": True, "algo": 8},
        # one decoder block's prefill
        {"name": "decoder-block-prefill", "kind": "block", "batch": 2, "seq": 1024, "dtype": "bf16"},
    ]


def _log(rng, lo: int, hi: int, step: int) -> int:
    """A multiple of ``step`` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 0.999)))
    return max(lo, min(hi, int(v) // step * step))


def draw(rng) -> dict:
    kind = rng.choice(["rmsnorm", "rmsnorm", "all_reduce", "all_reduce", "reduce_scatter", "reduce_scatter",
                       "all_gather", "all_to_all", "gemm", "overlap", "block"])
    dtype = rng.choice(sorted(DTYPES))
    if kind == "rmsnorm":
        n = _log(rng, 512, 32768, 8)  # any multiple of 8
        return {"kind": kind, "m": _log(rng, 1, min(32768, (1 << 28) // n), 1), "n": n, "dtype": dtype}
    if kind == "block":
        batch = rng.choice([1, 2, 3, 4])
        return {"kind": kind, "batch": batch, "seq": _log(rng, 256, 8192 // batch // 256 * 256, 256), "dtype": dtype}
    while True:
        # K in steps of 8 (any), rows in whole tiles of 128 (any number for the dispatch), columns in steps of 128
        m = _log(rng, 128, 16384, 128)
        n = _log(rng, 1024, 14336, 128)
        k = _log(rng, 256, 28672, 8)
        if m * n * k <= MOST:
            break
    if kind == "all_to_all":
        m = min(16384, m + rng.randrange(128))
        return {"kind": kind, "m": m, "n": n, "k": k, "dtype": dtype, "norm": False,
                "algo": gather_algo_candidates(m, n)[0]}
    if kind == "overlap":
        return {"kind": kind, "m": m, "n": n, "k": k, "dtype": dtype, "norm": True, "algo": _algo(m, n)}
    norm = kind in ("all_reduce", "reduce_scatter") and rng.random() < 0.75
    return _linear(kind, m, n, k, dtype, norm)


# ---------------------------------------------------------------------------
_impl = None
_blocks: dict = {}


def _shared_impl():
    """The one communication object a program keeps."""
    global _impl
    if _impl is None:
        _impl = torch.classes.flashoverlap_class.OverlapImpl()
        _impl.nccl_init(0, 1, [0] * 16)
        _impl.cutlass_init()
        _impl.overlap_init()
    return _impl


def _block(dtype):
    """The block whose weights a serving program loads once."""
    if dtype not in _blocks:
        hidden, ffn, heads, kv = BLOCK
        _blocks[dtype] = TPDecoderBlock(_shared_impl(), hidden, ffn, heads, kv, EPS, 8, dtype=dtype)
    return _blocks[dtype]


def _inputs(case: dict, seed: int) -> dict:
    """The tensors of a case, from the seed alone."""
    dt = DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(dt)

    kind = case["kind"]
    if kind == "block":
        tokens = case["batch"] * case["seq"]
        resid = normal(tokens, BLOCK[0])
        x = resid.float()
        return {"resid": resid, "h": (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS)).to(dt)}
    m, n = case["m"], case["n"]
    if kind == "rmsnorm":
        return {"x": normal(m, n), "w": (1 + 0.1 * torch.randn(n, device="cuda", generator=gen)).to(dt)}
    k = case["k"]
    x = normal(m, k)
    w = normal(n, k, scale=k ** -0.5)
    return {"x": x, "w": w, "g": (1 + 0.1 * torch.randn(n, device="cuda", generator=gen)).to(dt)}


def prepare(case: dict, seed: int) -> dict:
    dt = DTYPES[case["dtype"]]
    kind = case["kind"]
    t = _inputs(case, seed)
    if kind == "block":
        return {"kind": kind, "block": _block(dt), "batch": case["batch"], "seq": case["seq"], "resid": t["resid"],
                "h": t["h"]}
    m, n = case["m"], case["n"]
    if kind == "rmsnorm":
        return {"kind": kind, "x": t["x"], "w": t["w"]}
    k = case["k"]
    x, w, g = t["x"], t["w"], t["g"]
    if kind in ("all_reduce", "reduce_scatter"):
        layer = FusedRowParallelLinear(_shared_impl(), k, n, comm_op=kind, norm=case["norm"], eps=EPS,
                                       algo=case["algo"], dtype=dt)
        layer.weight = torch.nn.Parameter(w, requires_grad=False)
        if case["norm"]:
            layer.norm_weight = torch.nn.Parameter(g, requires_grad=False)
        return {"kind": kind, "layer": layer, "x": x}
    if kind == "overlap":
        bm, bn, _ = ALGO_TILES[case["algo"]]
        tm, tn = m // bm, n // bn
        # tiles in the order in which the kernel finishes them, in groups of one wave: a tuned file's hint and cSeg
        hint = list(torch.ops.flashoverlap_op.tile_walk(tm, tn, 2, True, 0, 1, 0, 0))
        wave = 148 * 128 // bm
        cseg = [min(wave, tm * tn - i) for i in range(0, tm * tn, wave)]
        config = {"BM": bm, "BN": bn, "Algo": case["algo"], "hint": hint, "cSeg": cseg}
        layer = OverlapRowParallelLayer(0, 1, k, n, m, config, "all_reduce", [0] * 16, dtype=dt)
        layer.weight = torch.nn.Parameter(w, requires_grad=False)
        norm = ReorderRMSNorm(n, m, bm, bn, hint, eps=EPS, dtype=dt)
        norm.weight = torch.nn.Parameter(g, requires_grad=False)
        return {"kind": kind, "layer": layer, "norm": norm, "x": x}
    state = {"kind": kind, "impl": _shared_impl(), "x": x, "w": w, "algo": case["algo"]}
    if kind == "all_to_all":
        state["mlen"] = torch.tensor([[m]], dtype=torch.int32)
    return state


def run(s: dict):
    kind = s["kind"]
    if kind == "rmsnorm":
        return ops.rmsnorm(s["x"], s["w"], EPS)
    if kind in ("all_reduce", "reduce_scatter"):
        return s["layer"](s["x"])
    if kind == "overlap":
        return s["norm"](s["layer"](s["x"]))
    if kind == "all_gather":
        return ops.allgather_gemm(s["impl"], s["x"], s["w"], 1, s["algo"])
    if kind == "all_to_all":
        return ops.a2a_dispatch_gemm(s["impl"], s["x"], s["w"], s["mlen"], 0, s["algo"])
    if kind == "gemm":
        return ops.gemm(s["impl"], s["x"], s["w"], s["algo"])
    return s["block"](s["h"], s["resid"], s["batch"], s["seq"])


def _norm64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w.double()


def exact(case: dict, seed: int):
    """What ``run`` returns, in 64 bits with torch's own operations."""
    t = _inputs(case, seed)
    kind = case["kind"]
    if kind == "rmsnorm":
        return _norm64(t["x"].double(), t["w"])
    if kind != "block":
        y = t["x"].double() @ t["w"].double().t()
        return _norm64(y, t["g"]) if case["norm"] else y
    hidden, ffn, heads, kv = BLOCK
    batch, seq, hd = case["batch"], case["seq"], hidden // heads
    p = _block(DTYPES[case["dtype"]])  # for its weights
    qkv = t["h"].double() @ p.w_qkv.double().t()
    q, k, v = (z.reshape(batch, seq, -1, hd) for z in qkv.split([hidden, kv * hd, kv * hd], dim=-1))
    hide = torch.ones(seq, seq, dtype=torch.bool, device="cuda").triu(1)
    attn = torch.empty(batch, seq, heads, hd, dtype=torch.float64, device="cuda")
    for b in range(batch):
        for h in range(heads):
            kh, vh = k[b, :, h * kv // heads], v[b, :, h * kv // heads]
            scores = (q[b, :, h] @ kh.t() / math.sqrt(hd)).masked_fill(hide, -math.inf)
            attn[b, :, h] = scores.softmax(-1) @ vh
    h2 = t["resid"].double() + attn.reshape(batch * seq, hidden) @ p.w_o.double().t()
    gate, up = (_norm64(h2, p.norm_attn) @ p.w_gate_up.double().t()).chunk(2, dim=-1)
    h3 = h2 + (torch.nn.functional.silu(gate) * up) @ p.w_down.double().t()
    return _norm64(h3, p.norm_next) @ p.w_qkv_next.double().t(), h3


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "block":
        hidden, ffn, heads, kv = BLOCK
        t = case["batch"] * case["seq"]
        qkv = hidden + 2 * kv * (hidden // heads)
        weights = 2 * qkv * hidden + hidden * hidden + 3 * ffn * hidden
        attention = 2 * case["batch"] * case["seq"] ** 2 * hidden  # causal: half of QK^T and PV
        return {"bytes": 2 * (weights + t * (3 * hidden + qkv)), "flops": 2 * t * weights + attention}
    m, n = case["m"], case["n"]
    if kind == "rmsnorm":
        return {"bytes": 2 * (2 * m * n + n), "flops": 4 * m * n}
    k = case["k"]
    norm = case["norm"]
    return {"bytes": 2 * (m * k + n * k + m * n + (n if norm else 0)), "flops": 2 * m * n * k + (4 * m * n if norm else 0)}


def tolerance(case: dict) -> dict:
    return TOLERANCE[case["dtype"]]["block" if case["kind"] == "block" else
                                    "norm" if case["kind"] == "rmsnorm" or case["norm"] else "gemm"]


# Measured against the same math in 64 bits (rel: 2-norm of the difference over that of the result; max: largest
# difference over the value or, where larger, the result's root mean square), times four.  fp16 then bf16, rel / max:
# GEMM 2.1e-4 / 5.0e-4 and 1.7e-3 / 3.9e-3; with RMSNorm (two roundings) 3.6e-4 / 1.4e-3 and 2.9e-3 / 1.1e-2;
# decoder block 4.7e-3 / 2.4e-2 in bf16, an eighth of it in fp16.
TOLERANCE = {
    "fp16": {"gemm": {"rel": 8e-4, "max": 2e-3}, "norm": {"rel": 1.4e-3, "max": 5.6e-3},
             "block": {"rel": 2.4e-3, "max": 1.2e-2}},
    "bf16": {"gemm": {"rel": 6.6e-3, "max": 1.6e-2}, "norm": {"rel": 1.1e-2, "max": 4.5e-2},
             "block": {"rel": 1.9e-2, "max": 9.6e-2}},
}
