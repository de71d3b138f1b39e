"""The work a program gives this library, as timed cases.

Every case goes through the public interface (`fe2o3_b200.prepare(...)` once, then `.launch(stream)` per pass, or
`MoeTop2Layer.forward()`), on buffers that stay on the GPU.  Sizes come from the benchmark's configurations and the
tests; `draw` spreads further cases over the ranges that they stand for.
"""
import math

import torch

import fe2o3_b200 as fe
from fe2o3_b200.moe import MoeTop2Layer


def listed():
    return [
        # -- bf16 GEMM, packed operands: a large training-size product, and the smallest one in use, where one
        #    launch is a few microseconds of loads, a few k steps and the output
        {"name": "gemm_8192", "op": "gemm", "m": 8192, "n": 8192, "k": 8192},
        {"name": "gemm_512", "op": "gemm", "m": 512, "n": 512, "k": 512},
        # -- C = alpha*A*B + beta*C on padded storage with sizes that end inside every tile
        {"name": "gemm_general_ragged", "op": "gemm_general", "m": 1000, "n": 3001, "k": 1111, "pad_a": 1, "pad_b": 15, "pad_c": 3,
         "alpha": 0.5, "beta": -0.25},
        # -- f32 GEMM with the reference's order of additions (the benchmark's first configuration)
        {"name": "scalar_gemm_512", "op": "scalar_gemm", "m": 512, "n": 512, "k": 512},
        # -- attention: the benchmark's shape, and a causal one of the wider common head size with a ragged length
        {"name": "attention_2048", "op": "attention", "batch": 4, "heads": 16, "seq": 2048, "dim": 64, "causal": False},
        {"name": "attention_causal_1900", "op": "attention", "batch": 2, "heads": 12, "seq": 1900, "dim": 128, "causal": True},
        # -- row softmax: the benchmark's shape, and long odd rows under an activity mask
        {"name": "softmax_65536x1024", "op": "softmax", "rows": 65536, "cols": 1024, "masked": False},
        {"name": "softmax_masked_5000x3001", "op": "softmax", "rows": 5000, "cols": 3001, "masked": True},
        # -- masked u32 sum at the benchmark's size
        {"name": "reduce_2p28", "op": "reduce", "n": 1 << 28, "packed": False},
        # -- prefix sum of a mid-size array: launches and carries count, not only the stream
        {"name": "scan_1m", "op": "scan", "n": (1 << 20) + 3, "dtype": "u32", "exclusive": False},
        # -- the MoE layer of the headline configuration: a whole batch, and a decode-size step in which the experts'
        #    weights are the work
        {"name": "moe_16384", "op": "moe", "tokens": 16384, "d": 2048, "f": 4096, "experts": 8, "capacity": 0},
        {"name": "moe_64", "op": "moe", "tokens": 64, "d": 2048, "f": 4096, "experts": 8, "capacity": 0},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["gemm", "gemm", "gemm_general", "scalar_gemm", "attention", "attention", "softmax", "softmax", "reduce", "scan",
                     "moe", "moe"])
    if op == "gemm":   # tiled_gemm_v1 admits multiples of 16
        m, n, k = (16 * _log(rng, 8, 512) for _ in range(3))
        return {"op": op, "m": m, "n": n, "k": k}
    if op == "gemm_general":
        # most callers pad their rows to whole 16-byte lines; packed odd rows come too
        m, n, k = (_log(rng, 16, 3000) for _ in range(3))
        packed = rng.random() < 0.2
        alpha, beta = rng.choice([(1.0, 0.0), (1.0, 1.0), (0.5, -0.25)])
        return {"op": op, "m": m, "n": n, "k": k, "pad_a": 0 if packed else -k % 8 + 8 * rng.randrange(3),
                "pad_b": 0 if packed else -n % 8 + 8 * rng.randrange(3), "pad_c": rng.randrange(8), "alpha": alpha, "beta": beta}
    if op == "scalar_gemm":
        m, n, k = (_log(rng, 32, 1024) for _ in range(3))
        return {"op": op, "m": m, "n": n, "k": k}
    if op == "attention":
        seq = _log(rng, 64, 4096)
        batch = _log(rng, 1, 8)
        heads = max(1, min(32, (4 * 16 * 2048 * 2048) // (batch * seq * seq), rng.randrange(1, 33)))
        return {"op": op, "batch": batch, "heads": heads, "seq": seq, "dim": rng.choice([64, 64, 64, 128, 128, 32, 96]),
                "causal": rng.random() < 0.5}
    if op == "softmax":
        cols = rng.choice([_log(rng, 16, 4096), 4 * _log(rng, 4, 1024)])
        rows = _log(rng, 16, min(65536, (1 << 26) // cols))
        return {"op": op, "rows": rows, "cols": cols, "masked": rng.random() < 0.4}
    if op == "reduce":
        return {"op": op, "n": _log(rng, 1 << 10, 1 << 28), "packed": rng.random() < 0.5}
    if op == "scan":
        return {"op": op, "n": _log(rng, 1 << 10, 1 << 28), "dtype": rng.choice(["u32", "f32"]), "exclusive": rng.random() < 0.5}
    d = rng.choice([256, 512, 1024, 2048, 2048])
    experts = rng.choice([8, 8, 16])
    tokens = _log(rng, 16, 16384)
    # 0: no route is dropped; otherwise the expert's share of the routes and a quarter more
    capacity = rng.choice([0, 0, max(1, (5 * tokens) // (2 * experts))])
    return {"op": op, "tokens": tokens, "d": d, "f": 2 * d, "experts": experts, "capacity": capacity}


_ctx = None


def _context():
    """One context and its default stream (shared with torch) per process, as a program keeps them."""
    global _ctx
    if _ctx is None:
        ctx = fe.GpuContext(torch.cuda.current_device())
        _ctx = (ctx, ctx.default_stream())
    return _ctx


def _uniform(g, n, dtype):   # [-1, 1)
    return torch.rand(n, generator=g, device="cuda").mul_(2).sub_(1).to(dtype)


class _Op:
    """One prepared launch, its buffers and what a pass of it returns."""

    def __init__(self, op, buffers, outputs, **kw):
        ctx, self.stream = _context()
        self.buffers, self.outputs = buffers, outputs
        self.prepared = fe.prepare(ctx, op, **buffers, **kw)

    def run(self):
        self.prepared.launch(self.stream)
        return self.outputs

    def __del__(self):
        self.prepared.destroy()


class _Layer:
    """A layer with its weights and tokens; kept for the life of the program, as are the buffers that it owns."""

    def __init__(self, case, g):
        ctx, stream = _context()
        self.layer = MoeTop2Layer(ctx, stream, case["tokens"], case["d"], case["f"], case["experts"],
                                  capacity=case["capacity"] or None)
        layer = self.layer
        layer.x.normal_(0, 1, generator=g)
        for w in (layer.wg, layer.w1, layer.w2):
            w.normal_(0, 0.02, generator=g)
        self.outputs = {"out": layer.out, "logits": layer.logits, "experts": layer.top2, "weights": layer.weights,
                        "admitted": layer.admitted}

    def run(self):
        self.layer.forward()
        return self.outputs


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    op = case["op"]
    if op == "moe":
        return _Layer(case, g)
    if op in ("gemm", "scalar_gemm"):
        m, n, k = case["m"], case["n"], case["k"]
        dtype = torch.bfloat16 if op == "gemm" else torch.float32
        c = torch.zeros(m * n, device="cuda")
        return _Op("tiled_gemm_v1" if op == "gemm" else "scalar_gemm_v1",
                   {"a": _uniform(g, m * k, dtype), "b": _uniform(g, k * n, dtype), "c": c}, c, m=m, n=n, k=k)
    if op == "gemm_general":
        m, n, k = case["m"], case["n"], case["k"]
        lda, ldb, ldc = k + case["pad_a"], n + case["pad_b"], n + case["pad_c"]
        c = _uniform(g, (m - 1) * ldc + n, torch.float32)
        return _Op("tiled_gemm_general_v1",
                   {"a": _uniform(g, (m - 1) * lda + k, torch.bfloat16), "b": _uniform(g, (k - 1) * ldb + n, torch.bfloat16), "c": c}, c,
                   m=m, n=n, k=k, lda=lda, ldb=ldb, ldc=ldc, alpha=case["alpha"], beta=case["beta"])
    if op == "attention":
        n = case["batch"] * case["heads"] * case["seq"] * case["dim"]
        q, k, v = (torch.randn(n, generator=g, device="cuda").to(torch.bfloat16) for _ in range(3))
        o = torch.zeros(n, device="cuda")
        return _Op("flash_attention_v1", {"q": q, "k": k, "v": v, "output": o}, o, batch=case["batch"], heads=case["heads"],
                   seq=case["seq"], dim=case["dim"], scale=1 / math.sqrt(case["dim"]), causal=int(case["causal"]),
                   input_dtype=fe.DTYPE_BF16)
    if op == "softmax":
        n = case["rows"] * case["cols"]
        buffers = {"input": torch.randn(n, generator=g, device="cuda").mul_(2), "output": torch.zeros(n, device="cuda")}
        if case["masked"]:
            mask = torch.rand(n, generator=g, device="cuda") < 0.75
            mask.view(case["rows"], case["cols"])[:, 0] = True   # a row without any active element is an error by contract
            buffers["mask"] = mask.to(torch.uint8)
        return _Op("row_softmax_v1", buffers, buffers["output"], rows=case["rows"], cols=case["cols"])
    n = case["n"]
    if op == "reduce":
        values = torch.randint(0, 1 << 16, (n,), generator=g, device="cuda", dtype=torch.int32)
        out = torch.zeros(1, dtype=torch.int32, device="cuda")
        if case["packed"]:   # either of two fair bits: active with probability 3/4
            words = [torch.randint(-(1 << 63), (1 << 63) - 1, ((n + 63) // 64,), generator=g, device="cuda") for _ in range(2)]
            return _Op("masked_reduce_u32_packed", {"values": values, "mask": words[0] | words[1], "output": out}, out)
        active = torch.randint(0, 4, (n,), generator=g, device="cuda", dtype=torch.int32).clamp_(0, 1).mul_(7)
        return _Op("masked_reduce_u32", {"values": values, "active": active, "output": out}, out)
    if case["dtype"] == "u32":
        values = torch.randint(0, 1 << 16, (n,), generator=g, device="cuda", dtype=torch.int32)
    else:
        values = torch.rand(n, generator=g, device="cuda")
    out = torch.zeros_like(values)
    return _Op("device_scan_" + case["dtype"], {"values": values, "output": out}, out, exclusive=int(case["exclusive"]))


def run(state):
    return state.run()


def work(case):
    op = case["op"]
    if op in ("gemm", "gemm_general", "scalar_gemm"):
        m, n, k = case["m"], case["n"], case["k"]
        e = 4 if op == "scalar_gemm" else 2
        reads_c = op == "gemm_general"   # beta*C is evaluated whatever beta is
        return {"bytes": e * (m * k + k * n) + (8 if reads_c else 4) * m * n, "flops": 2 * m * n * k}
    if op == "attention":
        heads, seq, dim = case["batch"] * case["heads"], case["seq"], case["dim"]
        pairs = seq * (seq + 1) // 2 if case["causal"] else seq * seq
        return {"bytes": heads * seq * dim * (3 * 2 + 4), "flops": 4 * heads * pairs * dim}
    if op == "softmax":
        return {"bytes": case["rows"] * case["cols"] * (9 if case["masked"] else 8), "flops": 0}
    if op == "reduce":
        return {"bytes": case["n"] * (4 + (0.125 if case["packed"] else 4)) + 4, "flops": 0}
    if op == "scan":
        return {"bytes": case["n"] * 8, "flops": 0}
    T, d, f, E = case["tokens"], case["d"], case["f"], case["experts"]
    rows = 2 * T
    if case["capacity"]:   # routes fall nearly evenly on the experts
        rows = min(rows, E * case["capacity"])
    hit = min(E, rows)     # experts whose weights are read
    return {"bytes": T * d * 2 + d * E * 2 + hit * d * f * 4 + T * d * 4 + T * (4 * E + 16), "flops": rows * 4 * d * f + 2 * T * d * E}


def tolerance(case):
    # each about four times the error measured against the same path in f64
    op = case["op"]
    if op in ("scalar_gemm", "reduce") or (op == "scan" and case["dtype"] == "u32"):
        return "exact"   # order of additions fixed by contract; whole numbers
    if op == "moe":      # hidden activations are bf16 (1.7e-3); routing is exact
        return {"rel": 8e-3, "max": 0.05, "differ": 0.0}
    if op == "attention" and case["dim"] == 64:   # probabilities are bf16 at this head size (1.9e-3)
        return {"rel": 8e-3, "max": 0.05}
    if op in ("gemm", "gemm_general", "attention"):   # f32 sums of exact products of up to 8192 terms (8.6e-6)
        return {"rel": 4e-5}
    return {"rel": 1e-5}   # shorter f32 sums
