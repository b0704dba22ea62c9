"""Workloads of the library as its users run them, for timing: linear layers on freshly quantised activations,
a BF16 training step, mixture-of-experts layers and the indexer's attention logits.

`listed()` names representative cases, `draw(rng)` picks another case of the same ranges, `prepare` makes what a
program holds before the call (inputs, resident weights), `run` is one pass through the public operators, `work` the
bytes and floating-point operations a pass cannot do without, `tolerance` how far two correct results may differ."""
import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "deepgemm-rs_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import deepgemm as dg  # noqa: E402
from deepgemm import Dtype, Operand, Output, SfGran, SfTensor, moe, synth  # noqa: E402

# (N, K) of the benchmark's dense projections
_PROJECTIONS = ((24576, 1536), (7168, 16384), (4096, 7168))
# the largest drawn linear layer: its FLOPs stay below the largest listed case
_MAX_LINEAR_FLOPS = 1.2e12


def listed():
    return [
        # one decode step of a projection: sixteen sequences, one token each; launch latency and the weight stream count
        dict(name="linear_decode", kind="linear", dtype="fp8", gran=128, m=16, n=4096, k=7168),
        # a large decode batch against a long contraction: the weights (117 MB) are streamed once
        dict(name="linear_decode_long_k", kind="linear", dtype="fp8", gran=128, m=100, n=7168, k=16384),
        # an ordinary prefill chunk of ragged length under per-32 scales, wide output and short contraction
        dict(name="linear_chunk_per32", kind="linear", dtype="fp8", gran=32, m=1021, n=24576, k=1536),
        # a full prefill batch, FP8 with per-128 scales
        dict(name="linear_prefill", kind="linear", dtype="fp8", gran=128, m=4096, n=7168, k=16384),
        # a full prefill batch with MXFP4 weights and activations
        dict(name="linear_prefill_fp4", kind="linear", dtype="fp4", gran=32, m=4096, n=7168, k=7168),
        # BF16 training step of a linear layer: forward, input gradient, weight gradient over two micro-batches
        dict(name="train_bf16", kind="train", m=2048, n=4096, k=7168),
        # prefill of an MoE projection: 256 experts, top-8, the largest batch
        dict(name="moe_prefill", kind="moe", tokens=16384, experts=256, topk=8, hidden=7168, n=4096),
        # the whole MoE feed-forward layer on a ragged chunk, the experts of one GPU of a group
        dict(name="moe_ffn_chunk", kind="moe_ffn", tokens=2019, experts=64, topk=8, hidden=7168, inter=2048),
        # decode of an MoE projection: 32 experts per GPU, up to 256 rows each, most of them partly filled
        dict(name="moe_decode", kind="moe_masked", groups=32, max_m=256, n=4096, k=7168),
        # indexer logits of a long prefill, f32 contract, causal over one sequence
        dict(name="indexer_prefill", kind="indexer", tokens=4096, kv=32768, heads=64, dim=128, sequences=1),
        # indexer logits of a packed chunk of three sequences under UE8M0 scales, ragged
        dict(name="indexer_chunk", kind="indexer_scaled", dtype="fp8", tokens=1000, kv=20011, heads=64, dim=128, sequences=3),
        # indexer logits of a decode step over a paged cache, contexts of different lengths
        dict(name="indexer_decode", kind="indexer_paged", dtype="fp8", requests=128, next_n=2, ctx=32768, page=64, heads=64, dim=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "train", "moe", "moe_ffn", "moe_masked", "indexer", "indexer_scaled",
                       "indexer_paged"])
    if kind == "linear":
        dtype, gran = rng.choice([("fp8", 128), ("fp8", 128), ("fp8", 32), ("fp4", 32)])
        if rng.random() < 0.5:
            n, k = rng.choice(_PROJECTIONS)
        else:
            n, k = 8 * _log_int(rng, 64, 3072), 256 * _log_int(rng, 4, 64)
        m = _log_int(rng, 1, 8192)
        m = max(1, min(m, int(_MAX_LINEAR_FLOPS / (2 * n * k))))
        return dict(kind=kind, dtype=dtype, gran=gran, m=m, n=n, k=k)
    if kind == "train":
        return dict(kind=kind, m=64 * _log_int(rng, 4, 64), n=64 * _log_int(rng, 16, 112), k=64 * _log_int(rng, 16, 112))
    if kind == "moe":
        return dict(kind=kind, tokens=_log_int(rng, 64, 16000), experts=rng.choice([16, 32, 64, 128, 256]),
                    topk=rng.choice([2, 4, 6, 8]), hidden=512 * rng.randint(4, 14), n=128 * rng.randint(8, 32))
    if kind == "moe_ffn":
        return dict(kind=kind, tokens=_log_int(rng, 64, 8000), experts=rng.choice([16, 32, 64, 128]),
                    topk=rng.choice([2, 4, 6, 8]), hidden=512 * rng.randint(4, 14), inter=512 * rng.randint(1, 4))
    if kind == "moe_masked":
        return dict(kind=kind, groups=rng.choice([4, 8, 16, 32, 64]), max_m=4 * _log_int(rng, 4, 128), n=128 * rng.randint(8, 56),
                    k=512 * rng.randint(3, 14))
    if kind == "indexer":
        tokens = _log_int(rng, 16, 4096)
        return dict(kind=kind, tokens=tokens, kv=max(tokens, _log_int(rng, 1024, 32768)), heads=rng.choice([32, 64, 64, 128]), dim=128,
                    sequences=rng.choice([1, 1, 2, 4]))
    if kind == "indexer_scaled":
        tokens = _log_int(rng, 16, 4096)
        return dict(kind=kind, dtype=rng.choice(["fp8", "fp8", "fp4"]), tokens=tokens, kv=max(tokens, _log_int(rng, 1024, 32768)),
                    heads=rng.choice([32, 64, 64]), dim=128, sequences=rng.choice([1, 1, 2, 4]))
    return dict(kind=kind, dtype=rng.choice(["fp8", "fp8", "fp4"]), requests=_log_int(rng, 1, 256), next_n=rng.choice([1, 1, 2, 3]),
                ctx=_log_int(rng, 512, 32768), page=rng.choice([16, 32, 64, 64, 128]), heads=rng.choice([32, 64, 64]), dim=128)


def _sequence_windows(tokens, kv, sequences):
    """Packed sequences: queries and kv rows are split evenly, query i of a sequence sees that sequence's kv rows up
    to its own position (the queries are the last rows of their sequence).  Lists of (start, end) over all queries."""
    win = []
    for s in range(sequences):
        q0, q1 = tokens * s // sequences, tokens * (s + 1) // sequences
        k0, k1 = kv * s // sequences, kv * (s + 1) // sequences
        for i in range(q1 - q0):
            win.append((k0, max(k0 + 1, k1 - (q1 - q0) + i + 1)))
    return win


def _weights(dtype, gran, n, k, gen, dev):
    """Resident weights of a linear layer: 128 x 128 blocks where the shape allows it, else one scale per row and group."""
    w = torch.randn((n, k), device=dev, generator=gen) * k ** -0.5
    if dtype == "fp8" and gran == 128 and n % 128 == 0 and k % 512 == 0:
        codes, sf = synth.block128_quant_fp8(w)
        return Operand.k_major(Dtype.Fp8, n, k, k, SfTensor(k // 512, n, SfGran.G128, sf), codes)
    kind = Dtype.Fp8 if dtype == "fp8" else Dtype.Fp4
    codes, sf = dg.quant_mx(w, n, k, kind, gran)
    return Operand.k_major(kind, n, k, k, sf, codes)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    c = dict(case)
    kind = c["kind"]

    def randn(*shape):
        return torch.randn(shape, device=dev, generator=gen)

    if kind == "linear":
        c["w"] = _weights(c["dtype"], c["gran"], c["n"], c["k"], gen, dev)
        c["x"] = randn(c["m"], c["k"])
    elif kind == "train":
        m, n, k = c["m"], c["n"], c["k"]
        c["w"] = (randn(n, k) * k ** -0.5).to(torch.bfloat16)
        c["x"] = [randn(m, k).to(torch.bfloat16) for _ in range(2)]
        c["dy"] = [randn(m, n).to(torch.bfloat16) for _ in range(2)]
        c["dw"] = torch.empty((n, k), dtype=torch.float32, device=dev)
    elif kind in ("moe", "moe_ffn"):
        e, h = c["experts"], c["hidden"]
        if kind == "moe":
            c["layer"] = moe.ExpertParallelMoE(synth.random_expert_weights(e, c["n"], h, seed, dev), e)
        else:
            c["layer"] = moe.GroupedMoEFfn(synth.random_expert_weights(e, 2 * c["inter"], h, seed, dev),
                                           synth.random_expert_weights(e, h, c["inter"], seed + 7, dev), e)
        c["x"] = randn(c["tokens"], h)
        c["idx"], c["topk_w"] = synth.random_topk_routing(c["tokens"], e, c["topk"], seed + 13, dev)
    elif kind == "moe_masked":
        g, mm, n, k = c["groups"], c["max_m"], c["n"], c["k"]
        c["w"] = synth.random_expert_weights(g, n, k, seed, dev)
        codes, sf = dg.quant_mx(randn(g * mm, k), g * mm, k, Dtype.Fp8, 128)
        c["a"] = Operand.k_major(Dtype.Fp8, mm, k, k, sf, codes)
        c["masked_m"] = torch.randint(0, mm + 1, (g,), device=dev, generator=gen, dtype=torch.int32)
        c["out"] = Output(Dtype.Bf16, mm, n, n, torch.zeros((g * mm, n), dtype=torch.bfloat16, device=dev))
    elif kind in ("indexer", "indexer_scaled"):
        t, s, heads, d = c["tokens"], c["kv"], c["heads"], c["dim"]
        win = _sequence_windows(t, s, c["sequences"])
        c["ks"] = torch.tensor([a for a, _ in win], dtype=torch.int32, device=dev)
        c["ke"] = torch.tensor([b for _, b in win], dtype=torch.int32, device=dev)
        c["width"] = (max(b - a for a, b in win) + 7) // 8 * 8
        if kind == "indexer":
            c["q"] = randn(t, heads, d).to(torch.float8_e4m3fn).view(torch.uint8)
            kvf = randn(s, d)
            c["scale"] = kvf.abs().amax(dim=1) / 448.0
            c["kv_codes"] = (kvf / c["scale"][:, None]).to(torch.float8_e4m3fn).view(torch.uint8)
            c["hw"] = randn(t, heads)
            c["logits"] = torch.zeros((t, c["width"]), dtype=torch.float32, device=dev)
        else:
            dt = Dtype.Fp8 if c["dtype"] == "fp8" else Dtype.Fp4
            codes, sf = dg.quant_mx(randn(t * heads, d), t * heads, d, dt, 32)
            c["q"] = Operand.k_major(dt, t * heads, d, d, sf, codes)
            codes, sf = dg.quant_mx(randn(s, d), s, d, dt, 32)
            c["kv_op"] = Operand.k_major(dt, s, d, d, sf, codes)
            c["hw"] = randn(t, heads).to(torch.bfloat16)
            c["logits"] = torch.zeros((t, c["width"]), dtype=torch.bfloat16, device=dev)
    else:
        b, nn, ctx, page, heads, d = c["requests"], c["next_n"], c["ctx"], c["page"], c["heads"], c["dim"]
        t = b * nn
        per = -(-ctx // page)
        pages = b * per + 3
        dt = Dtype.Fp8 if c["dtype"] == "fp8" else Dtype.Fp4
        codes, sf = dg.quant_mx(randn(t * heads, d), t * heads, d, dt, 32)
        c["q"] = Operand.k_major(dt, t * heads, d, d, sf, codes)
        codes, sf = dg.quant_mx(randn(pages * page, d), pages * page, d, dt, 32)
        c["kv_pages"], c["kv_words"], c["num_pages"] = codes, sf.buf[0, :pages * page].contiguous(), pages
        c["hw"] = randn(t, heads).to(torch.bfloat16)
        perm = torch.randperm(pages, device=dev, generator=gen).to(torch.int32)
        table = torch.zeros((t, per), dtype=torch.int32, device=dev)
        table[::nn] = perm[:b * per].view(b, per)
        c["table"], c["per"] = table, per
        c["req"] = torch.arange(b, device=dev, dtype=torch.int32).repeat_interleave(nn)
        last = torch.randint(max(nn, ctx // 4), ctx + 1, (b,), device=dev, generator=gen)     # context of a request's last token
        c["lens"] = (last[:, None] - (nn - 1) + torch.arange(nn, device=dev)[None, :]).reshape(-1).to(torch.int32)
        c["width"] = (ctx + 7) // 8 * 8
        c["logits"] = torch.zeros((t, c["width"]), dtype=torch.bfloat16, device=dev)
    return c


def run(s):
    kind = s["kind"]
    if kind == "linear":
        m, n, k, w = s["m"], s["n"], s["k"], s["w"]
        codes, sf = dg.quant_mx(s["x"], m, k, w.dtype, s["gran"])
        y = torch.empty((m, n), dtype=torch.bfloat16, device=codes.device)
        dg.gemm_nt(Operand.k_major(w.dtype, m, k, k, sf, codes), w, Output(Dtype.Bf16, m, n, n, y))
        return y, codes, sf.buf
    if kind == "train":
        m, n, k, w, dw = s["m"], s["n"], s["k"], s["w"], s["dw"]
        ys, dxs = [], []
        for i, (x, dy) in enumerate(zip(s["x"], s["dy"])):
            y = torch.empty((m, n), dtype=torch.bfloat16, device=x.device)
            dx = torch.empty((m, k), dtype=torch.bfloat16, device=x.device)
            dg.bf16_gemm_nt(Operand.k_major(Dtype.Bf16, m, k, k, None, x), Operand.k_major(Dtype.Bf16, n, k, k, None, w),
                            Output(Dtype.Bf16, m, n, n, y))
            # dx = dy . w, dw += dy^T . x: the transposed operands are MN-major views of the same buffers
            dg.gemm_nn(Operand.k_major(Dtype.Bf16, m, n, n, None, dy), Operand.mn_major(Dtype.Bf16, k, n, k, None, w),
                       Output(Dtype.Bf16, m, k, k, dx))
            dg.gemm_tt(Operand.mn_major(Dtype.Bf16, n, m, n, None, dy), Operand.mn_major(Dtype.Bf16, k, m, k, None, x),
                       Output(Dtype.F32, n, k, k, dw), accumulate=i > 0)
            ys.append(y)
            dxs.append(dx)
        return ys, dxs, dw
    if kind in ("moe", "moe_ffn"):
        codes, sf = dg.quant_mx(s["x"], s["tokens"], s["hidden"], Dtype.Fp8, 128)
        return s["layer"].forward(codes, sf, s["idx"], s["topk_w"])
    if kind == "moe_masked":
        dg.m_grouped_fp8_gemm_nt_masked(s["a"], s["w"], s["out"], s["masked_m"], s["groups"], max(1, s["max_m"] // 2))
        return s["out"].data
    if kind == "indexer":
        dg.mqa_logits_f32(s["q"], s["kv_codes"], s["scale"], s["hw"], s["ks"], s["ke"], s["tokens"], s["kv"], s["heads"], s["dim"],
                          s["logits"], s["width"])
    elif kind == "indexer_scaled":
        dg.mqa_logits(s["q"], s["kv_op"], s["hw"], s["ks"], s["ke"], s["tokens"], s["kv"], s["heads"], s["dim"], s["logits"], s["width"])
    else:
        dg.mqa_logits_paged(s["q"], s["kv_pages"], s["kv_words"], s["hw"], s["page"], s["num_pages"], s["lens"], s["req"], s["table"],
                            s["per"], s["requests"] * s["next_n"], s["heads"], s["dim"], s["logits"], s["width"])
    return s["logits"]


def work(case):
    c, kind = case, case["kind"]
    if kind == "linear":
        m, n, k, e = c["m"], c["n"], c["k"], 1.0 if c["dtype"] == "fp8" else 0.5
        sf = (m + n) * (k / c["gran"])
        return {"bytes": 4.0 * m * k + e * (m + n) * k + sf + 2.0 * m * n, "flops": 2.0 * m * n * k}
    if kind == "train":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2.0 * (2 * (2 * m * k + 2 * m * n) + n * k) + 4.0 * n * k, "flops": 2 * 6.0 * m * n * k}
    if kind == "moe":
        t, h, n = c["tokens"], c["hidden"], c["n"]
        used = c["experts"] * (1 - (1 - c["topk"] / c["experts"]) ** t)                    # expected experts with a token
        return {"bytes": 4.0 * t * h + used * n * h + 2.0 * t * n, "flops": 2.0 * t * c["topk"] * n * h}
    if kind == "moe_ffn":
        t, h, i = c["tokens"], c["hidden"], c["inter"]
        used = c["experts"] * (1 - (1 - c["topk"] / c["experts"]) ** t)
        return {"bytes": 4.0 * t * h + used * 3.0 * h * i + 2.0 * t * h, "flops": 6.0 * t * c["topk"] * h * i}
    if kind == "moe_masked":
        g, n, k = c["groups"], c["n"], c["k"]
        rows = g * c["max_m"] / 2.0                                                         # expected rows (uniform fill)
        used = g * c["max_m"] / (c["max_m"] + 1.0)
        return {"bytes": rows * k + used * n * k + 2.0 * rows * n, "flops": 2.0 * rows * n * k}
    heads, d = c["heads"], c["dim"]
    if kind in ("indexer", "indexer_scaled"):
        pairs = float(sum(b - a for a, b in _sequence_windows(c["tokens"], c["kv"], c["sequences"])))
        e = 0.5 if c.get("dtype") == "fp4" else 1.0
        out = 4.0 if kind == "indexer" else 2.0
        return {"bytes": e * d * (c["tokens"] * heads + c["kv"]) + out * pairs + 4.0 * c["kv"] + out * c["tokens"] * heads,
                "flops": 2.0 * heads * d * pairs}
    tokens = c["requests"] * (max(c["next_n"], c["ctx"] // 4) + c["ctx"]) / 2.0             # expected cached tokens
    e = 0.5 if c["dtype"] == "fp4" else 1.0
    return {"bytes": tokens * (e * d + 4) + 2.0 * c["next_n"] * tokens, "flops": 2.0 * heads * d * c["next_n"] * tokens}


def tolerance(case):
    """Largest differences between correct implementations, about four times what the library shows against the same
    path in float64: BF16 outputs of one rounding 1.7e-3 (largest element 3.9e-3), MoE layers, whose copies are rounded
    before they are combined, 2.3e-3 (1.4e-2), f32 logits 7e-8 (4e-7).  Codes and scale words are whole numbers and equal."""
    if case["kind"] in ("moe", "moe_ffn"):
        return {"rel": 9e-3, "max": 6e-2}
    if case["kind"] == "indexer":
        return {"rel": 1e-6, "max": 1e-5}
    return {"rel": 7e-3, "max": 2e-2}


def _scales(sf, col0, cols, k, gran):
    """The float64 factor of every row of [col0, col0 + cols) and group of `gran` columns: byte j of word row r is group 4 r + j."""
    words = sf[:, col0:col0 + cols].to(torch.int64) & 0xffffffff
    e = torch.stack([(words >> (8 * j)) & 0xff for j in range(4)], dim=1).reshape(-1, cols)[:k // gran]
    return torch.exp2(e.to(torch.float64) - 127.0).t()


def _decode(dtype, codes, sf, col0, rows, k, gran):
    """Rows [col0, col0 + rows) of a quantised operand as float64 values."""
    raw = codes.view(torch.uint8).reshape(-1, k // 2 if dtype == Dtype.Fp4 else k)[col0:col0 + rows]
    if dtype == Dtype.Fp4:
        table = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, -0.0, -.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64, device=raw.device)
        v = torch.stack([table[(raw & 15).long()], table[(raw >> 4).long()]], dim=-1).reshape(rows, k)
    else:
        v = raw.view(torch.float8_e4m3fn).to(torch.float64)
    return (v.view(rows, k // gran, gran) * _scales(sf, col0, rows, k, gran)[:, :, None]).view(rows, k)


def _rounded(x, dtype, gran):
    """x after quantisation: every group of `gran` columns scaled by the smallest power of two that brings its largest
    magnitude to the largest code or below, then rounded to the nearest code (ties to even)."""
    m, k = x.shape
    g = x.to(torch.float64).view(m, k // gran, gran)
    top = 6.0 if dtype == Dtype.Fp4 else 448.0
    s = torch.exp2(torch.ceil(torch.log2(g.abs().amax(dim=2, keepdim=True).clamp_min(1e-30) / top)))
    v = g / s
    if dtype == Dtype.Fp4:
        step = torch.where(v.abs() < 2, 0.5, torch.where(v.abs() < 4, 1.0, 2.0)).to(torch.float64)
        q = torch.round(v / step) * step
    else:
        q = v.to(torch.float32).to(torch.float8_e4m3fn).to(torch.float64)
    return (q * s).view(m, k)


def _relu_logits(q, kv, hw):
    """sum_h hw[i, h] relu(<q[i, h], kv[j]>) for [i, h, d], [j, d] and [i, h]."""
    s = torch.einsum("ihd,jd->ihj", q, kv).clamp_min_(0)
    return torch.einsum("ihj,ih->ij", s, hw)


def exact(case, seed):
    """What `run` returns, in float64 from the same inputs.  The codes and scale words of the linear layers are whole
    numbers that have no more exact value."""
    s = prepare(case, seed)
    kind = s["kind"]
    f64 = torch.float64
    if kind == "linear":
        m, n, k, w = s["m"], s["n"], s["k"], s["w"]
        x = _rounded(s["x"], w.dtype, s["gran"])
        return x @ _decode(w.dtype, w.data, w.sf.buf, 0, n, k, int(w.sf.gran)).t(), None, None
    if kind == "train":
        w = s["w"].to(f64)
        xs, dys = [x.to(f64) for x in s["x"]], [d.to(f64) for d in s["dy"]]
        return [x @ w.t() for x in xs], [d @ w for d in dys], sum(d.t() @ x for x, d in zip(xs, dys))
    if kind in ("moe", "moe_ffn"):
        x, idx, tw = _rounded(s["x"], Dtype.Fp8, 128), s["idx"].long(), s["topk_w"].to(f64)
        w1 = s["layer"].w if kind == "moe" else s["layer"].w13
        out = torch.zeros((s["tokens"], s["n"] if kind == "moe" else s["hidden"]), dtype=f64, device=x.device)
        for e in range(s["experts"]):
            t, j = (idx == e).nonzero(as_tuple=True)
            if t.numel() == 0:
                continue
            y = x[t] @ _decode(w1.dtype, w1.data, w1.sf.buf, e * w1.rows, w1.rows, w1.k, int(w1.sf.gran)).t()
            if kind == "moe_ffn":
                y, w2, i = y.to(torch.bfloat16).to(f64), s["layer"].w2, s["inter"]
                h = _rounded(y[:, :i] * torch.sigmoid(y[:, :i]) * y[:, i:], Dtype.Fp8, 128)
                y = h @ _decode(w2.dtype, w2.data, w2.sf.buf, e * w2.rows, w2.rows, w2.k, int(w2.sf.gran)).t()
            out.index_add_(0, t, y * tw[t, j][:, None])
        return out
    if kind == "moe_masked":
        a, w, mm = s["a"], s["w"], s["max_m"]
        out = torch.zeros(s["out"].data.shape, dtype=f64, device=s["out"].data.device)
        for g, r in enumerate(s["masked_m"].tolist()):
            if r:
                out[g * mm:g * mm + r] = _decode(a.dtype, a.data, a.sf.buf, g * mm, r, a.k, 128) @ \
                    _decode(w.dtype, w.data, w.sf.buf, g * w.rows, w.rows, w.k, int(w.sf.gran)).t()
        return out
    heads, d, hw = s["heads"], s["dim"], s["hw"].to(f64)
    logits = torch.zeros(s["logits"].shape, dtype=f64, device=hw.device)
    if kind == "indexer_paged":
        dt, per, page, nn = s["q"].dtype, s["per"], s["page"], s["next_n"]
        kv = _decode(dt, s["kv_pages"], s["kv_words"][None], 0, s["num_pages"] * page, d, 32).view(s["num_pages"], page, d)
        q = _decode(dt, s["q"].data, s["q"].sf.buf, 0, hw.shape[0] * heads, d, 32).view(-1, heads, d)
        lens = s["lens"].tolist()
        for b in range(s["requests"]):
            rows = kv[s["table"][b * nn, :per].long()].view(per * page, d)
            for t in range(b * nn, b * nn + nn):
                logits[t, :lens[t]] = _relu_logits(q[t:t + 1], rows[:lens[t]], hw[t:t + 1])[0]
        return logits
    if kind == "indexer":
        q = s["q"].view(torch.float8_e4m3fn).to(f64)
        kv = s["kv_codes"].view(torch.float8_e4m3fn).to(f64) * s["scale"].to(f64)[:, None]
    else:
        q = _decode(s["q"].dtype, s["q"].data, s["q"].sf.buf, 0, s["tokens"] * heads, d, 32).view(-1, heads, d)
        kv = _decode(s["kv_op"].dtype, s["kv_op"].data, s["kv_op"].sf.buf, 0, s["kv"], d, 32)
    ks, ke = s["ks"].tolist(), s["ke"].tolist()
    for t0 in range(0, s["tokens"], 64):
        t1 = min(s["tokens"], t0 + 64)
        lo, hi = min(ks[t0:t1]), max(ke[t0:t1])
        part = _relu_logits(q[t0:t1], kv[lo:hi], hw[t0:t1])
        for t in range(t0, t1):
            logits[t, :ke[t] - ks[t]] = part[t - t0, ks[t] - lo:ke[t] - lo]
    return logits
