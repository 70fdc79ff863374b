"""The work that a program built on this framework has it do, as timed cases: single layers of the model's MSA and pair
tracks (Q8, tf32, bf16 and exact fp32 Linears, forward and backward; attention, forward and backward; triangle
multiplication; outer-product-mean), each through the public entry points of `ops`.

Sizes are those of the model's full-size blocks (256 residues, MSA depth 256, extra MSA depth 1024: 65536 tokens), of its
development size (51 residues, MSA depth 8: 408 and 2601 tokens) and what lies between.  `math` says which arithmetic the
caller asked for: "exact" is fp32 on the CUDA cores (what the drop-in launchers run by default), "tf32" the tensor cores
behind fp32 tensors, "bf16" 16-bit operands.
"""
import math

import torch

from proteinpredictmachinelearning_b200 import ops
from proteinpredictmachinelearning_b200._lib import PATH_AUTO, PATH_SIMT


def listed():
    return [
        # Q8 projection of the development-size MSA (51 residues x 8 rows): the smallest call, latency and launches
        dict(name="q8_linear_dev", kind="q8", tokens=408, k=128, n=128),
        # Q, K, V and gate projections of an MSA attention as one Q8 Linear over all 65536 tokens
        dict(name="q8_linear_qkvg", kind="q8", tokens=65536, k=256, n=1024),
        # pair track: LayerNorm folded into a gate projection, sigmoid gate applied in the epilogue
        dict(name="linear_norm_gate", kind="norm_gate", tokens=65536, k=128, n=128),
        # feed-forward down projection with bf16 operands
        dict(name="linear_bf16", kind="linear", math="bf16", tokens=65536, k=1024, n=256),
        # training step of a 256 -> 256 Linear on the MSA: output, input gradient, weight gradient over 65536 tokens
        dict(name="linear_train_tf32", kind="linear_train", math="tf32", tokens=65536, k=256, n=256),
        # the same for a development-size pair Linear (51 x 51 tokens) in the default arithmetic of the drop-in launchers
        dict(name="linear_train_exact_dev", kind="linear_train", math="exact", tokens=2601, k=128, n=256),
        # MSA row attention with the pair bias and the gate, on the projection's output as it lies
        dict(name="attention_msa_gated", kind="attention", math="tf32", batch=256, heads=8, lq=256, lk=256, d=32,
             layout="tokens", bias=True, gate=True, causal=False),
        # extra-MSA row attention: 1024 rows, head dim 8
        dict(name="attention_extra_msa", kind="attention", math="tf32", batch=1024, heads=8, lq=256, lk=256, d=8,
             layout="dense", bias=True, gate=False, causal=False),
        # development-size pair attention in the default arithmetic of the drop-in launchers
        dict(name="attention_dev_exact", kind="attention", math="exact", batch=51, heads=8, lq=51, lk=51, d=32,
             layout="dense", bias=True, gate=False, causal=False),
        # training step of an attention: forward and all four gradients, exact fp32
        dict(name="attention_train_exact", kind="attention_train", batch=64, heads=8, l=256, d=32, bias=True, causal=False),
        # both triangle multiplications of a pair block
        dict(name="tri_mul_pair", kind="tri_mul", math="tf32", slabs=128, l=256),
        # outer-product-mean of a main block in the default arithmetic of the drop-in launchers
        dict(name="opm_exact", kind="opm", math="exact", slabs=16, l=256, rows=256),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["q8", "q8", "norm_gate", "linear", "linear", "linear_train", "linear_train", "attention", "attention",
                       "attention", "attention_train", "tri_mul", "opm"])
    if kind == "q8":                               # K in whole quant blocks; few output columns are the pair-bias projections
        return dict(kind=kind, tokens=_log(rng, 64, 65536), k=rng.choice([64, 96, 128, 256, 512, 1024]),
                    n=rng.choice([8, 16, _log(rng, 32, 1024), 128, 256, 512]))
    if kind == "norm_gate":
        return dict(kind=kind, tokens=_log(rng, 200, 65536), k=4 * _log(rng, 8, 64), n=_log(rng, 16, 384))
    if kind == "linear":
        m = rng.choice(["exact", "tf32", "bf16"])
        top = 256 if m == "exact" else 1024
        # K = 33 is the radial network's input width (no 16-byte rows: CUDA cores in every arithmetic)
        k = rng.choice([33, 64, 8 * _log(rng, 2, top // 8), _log(rng, 20, 200)])
        return dict(kind=kind, math=m, tokens=_log(rng, 100, 65536), k=k, n=rng.choice([_log(rng, 8, top), 128, 256]))
    if kind == "linear_train":
        return dict(kind=kind, math=rng.choice(["exact", "tf32"]), tokens=_log(rng, 100, 32768),
                    k=rng.choice([33, 64, 4 * _log(rng, 8, 64), 128, 256]), n=rng.choice([4 * _log(rng, 4, 64), 128, 256]))
    if kind == "attention":
        m = rng.choice(["exact", "tf32", "tf32", "bf16"])
        d = rng.choice([32, 32, 8, 8, 64, 16])
        lq = _log(rng, 17, 384)
        lk = rng.choice([lq, lq, 4 * _log(rng, 8, 96)])
        heads = rng.choice([1, 4, 8])
        budget = (1 << 26) if (m == "exact" or d not in (8, 32)) else (1 << 27)
        batch = max(1, min(256, budget // (heads * lq * lk * max(1, d // 16))))
        batch = _log(rng, max(1, batch // 8), batch)
        layout = "dense" if m == "bf16" else rng.choice(["dense", "tokens"])
        return dict(kind=kind, math=m, batch=batch, heads=heads, lq=lq, lk=lk, d=d, layout=layout, bias=rng.random() < 0.7,
                    gate=layout == "tokens" and rng.random() < 0.7, causal=lq == lk and rng.random() < 0.15)
    if kind == "attention_train":
        l, d, heads = _log(rng, 33, 256), rng.choice([32, 32, 8, 16, 64]), rng.choice([4, 8])
        batch = max(1, min(96, (1 << 25) // (heads * l * l * max(1, d // 32))))
        return dict(kind=kind, batch=_log(rng, max(1, batch // 6), batch), heads=heads, l=l, d=d, bias=rng.random() < 0.75,
                    causal=rng.random() < 0.15)
    if kind == "tri_mul":
        m = rng.choice(["exact", "tf32", "tf32", "bf16"])
        l = rng.choice([_log(rng, 40, 300), 8 * _log(rng, 6, 48)])
        return dict(kind=kind, math=m, slabs=rng.choice([16, 64, 128]), l=min(l, 256) if m == "exact" else l)
    m = rng.choice(["exact", "tf32", "bf16"])
    return dict(kind=kind, math=m, slabs=rng.choice([8, 16]), l=_log(rng, 48, 256), rows=rng.choice([8, 51, 128, 256, _log(rng, 16, 256)]))


# ---- inputs ------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, shape, scale=1.0):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).mul_(scale)


def _inputs(c, seed):
    """The tensors of a case, fp32, from the seed alone: activations behind a LayerNorm (unit variance), Linear weights
    N(0, 0.02), attention operands N(0, 1/32), pair biases and upstream gradients of unit variance."""
    g, k = _gen(seed), c["kind"]
    if k in ("q8", "linear", "linear_train"):
        t = dict(x=_randn(g, (c["tokens"], c["k"])), w=_randn(g, (c["n"], c["k"]), 0.02), b=_randn(g, (c["n"],), 0.1))
        if k == "linear_train":
            t["dy"] = _randn(g, (c["tokens"], c["n"]))
    elif k == "norm_gate":
        t = dict(x=_randn(g, (c["tokens"], c["k"])).add_(0.3), w=_randn(g, (c["n"], c["k"]), 0.02), b=_randn(g, (c["n"],), 0.1),
                 gamma=_randn(g, (c["k"],), 0.1).add_(1.0), beta=_randn(g, (c["k"],), 0.1), gate=_randn(g, (c["tokens"], c["n"])))
    elif k == "attention":
        s = 1.0 / math.sqrt(32.0)
        if c["layout"] == "tokens":                # [q | gate logits] and [k | v] as two projection outputs
            hd = c["heads"] * c["d"]
            t = dict(qg=_randn(g, (c["batch"], c["lq"], 2 * hd), s), kv=_randn(g, (c["batch"], c["lk"], 2 * hd), s))
            t["qg"][..., hd:].mul_(4.0)
        else:
            t = dict(q=_randn(g, (c["batch"], c["heads"], c["lq"], c["d"]), s), k=_randn(g, (c["batch"], c["heads"], c["lk"], c["d"]), s),
                     v=_randn(g, (c["batch"], c["heads"], c["lk"], c["d"]), s))
        t["bias"] = _randn(g, (c["heads"], c["lq"], c["lk"])) if c["bias"] else None
    elif k == "attention_train":
        s, shape = 1.0 / math.sqrt(32.0), (c["batch"], c["heads"], c["l"], c["d"])
        t = dict(q=_randn(g, shape, s), k=_randn(g, shape, s), v=_randn(g, shape, s), do=_randn(g, shape))
        t["bias"] = _randn(g, (c["heads"], c["l"], c["l"])) if c["bias"] else None
    elif k == "tri_mul":
        shape = (c["slabs"], c["l"], c["l"], 1)
        t = dict(left=_randn(g, shape), right=_randn(g, shape))
    else:
        shape = (c["slabs"], c["l"], c["rows"], 1)
        t = dict(left=_randn(g, shape), right=_randn(g, shape))
    if c.get("math") == "bf16":                    # 16-bit operands; biases stay fp32
        t = {n: (v if v is None or n in ("b", "bias") else v.to(torch.bfloat16)) for n, v in t.items()}
    return t


def prepare(case, seed):
    c, t = dict(case), _inputs(case, seed)
    c["path"] = PATH_SIMT if c.get("math") == "exact" else PATH_AUTO
    if c["kind"] == "q8":                          # the model keeps its weights quantized
        t["w"] = ops.quantize_q8_0r(t["w"])
    elif c["kind"] == "norm_gate":                 # and the LayerNorm terms folded into them
        t["wg"], t["u"], t["vv"] = ops.layernorm_fold(t["w"], t["gamma"], t["beta"], t["b"])
    elif c["kind"] == "linear_train":              # and a transposed copy for the input gradient
        t["wt"] = t["w"].t().contiguous()
    return c, t


def run(state):
    c, t = state
    k, path = c["kind"], c["path"]
    if k == "q8":
        return ops.mul_mat_q8_cuda(t["w"], t["x"], c["n"], bias=t["b"])[0]
    if k == "norm_gate":
        return ops.mul_mat_fused(t["x"], t["wg"], bias=t["vv"], ln_stats=ops.row_stats(t["x"]), ln_u=t["u"], gate=t["gate"], act="sigmoid")
    if k == "linear":
        if c["math"] == "bf16":
            return ops.mul_mat_16(t["x"], t["w"], bias=t["b"])
        return ops.mul_mat_cuda(t["x"], t["w"], bias=t["b"], path=path)
    if k == "linear_train":
        y = ops.mul_mat_cuda(t["x"], t["w"], bias=t["b"], path=path)
        dx = ops.mul_mat_cuda(t["dy"], t["wt"], path=path)
        dw = ops.out_prod_cuda(t["x"][None, None], t["dy"][None, None], path=path)[0, 0]
        return y, dx, dw
    if k == "attention":
        if c["layout"] == "tokens":
            hd = c["heads"] * c["d"]
            out = torch.empty((c["batch"], c["lq"], hd), device="cuda", dtype=torch.float32)
            return ops.flash_attn_tokens(t["qg"][..., :hd], t["kv"][..., :hd], t["kv"][..., hd:], c["heads"], bias=t["bias"],
                                         gate=t["qg"][..., hd:] if c["gate"] else None, causal=c["causal"], bias_bcast=c["bias"],
                                         path=path, out=out)
        return ops.flash_attn_forward_cuda(t["q"], t["k"], t["v"], t["bias"], causal=c["causal"], bias_bcast=c["bias"], path=path)
    if k == "attention_train":
        o, lse = ops.flash_attn_forward_cuda(t["q"], t["k"], t["v"], t["bias"], causal=c["causal"], bias_bcast=c["bias"], path=PATH_SIMT)
        g = ops.flash_attn_backward_cuda(t["q"], t["k"], t["v"], o, t["do"], lse, t["bias"], causal=c["causal"], bias_bcast=c["bias"])
        return o, lse, g["dQ"], g["dK"], g["dV"], g["dbias"]
    if k == "tri_mul":
        return (ops.tri_mul_cuda(t["left"], t["right"], c["l"], True, path=path),
                ops.tri_mul_cuda(t["left"], t["right"], c["l"], False, path=path))
    return ops.outer_prod_mean_cuda(t["left"], t["right"], path=path)


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def work(case):
    c, k = case, case["kind"]
    e = 2 if c.get("math") == "bf16" else 4
    if k == "q8":
        T, K, N = c["tokens"], c["k"], c["n"]
        return dict(bytes=34 * N * K // 32 + 4 * T * K + 4 * T * N + 4 * N, flops=2 * T * K * N)
    if k in ("linear", "norm_gate"):
        T, K, N = c["tokens"], c["k"], c["n"]
        return dict(bytes=e * (T * K + N * K) + 4 * N + (8 if k == "norm_gate" else 4) * T * N, flops=2 * T * K * N)
    if k == "linear_train":
        T, K, N = c["tokens"], c["k"], c["n"]
        return dict(bytes=4 * (2 * T * K + 2 * T * N + 2 * N * K + N), flops=6 * T * K * N)
    if k == "attention":
        B, h, lq, lk, d = c["batch"], c["heads"], c["lq"], c["lk"], c["d"]
        half = 0.5 if c["causal"] else 1.0
        nbytes = e * B * h * d * (lq + 2 * lk) + 4 * B * h * lq * (d + 1) + (4 * h * lq * lk if c["bias"] else 0)
        return dict(bytes=nbytes + (4 * B * h * lq * d if c["gate"] else 0), flops=int(half * 4 * B * h * lq * lk * d))
    if k == "attention_train":
        B, h, l, d = c["batch"], c["heads"], c["l"], c["d"]
        half = 0.5 if c["causal"] else 1.0
        return dict(bytes=4 * B * h * l * (8 * d + 1) + 4 * B * h * l * l + (4 * h * l * l if c["bias"] else 0),
                    flops=int(half * 14 * B * h * l * l * d))
    if k == "tri_mul":
        D, l = c["slabs"], c["l"]
        return dict(bytes=2 * e * D * l * l + 8 * D * l * l, flops=4 * D * l ** 3)
    D, l, n = c["slabs"], c["l"], c["rows"]
    return dict(bytes=2 * e * D * l * n + 4 * (D * l) ** 2, flops=2 * (D * l) ** 2 * n)


def tolerance(case):
    # measured against exact(): tf32 operands 2.4e-4 to 3.3e-4; behind a sigmoid of small logits 3.4e-5; fp32 sums 3e-8 to
    # 2.5e-6 (the longest: a weight gradient over 27000 tokens); bf16 probabilities 2e-3
    k, m = case["kind"], case.get("math")
    if k == "norm_gate":
        return {"rel": 2e-4}
    if m == "tf32":
        return {"rel": 1e-3}
    if k == "attention" and m == "bf16":
        return {"rel": 1e-2}
    return {"rel": 1e-5}


# ---- 64-bit results ----------------------------------------------------------------------------------------------------
def _quant(x, top, first_sign):
    """Blocks of 32 along the last axis as the block formats define them, in fp32: (integers, fp16-rounded scales)."""
    b = x.reshape(-1, 32)
    amax, idx = b.abs().max(dim=1)
    if first_sign:                                 # activations: scale from the first element of largest magnitude, sign kept
        hit = b.abs() == amax[:, None]
        idx = torch.argmax(hit.to(torch.int32), dim=1)
        d = b.gather(1, idx[:, None])[:, 0] / -128.0
        lo, hi = -128.0, 127.0
    else:
        d = amax / top
        lo, hi = -127.0, 127.0
    inv = torch.where(d == 0, torch.zeros_like(d), 1.0 / d)
    y = (b * inv[:, None]).double()
    q = torch.trunc(y + torch.copysign(torch.full_like(y, 0.5), y)).clamp_(lo, hi)
    return (q * d.to(torch.float16).double()[:, None]).reshape(x.shape)


def _sigmoid_gate(o, g):
    return torch.sigmoid(g.double()) * o


def _attention64(q, k, v, bias, scale, causal, do=None):
    """One chunk of batches in 64 bits; with `do` also dQ, dK, dV and dbias."""
    s = (q @ k.transpose(-1, -2)) * scale
    if bias is not None:
        s = s + bias
    if causal:
        lq, lk = s.shape[-2:]
        s = s.masked_fill(torch.ones(lq, lk, dtype=torch.bool, device=s.device).triu(1), -math.inf)
    lse = torch.logsumexp(s, dim=-1)
    p = torch.exp(s - lse[..., None])
    o = p @ v
    if do is None:
        return o, lse
    ds = p * (do @ v.transpose(-1, -2) - (do * o).sum(-1, keepdim=True))
    return o, lse, scale * (ds @ k), scale * (ds.transpose(-1, -2) @ q), p.transpose(-1, -2) @ do, ds


def exact(case, seed):
    c, t = case, _inputs(case, seed)
    k = c["kind"]
    if k == "q8":
        return _quant(t["x"], 128.0, True) @ _quant(t["w"], 127.0, False).t() + t["b"].double()
    t = {n: (v if v is None else v.double()) for n, v in t.items()}
    if k == "norm_gate":
        x = torch.nn.functional.layer_norm(t["x"], (c["k"],), t["gamma"], t["beta"], 1e-5)
        return _sigmoid_gate(t["gate"], x @ t["w"].t() + t["b"])
    if k == "linear":
        return t["x"] @ t["w"].t() + t["b"]
    if k == "linear_train":
        return t["x"] @ t["w"].t() + t["b"], t["dy"] @ t["w"], t["dy"].t() @ t["x"]
    if k == "attention":
        B, h, lq, lk, d = c["batch"], c["heads"], c["lq"], c["lk"], c["d"]
        scale = 1.0 / math.sqrt(d)
        if c["layout"] == "tokens":
            hd = h * d
            split = lambda x, n: x.reshape(B, n, h, d).transpose(1, 2)
            q, kk, v = split(t["qg"][..., :hd], lq), split(t["kv"][..., :hd], lk), split(t["kv"][..., hd:], lk)
        else:
            q, kk, v = t["q"], t["k"], t["v"]
        step = max(1, (1 << 27) // (h * lq * lk))
        parts = [_attention64(q[i:i + step], kk[i:i + step], v[i:i + step], t["bias"], scale, c["causal"]) for i in range(0, B, step)]
        o, lse = (torch.cat(p) for p in zip(*parts))
        if c["layout"] == "tokens":
            o = o.transpose(1, 2).reshape(B, lq, hd)
            if c["gate"]:
                o = _sigmoid_gate(o, t["qg"][..., hd:])
        return o, lse
    if k == "attention_train":
        scale, step = 1.0 / math.sqrt(c["d"]), max(1, (1 << 26) // (c["heads"] * c["l"] ** 2))
        parts = [_attention64(t["q"][i:i + step], t["k"][i:i + step], t["v"][i:i + step], t["bias"], scale, c["causal"], t["do"][i:i + step])
                 for i in range(0, c["batch"], step)]
        return tuple(torch.cat(p) for p in zip(*parts))
    left, right = t["left"][..., 0], t["right"][..., 0]
    if k == "tri_mul":
        out = (left @ right.transpose(1, 2)) / c["l"]
        inc = (left.transpose(1, 2) @ right) / c["l"]
        return out.clamp(-1e4, 1e4)[..., None], inc.clamp(-1e4, 1e4)[..., None]
    D, l, n = c["slabs"], c["l"], c["rows"]
    full = (left.reshape(D * l, n) @ right.reshape(D * l, n).t()) / n
    return full.reshape(D, l, D, l).permute(0, 2, 1, 3).reshape(D * D, l, l, 1)
