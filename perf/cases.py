"""The attention calls whose speed this repository cares about, as data: what is called, on which sizes, and what the
call cannot do without.

Every case goes through the public entry points as a model would: the two modules (`SparseLinearAttention`,
`SageSparseLinearAttention`), the mask predicted once and handed back (`norm_rope_and_predict` + `forward(block_map=)`),
and the operator pair `get_block_map` / `_attention.apply` of the reference's own kernel benchmark. The sizes are those
of the repository's benchmark configurations (`sla_b200/synthetic.py`), its README and its edge-shape tests.

A case's fields:
  call     "train": module forward + backward; "infer": module forward without gradients; "sage": quantized forward;
           "layer": QK norm + rotary embedding + mask prediction + forward on the predicted mask, without gradients;
           "kernel": sparse operator forward + backward on a mask made beforehand
  B, H, L, D, BLKQ, topk (kept fraction of KV blocks; KV blocks have 64 rows)
  dtype    of the tensors the caller passes; compute: the module's 16-bit type
  feature  feature map of the linear branch; scope: its summation scope
  values   "randn", or "grid": tokens of a (t, 30, 52) latent grid with a positional term, whose block scores are
           structured like those of video models
"""
import math

import torch

import sla_b200

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(call, B, H, L, D, BLKQ, topk, dtype="bf16", compute="bf16", feature="softmax", scope="all", values="grid", **kw):
    return dict(kw, call=call, B=B, H=H, L=L, D=D, BLKQ=BLKQ, topk=topk, dtype=dtype, compute=compute, feature=feature,
                scope=scope, values=values)


def listed():
    return [
        # one short clip or image in fp32, forward only: the smallest call, bound by launches and host work
        _case("infer", 1, 2, 1024, 64, 64, 0.25, dtype="fp32", values="randn", name="infer_small_fp32"),
        # the README's training shape
        _case("train", 2, 4, 4096, 128, 64, 0.2, values="randn", name="train_readme"),
        # a ragged fp16 training step: odd length, batch and heads that do not fill the chip
        _case("train", 2, 3, 2049, 128, 128, 0.2, dtype="fp16", compute="fp16", feature="elu", values="randn",
              name="train_ragged_fp16"),
        # quantized forward of a short ragged sequence at head dim 64
        _case("sage", 2, 4, 1931, 64, 128, 0.15, values="randn", name="sage_ragged_d64"),
        # self-attention of a 1.3B-like video model (21x30x52 latents): one training step
        _case("train", 1, 12, 32760, 128, 64, 0.05, name="train_video"),
        # the same attention in a sampler
        _case("infer", 1, 12, 32760, 128, 64, 0.05, name="infer_video"),
        # what one GPU does of that training step when the 12 heads are spread over 8 GPUs
        _case("train", 1, 2, 32760, 128, 64, 0.05, name="train_video_2heads"),
        # the sampler's whole attention layer: norm, rotary embedding, mask and attention
        _case("layer", 1, 12, 32760, 128, 64, 0.05, name="layer_video"),
        # training with the linear branch restricted to the blocks that were not selected
        _case("train", 1, 12, 32760, 128, 64, 0.05, scope="unselected", name="train_video_unselected"),
        # quantized forward of a 14B-like video model (75600 tokens, 40 heads)
        _case("sage", 1, 40, 75600, 128, 128, 0.05, name="sage_video_14b"),
        # the reference's kernel benchmark: sparse operator forward + backward, mask outside
        _case("kernel", 2, 16, 32760, 128, 128, 0.05, values="randn", name="kernel_bench"),
        # long-sequence training at head dim 64
        _case("train", 1, 16, 131072, 64, 128, 0.05, feature="relu", name="train_long_d64"),
    ]


# The ranges behind the listed cases: smallest and largest L, how the calls are spread, what a call may cost.
_RANGES = {"infer": (256, 131072), "train": (256, 131072), "sage": (512, 75600), "layer": (1024, 75600),
           "kernel": (512, 65536)}


def draw(rng):
    most_flops = 0.9 * max(work(c)["flops"] for c in listed())
    call = rng.choice(["infer", "train", "train", "sage", "layer", "kernel"])
    lo, hi = _RANGES[call]
    while True:
        L = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if rng.random() < 0.3:
            L = max(lo, L // 64 * 64)        # whole blocks, as padded sequences have
        D = rng.choice([64, 128, 128])
        BLKQ = 128 if call == "sage" else rng.choice([64, 128])
        B = rng.choice([1, 1, 1, 2, 3])
        H = rng.choice([1, 2, 3, 5, 8, 12, 16, 24, 40])
        # short sequences keep a larger share of their blocks than long ones
        topk = round(math.exp(rng.uniform(math.log(0.03 if L > 8192 else 0.08), math.log(0.2 if L > 8192 else 0.5))), 3)
        compute = rng.choice(["bf16", "bf16", "fp16"])
        dtype = compute if call in ("layer", "kernel") or rng.random() < 0.75 else "fp32"
        feature = rng.choice(["softmax", "softmax", "relu", "elu"])
        scope = "unselected" if call == "train" and rng.random() < 0.15 else "all"
        values = "grid" if L > 8192 and call != "kernel" else "randn"
        # at least one KV block is kept; the tcgen05 kernels' lists reach to L = 98304 at 64-row query blocks and head
        # dim 128; q stays within the largest listed tensor
        if int(topk * ((L + 63) // 64)) < 1 or (BLKQ == 64 and L > 98304) or B * H * L * D > 40 * 75600 * 128:
            continue
        c = _case(call, B, H, L, D, BLKQ, topk, dtype, compute, feature, scope, values)
        if work(c)["flops"] <= most_flops:
            return c


def _inputs(c, seed, count):
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (c["B"], c["H"], c["L"], c["D"])
    ts = [torch.randn(shape, generator=g, device="cuda") for _ in range(count)]
    if c["values"] == "grid":
        n = torch.arange(c["L"], device="cuda")
        theta = 10000.0 ** (-torch.arange(32, device="cuda", dtype=torch.float32) / 32.0)
        angles = [x.float()[:, None] * theta for x in (n // 1560, n // 52 % 30, n % 52)]
        feats = torch.cat([f(a) for a in angles for f in (torch.sin, torch.cos)], dim=-1)
        pos = feats @ (torch.randn(192, c["D"], generator=g, device="cuda") / 192 ** 0.5)
        for t in ts[:2]:
            t.mul_(0.5).add_(pos)
    return [t.to(_DTYPES[c["dtype"]]) for t in ts], g


def prepare(case, seed):
    c = case
    train = c["call"] in ("train", "kernel")
    (q, k, v, *rest), g = _inputs(c, seed, 4 if train else 3)
    s = {"call": c["call"], "q": q, "k": k, "v": v}
    if train:
        s["do"] = rest[0]
        for t in (q, k, v):
            t.requires_grad_(True)
    if c["call"] == "kernel":
        with torch.no_grad():
            s["map"] = sla_b200.get_block_map(q, k, c["topk"], c["BLKQ"], 64)
        s["BLKQ"] = c["BLKQ"]
        return s
    use_bf16 = c["compute"] == "bf16"
    if c["call"] == "sage":
        m = sla_b200.SageSparseLinearAttention(c["D"], c["topk"], c["feature"], use_bf16=use_bf16)
    else:
        m = sla_b200.SparseLinearAttention(c["D"], c["topk"], c["feature"], c["BLKQ"], 64, use_bf16=use_bf16,
                                           linear_scope=c["scope"])
    m = m.cuda()
    with torch.no_grad():
        m.proj_l.weight.copy_(torch.randn(c["D"], c["D"], generator=g, device="cuda") * 0.02)
        m.proj_l.bias.copy_(torch.randn(c["D"], generator=g, device="cuda") * 0.02)
    s["m"] = m
    if c["call"] == "layer":
        ang = torch.arange(c["L"], device="cuda")[:, None] * 10000.0 ** (-torch.arange(c["D"] // 2, device="cuda") / (c["D"] // 2))
        s["cos"], s["sin"] = torch.cos(ang), torch.sin(ang)
        s["gq"], s["gk"] = (1 + 0.1 * torch.randn(c["D"], generator=g, device="cuda") for _ in range(2))
    return s


def run(state):
    s = state
    q, k, v = s["q"], s["k"], s["v"]
    if s["call"] == "train":
        m = s["m"]
        params = (q, k, v, m.proj_l.weight, m.proj_l.bias)
        for t in params:
            t.grad = None
        o = m(q, k, v)
        o.backward(s["do"])
        return {"o": o, **{n: t.grad for n, t in zip(("dq", "dk", "dv", "dw", "db"), params)}}
    if s["call"] == "kernel":
        smap, lut, topk = s["map"]
        for t in (q, k, v):
            t.grad = None
        o = sla_b200._attention.apply(q, k, v, smap, lut, topk, s["BLKQ"], 64)
        o.backward(s["do"])
        return {"o": o, "dq": q.grad, "dk": k.grad, "dv": v.grad}
    with torch.no_grad():
        if s["call"] == "layer":
            qn, kn, bm = s["m"].norm_rope_and_predict(q, k, s["gq"], s["gk"], s["cos"], s["sin"], with_column_lists=False)
            return {"q": qn, "k": kn, "o": s["m"](qn, kn, v, block_map=bm)}
        return s["m"](q, k, v)


def work(case):
    """Tensors of the caller's type once in and once out, and the matrix work of the selected blocks (2 contractions
    forward, 5 backward) and of the linear branch (state and read-out forward; dO W H, G, and the two of dK, dV
    backward). The scope "unselected" adds the unnormalised pass over the selected blocks, 2 forward and 5 backward."""
    c = case
    B, H, L, D = c["B"], c["H"], c["L"], c["D"]
    kept = int(c["topk"] * ((L + 63) // 64)) * 64
    unit = 2.0 * B * H * L * min(kept, L) * D
    linear = 2.0 * B * H * L * D * D
    tensor = float(B * H * L * D * (4 if c["dtype"] == "fp32" else 2))
    tensors = {"train": 8, "kernel": 8, "infer": 4, "sage": 4, "layer": 6}[c["call"]]
    flops = unit * (7 if c["call"] in ("train", "kernel") else 2)
    if c["scope"] == "unselected":
        flops *= 2
    if c["call"] != "kernel":
        flops += linear * (6 if c["call"] == "train" else 2)
    return {"bytes": tensors * tensor, "flops": flops}


def tolerance(case):
    """16-bit outputs of contractions whose operands (P, dS, phi) are rounded to 16 bits: about 1e-2. The quantized
    forward rounds P to e4m3 (3 mantissa bits, 2.6% rms a value), at points that depend on the running maximum."""
    return {"rel": 3e-2 if case["call"] == "sage" else 1e-2}
