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
        _case("train", 2, 3, 2049, 128, 128, 0.2, dtype="fp16", compute="fp16", values="randn", name="train_ragged_fp16"),
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
        # phi(q) . z of the unnormalised maps leaves the fp16 range after some hundred tokens
        feature = rng.choice(["softmax", "softmax", "relu", "elu"]) if compute == "bf16" else "softmax"
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


def _rope(c):
    half = c["D"] // 2
    angles = torch.arange(c["L"], device="cuda")[:, None] * 10000.0 ** (-torch.arange(half, device="cuda") / half)
    return torch.cos(angles), torch.sin(angles)


def _gains(c, g):
    return [1 + 0.1 * torch.randn(c["D"], generator=g, device="cuda") for _ in range(2)]


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
        s["cos"], s["sin"] = _rope(c)
        s["gq"], s["gk"] = _gains(c, g)
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

def _phi(x, feature):
    if feature == "softmax":
        return torch.softmax(x, dim=-1)
    return torch.nn.functional.elu(x) + 1 if feature == "elu" else torch.relu(x)


def _block_means(x, rows):
    pad = -x.shape[0] % rows
    sums = torch.nn.functional.pad(x, (0, 0, 0, pad)).view(-1, rows, x.shape[1]).sum(1)
    sums /= rows
    if pad:
        sums[-1] *= rows / (rows - pad)
    return sums


def _selected(c, q, k):
    """The blocks that each query block keeps, (mb, topk), for one head: a discrete choice, hence with the 16-bit
    roundings that belong to its definition, and the lower index in a tie."""
    dt = _DTYPES[c["dtype"]]
    mean = k.double().mean(0).to(dt)
    if c["call"] == "layer":       # from block sums: the mean comes off the block's mean
        pk = (_block_means(k.double(), 64) - mean.double()).to(dt)
    else:
        pk = _block_means((k - mean).double(), 64).to(dt)
    pq = _block_means(q.double(), c["BLKQ"]).to(dt)
    score = (pq.double() @ pk.double().T).to(dt)
    keep = min(score.shape[1], int(c["topk"] * score.shape[1]))
    return torch.sort(score, dim=-1, descending=True, stable=True).indices[:, :keep].sort(dim=-1).values


def _exact_head(c, q, k, v, do, sel, w, b):
    """Output of one head in the type of q, k, v; with `do`, their gradients (and w's and b's) accumulate."""
    L, D, BQ = c["L"], c["D"], c["BLKQ"]
    scope = "none" if c["call"] == "kernel" else c["scope"]
    outs, lin = [], []
    if scope != "none":            # the state over all tokens, a leaf of its own for the chunks below
        phik = _phi(k, c["feature"])
        state = [phik.T @ v, phik.sum(0)]
        lin = [t.detach().requires_grad_(do is not None) for t in state]
    kept = sel.shape[1] * 64
    blocks = max(1, int(2 ** 27 / (BQ * kept)))
    for i0 in range(0, sel.shape[0], blocks):
        keys = (sel[i0:i0 + blocks, :, None] * 64 + torch.arange(64, device=q.device)).flatten(1)
        r0, r1 = i0 * BQ, min(L, (i0 + blocks) * BQ)
        n, there = keys.shape[0], (keys < L)
        keys = keys.clamp(max=L - 1)
        qb = torch.nn.functional.pad(q[r0:r1], (0, 0, 0, n * BQ - (r1 - r0))).view(n, BQ, D)
        kb, vb = k[keys], v[keys]
        s = (qb @ kb.transpose(1, 2) * D ** -0.5).masked_fill(~there[:, None], -math.inf)
        o = torch.softmax(s, dim=-1) @ vb
        if scope != "none":
            H, z = lin
            phiq = _phi(qb, c["feature"])
            if scope == "unselected":
                pk = _phi(kb, c["feature"]) * there[:, :, None]
                H, z = H - pk.transpose(1, 2) @ vb, z - pk.sum(1)[:, None]
            if scope == "all" or sel.shape[1] < (L + 63) // 64:
                o_l = (phiq @ H) / (1e-5 + (phiq * z).sum(-1, keepdim=True))
            else:
                o_l = 0 * phiq
            o = o + o_l @ w.T + b
        o = o.reshape(n * BQ, D)[:r1 - r0]
        if do is not None:
            o.backward(do[r0:r1])
        outs.append(o.detach())
    if do is not None and lin:
        torch.autograd.backward([s for s, t in zip(state, lin) if t.grad is not None], [t.grad for t in lin if t.grad is not None])
    return torch.cat(outs)


def exact(case, seed):
    """The formulas of the operator in 64 bits, one head and a few query blocks at a time; the quantized forward is
    measured against the attention without quantization."""
    c = case
    train = c["call"] in ("train", "kernel")
    (q, k, v, *rest), g = _inputs(c, seed, 4 if train else 3)
    D = c["D"]
    w = b = None
    if c["call"] != "kernel":
        w, b = ((torch.randn(*n, generator=g, device="cuda") * 0.02).double().requires_grad_(train) for n in ((D, D), (D,)))
    extra = {}
    if c["call"] == "layer":
        cos, sin = _rope(c)
        gq, gk = _gains(c, g)
        qk = []
        for x, gain in ((q, gq), (k, gk)):
            y = x.double()
            y = y * torch.rsqrt(y.square().mean(-1, keepdim=True) + 1e-6) * gain.double()
            e, o = y[..., 0::2], y[..., 1::2]
            qk.append(torch.stack([e * cos - o * sin, e * sin + o * cos], -1).flatten(-2))
        extra = {"q": qk[0], "k": qk[1]}
    out = {n: torch.empty(q.shape, dtype=torch.float64, device="cuda") for n in (("o", "dq", "dk", "dv") if train else ("o",))}
    for i in range(c["B"]):
        for h in range(c["H"]):
            if c["call"] == "layer":
                ts = [qk[0][i, h], qk[1][i, h], v[i, h].double()]
                sel = _selected(c, *(t.to(_DTYPES[c["dtype"]]) for t in ts[:2]))
            else:
                ts = [t[i, h].double().requires_grad_(train) for t in (q, k, v)]
                sel = _selected(c, q[i, h], k[i, h])
            with torch.set_grad_enabled(train):
                out["o"][i, h] = _exact_head(c, *ts, rest[0][i, h].double() if train else None, sel, w, b)
            if train:
                for n, t in zip(("dq", "dk", "dv"), ts):
                    out[n][i, h] = t.grad
    if c["call"] == "train":
        out["dw"], out["db"] = w.grad, b.grad
    if train or c["call"] == "layer":
        return {**extra, **out}
    return out["o"]
