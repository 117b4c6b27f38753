"""The row passes whose CTAs walk several tiles or heads through a ring of copies: against the same unit in a call so small
that a CTA has one, and against the formulas."""
import ctypes as C

import pytest
import torch

from sla_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _randn(shape, seed, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(dtype)


def _up(n):
    return (n + 255) // 256 * 256


def _quantized(q, k):
    """INT8 rows, scales and the mean of k that the quantized forward makes of q and k, from its workspace
    (csrc/workspace.h, WsSage)."""
    B, H, L, D = q.shape
    bh, mb, nb = B * H, (L + 127) // 128, (L + 63) // 64
    w = torch.zeros(D, D, device="cuda")
    ws = ops.sage_prepare(q, k, torch.zeros_like(q), w, None, 1).ws
    shape = ops.make_shape(B, H, L, D, 128, 64, 1, q.dtype)
    o = int(_lib.lib.sla_workspace_bytes(C.byref(shape), _lib.OP_LINEAR_STATE)) + _up(D * D * 2 + D * 2)
    mean = ws[o:o + bh * D * 4].view(torch.float32).view(B, H, D)      # made where L > 4096
    o += _up(bh * D * 4) + _up(bh * ((L + 511) // 512) * D * 4 * 2)
    rows = _up(bh * L * 128)

    def rows8(at):
        return ws[at:at + bh * L * 128].view(torch.int8).view(B, H, L, 128)[..., :D]

    q8, k8 = rows8(o), rows8(o + rows)
    o += 3 * rows
    qs = ws[o:o + bh * mb * 4].view(torch.float32).view(B, H, mb)
    o += _up(bh * mb * 4)
    ks = ws[o:o + bh * nb * 4].view(torch.float32).view(B, H, nb)
    return q8, k8, qs, ks, mean


def _check_rounding(x, x8, scale, blk):
    """Every scale is its block's largest magnitude over 127 (three units for the division and its operands), every value
    its element over the scale, half a step plus the rounding of the reciprocal and the product off at most."""
    L = x.shape[2]
    pad = -L % blk
    blocks = torch.nn.functional.pad(x, (0, 0, 0, pad)).unflatten(2, (-1, blk))
    amax = blocks.abs().amax(dim=(3, 4)).clamp_min(1e-8)
    assert bool(((scale * 127 - amax).abs() <= 3 * 2.0 ** -23 * amax).all())
    steps = blocks / scale[..., None, None]
    got = torch.nn.functional.pad(x8.float(), (0, 0, 0, pad)).unflatten(2, (-1, blk))
    assert float((steps - got).abs().max()) <= 0.5 + 127 * 4 * 2.0 ** -23


# tiles of 128 rows in q and k together, over 888: tiles a CTA walks
@pytest.mark.parametrize("units,L,D,dtype,per_cta", [
    (13, 9000, 64, torch.bfloat16, 2), (60, 5130, 128, torch.bfloat16, 5), (60, 5130, 128, torch.float16, 5),
    (100, 5100, 64, torch.bfloat16, 8),
])
def test_int8_pass_of_several_tiles_a_cta(units, L, D, dtype, per_cta):
    """Chunks of tiles that do not divide a head, an odd number of 64-row blocks, a ragged last row block."""
    mb = (L + 127) // 128
    assert min(8, 2 * mb * units // 888) == per_cta and 2 * mb // 888 <= 1
    q, k = _randn((1, units, L, D), 1, dtype), _randn((1, units, L, D), 2, dtype)
    k += 0.5
    q[:, :, ::97] *= 5
    q8, k8, qs, ks, mean = whole = _quantized(q, k)
    exact = k.double().mean(2)
    ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert bool(((mean - exact).abs() <= 1.01 * ulp * exact.abs() + 1e-6).all())      # rounded once to 16 bits
    for u in sorted({0, 1, units // 2, units - 1}):
        alone = _quantized(q[:, u:u + 1].contiguous(), k[:, u:u + 1].contiguous())
        for a, b in zip(whole, alone):
            assert torch.equal(a[:, u], b[:, 0])
        one = slice(u, u + 1)
        _check_rounding(q[:, one].float(), q8[:, one], qs[:, one], 128)
        _check_rounding(k[:, one].float() - mean[:, one, None], k8[:, one], ks[:, one], 64)


@pytest.mark.parametrize("D", [64, 128])
def test_int8_rounding_of_halves(D):
    """With a scale of one the elements n + 1/2 are products half-way between two integers: they go to the even one, as a
    conversion takes them."""
    L = 128
    n = torch.arange(-127, 127, device="cuda").float() + 0.5
    q = n[torch.arange(L * D, device="cuda") % n.numel()].view(1, 1, L, D).clone()
    q[..., 0, 0] = 127.0
    q8, _, qs, _, _ = _quantized(q.bfloat16(), torch.zeros_like(q).bfloat16())
    assert float(qs) == 1.0
    assert torch.equal(q8.float(), torch.round(q))            # torch.round: ties to even


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_int8_of_infinities_and_nan(dtype):
    """NaN becomes 0 and leaves the rest of its block alone; an infinity makes its block's scale infinite and its values 0;
    other blocks, of the same CTA too, are what they are without either."""
    q, k = _randn((1, 1, 900, 128), 3, dtype), _randn((1, 1, 900, 128), 4, dtype)
    clean = _quantized(q, k)
    bad = q.clone()
    bad[0, 0, 130, 5] = float("nan")
    bad[0, 0, 300, 17], bad[0, 0, 301, 17] = float("inf"), float("-inf")
    q8, k8, qs, ks, _ = _quantized(bad, k)
    assert torch.equal(k8, clean[1]) and torch.equal(ks, clean[3])
    for b in range(8):
        rows = slice(128 * b, min(900, 128 * b + 128))
        want, scale = clean[0][0, 0, rows].clone(), clean[2][0, 0, b]
        if b == 1:
            assert float(q[0, 0, 130, 5].abs()) < float(q[0, 0, rows].abs().max())      # the block's scale is another's
            want[2, 5] = 0
        if b == 2:
            want.zero_()
            scale = torch.full_like(scale, float("inf"))
        assert torch.equal(q8[0, 0, rows], want) and torch.equal(qs[0, 0, b], scale)
    # in k one NaN makes the column's mean, and with it the column, NaN
    bad = k.clone()
    bad[0, 0, 10, 3] = float("nan")
    _, k8, _, _, _ = _quantized(q, bad)
    assert bool((k8[..., 3] == 0).all()) and bool((k8[..., 4] == clean[1][..., 4]).float().mean() > 0.9)


def _norm(units, L, D, BLKQ, inplace, x):
    q, k, gq, gk, cos, sin = x
    q, k = q.clone(), k.clone()
    qo, ko, pooled = ops.qk_norm_rope_pool(q, k, gq, gk, cos, sin, 1e-6, True, BLKQ, 64, inplace)
    mb, nb = (L + BLKQ - 1) // BLKQ, (L + 63) // 64
    sums = pooled.buf.view(torch.uint8)
    qsum = sums[:units * mb * D * 4].view(torch.float32).view(units, mb, D)
    at = _up(units * mb * D * 4)
    return qo, ko, qsum, sums[at:at + units * nb * D * 4].view(torch.float32).view(units, nb, D)


# CTAs of one head, 2 * max(q blocks, k blocks) * units: two heads a CTA from 4096 on, four from 8192
@pytest.mark.parametrize("units,L,D,BLKQ,heads", [
    (5, 32700, 128, 64, 2), (5, 30001, 64, 128, 2), (9, 30000, 128, 128, 4), (10, 30000, 64, 64, 4), (75, 3600, 128, 64, 4),
])
def test_norm_and_rotation_of_several_heads_a_cta(units, L, D, BLKQ, heads):
    """A number of heads that is no multiple of a CTA's, ragged blocks, one batch of rows and two, in place and not."""
    ctas = 2 * ((L + 63) // 64) * units
    assert (4 if ctas >= 8192 else 2 if ctas >= 4096 else 1) == heads and units % heads != 0
    assert ctas // units < 4096
    q, k = _randn((1, units, L, D), 5), _randn((1, units, L, D), 6)
    gq, gk = (1 + 0.1 * _randn((D,), 7 + i, torch.float32) for i in range(2))
    angles = torch.arange(L, device="cuda")[:, None] * 10000.0 ** (-torch.arange(D // 2, device="cuda") / (D // 2))
    tables = (gq, gk, torch.cos(angles), torch.sin(angles))
    whole = _norm(units, L, D, BLKQ, False, (q, k, *tables))
    inplace = _norm(units, L, D, BLKQ, True, (q, k, *tables))
    for a, b in zip(whole, inplace):
        assert torch.equal(a, b)
    for u in sorted({0, 1, heads - 1, heads, units // 2, units - 1}):
        alone = _norm(1, L, D, BLKQ, False, (q[:, u:u + 1].contiguous(), k[:, u:u + 1].contiguous(), *tables))
        for a, b in zip(whole[:2], alone[:2]):
            assert torch.equal(a[:, u], b[:, 0])
        for a, b in zip(whole[2:], alone[2:]):
            assert torch.equal(a[u], b[0])
