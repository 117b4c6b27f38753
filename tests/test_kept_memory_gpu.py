"""What the scope "unselected" holds between a forward and its backward."""
import pytest
import torch

import sla_b200
from sla_b200 import _lib

pytestmark = pytest.mark.gpu


def _module(D, BLKQ=64):
    m = sla_b200.SparseLinearAttention(D, 0.25, "softmax", BLKQ, 64, linear_scope="unselected").cuda()
    with torch.no_grad():
        m.proj_l.weight.normal_(0, 0.05)
    return m


def _inputs(B, H, L, D):
    g = torch.Generator(device="cuda").manual_seed(50)
    return [torch.randn(B, H, L, D, generator=g, device="cuda").to(torch.bfloat16).requires_grad_(True) for _ in range(3)]


def _kept(o):
    return [t for t in o.grad_fn.saved_tensors if t is not None and t.dtype == torch.uint8]


@pytest.mark.parametrize("L,D", [(777, 64), (4096, 128), (5000, 128)])
def test_kept_buffer_is_three_times_q(L, D):
    """phi(q), phi(k), C_num in 16 bits, C_den in 32, the 16-bit proj_l and the rounding of six regions."""
    q, k, v = _inputs(1, 3, L, D)
    kept = _kept(_module(D)(q, k, v))
    rows = q.numel() // D
    assert [t.numel() for t in kept] and sum(t.numel() for t in kept) <= rows * (3 * 2 * D + 4) + 2 * D * (D + 1) + 6 * 256


def _launches_of_backward(m, ts):
    o = m(*ts)
    kept = len(_kept(o))
    before = _lib.lib.sla_launch_count()
    o.backward(torch.ones_like(o))
    return kept, _lib.lib.sla_launch_count() - before


def test_the_caller_chooses_between_memory_and_recomputation():
    """Without the kept buffer the backward has two launches more, the feature maps and the product over the selected
    blocks, and the same gradients."""
    m = _module(128)
    grads, seen = [], []
    for keep in (True, False):
        m.keep_linear_intermediates = keep
        m.zero_grad()
        ts = _inputs(1, 2, 900, 128)
        seen.append(_launches_of_backward(m, ts))
        grads.append([t.grad for t in (*ts, m.proj_l.weight, m.proj_l.bias)])
    (kept, launches), (kept_not, launches_more) = seen
    assert (kept, kept_not) == (1, 0)
    assert launches_more == launches + 2
    for a, b in zip(*grads):
        assert torch.equal(a, b)
