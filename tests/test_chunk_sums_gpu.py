"""The sums over chunks of rows that the mask prediction and the quantization start from, at the chunk counts where their
kernels change."""
import pytest
import torch

import sla_b200
from oracle import sla_oracle as O
from sla_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _randn(shape, seed, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(dtype)


def _kernel_us(fn, name, calls=50):
    """Shortest device time of the kernel `name` over some calls of fn."""
    from torch.profiler import ProfilerActivity, profile
    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        for _ in range(calls):
            fn()
        torch.cuda.synchronize()
    times = [e.device_time for e in p.events() if name in e.name and e.device_time > 0]
    if not times:
        pytest.skip("no kernel times from the profiler here")
    return min(times)


# 512 rows a chunk, sixteen chunks a batch: one chunk into a batch, one short of it, all of it, one more
@pytest.mark.parametrize("L", [4609, 7680, 8192, 8193])
def test_block_map_at_the_mean_batch_edges(L):
    q, k = _randn((1, 2, L, 64), 5), _randn((1, 2, L, 64), 6) + 0.5
    lut = ops.block_map(q, k, 0.25, 64, 64).lut.cpu()
    score = O.pooled_scores(q.cpu(), k.cpu(), 64, 64)
    want = O.select_topk(score, lut.shape[-1])
    _, _, bad = O.lut_rows_equal_up_to_ties(score, lut, want, ulps=2)   # sums of another order: one unit either way
    assert bad == 0


def test_mean_of_an_unfilled_batch_takes_no_longer():
    """Fifteen chunks have less to add than sixteen; one load after another they take 2.5 to 3 times as long."""
    def run(L):
        q, k = _randn((1, 8, L, 128), 7), _randn((1, 8, L, 128), 8)
        return _kernel_us(lambda: ops.block_map(q, k, 0.25, 64, 64), "kmean_finalize_kernel")
    full, short = run(8192), run(7680)
    print(f"kmean_finalize: 15 chunks {short:.2f} us, 16 chunks {full:.2f} us")
    assert short < 1.8 * full, (short, full)


def _launches(fn):
    before = _lib.lib.sla_launch_count()
    out = fn()
    return _lib.lib.sla_launch_count() - before, out


# 64 blocks of 8 chunks a unit: the line lies at 16 units
@pytest.mark.parametrize("D,units", [(64, 17), (128, 24)])
def test_many_units_do_not_repeat_the_maxima_of_v(D, units):
    """Above the line V's scales come from a kernel of their own, with the same bits as where every block makes them."""
    q, k, v = (_randn((1, units, 4096, D), 30 + i) for i in range(3))
    m = sla_b200.SageSparseLinearAttention(D, 0.1).cuda()
    m.overlap_prepare = False
    with torch.no_grad():
        n_all, out = _launches(lambda: m(q, k, v))
        n_few, few = _launches(lambda: m(*(t[:, :16].contiguous() for t in (q, k, v))))
    assert n_all == n_few + 1
    assert torch.equal(out[:, :16], few)
