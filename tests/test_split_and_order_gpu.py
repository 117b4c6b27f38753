"""Dispatch edges of the preparation and ordering kernels: each result against another route to the same values."""
import ctypes as C
import gc
import subprocess
import sys

import pytest
import torch

import sla_b200
from oracle import sla_oracle as O
from sla_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _collect_maps_afterwards():
    """A block map and its 0/1 tensor refer to each other: their memory goes here, not in the middle of a later test
    that watches the allocator."""
    yield
    gc.collect()


def _randn(shape, seed, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("L,BLKQ,topk", [
    (64, 64, 1.0), (2049, 64, 0.2), (2111, 128, 0.5), (16384, 64, 0.05),    # lists in one kernel
    (16385, 64, 0.05), (32700, 128, 0.03),                                  # counted, scanned, filled
])
def test_column_lists_match_the_map(L, BLKQ, topk):
    q, k = _randn((2, 3, L, 64), 1), _randn((2, 3, L, 64), 2)
    bm = ops.block_map(q, k, topk, BLKQ, 64, want_map=True, want_cols=True)
    co, ci = ops.column_lists(bm.sparse_map, L, BLKQ, 64, bm.topk)
    assert torch.equal(bm.col_offsets, co)
    assert torch.equal(bm.col_index, ci)


@pytest.mark.parametrize("L", [500, 4096, 4097])       # one chunk of K sums, the most that are added inline, one more
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_block_map_at_the_inline_mean_edge(L, dtype):
    q, k = _randn((1, 2, L, 64), 3, dtype), _randn((1, 2, L, 64), 4, dtype) + 0.5
    lut = ops.block_map(q, k, 0.25, 64, 64).lut.cpu()
    score = O.pooled_scores(q.cpu(), k.cpu(), 64, 64)
    want = O.select_topk(score, lut.shape[-1])
    _, _, bad = O.lut_rows_equal_up_to_ties(score, lut, want, ulps=2)   # sums of another order: one unit either way
    assert bad == 0


@pytest.mark.parametrize("L,D,BLKQ,heads", [(1000, 64, 64, 24), (2500, 128, 128, 9), (19000, 64, 128, 3)])
def test_tile_order_leaves_the_gradients_alone(L, D, BLKQ, heads):
    """All heads in one call take the ordered tiles (more than one per SM), a head by itself the sequence order."""
    # At L = 19000 a single head has 149 tiles and an order of its own. Here every head is ordered; the calls whose first
    # heads are not are in test_tile_order_of_the_last_heads.
    q, k, v, do = (_randn((1, heads, L, D), 10 + i) for i in range(4))
    k[:, :, : L // 3] *= 3                                # popular and unpopular blocks

    def grads(h0, h1):
        qs, ks, vs = (t[:, h0:h1].contiguous().requires_grad_(True) for t in (q, k, v))
        smap, lut, topk = sla_b200.get_block_map(qs.detach(), ks.detach(), 0.2, BLKQ, 64)
        sla_b200._attention.apply(qs, ks, vs, smap, lut, topk, BLKQ, 64).backward(do[:, h0:h1].contiguous())
        return qs.grad, ks.grad, vs.grad

    tiles = (((L + 63) // 64) + 1) // 2
    assert tiles * heads > 148 and (tiles <= 148 or D == 64)
    whole = grads(0, heads)
    for h in range(heads):
        for a, b in zip(whole, grads(h, h + 1)):
            assert torch.equal(a[:, h], b[:, 0])


@pytest.mark.parametrize("L,D,BLKQ,feature", [(777, 64, 64, "relu"), (1500, 128, 128, "softmax")])
def test_saved_workspace_backward_equals_the_recomputing_one(L, D, BLKQ, feature):
    m = sla_b200.SparseLinearAttention(D, 0.25, feature, BLKQ, 64, linear_scope="unselected").cuda()
    with torch.no_grad():
        m.proj_l.weight.copy_(_randn((D, D), 5, torch.float32) * 0.05)
    q, k, v, do = (_randn((2, 2, L, D), 20 + i) for i in range(4))
    ts = [t.clone().requires_grad_(True) for t in (q, k, v)]
    m(*ts).backward(do)

    bm = ops.block_map(q, k, 0.25, BLKQ, 64, want_cols=True)
    shape = ops.make_shape(2, 2, L, D, BLKQ, 64, bm.topk, q.dtype, feature, flags=m.impl_flags)
    o, o_s, lse = torch.empty_like(q), torch.empty_like(q), torch.empty(q.shape[:-1], device="cuda")
    state = torch.empty((2, 2, 2 * D * D + D), dtype=q.dtype, device="cuda")
    w, b, p = m.proj_l.weight.detach(), m.proj_l.bias.detach(), ops._p
    ws = ops._workspace(shape, _lib.OP_FWD, q.device)
    st = ops._stream(q)
    _lib.check(_lib.lib.sla_fwd(C.byref(shape), p(q), p(k), p(v), p(bm.lut), p(w), p(b), p(o), p(o_s), p(lse), p(state),
                                p(ws), ws.numel(), st))
    out = [torch.empty_like(q) for _ in range(3)]
    dw, db = torch.empty((D, D), device="cuda"), torch.empty((D,), device="cuda")
    ws = ops._workspace(shape, _lib.OP_BWD, q.device)
    _lib.check(_lib.lib.sla_bwd(C.byref(shape), p(q), p(k), p(v), p(o_s), p(lse), p(do), p(bm.lut), p(bm.col_offsets),
                                p(bm.col_index), p(w), p(state), *(p(t) for t in out), p(dw), p(db), p(ws), ws.numel(), st))
    for a, t in zip(out, ts):
        assert torch.equal(a, t.grad)
    assert torch.equal(dw, m.proj_l.weight.grad) and torch.equal(db, m.proj_l.bias.grad)


def test_one_preparation_serves_two_forwards_before_their_backwards():
    L, D = 900, 64
    m = sla_b200.SparseLinearAttention(D, 0.25, "elu", linear_scope="unselected").cuda()
    w, b = m.proj_l.weight.detach().normal_(0, 0.05), m.proj_l.bias.detach()
    k, v, do = (_randn((1, 2, L, D), 30 + i) for i in range(3))
    qs = [_randn((1, 2, L, D), 40 + i).requires_grad_(True) for i in range(2)]
    bms = [ops.block_map(q.detach(), k, 0.25, 64, 64, want_cols=True) for q in qs]
    prep = ops.prepare_linear(k, v, w, b, bms[0].topk, 64, 64, "elu", m.impl_flags)
    outs = [ops.sla_attention(q, k, v, w, b, bm, 64, 64, "elu", m.impl_flags, prep) for q, bm in zip(qs, bms)]
    for o in outs:
        o.backward(do)
    for q, bm in zip(qs, bms):
        alone = q.detach().requires_grad_(True)
        ops.sla_attention(alone, k, v, w, b, bm, 64, 64, "elu", m.impl_flags).backward(do)
        assert torch.equal(alone.grad, q.grad)



def test_first_call_of_a_thread_may_be_a_backward():
    """A new process, whose autograd thread has made no CUDA call when the backward encodes its tensor maps."""
    code = """
import torch, sla_b200
m = sla_b200.SparseLinearAttention(128, 0.25).cuda()
q, k, v = (torch.randn(1, 2, 1000, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
smap, lut, topk = sla_b200.get_block_map(q.detach(), k.detach(), 0.25, 64, 64)
sla_b200._attention.apply(q, k, v, smap, lut, topk, 64, 64).backward(torch.ones_like(q))
m(q, k, v).backward(torch.ones_like(q))
torch.cuda.synchronize()
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def _first_ordered_head(L, D, heads):
    """order_heads of the library: the last heads with at most 64 MB of 16-bit Q and dO rows."""
    tiles = ((L + 63) // 64 + 1) // 2
    assert tiles <= 148 < tiles * heads          # a head by itself takes the sequence order, all of them do not
    return heads - min(heads, max(1, 1024 * 128 // D // tiles))


@pytest.mark.parametrize("scope", ["sparse", "all", "unselected"])
@pytest.mark.parametrize("L,D,BLKQ,heads", [(16384, 128, 64, 10), (18944, 64, 128, 15), (16300, 128, 128, 9)])
def test_tile_order_of_the_last_heads(L, D, BLKQ, heads, scope):
    """The first heads run in sequence and the last ones by length; a head by itself always in sequence."""
    assert 0 < _first_ordered_head(L, D, heads) < heads
    q, k, v, do = (_randn((1, heads, L, D), 60 + i) for i in range(4))
    k[:, :, : L // 3] *= 3                                # popular and unpopular blocks
    if scope != "sparse":
        m = sla_b200.SparseLinearAttention(D, 0.1, "softmax", BLKQ, 64, linear_scope=scope).cuda()
        with torch.no_grad():
            m.proj_l.weight.copy_(_randn((D, D), 70, torch.float32) * 0.05)

    def grads(h0, h1):
        qs, ks, vs = (t[:, h0:h1].contiguous().requires_grad_(True) for t in (q, k, v))
        if scope == "sparse":
            smap, lut, topk = sla_b200.get_block_map(qs.detach(), ks.detach(), 0.1, BLKQ, 64)
            o = sla_b200._attention.apply(qs, ks, vs, smap, lut, topk, BLKQ, 64)
        else:
            o = m(qs, ks, vs)
        o.backward(do[:, h0:h1].contiguous())
        return qs.grad, ks.grad, vs.grad

    whole = grads(0, heads)
    for h in range(heads):
        for a, b in zip(whole, grads(h, h + 1)):
            assert torch.equal(a[:, h], b[:, 0])
