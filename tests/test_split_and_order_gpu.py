"""Dispatch edges of the preparation and ordering kernels: each result against another route to the same values."""
import ctypes as C
import subprocess
import sys

import pytest
import torch

import sla_b200
from oracle import sla_oracle as O
from sla_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _randn(shape, seed, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(dtype)


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
