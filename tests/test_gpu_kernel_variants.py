"""Kernels that exist in more than one form, chosen by size: every form against a plain computation, or against the other form
where both take the size, at the sizes where a form can go wrong (tile edges, remainders, smallest and largest)."""
import math

import pytest
import torch

import helpers
from plain import qwen2_plain as plain
from test_gpu_kernels import paged_cache

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F = torch.float64


def ops():
    from vt_transformer_b200 import ops as o
    return o


# (rows around the bounds of the two 32-bit kernels and of a tile of 64; columns in one, four and a part of four rows of w a warp;
# inner sizes below, at and beyond a chunk of 512 and a tile's 64)
@pytest.mark.parametrize("n,k", [(1, 8), (7, 520), (65, 512), (130, 1000), (4739, 72), (300, 4864)])
def test_32_bit_products_are_the_same_in_both_kernels(n, k):
    """A row's results bit for bit in steps of every size, and within the rounding of sums in runs of 16."""
    g = torch.Generator(device=DEV).manual_seed(n + k)
    a = torch.randn((130, k), generator=g, device=DEV)
    w = torch.randn((n, k), generator=g, device=DEV)
    bias = torch.randn(n, generator=g, device=DEV)
    ref = plain.linear(a.cpu().double(), w.cpu().double(), bias.cpu().double())
    whole = ops().linear(a, w, bias, torch.empty((130, n), device=DEV))
    size = (a.abs().double() @ w.abs().double().T + bias.abs()).cpu()
    assert float(((whole.cpu().double() - ref).abs() / size).max()) <= (16 + k / 16) * 2.0 ** -24
    for m in (1, 2, 3, 4, 5, 8, 9, 31, 32, 33, 64, 65, 129):
        part = ops().linear(a[:m].contiguous(), w, bias, torch.full((m, n), float("nan"), device=DEV))
        assert torch.equal(part, whole[:m]), m
