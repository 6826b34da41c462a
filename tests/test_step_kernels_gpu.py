"""Kernels that a step takes by its size, each against the kernel it stands in for (the same bits, where it keeps every sum)
or against a float64 statement, at the sizes where it can go wrong: edges of tiles and chunks, remainders, one row and the most."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def ops():
    from supersonic_b200.csrc import ops as o
    return o


def rnd(*shape, seed=0, scale=1.0, dtype=torch.float32):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (scale * torch.randn(*shape, device=DEV, generator=g)).to(dtype)


def off_by_one(t):
    """The same values at an address that no 16-byte access can take: the general kernel's operands."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    view = flat[1:].view(t.shape)
    view.copy_(t)
    return view


# rows that every form takes (one to sixteen rows a group, tiles), around the edges of groups, tiles, turns of 512 and chunks of 16
@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (1, 9, 2052), (2, 130, 516), (3, 65, 20), (4, 8, 512), (5, 33, 1000), (8, 16, 528),
                                   (9, 200, 2048), (16, 64, 1028), (17, 100, 520), (33, 257, 300), (65, 130, 36), (129, 127, 44),
                                   (300, 2500, 516), (257, 129, 64), (64, 3, 4), (1000, 129, 12)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_float32_products_are_the_general_kernels_bit_for_bit(m, n, k, accumulate):
    a, w, c = rnd(m, k, seed=m), rnd(n, k, seed=n), rnd(m, n, seed=k)
    a[0, k // 2] = 3e38                                             # a sum that overflows spreads the same way
    want, got = c.clone(), c.clone()
    ops().gemm_nt_plain(off_by_one(a), w, want, accumulate)
    ops().gemm_nt_plain(a, w, got, accumulate)
    assert torch.equal(torch.nan_to_num(got, nan=7.0), torch.nan_to_num(want, nan=7.0))
    wide = torch.full((m, n + 3), 5.0, device=DEV)                  # rows wider than the result: nothing beside it is touched
    ops().gemm_nt_plain(a, w, wide[:, :n], False)
    assert bool((wide[:, n:] == 5.0).all())


@pytest.mark.parametrize("T,H,K,N", [(1, 6, 64, 128), (133, 3, 128, 48), (70, 4, 24, 72), (8, 2, 16, 260)])
def test_float32_head_products_are_the_general_kernels_bit_for_bit(T, H, K, N):
    x, w = rnd(T, H, K + 4, seed=T)[:, :, :K], rnd(H, N, K, seed=N)
    want, got = torch.empty(T, H, N, device=DEV), torch.empty(T, H, N, device=DEV)
    ops().head_linear_plain(off_by_one(x.contiguous()), w, want)
    ops().head_linear_plain(x, w, got)
    assert torch.equal(got, want)
