"""Edges of the kernels' tiles and of the rules that choose between kernels, against plain 64-bit references."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def K():
    from dllama_b200.ops import kernels
    return kernels


def L():
    from dllama_b200.ops import layers
    return layers


@pytest.mark.parametrize("heads,kv,hs,n_splits", [(4, 1, 128, 1), (3, 1, 128, 4), (4, 2, 64, 1), (8, 2, 64, 3), (2, 2, 128, 2)])
def test_decode_attention_half_pages(heads, kv, hs, n_splits):
    """Contexts around the borders of half pages, of the warps' turns and of the split rule (24 pages); an infinite key that a head's
    score sends to -inf takes no weight and leaves the rest finite, as in f32.  Bound: f32 sums of some hundred terms and an
    exponential of relative error 2^-22 on scores below 8 in units of log2: 2e-6 of the largest value is several times that."""
    positions = [0, 14, 15, 16, 31, 32, 63, 64, 127, 767, 768, 901]
    M, pages = len(positions), 30
    g = torch.Generator().manual_seed(heads * 1000 + hs)
    q = torch.randn(M, heads * hs, generator=g)
    kc, vc = (torch.randn(M * pages, kv, 32, hs, generator=g).half() for _ in range(2))
    bt = torch.randperm(M * pages, generator=g).int().view(M, pages)
    kc[bt[11, 3], :, 5] = 0                        # one key of the last row: -inf along its first dimension
    kc[bt[11, 3], :, 5, 0] = -float("inf")
    q[11].view(heads, hs)[:, 0] = 1.5
    y = torch.zeros(M, heads * hs, device="cuda")
    scratch = torch.zeros(K().attention_scratch_bytes(M, heads, hs, n_splits), dtype=torch.uint8, device="cuda")
    for _ in range(2):                              # twice: the split counters reset themselves
        K().attention(q.cuda(), M, heads, kv, hs, kc.cuda(), vc.cuda(), torch.tensor(positions, dtype=torch.int32, device="cuda"),
                      torch.arange(M, dtype=torch.int32, device="cuda"), bt.cuda(), pages, n_splits, scratch, None, None, M, y)
    want = torch.empty(M, heads, hs, dtype=torch.float64)
    for m, p in enumerate(positions):
        k, v = (c[bt[m].long()].transpose(1, 2).reshape(-1, kv, hs)[:p + 1].double().repeat_interleave(heads // kv, dim=1) for c in (kc, vc))
        s = torch.einsum("hd,thd->ht", q[m].double().view(heads, hs), k) * hs ** -0.5
        want[m] = torch.einsum("ht,thd->hd", s.softmax(dim=1), v)
    got = y.cpu().double().view(M, heads, hs)
    assert torch.isfinite(got).all()
    assert (got - want).abs().max() <= 2e-6 * want.abs().max()
