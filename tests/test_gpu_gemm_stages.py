"""Staged products (an MN-major A, or a long contraction) by their chunks.

A launch allots a buffer for each 64-wide contraction chunk, four at most:
products of less than one chunk to more than four, in one and several
splits, with the last 128-row tile full, partial and of one 8-row group.
Small whole numbers as inputs: every sum is exact in f32.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k, k_split", [(8, 0), (16, 0), (64, 0), (72, 0), (128, 0), (184, 0), (256, 0), (264, 0),
                                        (520, 0), (72, 64), (520, 128), (456, 256)])
@pytest.mark.parametrize("m, n", [(8, 16), (128, 64), (136, 80), (200, 256)])
@pytest.mark.parametrize("a_mn, b_mn", [(1, 1), (1, 0), (0, 1)])
def test_products_of_few_and_many_chunks(m, n, k, k_split, a_mn, b_mn, cuda_lib, monkeypatch):
    import torch

    from tangle_b200 import warmstart

    monkeypatch.setenv("TGL_GEMM_STAGED", "1")
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    rows, columns = (torch.randint(-8, 9, size, device="cuda", generator=gen).to(torch.bfloat16) for size in ((m, k), (n, k)))
    a, b = rows.T.contiguous() if a_mn else rows, columns.T.contiguous() if b_mn else columns
    out = torch.full((-(-k // k_split) if k_split else 1, m, n), float("nan"), device="cuda")
    warmstart.gemm(a, b, m, n, k, a_mn=bool(a_mn), b_mn=bool(b_mn), lda=a.shape[1], ldb=b.shape[1], out_f32=out, ldo=n,
                   k_split=k_split)
    assert torch.equal(out.sum(0), (rows.double() @ columns.double().T).float())
