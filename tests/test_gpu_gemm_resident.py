"""Data-gradient products (K-major A, MN-major B) keep B in shared memory.

At the sizes where that layout can go wrong -- one and several contraction
chunks, a last chunk that K does not fill, every multiple of 16 columns near
the swizzle's 8-row atoms, a last tile that M does not fill, more tiles than
CTAs, and a B too large to stay resident -- the product must be that of the
staged kernel (the same MMAs in the same order) bit for bit.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 16, 8), (127, 16, 16), (129, 48, 24), (300, 80, 64), (40001, 64, 64),
                                   (1000, 192, 72), (5000, 256, 200), (700, 256, 256), (260, 256, 520)])
def test_resident_b_matches_the_staged_kernel(m, n, k, cuda_lib, monkeypatch):
    import torch

    from tangle_b200 import warmstart

    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=gen).bfloat16()
    b = torch.randn(k, n, device="cuda", generator=gen).bfloat16()
    mask = torch.randn(m, n, device="cuda", generator=gen).bfloat16()
    out = []
    for staged in (False, True):
        if staged:
            monkeypatch.setenv("TGL_GEMM_STAGED", "1")
        f32 = torch.full((m, n), float("nan"), device="cuda")
        bf16 = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16)
        warmstart.gemm(a, b, m, n, k, b_mn=True, lda=k, ldb=n, mask=mask, ld_mask=n, out_f32=f32, ldo=n,
                       out_bf16=bf16, ldo_bf16=n)
        out.append((f32, bf16))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert torch.isfinite(out[0][0]).all()
