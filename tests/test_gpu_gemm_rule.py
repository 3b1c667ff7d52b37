"""Data-gradient products on both sides of the line between their kernels.

A K-major A and an MN-major B take the kernel that keeps B in shared memory
from so many 128-row tiles per SM as repay writing B there (one to 64
columns, three to 128 or for a contraction as long as the columns, four to
192, sixteen else; never beyond 128 columns for less than 64), the staged
kernel below. Both run the same MMAs in the same order: equal bits.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm, n, k", [(1, 16, 8), (1, 48, 24), (1, 64, 200), (3, 80, 64), (3, 128, 136), (3, 192, 200),
                                          (3, 256, 256), (4, 192, 72), (16, 256, 64), (16, 144, 16)])
@pytest.mark.parametrize("below", [True, False], ids=["below", "from"])
def test_both_kernels_give_the_same_bits(per_sm, n, k, below, cuda_lib, monkeypatch):
    import torch

    from tangle_b200 import warmstart

    m = per_sm * torch.cuda.get_device_properties(0).multi_processor_count * 128 - (128 if below else 55)
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
