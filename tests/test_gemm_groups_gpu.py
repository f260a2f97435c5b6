"""Several products of one size in one launch (bfi_gemm_groups_bf16) against a 64-bit product, at the edges of its tiles and with
groups whose columns end inside a block of k, beside values that must not enter."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("groups,m,n,k,pad", [(1, 1, 8, 8, 0), (3, 17, 40, 24, 8), (16, 64, 512, 64, 64), (5, 129, 128, 512, 0), (12, 300, 136, 72, 16),
                                              (2, 128, 264, 128, 8)])
def test_groups(out_dtype, groups, m, n, k, pad):
    from builderforce_inference_b200.kernels import fast_ops
    g = torch.Generator(device=DEV).manual_seed(groups * m + n + k)
    a = torch.full((m, groups * (k + pad)), float("nan"), device=DEV, dtype=torch.bfloat16)      # what lies between groups is not read
    a.view(m, groups, k + pad)[..., :k] = torch.randn(m, groups, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(groups, n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    out = torch.full((m, groups * (n + 8)), 7.0, device=DEV, dtype=out_dtype)
    assert fast_ops.gemm_groups(a[:, :k], k + pad, w, out[:, :n], n + 8)
    ref = torch.einsum("mgk,gnk->mgn", a.view(m, groups, k + pad)[..., :k].double(), w.double())
    got = out.view(m, groups, n + 8)
    assert float((got[..., :n].double() - ref).norm() / ref.norm()) < (2.0 ** -8 if out_dtype == torch.bfloat16 else 1e-6)
    assert bool((got[..., n:] == 7.0).all())
    assert int(fast_ops.tc_status(DEV)[0].item()) == 0


def test_refusals():
    from builderforce_inference_b200.kernels import fast_ops
    from builderforce_inference_b200.kernels.library import KernelError
    a, w = torch.zeros(4, 64, device=DEV, dtype=torch.bfloat16), torch.zeros(4, 16, 16, device=DEV, dtype=torch.bfloat16)
    out = torch.zeros(4, 64, device=DEV, dtype=torch.bfloat16)
    assert not fast_ops.gemm_groups(a[:, :16], 12, w, out[:, :16], 16)                          # groups that do not start on 16 bytes
    with pytest.raises(KernelError):
        fast_ops.gemm_groups(a[:, :16], 24, w, out[:, :16], 16)                                 # the last group ends outside
