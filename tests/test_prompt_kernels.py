"""Prompt-pass kernels whose tiles or rows were cut anew, against plain 64-bit forms at the edges of their tiles."""
import pytest
import torch
import torch.nn.functional as F

from b200serve.ops import gemm as G
from b200serve.ops import lib as K
from b200serve.utils import quant as Q

pytestmark = pytest.mark.gpu


# rows: one and two 128-row halves, a pair's second half empty, several pairs; columns that end inside a tile, inside a CTA's half, at
# a W4B block's end; k shorter than the ring and longer
@pytest.mark.parametrize("m,n,k", [(129, 256, 64), (128, 512, 128), (256, 264, 320), (257, 640, 576), (300, 1000, 64), (511, 384, 1088), (40, 256, 128),
                                   (1024, 5120, 512), (2049, 776, 256), (130, 40960, 64)])
@pytest.mark.parametrize("bn", [-256, 0])
def test_two_sm_gemm(m, n, k, bn):
    torch.manual_seed(m + n)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), (torch.randn(n, k, device="cuda") * k ** -0.5).bfloat16()
    ref = a.double() @ b.double().T
    # exact products, fp32 sums: a few 2^-24 of the absolute terms; one rounding to bf16 on the way out
    bound = 16 * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T)
    out = torch.full((m + 1, n), float("nan"), device="cuda")
    G.gemm_bf16(a, b, out[:m], epi=G.EPI_F32, bn=bn)
    one = torch.empty(m, n, device="cuda")
    G.gemm_bf16(a, b, one, epi=G.EPI_F32, bn=128)
    torch.cuda.synchronize()
    K.check_status()
    assert ((out[:m].double() - ref).abs() <= bound + 1e-9).all() and torch.isnan(out[m]).all()
    assert torch.equal(out[:m], one)            # the same products in the same order as the one-SM form
    resid = torch.randn(m, n, device="cuda").bfloat16()
    got = resid.clone()
    G.gemm_bf16(a, b, got, epi=G.EPI_RESID_ADD, resid=got, bn=bn)
    assert ((got.double() - resid.double() - ref).abs() <= 2.0 ** -8 * (resid.double() + ref).abs() + bound + 1e-9).all()
    if n % 32 == 0:
        act = torch.empty(m, n // 2, dtype=torch.bfloat16, device="cuda")
        G.gemm_bf16(a, b, act, epi=G.EPI_SILU_MUL, bn=bn)
        v = ref.view(m, n // 32, 2, 16)
        want = (F.silu(v[:, :, 0]) * v[:, :, 1]).reshape(m, n // 2)
        assert ((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()


@pytest.mark.parametrize("n,k", [(128, 64), (100, 256), (1000, 320), (256, 4096), (5120, 1088)])
def test_expanded_weights(n, k):
    """Four blocks per CTA and what is left of them, rows behind the matrix untouched."""
    w = Q.random_w4b(n, k, "cuda", 3)
    out = torch.full((n + 1, k), float("nan"), dtype=torch.bfloat16, device="cuda")
    G.dequant_w4b(w, n, k, out[:n])
    torch.cuda.synchronize()
    assert torch.equal(out[:n], Q.dequant_w4b(w, n).bfloat16()) and torch.isnan(out[n]).all()
