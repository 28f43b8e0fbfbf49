"""Split path at N an odd multiple of 128: the last column tile is half a tile whose other half must neither be stored nor
disturb anything (the columns after N of a wider output buffer, the rows of the next expert)."""
import pytest
import torch

import nvfp4_gemm
from nvfp4_cutlass_b200 import _C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("n,k,align", [(640, 256, 128), (1152, 384, 128), (1408, 512, 256)])
def test_last_half_tile(oracle, n, k, align, residual):
    sizes = [align, 2 * align, 0, align]
    g = torch.Generator().manual_seed(n + k)
    b, sfb, gw = nvfp4_gemm.quantize_weight_nvfp4((torch.randn(len(sizes), n, k, generator=g) * 0.05).to(torch.bfloat16).cuda())
    a = torch.randn(sum(sizes), k, generator=g).to(torch.bfloat16)
    mi = nvfp4_gemm.make_m_indices(sizes, alignment=align)
    wide = torch.full((sum(sizes), n + 128), 7.0, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a.cuda(), b, sfb, gw, wide[:, :n], mi.cuda(), enable_residual_pass=residual,
                                                         m_alignment=align, device_status=status)
    assert _C.read_status(status) == 0
    want = oracle.grouped_gemm(a, b.cpu(), sfb.cpu(), gw.cpu(), mi, n, mode="dual" if residual else "single").float()
    got = wide[:, :n].float().cpu()
    assert float((got - want).norm() / want.norm()) < 2.5e-3               # BF16 ties of FP32 sums in another order
    assert bool((wide[:, n:] == 7.0).all())
