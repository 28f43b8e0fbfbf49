"""Decode GEMM where its general form begins: K that the large K blocks do not divide (the last one in part), and runs of weight
tiles that share one transformed token tile.  The K atoms are added in the same order whatever the block, so blocks of 128 (asked for
by tune_block_k) give the same bits."""
import pytest
import torch

import nvfp4_gemm
from nvfp4_cutlass_b200 import _C

pytestmark = pytest.mark.gpu


def both(sizes, n, k, tile, residual=True, policy="derived_div8"):
    g = torch.Generator(device="cuda").manual_seed(n + k + len(sizes))
    w = (torch.randn(len(sizes), n, k, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    b, sfb, gw = nvfp4_gemm.quantize_weight_nvfp4(w)
    a = torch.randn(sum(sizes), k, generator=g, device="cuda").to(torch.bfloat16)
    mi = nvfp4_gemm.make_m_indices(sizes, device="cuda", alignment=tile)
    out, status = [], torch.zeros(1, dtype=torch.int32, device="cuda")
    for block_k in (0, 128):
        wide = torch.full((sum(sizes), n + 8), 7.0, dtype=torch.bfloat16, device="cuda")
        for _ in range(2):
            nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a, b, sfb, gw, wide[:, :n], mi, policy, residual, device_status=status, m_alignment=tile,
                                                                 tune_swap_ab=1, tune_block_k=block_k, tune_split_transform=2)
        assert _C.read_status(status) == 0 and bool((wide[:, n:] == 7.0).all())
        out.append(wide[:, :n].clone())
    assert torch.equal(out[0], out[1])
    return a, b, sfb, gw, mi, out[0]


@pytest.mark.parametrize("tile", [16, 32, 64])
@pytest.mark.parametrize("k", [896, 1024 + 128, 1408, 2048 - 128])
@pytest.mark.parametrize("residual", [True, False])
def test_last_k_block_in_part(oracle, tile, k, residual):
    a, b, sfb, gw, mi, d = both([tile, 0, 2 * tile, tile], 384, k, tile, residual)
    want = oracle.grouped_gemm(a.cpu(), b.cpu(), sfb.cpu(), gw.cpu(), mi.cpu(), 384, mode="dual" if residual else "single").float()
    assert float((d.float().cpu() - want).norm() / want.norm()) < 2.5e-3       # BF16 ties of FP32 sums in another order


def test_scales_past_the_end_of_k_are_not_used():
    """An expert whose scales are NaN follows one whose K ends inside a K block: the first one's output stays finite."""
    a, b, sfb, gw, mi, d = both([16, 16], 256, 896, 16)
    poisoned = sfb.clone()
    poisoned[896 // 64:] = 0x7f7f7f7f
    got = torch.zeros_like(d)
    nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a, b, poisoned, gw, got, mi, m_alignment=16, tune_swap_ab=1)
    assert torch.equal(got[:16], d[:16]) and bool(got[16:].isnan().all())


# token tiles x column tiles: runs of four (480 weight tiles on 148 SMs), of two (580), none (odd column tiles; few tiles)
@pytest.mark.parametrize("experts,n", [(30, 2048), (58, 1280), (58, 1152), (5, 512)])
@pytest.mark.parametrize("tile,k", [(16, 1024), (32, 512), (32, 1024), (32, 896), (64, 768), (64, 256)])
def test_runs_of_weight_tiles(experts, n, tile, k):
    both([tile] * experts, n, k, tile)


@pytest.mark.parametrize("policy", ["residual_amax", "derived_div4", "div4_radix8"])
def test_other_policies(policy):
    both([32] * 30, 2048, 512, 32, policy=policy)
    both([16, 32], 256, 1408, 16, policy=policy)
