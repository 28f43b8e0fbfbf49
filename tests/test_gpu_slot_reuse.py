"""Kernels that transform activations in shared memory, at sizes where every block refills its slots many times: a slot handed back
before its loads are over shows as a row of another tile now and then, so every call's whole output is compared."""
import pytest
import torch

import nvfp4_gemm
from nvfp4_cutlass_b200 import _C

pytestmark = pytest.mark.gpu

CALLS = 40
# Two BF16 results of FP32 sums in different orders differ by one unit in the last place at most, 2^-8 of the value
ROW = 2.0 ** -8


def operands(sizes, n, k, alignment):
    g = torch.Generator(device="cuda").manual_seed(n + k + len(sizes))
    b, sfb, gw = nvfp4_gemm.quantize_weight_nvfp4((torch.randn(len(sizes), n, k, generator=g, device="cuda") * 0.05).to(torch.bfloat16))
    a = torch.randn(sum(sizes), k, generator=g, device="cuda").to(torch.bfloat16)
    return a, b, sfb, gw, nvfp4_gemm.make_m_indices(sizes, device="cuda", alignment=alignment)


def calls(a, b, sfb, gw, mi, n, count, **kw):
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for _ in range(count):
        d = torch.full((a.shape[0], n), float("nan"), dtype=torch.bfloat16, device="cuda")
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a, b, sfb, gw, d, mi, device_status=status, **kw)
        yield d
    assert _C.read_status(status) == 0


def wrong_rows(got, want):
    return torch.nonzero((got.view(torch.int16) != want.view(torch.int16)).any(dim=1)).flatten().tolist()


def assert_rows_match(oracle, d, a, b, sfb, gw, mi, residual, experts, columns=128):
    """Rows of a few experts, the first columns, against the oracle."""
    n, k = d.shape[1], a.shape[1]
    for e in experts:
        rows = torch.nonzero(mi == e).flatten()
        want = oracle.grouped_gemm(a[rows].cpu(), b[e * n:e * n + columns].cpu(), sfb[e * (k // 64):(e + 1) * (k // 64), :columns].contiguous().cpu(),
                                   gw[e:e + 1].cpu(), torch.zeros(rows.numel(), dtype=torch.int32), columns, mode="dual" if residual else "single").float()
        err = (d[rows, :columns].float().cpu() - want).norm(dim=1) / want.norm(dim=1)
        assert float(err.max()) < ROW, (e, err.tolist())


@pytest.mark.parametrize("tile", [16, 32, 64])
@pytest.mark.parametrize("k", [3456, 3584])
@pytest.mark.parametrize("residual", [True, False])
def test_decode_rows_stay_in_their_tile(oracle, tile, k, residual):
    """Eight weight tiles a block, seven K blocks (fourteen at 64 tokens), of 3456 the last one in part, a P ring of two (three): the two
    forms of the kernel, which hand the slot back at different times."""
    n = 1280
    t = operands([tile] * 120, n, k, tile)
    kw = dict(enable_residual_pass=residual, m_alignment=tile, tune_swap_ab=1, tune_split_transform=2)
    (want,) = calls(*t, n, 1, tune_block_k=128, **kw)
    assert_rows_match(oracle, want, *t, residual, (0, 57, 119))
    for i, d in enumerate(calls(*t, n, CALLS, **kw)):
        assert wrong_rows(d, want) == [], i


@pytest.mark.parametrize("n,k,tune", [(1024, 2048, {}), (512, 2048, {}), (512, 2048, dict(tune_split_transform=2, tune_cluster=1))],
                         ids=["quads", "pairs", "single CTAs"])
@pytest.mark.parametrize("residual", [False, True])
def test_fused_rows_stay_in_their_tile(oracle, n, k, tune, residual):
    t = operands([256] * 4 if not tune else [512] * 40, n, k, 128)
    want = None
    for i, d in enumerate(calls(*t, n, CALLS, enable_residual_pass=residual, **tune)):
        if want is None:
            assert_rows_match(oracle, d, *t, residual, (0, 3))
            want = d
        assert wrong_rows(d, want) == [], i
