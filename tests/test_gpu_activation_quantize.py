"""Activation quantiser of the split path where its loads and tiles (128 rows x 128 K) change: rows that are only 16-byte
aligned, one tile, K that is an odd multiple of the tile.  The aligned call is pinned to the oracle elsewhere, for
K a multiple of 256; here also for one tile."""
import pytest
import torch

from nvfp4_gemm import _C
from conftest import grid_i8_from_codes

pytestmark = pytest.mark.gpu


def codes(packed):
    u = packed.cpu()
    return torch.stack([u & 0xF, u >> 4], dim=-1).reshape(u.shape[0], -1)


@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("m,k", [(128, 128), (384, 384), (256, 1152)])
def test_unaligned_rows_and_tile_edges(oracle, m, k, residual):
    g = torch.Generator().manual_seed(m + k)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    q0, q1, s0, s1 = oracle.decompose(x)
    r = torch.arange(m) % 128
    for offset, pad in ((0, 0), (8, 0), (0, 8), (8, 24)):                # elements: base, row stride
        flat = torch.full((m * (k + pad) + offset,), float("nan"), dtype=torch.bfloat16, device="cuda")
        a = flat[offset:].view(m, k + pad)[:, :k]
        a.copy_(x)
        a0, a1, sfa = _C.debug_split_workspace(a, enable_residual_pass=residual)
        for got, want in ((a0, q0), (a1, q1))[:2 if residual else 1]:
            assert torch.equal(grid_i8_from_codes(codes(got)), grid_i8_from_codes(want)), (offset, pad)
        for p, plane in enumerate((s0, s1)[:2 if residual else 1]):
            at = (r % 32) * 16 + (r // 32) * 4
            for j in range(4):
                got = sfa.cpu()[torch.arange(m) // 128, :, p, at + j]
                assert torch.equal(got, plane.reshape(m, k // 64, 4)[:, :, j]), (offset, pad, p)
