"""Weight quantiser at the edges of its tiles (64 rows x 512 K, 128 KB of maxima) and of its arithmetic (kept-reciprocal
quotients instead of divisions): byte for byte against the oracle, which divides."""
import pytest
import torch

import nvfp4_gemm
from nvfp4_cutlass_b200 import _C

pytestmark = pytest.mark.gpu


def check(oracle, w, wd):
    got, want = nvfp4_gemm.quantize_weight_nvfp4(wd), oracle.quantize_weight(w.contiguous())
    for name, x, y in zip(("b", "sfb", "gw"), got, want):
        assert torch.equal(x.cpu(), y), name


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape,offset", [((1, 1, 64), 0), ((3, 63, 576), 0), ((2, 65, 448), 1), ((40, 64, 512), 0), ((2, 200, 4160), 3)])
def test_tile_edges_and_unaligned_views(oracle, dtype, shape, offset):
    g = torch.Generator().manual_seed(sum(shape) + offset)
    flat = torch.randn(shape[0] * shape[1] * shape[2] + offset, generator=g) * 0.02
    flat[::5] *= 0.0                                         # zeros of both signs: the sign bit is part of the code
    flat = flat.to(dtype)
    check(oracle, flat[offset:].view(shape), flat.cuda()[offset:].view(shape))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -70, 2.0 ** 70, 2.0 ** -120])
def test_every_global_scale_mantissa(oracle, dtype, scale):
    g = torch.Generator().manual_seed(7)
    w = torch.randint(-128, 128, (128, 16, 128), generator=g).to(torch.float32) * 2.0 ** torch.randint(-12, -7, (128, 16, 1), generator=g)
    if dtype == torch.float32:
        w = w * (1 + torch.rand(w.shape, generator=g))
    w[:, 0, 0] = 1.0 + torch.arange(128) / 128.0             # one expert per BF16 mantissa of the largest magnitude
    w = (w * scale).to(dtype)
    check(oracle, w, w.cuda())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(1, 16, 64), (70, 64, 512), (3, 2048, 4096)])
def test_a_wait_that_runs_out_shows(oracle, dtype, shape):
    """Waits that can only run out (after half a millisecond): the kernel ends, and no global scale looks like one."""
    w = (torch.randn(shape, generator=torch.Generator().manual_seed(9)) * 0.02).to(dtype)
    wd = w.cuda()
    gw = _C.debug_quantize_weight_expired(wd, 1_000_000)[2]
    assert bool(torch.isnan(gw).all())
    check(oracle, w[:2, :64], wd[:2, :64])                   # and the next call is an ordinary one


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -70])         # kept reciprocals, divisions
def test_nan_and_infinity(oracle, dtype, scale):
    """A NaN does not count for a maximum and gets the largest positive code whatever its sign (the conversion's rule; the oracle
    keeps the sign); the elements around it get the codes they would get beside a zero.  Infinities make G infinite."""
    g = torch.Generator().manual_seed(11)
    clean = (torch.randn(2, 70, 640, generator=g) * 0.02 * scale).to(dtype)
    at = torch.rand(clean.shape, generator=g) < 0.02
    at[0, 3, 16:32] = True                                   # a block of nothing else
    clean[at] = 0.0
    nan = torch.where(torch.rand(clean.shape, generator=g) < 0.5, torch.tensor(float("nan")), -torch.tensor(float("nan"))).to(dtype)
    w = torch.where(at, nan, clean)
    b, sfb, gw = nvfp4_gemm.quantize_weight_nvfp4(w.cuda())
    want_b, want_sfb, want_gw = oracle.quantize_weight(clean)
    codes = want_b.view(torch.uint8).view(2, 70, 320)
    codes = torch.stack((codes & 15, codes >> 4), dim=-1).view(2, 70, 640)
    codes[at] = 7
    want_b = (codes[..., 0::2] | codes[..., 1::2] << 4).view(140, 320)
    assert torch.equal(b.cpu().view(torch.uint8), want_b) and torch.equal(sfb.cpu(), want_sfb) and torch.equal(gw.cpu(), want_gw)
    w[1, 5, 7], w[1, 60, 639] = float("inf"), -float("inf")
    b, sfb, gw = nvfp4_gemm.quantize_weight_nvfp4(w.cuda())
    assert torch.equal(gw.cpu(), torch.stack((want_gw[0], torch.tensor(float("inf")))))
    assert torch.equal(b.cpu().view(torch.uint8)[:70], want_b[:70])


@pytest.mark.parametrize("shape", [(5, 2048, 4096), (7, 1000, 4160), (4, 4096, 4096)])     # batches of 24 MB: one expert each,
def test_stages_of_several_batches(oracle, shape):                                         # 3 + 3 + 1, one each
    w = (torch.randn(*shape, generator=torch.Generator().manual_seed(sum(shape))) * 0.02).to(torch.bfloat16)
    w *= torch.arange(1, shape[0] + 1).reshape(-1, 1, 1)                                   # every expert a global scale of its own
    for got, want in zip(nvfp4_gemm.quantize_weight_nvfp4(w.cuda()), oracle.quantize_weight(w)):
        assert torch.equal(got.cpu(), want)
