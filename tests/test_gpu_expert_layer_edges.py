"""Kernels around the expert GEMMs where their paths change: the routing plan (one block up to 8192 pairs, chunks above;
a table of counts up to 512 experts, turns above) and the scale relay (chunks of eight K atoms, whole or not)."""
import pytest
import torch

from nvfp4_cutlass_b200 import _C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,experts", [(1, 1), (1025, 512), (3000, 513), (8192, 64), (8193, 64), (20000, 600)])
def test_plan_keeps_the_order_of_pairs(n, experts):
    g = torch.Generator().manual_seed(n + experts)
    ids = (torch.rand(n, generator=g) ** 2 * experts).long()              # low experts more often: some overflow the cap
    counts = torch.bincount(ids, minlength=experts)
    cap_m = 128
    order = torch.argsort(ids, stable=True)
    within = torch.empty_like(ids)
    within[order] = torch.arange(n) - (torch.cumsum(counts, 0) - counts)[ids[order]]
    want = torch.where(within < cap_m, ids * cap_m + within, torch.full_like(ids, -1))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ids_dev = ids.cuda()
    assert torch.equal(_C.expert_histogram(ids_dev, experts).cpu(), counts)
    masked_m, dst_row = _C.plan_peer_masked(counts.cuda(), ids_dev, 1, 0, cap_m, status)
    assert torch.equal(dst_row.cpu(), want)
    assert torch.equal(masked_m.cpu(), counts.clamp(max=cap_m).int())
    assert bool(int(status.item()) & 4) == bool((counts > cap_m).any())


@pytest.mark.parametrize("k", [128, 512, 640, 1024])
def test_scale_relay_moves_every_byte(k):
    e, max_m, counts = 3, 256, [256, 0, 129]
    g = torch.Generator().manual_seed(k)
    store = torch.randint(0, 256, (e * max_m * (k + k // 8),), generator=g, dtype=torch.uint8).cuda()
    rows = _C.QuantizedRows(store, e, max_m, k)
    rows.scale_atoms.fill_(0xA5)
    _C.relayout_scales(rows, torch.tensor(counts, dtype=torch.int32, device="cuda"))
    got, src = rows.scale_atoms.cpu(), rows.scale_rows.cpu().view(e * max_m // 128, 4, 32, 2, k // 64, 4)
    want = src.permute(0, 4, 3, 2, 1, 5).reshape(got.shape)               # [row block][K atom][pass][r % 32][r / 32][byte]
    for block in range(e * max_m // 128):
        live = block * 128 % max_m < counts[block * 128 // max_m]
        assert torch.equal(got[block], want[block] if live else torch.full_like(got[block], 0xA5)), block


@pytest.mark.parametrize("n,experts", [(0, 3), (1, 1), (1024, 512), (1025, 513), (8192, 64), (8193, 64), (20000, 600), (131072, 128)])
@pytest.mark.parametrize("stray", [False, True])
def test_one_rank_plan_is_the_plan_of_the_histogram(n, experts, stray):
    """plan_one_rank counts while it hands out rows; ids out of range get owners out of range and no row."""
    g = torch.Generator().manual_seed(n + experts)
    ids = (torch.rand(n, generator=g) ** 2 * experts).long()
    if stray:
        ids[::7] = torch.tensor([-1, -experts - 1, experts, 2 * experts + 3]).repeat(n // 28 + 1)[:ids[::7].numel()]
    valid, cap_m = (ids >= 0) & (ids < experts), 1024 if n > 20000 else 128
    ids = ids.cuda()
    counts = _C.expert_histogram(ids, experts)
    status, want_status = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
    want_m, want_row = _C.plan_peer_masked(counts, ids, 1, 0, cap_m, want_status)
    masked_m, dst_rank, dst_row = _C.plan_one_rank(ids, experts, cap_m, status)
    assert torch.equal(masked_m, want_m) and int(status.item()) == int(want_status.item())
    assert torch.equal(dst_rank, torch.div(ids, experts, rounding_mode="floor"))
    assert torch.equal(dst_row.cpu()[valid], want_row.cpu()[valid])
