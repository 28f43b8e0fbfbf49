"""The decode GEMM over quantised rows (gemm_stream.cu): every token tile and K block against the oracle, the masked form
and the layer that uses it against the 128-row kernels, which differ from it in the order of the FP32 sums only."""
import pytest
import torch

import nvfp4_gemm
from nvfp4_cutlass_b200 import _C
from nvfp4_cutlass_b200.ep import ExpertParallelMoE, route_topk

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def weights(e, n, k, seed):
    g = torch.Generator().manual_seed(seed)
    return nvfp4_gemm.quantize_weight_nvfp4((torch.randn(e, n, k, generator=g) * 0.05).to(torch.bfloat16).cuda())


@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("align,n,k", [(16, 128, 256), (16, 640, 1536), (32, 256, 512), (32, 128, 768), (64, 384, 1024), (128, 128, 256)])
def test_contiguous_matches_oracle(oracle, align, n, k, residual):
    sizes = [align, 0, 3 * align, align, 2 * align]
    b, sfb, gw = weights(len(sizes), n, k, n + k)
    mi = nvfp4_gemm.make_m_indices(sizes, alignment=align)
    a = torch.randn(sum(sizes), k, generator=torch.Generator().manual_seed(k)).to(torch.bfloat16)
    d = torch.full((sum(sizes), n), float("nan"), dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a.cuda(), b, sfb, gw, d, mi.cuda(), enable_residual_pass=residual, m_alignment=align,
                                                         tune_swap_ab=1, tune_split_transform=1, device_status=status)
    assert _C.read_status(status) == 0
    want = oracle.grouped_gemm(a, b.cpu(), sfb.cpu(), gw.cpu(), mi, n, mode="dual" if residual else "single")
    # FP32 sums in another order move a BF16 output by one ulp (2^-8) where it sits at a tie: far less than one in ten
    assert rel_l2(d, want) < 2.5e-3


POLICIES = ["derived_div8", "residual_amax", "derived_div4", "div4_radix8"]


@pytest.mark.parametrize("policy", POLICIES)
@pytest.mark.parametrize("align,n,k,residual", [(16, 256, 768, True), (32, 384, 1024, False), (64, 128, 512, True)])
def test_policies_and_row_strides(oracle, policy, align, n, k, residual):
    """The quantisation pass in all its scale policies, activations and output as column ranges of wider tensors."""
    sizes = [2 * align, align, 0, align]
    m = sum(sizes)
    b, sfb, gw = weights(len(sizes), n, k, n + k)
    mi = nvfp4_gemm.make_m_indices(sizes, alignment=align)
    wide = torch.randn(m, k + 72, generator=torch.Generator().manual_seed(k)).to(torch.bfloat16)
    a, d = wide.cuda()[:, 24:24 + k], torch.full((m, n + 40), 7.0, dtype=torch.bfloat16, device="cuda")
    nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a, b, sfb, gw, d[:, 16:16 + n], mi.cuda(), policy, residual, m_alignment=align,
                                                         tune_swap_ab=1, tune_split_transform=1)
    want = oracle.grouped_gemm(wide[:, 24:24 + k].contiguous(), b.cpu(), sfb.cpu(), gw.cpu(), mi, n, mode="dual" if residual else "single",
                               scale_policy=policy)
    assert rel_l2(d[:, 16:16 + n], want) < 2.5e-3                          # as above
    assert bool((d[:, :16] == 7.0).all()) and bool((d[:, 16 + n:] == 7.0).all())


@pytest.mark.parametrize("align,tiles,n,k", [(16, 256, 4096, 1792), (32, 4, 6400, 4608), (64, 4, 4096, 3584), (16, 8, 640, 1024), (64, 2, 640, 1024)])
@pytest.mark.parametrize("policy", ["derived_div8", "div4_radix8"])
def test_the_default_is_one_of_the_two_paths(align, tiles, n, k, policy):
    """Calls on either side of the limits from which the library takes this path by itself: both paths sum every pass in ascending K
    and add the two at the end, so whichever it is, the bits are the same."""
    experts = min(4, tiles)
    b, sfb, gw = weights(experts, n, k, 3)
    mi = nvfp4_gemm.make_m_indices([tiles // experts * align] * experts, alignment=align).cuda()
    a = torch.randn(tiles * align, k, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).cuda()
    d = torch.full((3, tiles * align, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    for split in range(3):
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a, b, sfb, gw, d[split], mi, policy, m_alignment=align, tune_swap_ab=1,
                                                             tune_split_transform=split)
    assert bool(torch.isfinite(d[0].float()).all()) and torch.equal(d[0], d[1]) and torch.equal(d[0], d[2])


def test_workspace_under_capture_and_on_two_streams():
    """The quantisation pass takes its workspace from a pool in stream order: inside a captured graph that is replayed with other
    activations, and with calls in flight on two streams."""
    align, n, k, sizes = 32, 512, 1024, [64, 32, 0, 96]
    m = sum(sizes)
    b, sfb, gw = weights(len(sizes), n, k, 4)
    mi = nvfp4_gemm.make_m_indices(sizes, alignment=align).cuda()
    inputs = [torch.randn(m, k, generator=torch.Generator().manual_seed(i)).to(torch.bfloat16).cuda() for i in range(2)]

    def call(a, d, split=1):
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a, b, sfb, gw, d, mi, m_alignment=align, tune_swap_ab=1, tune_split_transform=split)

    want = [torch.zeros(m, n, dtype=torch.bfloat16, device="cuda") for _ in inputs]
    for a, d in zip(inputs, want):
        call(a, d, split=2)                              # without a workspace
    a, d = inputs[0].clone(), torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(a, d)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(a, d)
        call(a, d)
    for i in (1, 0, 1):
        a.copy_(inputs[i])
        d.zero_()
        graph.replay()
        assert torch.equal(d, want[i])
    streams, outs = [torch.cuda.Stream(), torch.cuda.Stream()], [torch.zeros(20, m, n, dtype=torch.bfloat16, device="cuda") for _ in inputs]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    for i in range(20):
        for s, a, d in zip(streams, inputs, outs):
            with torch.cuda.stream(s):
                call(a, d[i])
    torch.cuda.synchronize()
    for d, w in zip(outs, want):
        assert bool((d == w).all())


@pytest.mark.parametrize("k,inter,tile", [(1024, 256, 32), (256, 512, 32), (512, 256, 64)])
def test_masked_rows_match_the_128_row_kernels(k, inter, tile):
    e, max_m, hidden, counts = 5, 256, 512, [1, 0, tile - 1, tile + 1, 256]
    up, down = weights(e, 2 * inter, k, 1), weights(e, hidden, inter, 2)
    up = (*_C.interleave_gate_up(up[0], up[1], e, inter), up[2])
    a = torch.randn(e * max_m, k, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16).cuda()
    masked_m = torch.tensor(counts, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def planes(width):
        return _C.QuantizedRows(torch.zeros(e * max_m * (width + width // 8), dtype=torch.uint8, device="cuda"), e, max_m, width)

    rows = planes(k)
    a0, a1, sfa = _C.debug_split_workspace(a)
    rows.a0.copy_(a0), rows.a1.copy_(a1), rows.scale_atoms.copy_(sfa)
    rows.scale_rows.copy_(sfa.view(e * max_m // 128, k // 64, 2, 32, 4, 4).permute(0, 4, 3, 2, 1, 5).reshape(rows.scale_rows.shape))
    live = torch.cat([torch.arange(c) + i * max_m for i, c in enumerate(counts)]).cuda()
    # one GEMM, BF16 out
    got, want = (torch.zeros(e, max_m, 2 * inter, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    _C.m_grouped_few_quantized_rows_gemm_masked(rows, *up, got, masked_m, token_tile=tile, device_status=status)
    _C.m_grouped_quantized_dual_nvfp4_gemm_masked(rows, *up, want, masked_m, device_status=status)
    assert _C.read_status(status) == 0
    assert rel_l2(got.view(-1, 2 * inter)[live], want.view(-1, 2 * inter)[live]) < 2.5e-3
    assert float(got[1].abs().max()) == 0.0 and float(got[0, tile:].abs().max()) == 0.0        # past the token tiles: untouched
    # SwiGLU and quantisation in the epilogue, then the down-projection
    hq, hw = planes(inter), planes(inter)
    _C.m_grouped_few_quantized_rows_gemm_masked(rows, *up, hq, masked_m, token_tile=tile, device_status=status)
    _C.m_grouped_quantized_swiglu_dual_nvfp4_gemm_masked(rows, *up, hw, masked_m, device_status=status)
    assert _C.read_status(status) == 0
    atoms = hw.scale_atoms.view(e * max_m // 128, inter // 64, 2, 32, 4, 4).permute(0, 4, 3, 2, 1, 5).reshape(hq.scale_rows.shape)
    for x, y in ((hq.a0, hw.a0), (hq.a1, hw.a1), (hq.scale_rows, atoms)):
        # an FP32 sum in another order is off by some 2^-20 of its value at most, so one gate or up value in 2^12 crosses a BF16
        # rounding boundary and moves its product by an ulp, which the residual code sees: one byte of two codes in 2^10
        assert float((x[live] != y[live]).float().mean()) < 0.002
    out, ref = (torch.zeros(e, max_m, hidden, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    _C.m_grouped_few_quantized_rows_gemm_masked(hq, *down, out, masked_m, token_tile=tile, device_status=status)
    _C.m_grouped_quantized_dual_nvfp4_gemm_masked(hw, *down, ref, masked_m, device_status=status)
    assert _C.read_status(status) == 0
    assert rel_l2(out.view(-1, hidden)[live], ref.view(-1, hidden)[live]) < 4e-3


@pytest.mark.parametrize("counts,tile,few", [([1, 0, 31, 33, 5], 32, True), ([256, 200, 0, 3, 128], 32, False), ([0, 0, 0, 0, 0], 32, True),
                                             ([160, 0, 0, 0, 0], 32, True), ([161, 0, 0, 0, 0], 32, False), ([96, 64, 0, 0, 0], 32, True),
                                             ([65, 1, 0, 0, 0], 64, True), ([65, 65, 0, 0, 0], 64, False)])
def test_the_counts_decide_between_the_kernels(counts, tile, few):
    """One of the two families takes the call, by the rule of gemm::Family (up to five token tiles of 32, or three of 64, to two blocks
    of 128 rows the decode kernels): the output has that family's bits, and of the two forms of the activation's scales
    only the one that the family writes is written."""
    e, max_m, hidden, inter = 5, 256, 512, 256
    up, down = weights(e, 2 * inter, hidden, 1), weights(e, hidden, inter, 2)
    up = (*_C.interleave_gate_up(up[0], up[1], e, inter), up[2])
    a = torch.randn(e * max_m, hidden, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16).cuda()
    masked_m = torch.tensor(counts, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def planes(width):
        return _C.QuantizedRows(torch.zeros(e * max_m * (width + width // 8), dtype=torch.uint8, device="cuda"), e, max_m, width)

    def outputs(call):
        rows, h, out = planes(hidden), planes(inter), torch.zeros(e, max_m, hidden, dtype=torch.bfloat16, device="cuda")
        a0, a1, sfa = _C.debug_split_workspace(a)
        rows.a0.copy_(a0), rows.a1.copy_(a1)
        rows.scale_rows.copy_(sfa.view(e * max_m // 128, hidden // 64, 2, 32, 4, 4).permute(0, 4, 3, 2, 1, 5).reshape(rows.scale_rows.shape))
        call(rows, h, out)
        assert _C.read_status(status) == 0
        return torch.cat([out[i, :c] for i, c in enumerate(counts)]), bool(h.scale_rows.any()), bool(h.scale_atoms.any())

    def by_decode(rows, h, out):
        _C.m_grouped_few_quantized_rows_gemm_masked(rows, *up, h, masked_m, token_tile=tile, device_status=status)
        _C.m_grouped_few_quantized_rows_gemm_masked(h, *down, out, masked_m, token_tile=tile, device_status=status)

    def by_128_rows(rows, h, out):
        _C.relayout_scales(rows, masked_m)
        _C.m_grouped_quantized_swiglu_dual_nvfp4_gemm_masked(rows, *up, h, masked_m, device_status=status)
        _C.m_grouped_quantized_dual_nvfp4_gemm_masked(h, *down, out, masked_m, device_status=status)

    either = lambda decide: lambda rows, h, out: _C.expert_mlp_few_rows(rows, up, h, down, out, masked_m, token_tile=tile, decide=decide,
                                                                       device_status=status)
    want, live = {True: outputs(by_decode)[0], False: outputs(by_128_rows)[0]}, sum(counts) > 0
    y, as_rows, as_atoms = outputs(either(True))
    assert torch.equal(y, want[few]) and (as_rows, as_atoms) == (few and live, not few and live)
    y, as_rows, as_atoms = outputs(either(False))
    assert torch.equal(y, want[True]) and (as_rows, as_atoms) == (live, False)


def test_layer_with_all_tokens_on_a_few_experts_runs_the_128_row_kernels():
    e, hidden, inter, tokens, k = 32, 1024, 256, 200, 4
    up, down = weights(e, 2 * inter, hidden, 5), weights(e, hidden, inter, 6)
    g = torch.Generator().manual_seed(8)
    x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16).cuda()
    uniform = torch.randn(tokens, e, generator=g).cuda()
    skewed = uniform + 50.0 * (torch.arange(e, device="cuda") < k)
    layer, other = (ExpertParallelMoE(e, hidden, inter, up, down, peer_rows_cap=256) for _ in range(2))
    other.FEW_ROWS = ()
    for logits, by_128_rows in ((uniform, False), (skewed, True)):
        ids, w = route_topk(logits, k)
        assert layer._few_rows_tile(ids.numel()) == 32
        y, want = layer(x, ids, w), other(x, ids, w)
        assert bool(layer.peer[0].hq.scale_atoms.any()) == by_128_rows         # only those kernels write them
        assert torch.equal(y, want) if by_128_rows else rel_l2(y, want) < 4e-3


def test_layer_of_few_tokens_matches_the_bf16_dispatch():
    e, hidden, inter, tokens, k = 16, 1024, 256, 40, 4
    up, down = weights(e, 2 * inter, hidden, 5), weights(e, hidden, inter, 6)
    g = torch.Generator().manual_seed(7)
    x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16).cuda()
    logits = torch.randn(tokens, e, generator=g)
    logits[:, 3] += 4.0                                                    # one expert gets nearly every token
    ids, w = route_topk(logits.cuda(), k)
    few = ExpertParallelMoE(e, hidden, inter, up, down, peer_rows_cap=128)
    assert few._few_rows_tile(ids.numel()) == 32 and few.peer[0].hq is not None
    y = [few(x, ids, w) for _ in range(2)]
    want = ExpertParallelMoE(e, hidden, inter, up, down, peer_rows_cap=128, quantized_dispatch=False)(x, ids, w)
    halves = ExpertParallelMoE(e, hidden, inter, up, down, peer_rows_cap=128, micro_batches=2)(x, ids, w)
    assert few.steps_repeated == 0 and torch.equal(y[0], y[1]) and torch.equal(y[0], halves) and rel_l2(y[0], want) < 4e-3
