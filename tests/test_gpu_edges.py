"""The edges of the kernels whose tiles, boxes and tables depend on the call's sizes."""

from __future__ import annotations

import pytest
import torch

from aklr_b200 import workloads as wl
from oracle import moe_oracle as orc

pytestmark = pytest.mark.gpu


def dev():
    return torch.device("cuda:0")


def router_case(tokens, hidden, experts, dtype):
    g = torch.Generator().manual_seed(tokens * 1000 + hidden + experts)
    x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16)
    w = (torch.randn(experts, hidden, generator=g) * hidden**-0.5).to(dtype)
    exact = x.double() @ w.double().T
    return x, w, exact, x.double().abs() @ w.double().abs().T


@pytest.mark.parametrize("tokens", [1, 2, 3, 16, 17, 63, 64, 129])
@pytest.mark.parametrize("hidden,experts", [(136, 7), (192, 33), (2048, 512), (7168, 256)])
def test_bf16_router_at_every_shape_of_its_kernels(tokens, hidden, experts):
    """One token, 2 x 2 and 2 x 4 dot products per warp (at 136 columns, no whole boxes of K, for every batch size), the
    tensor-core tiles of 16 experts with one and two boxes of K per stage.
    Bound: the rounding to bf16 (2^-8 of the value) and at most 2^-23 of the sum of magnitudes for every 16th of the chain."""
    from aklr_b200.moe import router_logits

    x, w, exact, magnitude = router_case(tokens, hidden, experts, torch.bfloat16)
    got = router_logits(x.to(dev()), w.to(dev())).cpu().double()
    assert ((got - exact).abs() <= 2.0**-8 * exact.abs() + (hidden / 16 + 16) * 2.0**-23 * magnitude).all()


def router_tile(tokens, experts, sms):
    """Experts per CTA of the bf16 tensor-core router: the fewest, a power of two from 16, whose CTAs fit the chip at once."""
    tile = 16
    while tile < 256 and tile < experts and -(-tokens // 128) * -(-experts // tile) > sms:
        tile *= 2
    return tile


@pytest.mark.parametrize("hidden", [192, 256])
@pytest.mark.parametrize("tokens,experts,tile", [(1153, 256, 32), (3999, 250, 64), (4097, 257, 128), (9601, 257, 256), (16385, 256, 256)])
def test_bf16_router_at_every_width_of_its_tiles(hidden, tokens, experts, tile):
    """Tiles of 32 to 256 experts, ragged in experts and in tokens: the bound of the test above, and bit for bit the logits
    that the same rows get from calls small enough for 16-expert tiles (one accumulation over K whatever the tile)."""
    from aklr_b200.moe import router_logits

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert router_tile(tokens, experts, sms) == tile
    x, w, exact, magnitude = router_case(tokens, hidden, experts, torch.bfloat16)
    x, w = x.to(dev()), w.to(dev())
    got = router_logits(x, w)
    error = (got.cpu().double() - exact).abs()
    assert (error <= 2.0**-8 * exact.abs() + (hidden / 16 + 16) * 2.0**-23 * magnitude).all()
    for rows in (slice(0, 512), slice(tokens - 129, tokens)):
        assert router_tile(x[rows].shape[0], experts, sms) == 16
        assert torch.equal(got[rows], router_logits(x[rows].contiguous(), w))


@pytest.mark.parametrize("tokens", [1, 16, 17, 128, 129, 300])
@pytest.mark.parametrize("hidden,experts", [(128, 1), (384, 33), (768, 40), (3072, 256)])
def test_float32_router_keeps_float32_accuracy(tokens, hidden, experts):
    """Dot products up to 16 tokens, three bf16 terms on the tensor cores from 17; fewer K steps than accumulators (128),
    ragged expert tiles.  Bound: a truncation of 2^-23 of the partial sum, itself at most the sum of magnitudes, per
    16 products, and the final additions."""
    from aklr_b200.moe import router_logits_f32

    x, w, exact, magnitude = router_case(tokens, hidden, experts, torch.float32)
    got = router_logits_f32(x.to(dev()), w.to(dev())).cpu().double()
    assert ((got - exact).abs() <= (hidden / 16 + 32) * 2.0**-23 * magnitude).all()
    if tokens > 16:  # token rows at 8-byte alignment cannot be a TMA operand: the CUDA-core tile serves them
        shifted = torch.empty(x.numel() + 4, dtype=torch.bfloat16, device=dev())[4:].view(x.shape)
        shifted.copy_(x)
        again = router_logits_f32(shifted, w.to(dev())).cpu().double()
        assert ((again - exact).abs() <= (hidden + 32) * 2.0**-24 * magnitude).all()


@pytest.mark.parametrize("tokens", [1, 16, 17, 300])
def test_float32_router_refuses_widths_it_has_no_kernel_for(tokens):
    from aklr_b200 import _lib
    from aklr_b200.moe import router_logits_f32

    x, w, _, _ = router_case(tokens, 192, 8, torch.float32)
    with pytest.raises(_lib.AklrError) as err:
        router_logits_f32(x.to(dev()), w.to(dev()))
    assert err.value.code == -4  # AKLR_ERR_UNSUPPORTED_SHAPE: hidden is not a multiple of 128


@pytest.mark.parametrize("tokens", [17, 128, 300])
@pytest.mark.parametrize("hidden,experts", [(128, 33), (768, 40), (3072, 96), (7168, 257)])
def test_float32_router_adds_every_term_exactly_once(tokens, hidden, experts):
    """Weights 1 + m 2^-17, m < 1024: the first bf16 term is 1, the second holds m's leading eight bits and the third the
    rest.  Activations +a, -a in pairs, the last pair of every 64 is +a, 0, so that every K step adds one to the first term's
    sum.  Every partial sum of every term is a multiple of 2^-17 below 2^7 (times a), so float32 holds all of them exactly in
    any order: a term, a K step or an accumulator left out or added twice shows in the bits, in each expert tile."""
    from aklr_b200.moe import router_logits_f32

    g = torch.Generator().manual_seed(hidden + tokens)
    w = 1.0 + torch.randint(0, 1024, (experts, hidden), generator=g).double() * 2.0**-17
    sign = torch.randint(0, 2, (tokens, hidden // 2, 1), generator=g).double() * 2 - 1
    x = torch.cat([sign, -sign], dim=2)
    x[:, 31::32, 0], x[:, 31::32, 1] = 1.0, 0.0
    x = x.view(tokens, hidden) * 2.0 ** (torch.arange(tokens) % 3 - 1).double()[:, None]
    exact = x @ w.T
    got = router_logits_f32(x.to(torch.bfloat16).to(dev()), w.float().to(dev()))
    assert torch.equal(got.cpu().double(), exact)


@pytest.mark.parametrize("tokens", [1, 16, 17, 130])
@pytest.mark.parametrize("experts", [33, 256])
def test_router_infinities_do_not_depend_on_the_batch_size(tokens, experts):
    """An infinite activation or weight gives +-inf, NaN where it meets a zero or the opposite infinity, and a NaN gives
    NaN, from the dot products (up to 16 tokens) and from the tensor cores alike; all other logits are as without them."""
    from aklr_b200.moe import router_logits, router_logits_f32

    g = torch.Generator().manual_seed(tokens + experts)
    x = torch.randn(tokens, 384, generator=g).to(torch.bfloat16)
    w = (torch.randn(experts, 384, generator=g) * 0.05).to(torch.bfloat16).float()
    w[7, 100] = 0.0
    w[9, 200], w[10, 300], w[11, 44] = float("inf"), float("-inf"), float("nan")
    x[0, 100] = float("inf")
    if tokens > 1:
        x[1, 5], x[2, 5], x[2, 333] = float("-inf"), float("inf"), float("inf")
        x[3, 17], x[tokens - 1, 200] = float("nan"), float("-inf")
    products = x.double()[:, None, :] * w.double()[None]
    exact = products.sum(-1)
    finite = exact.isfinite()
    assert exact.isposinf().any() and exact.isneginf().any() and exact.isnan().any()
    bound = (384 / 16 + 32) * 2.0**-23 * products.abs().nan_to_num(0.0, 0.0, 0.0).sum(-1)
    for weight, logits, rounding in ((w, router_logits_f32, 0.0), (w.to(torch.bfloat16), router_logits, 2.0**-8)):
        got = logits(x.to(dev()), weight.to(dev())).cpu().double()
        assert torch.equal(got.isnan(), exact.isnan())
        assert torch.equal(got.isposinf(), exact.isposinf()) and torch.equal(got.isneginf(), exact.isneginf())
        assert ((got - exact).abs()[finite] <= (rounding * exact.abs() + bound)[finite]).all()


@pytest.mark.parametrize("n_experts", [1, 31, 543, 544, 545, 1025])
@pytest.mark.parametrize("n_tokens,k,block_m", [(1, 1, 16), (33, 1, 128), (1025, 1, 16), (4096, 1, 32), (4097, 1, 128)])
def test_sort_with_and_without_the_per_warp_counts(n_experts, n_tokens, k, block_m):
    """The per-warp count table serves up to 544 experts; one CTA up to 4096 routes, chunks of 1024 beyond."""
    from aklr_b200.moe import moe_align

    g = torch.Generator().manual_seed(n_experts + n_tokens)
    ids = torch.randint(0, n_experts, (n_tokens, k), generator=g).to(torch.int32)
    sorted_ids, block_expert, counts, nb = moe_align(ids.to(dev()), n_experts, block_m)
    ref_sorted, ref_blocks, ref_counts = orc.moe_align(ids, n_experts, block_m)
    assert torch.equal(counts.cpu().long(), ref_counts) and nb == ref_blocks.numel()
    assert torch.equal(block_expert.cpu(), ref_blocks)
    assert torch.equal(sorted_ids.cpu(), ref_sorted)


@pytest.mark.parametrize("inter", [128, 256, 384])
@pytest.mark.parametrize("act_bits", [4, 8, 16])
@pytest.mark.parametrize("copies", [1, 3])
def test_mxfp4_boxes_at_their_edges(inter, act_bits, copies):
    """Experts with 1, 8, 9, 16, 17, ... routed rows (boxes of 16, 32, 64 and 128 rows, direct and staged output rows, warps
    without a row): bit for bit the output of loading all 128 rows, and the oracle's within its gates.  With three routes per
    token and more than 512 tokens the same rows are quantised once per token, then copied."""
    from aklr_b200 import _lib
    from aklr_b200.moe import fused_experts_mxfp4

    rows = [1, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129]
    fillers = 4  # experts after them that take the other routes of a token with three
    cfg = wl.MoEConfig("mx", hidden=256, inter=inter, n_routed=len(rows) + fillers + 1, topk=copies)
    weights = [t.to(dev()) for t in wl.mx_expert_weights(cfg, 5)]
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(rows)])  # the last expert gets none
    g = torch.Generator().manual_seed(inter + act_bits)
    ids = ids[torch.randperm(ids.numel(), generator=g)].view(-1, 1)
    if copies == 3:  # one route to an edge-sized expert in a random slot, two to the fillers
        t = torch.arange(ids.shape[0], dtype=torch.int32).view(-1, 1)
        ids = torch.cat([ids, len(rows) + t % 2, len(rows) + 2 + t % 2], dim=1)
        ids = ids.gather(1, torch.rand(ids.shape, generator=g).argsort(1)).contiguous()
    assert torch.bincount(ids.flatten(), minlength=cfg.n_routed)[: len(rows)].tolist() == rows
    x = torch.randn(ids.shape[0], 256, generator=g).to(torch.bfloat16)
    route_weights = torch.rand(ids.shape, generator=g)
    outs = []
    for variant in (0, _lib.VARIANT_FULL_ACTIVATION_BOXES):
        out, ws = fused_experts_mxfp4(x.to(dev()), ids.to(dev()), route_weights.to(dev()), *weights, return_workspace=True,
                                      variant=variant, act_bits=act_bits)
        ws.check_status()
        outs.append(out.cpu())
    assert torch.equal(outs[0], outs[1])
    ref = orc.mx_experts(x, ids.long(), route_weights, *[t.cpu() for t in weights], act_bits=act_bits)
    gates = orc.output_gates(outs[0], ref)
    assert orc.gates_pass(gates, min_sqnr_db=30.0 if act_bits != 4 else 20.0), gates


@pytest.mark.parametrize("rows,hidden", [(1, 128), (37, 384), (600, 7168)])
def test_quantised_codes_do_not_depend_on_the_outputs_alignment(rows, hidden):
    """Sixteen codes in one store where the buffer is 16-byte aligned, in two where it is only 8-byte aligned."""
    from aklr_b200.moe import per_group_quant_fp8

    x = torch.randn(rows, hidden, generator=torch.Generator().manual_seed(rows)).to(torch.bfloat16).to(dev())
    codes, scales = per_group_quant_fp8(x)
    shifted = torch.empty(rows * hidden + 8, dtype=torch.uint8, device=dev())[8:].view(torch.float8_e4m3fn).view(rows, hidden)
    codes8, scales8 = per_group_quant_fp8(x, quantized=shifted)
    assert torch.equal(codes.view(torch.uint8), codes8.view(torch.uint8)) and torch.equal(scales, scales8)
    amax = x.float().cpu().view(rows, hidden // 128, 128).abs().amax(-1)
    assert torch.equal(scales.cpu(), (amax.clamp_min(1e-10) * torch.tensor(1.0 / 448.0)).T.contiguous())


@pytest.mark.parametrize("rows,hidden", [(1, 128), (63, 16384), (64, 16384), (65, 16384), (1100, 1024)])
def test_quantised_rows_do_not_depend_on_the_rows_beside_them(rows, hidden):
    """Sixteen lanes per group in launches below 8192 groups (63 rows of 16384 and less), eight from there: the same codes and
    scales, bit for bit, for the same rows in a call of their own -- infinities, NaN, zeros, the largest and the smallest
    values among them.  The MXFP8 quantiser of per-token rows changes its warps' share of a row with the call's size, too."""
    from aklr_b200 import _lib
    from aklr_b200.moe import act_quant_fp8, per_group_quant_fp8

    def mx_rows(x):
        codes = torch.empty(x.shape, dtype=torch.uint8, device=dev())
        scales = torch.empty((x.shape[0], hidden // 32), dtype=torch.uint8, device=dev())
        order = torch.arange(x.shape[0], dtype=torch.int32, device=dev())
        stream = torch.cuda.current_stream().cuda_stream
        _lib.check(_lib.load().aklr_ep_gather_quant_mxfp8(x.data_ptr(), order.data_ptr(), x.shape[0], hidden, 1,
                                                          codes.data_ptr(), scales.data_ptr(), stream))
        return codes, scales

    x = torch.randn(rows, hidden, generator=torch.Generator().manual_seed(rows)).to(torch.bfloat16)
    special = [float("inf"), float("-inf"), float("nan"), 0.0, torch.finfo(torch.bfloat16).max, 2.0**-126, 2.0**-133, -3.0e-30]
    for i, value in enumerate(special[: hidden // 16]):
        x[0, 16 * i] = value
    x[rows - 1, :128] = 0.0
    x = x.to(dev())
    for quantise, by_group in ((act_quant_fp8, False), (per_group_quant_fp8, True), (mx_rows, False)):
        codes, scales = quantise(x)
        scales = scales.T if by_group else scales
        for row in {0, rows // 2, rows - 1}:
            alone, alone_scales = quantise(x[row : row + 1].contiguous())
            alone_scales = alone_scales.T if by_group else alone_scales
            assert torch.equal(alone.view(torch.uint8), codes[row : row + 1].view(torch.uint8)), quantise
            assert torch.equal(alone_scales.contiguous().view(torch.uint8), scales[row : row + 1].contiguous().view(torch.uint8))


@pytest.mark.parametrize("groups,limit", [(1, 256), (8, 1536)])
def test_routing_is_the_same_on_both_sides_of_the_kernels_line(groups, limit):
    """256 experts, sigmoid: counted up to 256 tokens without groups and 1536 with them, warp arg-maxes past that.  The
    tables of the first tokens agree bit for bit."""
    from aklr_b200.moe import Routing, route

    g = torch.Generator().manual_seed(limit)
    logits = torch.randn(limit + 1, 256, generator=g).to(torch.bfloat16).to(dev())
    bias = (torch.randn(256, generator=g) * 0.01).to(dev())
    routing = Routing(topk=8, scoring="sigmoid", num_expert_group=groups, topk_group=max(1, groups // 2), routed_scaling_factor=2.5)
    ids, weights = route(logits, bias, routing)
    ids_few, weights_few = route(logits[:limit].contiguous(), bias, routing)
    assert torch.equal(ids[:limit], ids_few) and torch.equal(weights[:limit], weights_few)


@pytest.mark.parametrize("tokens,experts", [(63, 64), (64, 64), (130, 256), (130, 33)])
def test_bf16_router_writes_logits_of_any_address(tokens, experts):
    """Logits that 16-byte stores cannot start at: bit for bit those of an aligned buffer, and nothing beside them."""
    from aklr_b200 import _lib
    from aklr_b200.moe import router_logits

    x, w, _, _ = router_case(tokens, 256, experts, torch.bfloat16)
    x, w = x.to(dev()), w.to(dev())
    want = router_logits(x, w)
    buffer = torch.full((tokens * experts + 16,), 7.0, dtype=torch.bfloat16, device=dev())
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.load().aklr_router_gemm_bf16(x.data_ptr(), w.data_ptr(), buffer.data_ptr() + 6, tokens, 256, experts, stream))
    assert torch.equal(buffer[3 : 3 + tokens * experts].view(tokens, experts), want)
    assert (buffer[:3] == 7.0).all() and (buffer[3 + tokens * experts :] == 7.0).all()
