"""GPU parity of the routed-MoE path (routing -> permutation -> NVFP4 grouped GEMMs ->
SwiGLU -> combine) against the CPU oracle, which runs the reference's expert loop on
dequantised NVFP4 operands."""
from __future__ import annotations

import pytest
import torch

from oracle import inputs as I
from oracle import ref_ops as R
from helpers import assert_bit_exact, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods():
    from racetrack_b200 import moe, ops
    return ops, moe


def _setup(tokens, hidden, inter, n_experts, topk, seed=0):
    x = I.randn((tokens, hidden), seed + 1)
    w13 = I.randn((n_experts, 2 * inter, hidden), seed + 2, std=0.05)
    w2 = I.randn((n_experts, hidden, inter), seed + 3, std=0.05)
    g = torch.Generator().manual_seed(seed + 4)
    indices = torch.rand(tokens, n_experts, generator=g).topk(topk, dim=-1)[1]
    weights = torch.rand(tokens, topk, generator=g) + 0.1
    return x, w13, w2, weights, indices


def test_moe_quant_nvfp4_matches_plain_quantiser(mods):
    """The tile-aware, gather-fused quantiser writes the same codes and scales as the plain one
    run on the gathered rows; scales land in each expert's own 128-row tiles."""
    ops, moe = mods
    tokens, hidden, n_experts, topk = 300, 512, 8, 2
    x, _, _, _, indices = _setup(tokens, hidden, 256, n_experts, topk)
    xc, idx = x.cuda(), indices.cuda()
    offsets, sorted_pairs, _ = ops.fused_moe_permute(idx, n_experts)
    pairs = tokens * topk
    tile_map, tile_base, tile_count = ops.moe_tile_map(offsets, 0, n_experts, pairs // 128 + n_experts + 1)
    amax = ops.tensor_absmax(xc)
    codes, sf, gs = moe.moe_quant_nvfp4(xc, tile_map, tile_count, pairs, amax=amax,
                                        sorted_pairs=sorted_pairs, topk=topk)
    gathered = xc[(sorted_pairs // topk).long()]
    ref_codes, ref_sf, ref_gs = ops.fused_nvfp4_quant(gathered, amax=amax)
    assert_bit_exact(codes, ref_codes, "codes")
    assert_bit_exact(gs, ref_gs, "global scale")
    off = offsets.cpu().tolist()
    tb = tile_base.cpu().tolist()
    sf_cpu, ref_sf_cpu = sf.cpu(), ref_sf.view(torch.uint8).cpu()
    kt = hidden // 64
    for e in range(n_experts):
        rows = off[e + 1] - off[e]
        if rows == 0:
            continue
        tiles = (rows + 127) // 128
        seg = sf_cpu[tb[e] * kt * 512:(tb[e] + tiles) * kt * 512]
        o = R.sf_tiled_offsets(rows, hidden // 16)
        assert torch.equal(seg[o], ref_sf_cpu[off[e]:off[e + 1]]), f"scales of expert {e}"
        pad = torch.ones(seg.numel(), dtype=torch.bool)
        pad[o.flatten()] = False
        assert int(seg[pad].sum()) == 0, "padding rows of a scale tile must be zero"


@pytest.mark.parametrize("tokens,hidden,inter,n_experts,topk", [
    (64, 512, 256, 16, 4),
    (300, 1024, 512, 8, 2),      # several m-tiles per expert
    (5, 512, 256, 16, 4),        # most experts empty
])
def test_fused_moe_experts_matches_oracle(mods, tokens, hidden, inter, n_experts, topk):
    ops, moe = mods
    x, w13, w2, weights, indices = _setup(tokens, hidden, inter, n_experts, topk, seed=tokens)
    shared = I.randn((tokens, hidden), 99)
    experts = moe.quantize_experts(w13.cuda(), w2.cuda())
    y = moe.fused_moe_experts(x.cuda(), weights.cuda(), indices.cuda(), experts,
                              n_experts=n_experts, shared=shared.cuda())
    ops.tc_error_state()
    ref = R.moe_experts_nvfp4(x, weights, indices, w13, w2, shared_out=shared)
    err = rel_err(y, ref)
    assert err <= 1e-2, f"relative error {err}"
    # expert parallelism: two ranks owning half of the experts each sum to the full result
    # (each rank quantises swiglu(h) with the amax of ITS rows, so a rank is checked against the
    # oracle restricted to the same experts, and the sum against the full result more loosely)
    half = n_experts // 2
    parts = []
    for r in range(2):
        lo, hi = r * half, (r + 1) * half
        ex = moe.quantize_experts(w13[lo:hi].cuda(), w2[lo:hi].cuda())
        part = moe.fused_moe_experts(x.cuda(), weights.cuda(), indices.cuda(), ex,
                                     n_experts=n_experts, expert_begin=lo)
        ops.tc_error_state()
        ref_r = R.moe_experts_nvfp4(x, weights, indices, w13, w2, expert_range=(lo, hi))
        assert rel_err(part, ref_r) <= 1e-2, f"rank {r}"
        parts.append(part.float())
    total = parts[0] + parts[1] + shared.cuda().float()
    assert rel_err(total, ref) <= 1e-1


def test_fused_moe_forward_routes_and_combines(mods):
    """Gate + routing + experts at DeepSeek-V3.2 routing shape (256 experts, 8 groups, top-8),
    small expert matrices."""
    ops, moe = mods
    tokens, hidden, inter = 256, 1024, 256
    d = I.gate_inputs(tokens, hidden=hidden)
    w13 = I.randn((I.N_EXPERTS, 2 * inter, hidden), 5, std=0.02)
    w2 = I.randn((I.N_EXPERTS, hidden, inter), 6, std=0.02)
    experts = moe.quantize_experts(w13.cuda(), w2.cuda())
    kw = dict(n_groups=d["n_groups"], topk_groups=d["topk_groups"], topk=d["topk"],
              route_scale=d["route_scale"])
    y = moe.fused_moe_forward(d["hidden"].cuda(), d["w_gate"].cuda(), d["bias"].cuda(), experts,
                              n_experts=I.N_EXPERTS, **kw)
    ops.tc_error_state()
    # the oracle gets the GPU's routing decision: the logits GEMM differs in summation order
    logits = torch.nn.functional.linear(d["hidden"].cuda().float(), d["w_gate"].cuda().float())
    w, idx = ops.fused_moe_route(logits, d["bias"].cuda(), **kw)
    ref = R.moe_experts_nvfp4(d["hidden"], w.cpu(), idx.cpu(), w13, w2)
    assert rel_err(y, ref) <= 1e-2


@pytest.mark.parametrize("window", [None, (37, 211)])
def test_swiglu_absmax_rows_writes_h_and_its_amax(mods, window):
    """One pass: h = bf16(silu(gate) * up) for the rows of the window and max |h| over them,
    bit for bit what the SwiGLU kernel and the windowed amax kernel give separately."""
    ops, moe = mods
    rows, inter = 300, 512
    gate_up = I.randn((rows, 2 * inter), 31, std=2.0).cuda()
    gate, up = gate_up[:, :inter], gate_up[:, inter:]
    win = None
    if window is not None:
        win = (torch.tensor([window[0]], dtype=torch.int32).cuda(),
               torch.tensor([window[1]], dtype=torch.int32).cuda())
    h, amax = moe.swiglu_absmax_rows(gate, up, win)
    lo, hi = window if window is not None else (0, rows)
    ref = ops.fused_swiglu(gate, up)
    assert_bit_exact(h[lo:hi], ref[lo:hi], "h")
    assert_bit_exact(amax, moe._absmax_rows(gate, up, win), "amax")
    assert_bit_exact(amax, ref[lo:hi].float().abs().max().reshape(1), "amax of h")


@pytest.mark.parametrize("tokens,hidden,n_experts,topk", [(300, 512, 8, 2), (5, 7168, 16, 4),
                                                           (1000, 1024, 4, 1)])
def test_moe_gather_nvfp4_equals_gather_fused_quantiser(mods, tokens, hidden, n_experts, topk):
    """Quantising every token once and copying codes and scales into expert order gives the
    bytes the gather-fused quantiser writes (quantisation is per row), padding rows included."""
    ops, moe = mods
    x, _, _, _, indices = _setup(tokens, hidden, 256, n_experts, topk, seed=tokens)
    xc = x.cuda()
    offsets, sorted_pairs, _ = ops.fused_moe_permute(indices.cuda(), n_experts)
    pairs = tokens * topk
    tile_map, _, tile_count = ops.moe_tile_map(offsets, 0, n_experts, pairs // 128 + n_experts + 1)
    amax = ops.tensor_absmax(xc)
    ref_codes, ref_sf, ref_gs = moe.moe_quant_nvfp4(xc, tile_map, tile_count, pairs, amax=amax,
                                                   sorted_pairs=sorted_pairs, topk=topk)
    q_codes, q_sf, q_gs = ops.fused_nvfp4_quant(xc, amax=amax)
    codes, sf = moe.moe_gather_nvfp4(q_codes, q_sf.view(torch.uint8), sorted_pairs, topk, tile_map,
                                     tile_count, pairs)
    assert_bit_exact(q_gs, ref_gs, "global scale")
    assert_bit_exact(codes, ref_codes, "codes")
    used = int(tile_count[0]) * (hidden // 64) * 512
    assert_bit_exact(sf[:used], ref_sf[:used], "tiled scales")


@pytest.mark.parametrize("rows", [[1], [8, 9], [16, 0, 17], [64, 65, 33], [128, 129, 1], [3, 255]])
def test_grouped_gemm_token_box_fits_the_rows(mods, rows):
    """Groups around the sizes of the token box (8, 16, ... 128 rows) on the single-CTA schedule, with
    other groups' rows behind each: against fp64 of the dequantised operands. Sums of K exact e2m1
    products times two e4m3 scales: K * 2^-24 of their magnitudes, bf16 rounds once."""
    ops, moe = mods
    groups, n, k = len(rows), 128, 512
    g = torch.Generator().manual_seed(sum(rows))
    total = sum(rows)
    x = torch.randn(total, k, generator=g).bfloat16().cuda()
    w = (torch.randn(groups, n, k, generator=g) * 0.1).bfloat16().cuda()
    offsets = torch.tensor([sum(rows[:i]) for i in range(groups + 1)], dtype=torch.int32, device="cuda")
    max_tiles = (total + 127) // 128 + groups
    tile_map, _, tile_count = ops.moe_tile_map(offsets, 0, groups, max_tiles)
    a_codes, a_sf, a_gs = moe.moe_quant_nvfp4(x, tile_map, tile_count, total, amax=ops.tensor_absmax(x))
    parts = [ops.fused_nvfp4_quant(w[i], tiled_scales=True) for i in range(groups)]
    prev = ops.gemm_nvfp4_schedule(1)
    try:
        out = ops.gemm_nvfp4_grouped(a_codes, a_sf, a_gs, torch.cat([p[0] for p in parts]),
                                     torch.cat([p[1].view(torch.uint8) for p in parts]),
                                     torch.cat([p[2] for p in parts]), tile_map, tile_count, n=n, groups=groups)
    finally:
        ops.gemm_nvfp4_schedule(prev)
    ops.tc_error_state()

    def dequant(t, amax):
        codes, sf, gs = (v.cpu() for v in ops.fused_nvfp4_quant(t, amax=amax))
        table = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])
        table = torch.cat([table, -table]).double()
        both = torch.stack([codes & 15, codes >> 4], dim=-1).reshape(t.shape[0], -1).long()
        return table[both] * sf.double().repeat_interleave(16, dim=1) * gs.double()
    a = dequant(x, ops.tensor_absmax(x))
    lo = 0
    for i, r in enumerate(rows):
        b = dequant(w[i], ops.tensor_absmax(w[i]))
        ref = a[lo:lo + r] @ b.t()
        bound = 2 * k * 2.0 ** -24 * (a[lo:lo + r].abs() @ b.abs().t()) + 2.0 ** -8 * ref.abs()
        assert bool(((out[lo:lo + r].cpu().double() - ref).abs() <= bound).all()), (i, r)
        lo += r


@pytest.mark.parametrize("tokens,topk,n_experts,begin,count", [
    (1, 8, 256, 0, 256), (13, 8, 256, 64, 128), (128, 8, 256, 0, 256),   # one launch: up to 1024 pairs
    (31, 33, 40, 0, 40), (1024, 1, 3, 1, 2), (5, 2, 1024, 1000, 24),
    (129, 8, 256, 0, 256), (341, 3, 7, 2, 5),                           # one block does not hold the pairs
])
def test_moe_plan_equals_permute_and_tile_map(mods, tokens, topk, n_experts, begin, count):
    from racetrack_b200 import _lib
    ops, _ = mods
    lib = _lib.load()
    g = torch.Generator().manual_seed(tokens)
    idx = torch.randint(0, n_experts, (tokens, topk), generator=g).cuda()
    want = ops.fused_moe_permute(idx, n_experts)
    pairs = tokens * topk
    max_tiles = (pairs + 127) // 128 + count
    tm, tb, tc = ops.moe_tile_map(want[0], begin, begin + count, max_tiles)
    new = [torch.full_like(t, -7) for t in (*want, tm, tb, tc)]
    amax2 = torch.full((2,), 5.0, device="cuda")
    ws = torch.empty(int(lib.rt_moe_permute_workspace_bytes(tokens, topk, n_experts)), dtype=torch.uint8, device="cuda")
    o, sp, pp, m, b, c = (t.data_ptr() for t in new)
    _lib.check(lib.rt_moe_plan(idx.data_ptr(), o, sp, pp, ws.data_ptr(), m, b, c, amax2.data_ptr(), max_tiles, begin,
                               begin + count, tokens, topk, n_experts, torch.cuda.current_stream().cuda_stream), "plan")
    for got, ref in zip((new[0], new[1], new[2], new[4], new[5]), (*want, tb, tc)):
        assert torch.equal(got, ref)
    n128, n256 = int(tc[0]), int(tc[1])
    assert torch.equal(new[3][:n128], tm[:n128])
    assert torch.equal(new[3][max_tiles:max_tiles + n256], tm[max_tiles:max_tiles + n256])
    assert amax2.tolist() == [0.0, 0.0]


@pytest.mark.parametrize("tokens", [1, 32, 33])
def test_experts_quantise_few_rows_in_expert_order(mods, tokens):
    """Up to 256 pairs the rows are quantised straight into expert order, beyond once per token and
    copied: the same bits as handing the rows over already quantised."""
    ops, moe = mods
    g = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, 512, generator=g).bfloat16().cuda()
    w13 = (torch.randn(16, 512, 512, generator=g) * 0.05).bfloat16().cuda()
    w2 = (torch.randn(16, 512, 256, generator=g) * 0.05).bfloat16().cuda()
    experts = moe.quantize_experts(w13, w2)
    weights, indices = ops.fused_moe_route(torch.randn(tokens, 16, generator=g).cuda(), None, n_groups=1,
                                           topk_groups=1, topk=8, route_scale=1.0, score_func="topk_softmax")
    got = moe.fused_moe_experts(x, weights, indices, experts, n_experts=16)
    codes, sf, gs = ops.fused_nvfp4_quant(x)
    want = moe.fused_moe_experts(None, weights, indices, experts, n_experts=16,
                                 x_quant=(codes, sf.view(torch.uint8), gs))
    assert torch.equal(got, want)


def test_a_token_is_routed_alike_in_calls_of_different_length(mods):
    """The experts and weights of a token do not depend on how many tokens a prefill chunk holds."""
    ops, _moe = mods
    g = torch.Generator(device="cuda").manual_seed(17)
    x = torch.empty(4096, 7168, device="cuda").normal_(generator=g).bfloat16()
    gate = torch.empty(256, 7168, device="cuda").normal_(0.0, 0.02, generator=g).bfloat16()
    bias = torch.empty(256, device="cuda").uniform_(-0.1, 0.1, generator=g)

    def route(m):
        logits = ops.linear_bf16(x[:m], gate, out_dtype=torch.float32)
        return ops.fused_moe_route(logits, bias, n_groups=8, topk_groups=4, topk=8, route_scale=2.5)
    weights, indices = route(4096)
    for m in (200, 777, 2048):
        w, i = route(m)
        assert torch.equal(i, indices[:m]) and torch.equal(w, weights[:m]), m


def test_expert_mlp_of_the_first_rows_of_a_buffer(mods):
    """Routing of fewer rows than x has (a padded token buffer): the routed rows' outputs, those of a
    call with these rows alone where the padding holds nothing larger."""
    ops, moe = mods
    tokens, hidden, inter, n_experts, topk = 200, 512, 256, 8, 2
    x, w13, w2 = _setup(tokens, hidden, inter, n_experts, topk)[:3]
    experts = moe.quantize_experts(w13.cuda(), w2.cuda())
    g = torch.Generator().manual_seed(3)
    x = x.cuda()
    for rows in (1, 40, 150):                 # few and many pairs
        indices = torch.randint(0, n_experts, (rows, topk), generator=g).cuda()
        weights = torch.rand(rows, topk, generator=g).cuda()
        padded = x.clone()
        padded[rows:] = 0
        want = moe.fused_moe_experts(x[:rows], weights, indices, experts, n_experts=n_experts)
        got = moe.fused_moe_experts(padded, weights, indices, experts, n_experts=n_experts)
        assert got.shape == (rows, hidden) and torch.equal(got, want)
    ops.tc_error_state()


@pytest.mark.parametrize("offset", [1, 4, 8])
@pytest.mark.parametrize("sizes", [(1, 7), (40, 0, 129), (200, 33, 96)])
def test_block_scales_at_any_address(mods, offset, sizes):
    """rt_moe_quant_nvfp4 writes the same codes and scales to scale buffers of any alignment."""
    from racetrack_b200 import _lib
    ops, _moe = mods
    rows, cols = sum(sizes), 512
    x = I.randn((rows, cols), 31).cuda()
    offsets = torch.tensor([0, *torch.tensor(sizes).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    max_tiles = rows // 128 + len(sizes) + 1
    tile_map, _, tile_count = ops.moe_tile_map(offsets, 0, len(sizes), max_tiles)
    amax = ops.tensor_absmax(x)

    def quantise(shift):
        codes = torch.zeros(rows, cols // 2, dtype=torch.uint8, device="cuda")
        sf = torch.full((max_tiles * (cols // 64) * 512 + 32,), 0xee, dtype=torch.uint8, device="cuda")
        _lib.check(_lib.load().rt_moe_quant_nvfp4(
            x.data_ptr(), None, None, 1, amax.data_ptr(), codes.data_ptr(), sf.data_ptr() + shift, None,
            tile_map.data_ptr(), tile_count.data_ptr(), max_tiles, cols, x.stride(0), 0, _lib.RT_BF16,
            torch.cuda.current_stream().cuda_stream), "rt_moe_quant_nvfp4")
        assert (sf[:shift] == 0xee).all()
        return codes, sf[shift:shift + max_tiles * (cols // 64) * 512]
    want, got = quantise(0), quantise(offset)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
