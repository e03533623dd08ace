"""The many-row paths of a prompt against the decode operators, row for row and bit for bit: the prompt attention
(history tiles + one merge per slab) against slab-by-slab verify attention, and the packed linear module against the
GEMV in slabs; whole prompts against the operator-by-operator forward."""
import numpy as np
import pytest
import torch

from bitmtp_b200 import generate, native, ops, synthetic
from bitmtp_b200.fast_runtime import GraphAtlas
from bitmtp_b200.model import T2LinearKernel, make_sdlm_cache
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SLAB = 16


def _attention_inputs(T, hist0, H, Hkv, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rows = hist0 + T + 40
    q = torch.randn(T, H, 128, generator=gen, device=DEV).to(torch.bfloat16)
    k = torch.randn(Hkv, rows, 128, generator=gen, device=DEV).to(torch.bfloat16)
    v = torch.randn(Hkv, rows, 128, generator=gen, device=DEV).to(torch.bfloat16)
    return q, k, v


def _by_slab(q, k, v, hist0):
    T, H, _ = q.shape
    state = ops.new_step_state(torch.device(DEV))
    att = torch.empty(T, H * 128, dtype=torch.bfloat16, device=DEV)
    for r0 in range(0, T, SLAB):
        n, h = min(SLAB, T - r0), hist0 + r0
        ops.set_step_state(state, h, 0, native.ROLE_AR, 0)
        att[r0:r0 + n] = ops.verify_attention(q[r0:r0 + n].contiguous(), k, v, h, state,
                                              ops.attention_scratch(SLAB, H, h, DEV))[0]
    return att


def _prompt(q, k, v, hist0, calls=1):
    T, H, _ = q.shape
    scratch = ops.prompt_attention_scratch(T, hist0, SLAB, H, k.shape[0], DEV)
    att = torch.full((T + 1, H * 128), 7.0, dtype=torch.bfloat16, device=DEV)
    for _ in range(calls):
        amax = torch.zeros(T, dtype=torch.int32, device=DEV)
        ops.prompt_attention(q, k, v, hist0, SLAB, scratch, att=att[:T], amax=amax)
    torch.cuda.synchronize()
    assert native.lib().bm_device_error() == 0
    assert bool((att[T] == 7.0).all())
    finite = att[:T].float().isfinite().all(dim=1)
    assert torch.equal(amax.view(torch.float32)[finite], att[:T].float().abs().amax(dim=1)[finite])
    return att[:T]


@pytest.mark.parametrize("H,Hkv", [(2, 2), (8, 8), (16, 8), (32, 8), (8, 1), (6, 2)])      # 1, 1, 2, 4, 8 and (general kernel) 3 heads per group
@pytest.mark.parametrize("T,hist0", [(1, 0), (16, 0), (17, 0), (33, 112), (64, 128), (100, 129), (31, 500), (256, 1024),
                                     (500, 129), (1000, 16), (47, 4096)])
def test_prompt_attention_equals_the_slabs(T, hist0, H, Hkv):
    """Calls on both sides of the line between the tiles and the general kernel, ragged last tiles and slabs."""
    q, k, v = _attention_inputs(T, hist0, H, Hkv, T + hist0 + H)
    want = _by_slab(q, k, v, hist0)
    assert torch.equal(_prompt(q, k, v, hist0, calls=2).view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("T,H,Hkv", [(357, 8, 8), (340, 16, 8), (341, 32, 8), (511, 8, 1)])
def test_prompts_that_end_inside_a_warp(T, H, Hkv):
    """The last warp with rows holds one vector group of the prompt and one past its end, behind whole super-chunks."""
    q, k, v = _attention_inputs(T, 2560, H, Hkv, T)
    assert torch.equal(_prompt(q, k, v, 2560).view(torch.int16), _by_slab(q, k, v, 2560).view(torch.int16))


@pytest.mark.parametrize("T,hist0,H,Hkv", [(64, 2048, 16, 8), (207, 1025, 16, 8), (209, 1025, 16, 8), (96, 1300, 32, 8), (97, 1300, 32, 8),
                                           (432, 1100, 8, 1), (433, 1100, 8, 1)])
def test_tiles_then_few_or_many_slab_blocks(T, hist0, H, Hkv):
    """Both builds of the slab kernel behind the tiles, next to the line between them (three blocks per SM)."""
    q, k, v = _attention_inputs(T, hist0, H, Hkv, T)
    assert torch.equal(_prompt(q, k, v, hist0, calls=2).view(torch.int16), _by_slab(q, k, v, hist0).view(torch.int16))


def test_rows_past_a_history_do_not_reach_it():
    """Infinities and NaN in K / V rows that a slab may not see stay out of its results."""
    for T, hist0, keep in ((64, 160, 32), (512, 160, 400)):       # the general kernel, the tiles
        q, k, v = _attention_inputs(T, hist0, 16, 8, 3)
        clean = _prompt(q, k, v, hist0)
        k[:, hist0 + keep:] = float("nan")
        v[:, hist0 + keep:] = float("inf")
        got = _prompt(q, k, v, hist0)[:keep]
        assert bool(clean.isfinite().all()) and torch.equal(got.view(torch.int16), clean[:keep].view(torch.int16))


@pytest.mark.parametrize("what", [float("nan"), float("inf"), float("-inf"), 3.0e38])
def test_odd_values_in_a_history(what):
    """Infinities, NaN and the largest values in K rows that the slabs see: the same bits as slab by slab."""
    T, hist0 = 512, 176
    q, k, v = _attention_inputs(T, hist0, 16, 8, 9)
    k[0, 40:44], k[1, 0:160], k[2, 5, 7] = what, what, what
    q[8, 6] = 0.0
    want, got = _by_slab(q, k, v, hist0), _prompt(q, k, v, hist0)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


def _module(N, K, rows, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    packed, scale = synthetic.device_ternary(N, K, gen, torch.device(DEV))
    layer = T2LinearKernel(K, N).to(DEV)
    layer.weight.data, layer.weight_scale = packed, scale
    return layer, torch.randn(1, rows, K, generator=gen, device=DEV).to(torch.bfloat16)


def _gemv_by_row(layer, x):
    q, s = ops.quant_rows(x)
    return torch.cat([ops.t2_gemv(q[r:r + 1], layer.weight.data, s[r:r + 1], layer.weight_scale) for r in range(x.shape[0])])


@pytest.mark.parametrize("N,K", [(8, 128), (136, 384), (200, 2048), (504, 2560), (1024, 9728), (512, 2048)])
@pytest.mark.parametrize("rows", [16, 17, 33, 333])
def test_linear_module_equals_the_gemv_in_slabs(N, K, rows):
    """Row counts on both sides of the module's change to the many-row kernel, weights that end inside one of its
    tiles of 128 rows, K with and without a whole number of its stages."""
    layer, x = _module(N, K, rows, N + K + rows)
    q, s = ops.quant_rows(x[0])
    want = torch.cat([ops.t2_gemv(q[r:r + SLAB], layer.weight.data, s[r:r + SLAB], layer.weight_scale)
                      for r in range(0, rows, SLAB)])
    got = layer(x)
    torch.cuda.synchronize()
    assert native.lib().bm_device_error() == 0
    assert got.shape == (1, rows, N) and torch.equal(got[0].view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("N,K", [(4096, 1024), (4104, 1024), (264, 768), (72, 1152), (72, 2048), (8, ops.GEMV_MAX_K),
                                 (8, ops.GEMV_MAX_K + 256)])
@pytest.mark.parametrize("rows", [17, 24, 25, 32, 33])
def test_linear_module_on_both_sides_of_its_lines(N, K, rows):
    """The kernel that ops.gemv_serves_rows names is the one that runs (one launch, or two of the GEMV's 16 rows), and the
    other gives the same bits."""
    layer, x = _module(N, K, rows, N + K + rows)
    gemv, before = ops.gemv_serves_rows(rows, N, K), native.lib().bm_launch_count()
    got = layer(x)[0]
    assert native.lib().bm_launch_count() - before == (3 if gemv else 2)
    qp, sums, s = ops.quant_rows(x[0], prepared=True)
    other = torch.empty_like(got)
    if gemv:
        ops.t2_gemm_wide(qp, sums, layer.weight.data, s, layer.weight_scale, out=other)
    elif K % 256 == 0 and K <= ops.GEMV_MAX_K:
        for r in range(0, rows, 32):
            ops.t2_gemv_prepared(qp[r:r + 32], sums[r:r + 32], layer.weight.data, s[r:r + 32], layer.weight_scale,
                                 out=other[r:r + 32])
    else:
        other = _gemv_by_row(layer, x[0])
    torch.cuda.synchronize()
    assert native.lib().bm_device_error() == 0
    assert torch.equal(got.view(torch.int16), other.view(torch.int16))


def test_linear_module_at_its_limits():
    """The largest K of the many-row kernel, more rows than one of its grids has, and what stays refused."""
    layer, x = _module(8, 51200, 17, 5)
    got = layer(x)[0]
    q, s = (t.cpu().numpy() for t in ops.quant_rows(x[0]))
    _, want, _ = O.t2_gemv(q, layer.weight.data.cpu().numpy(), O.torch_to_u16(layer.weight_scale), s)
    assert np.array_equal(O.torch_to_u16(got), want)
    layer, x = _module(8, 51328, 17, 5)
    with pytest.raises(native.NativeError):
        layer(x)
    for N, K in ((12, 1024), (12, 512)):
        layer, x = _module(N, K, 17, 5)
        with pytest.raises(native.NativeError):
            layer(x)
    layer, x = _module(8, 128, 17, 5)
    layer.weight_scale = torch.cat([layer.weight_scale.view(-1)[:4], layer.weight_scale.view(-1)])[4:].view(8, 1)
    assert layer.weight_scale.data_ptr() % 16
    with pytest.raises(native.NativeError):
        layer(x)
    rows = ops.GEMM_WIDE_MAX_ROWS + 33
    layer, x = _module(8, 128, 1, 5)
    x = x[0].expand(rows, -1).contiguous()
    x[-1] *= -3.0
    got = layer(x)
    torch.cuda.synchronize()
    assert native.lib().bm_device_error() == 0
    ends = torch.cat([x[:1], x[-34:]])
    assert torch.equal(got[[0, *range(rows - 34, rows)]].view(torch.int16), _gemv_by_row(layer, ends).view(torch.int16))
    assert bool((got[:-1] == got[0]).all())


@pytest.mark.parametrize("N,K", [(8, 128), (128, 1152), (136, 2048), (128, 2176), (264, 4096), (19000, 2048)])
@pytest.mark.parametrize("T", [1, 31, 32, 33, 63, 64, 65, 130, 300])
def test_many_row_product_at_tile_edges(N, K, T):
    """Row counts and weight rows on both sides of a tile, fewer than 16 groups, an odd number of them, two and three per
    slot, more tiles than CTAs; scales of either sign, rows of zeros and weights of zeros (the sign of a zero counts)."""
    gen = torch.Generator(device=DEV).manual_seed(N + K + T)
    packed, scale = synthetic.device_ternary(N, K, gen, torch.device(DEV))
    packed[N // 2] = -86                                   # 0b10101010: codes of zero
    scale[::3] *= -1.0
    x = torch.randn(T, K, generator=gen, device=DEV).to(torch.bfloat16)
    x[T // 2] = 0.0
    qp, sums, s = ops.quant_rows(x, prepared=True)
    out = torch.full((T + 1, N), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.t2_gemm_wide(qp, sums, packed, s, scale, out=out[:T])
    q, s = ops.quant_rows(x)
    want = torch.cat([ops.t2_gemv(q[r:r + SLAB], packed, s[r:r + SLAB], scale) for r in range(0, T, SLAB)])
    torch.cuda.synchronize()
    assert native.lib().bm_device_error() == 0
    assert torch.equal(out[:T].view(torch.int16), want.view(torch.int16)) and bool((out[T] == 7.0).all())


@pytest.mark.parametrize("N,K,T", [(40008, 384, 17), (40008, 2176, 17), (19000, 1152, 130), (19000, 2176, 130)])
def test_many_row_product_over_several_tiles_with_an_odd_step(N, K, T):
    """CTAs that walk several tiles whose last step holds one group of its two, so that the rings and the prefetch go on from
    it: tiles of 32 and of 64 prompt rows, one and several groups per slot."""
    gen = torch.Generator(device=DEV).manual_seed(N + K + T)
    packed, scale = synthetic.device_ternary(N, K, gen, torch.device(DEV))
    x = torch.randn(T, K, generator=gen, device=DEV).to(torch.bfloat16)
    qp, sums, s = ops.quant_rows(x, prepared=True)
    q, _ = ops.quant_rows(x)
    want = torch.cat([ops.t2_gemv(q[r:r + SLAB], packed, s[r:r + SLAB], scale) for r in range(0, T, SLAB)])
    out = torch.full((T + 1, N), 7.0, dtype=torch.bfloat16, device=DEV)
    for _ in range(2):
        ops.t2_gemm_wide(qp, sums, packed, s, scale, out=out[:T])
    torch.cuda.synchronize()
    assert native.lib().bm_device_error() == 0
    assert torch.equal(out[:T].view(torch.int16), want.view(torch.int16)) and bool((out[T] == 7.0).all())


def _packed_model(geo, max_positions):
    cfg = synthetic.make_config(geo, block_size=8)
    state = synthetic.make_state(cfg, seed=4)
    model = generate.model_from_state(generate.args_from_config(cfg), state, DEV)
    model.prepare_merged_weights(max_positions=max_positions)
    return cfg, model


@pytest.mark.parametrize("heads", [(16, 8), (6, 2)])
def test_long_prompts_equal_the_operator_prefill(heads):
    """Prompts of one pass with several attention calls (600, 1200 rows) and of two passes (1300), an AR-only atlas,
    and short prompts before and after the workspace has grown (a pass captured with the old one must not come
    back): last-row logits and K / V rows bit for bit those of the operator-by-operator forward."""
    geo = dict(synthetic.TINY, n_heads=heads[0], n_kv_heads=heads[1], dim=512, ffn_dim=512)
    cfg, model = _packed_model(geo, 1601)
    sigma = 1600
    atlas = GraphAtlas(model, model.args, torch.device(DEV), segment_ladder=(sigma,), m_set=(1,), roles=("ar",),
                       capture_verbose=False)
    for seq in (40, 40, 600, 40, 1200, 1300, 1300, 40):
        assert atlas.takes_prompt(seq, sigma)
        prompt = synthetic.random_prompt(seq, cfg["vocab_size"], seed=seq)[0].to(DEV)
        cache = make_sdlm_cache(model.args, device=torch.device(DEV))
        want = model.forward_sdlm_prefill(token_values=prompt, cache=cache)[-1:].clone()
        atlas.kv_buffers[sigma].zero_()
        got = atlas.prefill(prompt, sigma)
        torch.cuda.synchronize()
        assert native.lib().bm_device_error() == 0
        assert torch.equal(got.view(torch.int32), want.view(torch.int32)), seq
        for i, (ck, cv) in enumerate(cache):
            for j, c in enumerate((ck, cv)):
                assert torch.equal(atlas.kv_buffers[sigma][j, i, 0, :, :seq].view(torch.int16), c[0].view(torch.int16)), (seq, i)
