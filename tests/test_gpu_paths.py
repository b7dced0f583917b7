"""Packed layers, single-token attention and the layer encoder at the sizes where their kernels and
dispatch rules begin and end: edges of tiles and stages, remainders, smallest and largest rows."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from conftest import ORDER, streaming_tiles
from oracle import oracle_np as onp
from rdquant_b200 import _lib
from rdquant_b200 import rdquant_cuda as rc
from rdquant_b200.inference import FusedMixedLinear, GraphedDecodeStep
from rdquant_b200.integrations.hf_export import pack_layer
from rdquant_b200.quantize import quantize_weight, quantize_weight_packed
from rdquant_b200.synthetic import random_packed_layer
from test_gpu_quantize import _special, _weights

pytestmark = pytest.mark.gpu


def _check_linear(n4, n8, n16, k, rows, dtype, bias, lead=()):
    layer = random_packed_layer(n4, n8, n16, k, seed=n4 + n8 + k + rows)
    splits = dict(zip(ORDER, (n4, n8, n16)))
    n = n4 + n8 + n16
    gen = torch.Generator().manual_seed(rows)
    if bias:
        layer["bias"] = (torch.randn(n, generator=gen) * 0.5).half()
    mod = FusedMixedLinear.from_layer_data(layer, splits, k, "cuda")
    x = torch.randn(rows, k, generator=gen).to(dtype).cuda()
    y = mod(x.view(*lead, -1, k) if lead else x)
    assert y.dtype == dtype and y.shape == (*(x.view(*lead, -1, k) if lead else x).shape[:-1], n)
    assert torch.equal(mod(x), y.view(rows, n)), "two calls differ"
    w = torch.from_numpy(onp.dequantize_layer_f32(onp.torch_layer_to_np(layer), splits, k)).cuda().double()
    xd = x.double()
    ref = xd @ w.t() + (layer["bias"].cuda().double() if bias else 0.0)
    # a sum of k exact products in FP32: at most k rounding errors of 2^-24 of the sum of magnitudes (and
    # one per weight for its channel scale); bf16 rows become f16 rows (below 2^-14 a step of 2^-24); then
    # the rounding of the result
    mags = xd.abs() @ w.abs().t()
    bound = (k + 2) * 2.0 ** -24 * mags + (2.0 ** -25 * w.abs().sum(1) if dtype == torch.bfloat16 else 0.0)
    bound = bound + (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) * (ref.abs() + bound) + 2.0 ** -25
    assert bool(((y.view(rows, n).double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("rows", [1, 16, 17, 64, 65, 128, 129, 256, 257])
@pytest.mark.parametrize("shape", [
    (256, 128, 128, 320),    # k past the last whole chunk of every format; one CTA's worth of chunks
    (300, 130, 20, 576),     # ragged groups
    (0, 130, 0, 128), (64, 0, 0, 64), (0, 0, 200, 192),  # one format, a single stage
    (1280, 896, 128, 1088),  # tiles cut by ranges
])
def test_streaming_gemm_edges(shape, rows):
    _check_linear(*shape, rows, torch.float16 if rows % 2 else torch.bfloat16, bias=rows in (16, 65, 129))


@pytest.mark.parametrize("shape,rows", [
    ((128, 64, 16, 208), 17),      # k a multiple of 16 only: decoded once from the first GEMM row on
    ((600, 303, 100, 336), 700),   # odd number of channels, partial tiles of both kinds
    ((768, 256, 0, 256), 2049),    # beyond the streaming GEMM
    ((2048, 384, 128, 2560), 1280),  # tiles split along k
])
def test_decoded_once_gemm_edges(shape, rows):
    _check_linear(*shape, rows, torch.float16, bias=True)
    _check_linear(*shape, rows, torch.bfloat16, bias=False)


@pytest.mark.parametrize("rows", [1, 8, 9, 16])
@pytest.mark.parametrize("shape", [(201, 90, 10, 4112), (17, 0, 0, 16), (0, 33, 0, 48), (5, 3, 1, 1040)])
def test_row_major_gemv_edges(shape, rows):
    _check_linear(*shape, rows, torch.float16, bias=rows == 9)
    _check_linear(*shape, rows, torch.bfloat16, bias=False)


@pytest.mark.parametrize("rows,lead", [(1, ()), (3, (3,)), (8, (2, 2)), (5, ())])
@pytest.mark.parametrize("shape", [(16, 16, 16, 64), (1328, 640, 80, 2560), (320, 160, 32, 9728)])
def test_tiled_gemv_edges(shape, rows, lead):
    """Fewer images than warp groups, tiles shared by groups and CTAs, bf16 rows."""
    _check_linear(*shape, rows, torch.float16, bias=False, lead=lead)
    _check_linear(*shape, rows, torch.bfloat16, bias=True, lead=lead)


@pytest.mark.parametrize("k", [64, 2560, 6144, 12288])
@pytest.mark.parametrize("rows", [1, 2, 5])
def test_norm_prologue_edges(k, rows):
    """The norm inside the GEMV with rows in registers and through shared memory: the same as the
    separate kernel up to the order of the mean square's sum."""
    if not rc.gemv_stages_x(rows, k):
        pytest.skip("rows do not fit")
    layer = random_packed_layer(64, 32, 16, k, seed=k)
    mod = FusedMixedLinear.from_layer_data(layer, dict(zip(ORDER, (64, 32, 16))), k, "cuda")
    gen = torch.Generator().manual_seed(k + rows)
    x, d = (torch.randn(rows, k, generator=gen).half().cuda() for _ in range(2))
    w = (1 + 0.1 * torch.randn(k, generator=gen)).half().cuda()
    res = torch.empty_like(x)
    y = rc.mixed_gemv_norm(x, d, w, 1e-6, mod._fd(), residual_out=res, flags=_lib.RDQ_GEMV_PDL)
    assert torch.equal(y, rc.mixed_gemv_norm(x, d, w, 1e-6, mod._fd()))
    h, r = torch.empty_like(x), x.clone()
    rc.add_rmsnorm(r, d, w, h, 1e-6, 0)
    assert torch.equal(res, r)
    ref = rc.mixed_gemv(h, mod._fd()).float()
    # a normalised value may move by one f16 step (2^-10 of it), twice (norm, weight)
    w_abs = torch.from_numpy(np.abs(onp.dequantize_layer_f32(onp.torch_layer_to_np(layer), dict(zip(ORDER, (64, 32, 16))), k))).cuda()
    assert bool(((y.float() - ref).abs() <= 2.0 ** -9 * (h.float().abs() @ w_abs.t()) + 2.0 ** -10 * ref.abs()).all())


@pytest.mark.parametrize("b,nq,nkv,dh,s,pos_v", [
    (1, 24, 2, 64, 40, 0),       # one row, twelve query heads per KV head
    (1, 16, 1, 256, 300, 255),   # one KV head: most splits
    (2, 32, 8, 128, 530, 512),   # the new row opens a block
    (40, 16, 8, 64, 50, 47),     # more sequences than two CTAs per SM
    (19, 32, 8, 128, 90, 77),    # one split per KV head, one wave
])
def test_single_token_attention_edges(b, nq, nkv, dh, s, pos_v):
    gen = torch.Generator().manual_seed(b + nq + pos_v)
    qkv = torch.randn(b, (nq + 2 * nkv) * dh, generator=gen).half().cuda()
    k_cache, v_cache = (torch.randn(b, nkv, s, dh, generator=gen).half().cuda() for _ in range(2))
    ang = torch.arange(s).float()[:, None] / 1e4 ** (torch.arange(0, dh, 2).float() / dh)[None, :]
    cos, sin = (torch.cat([f(ang), f(ang)], -1).half().cuda() for f in (torch.cos, torch.sin))
    pos = torch.tensor([pos_v], dtype=torch.long, device="cuda")
    k1, v1 = k_cache.clone(), v_cache.clone()
    q = torch.empty(b, nq, dh, dtype=torch.float16, device="cuda")
    rc.qk_rope_cache(qkv, None, None, cos, sin, pos, q, k1, v1, 1e-6, 0)
    scratch = rc.rope_attn_scratch(b, nq, nkv, dh, s, "cuda")
    for flags in (0, _lib.RDQ_GEMV_PDL):
        k2, v2 = k_cache.clone(), v_cache.clone()
        out = torch.full((b, nq * dh), float("nan"), dtype=torch.float16, device="cuda")
        rc.rope_attn_decode(qkv, None, None, cos, sin, pos, k2, v2, scratch, out, nq, dh ** -0.5, 1e-6, flags)
        assert torch.equal(k2, k1) and torch.equal(v2, v1)
        assert int(scratch.view(torch.int32).abs().sum()) == 0, "scratch not idle"
        kd, vd = k1[:, :, :pos_v + 1].double(), v1[:, :, :pos_v + 1].double()
        ref = F.scaled_dot_product_attention(q[:, :, None].double(), kd, vd, enable_gqa=True).reshape(b, nq * dh)
        # scores are FP32 sums of dh products (and the exponential a few 2^-22): a relative error e of every
        # weight moves the average by at most 2 e max |v|; the weights' own rounding is 2^-22; then f16
        mags = (q.double().abs().amax() * kd.abs().amax() * dh * dh ** -0.5).item()
        e = dh * 2.0 ** -24 * mags + 2.0 ** -20
        assert bool(((out.double() - ref).abs() <= 2.0 ** -11 * ref.abs() + 2 * e * vd.abs().max()).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("n4,n8,n16,k", [(12, 0, 0, 32), (40, 25, 3, 16), (0, 70, 0, 528), (30, 20, 10, 1040), (600, 500, 0, 512),
                                         (0, 0, 9, 48)])
def test_layer_encoder_edges(n4, n8, n16, k, dtype):
    """The whole layer in two launches: byte for byte the host route."""
    n = n4 + n8 + n16
    w = _special(dtype).repeat(2, 1)[:n] if k == 32 else _weights(n, k, n + k, dtype)
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(n))
    splits = dict(zip(ORDER, (n4, n8, n16)))
    host = pack_layer(quantize_weight(w, perm, splits), None)
    dev = quantize_weight_packed(w.cuda(), perm, splits)
    assert set(host) == set(dev)
    for key in host:
        a, b = host[key], dev[key].cpu()
        assert a.dtype == b.dtype and torch.equal(a, b), key


@pytest.mark.parametrize("n4,n8,n16,k", [(5000, 2150, 50, 1280), (4000, 2000, 0, 1296), (4000, 1200, 13, 1552), (0, 36000, 0, 16)])
def test_layer_encoder_long_pieces(n4, n8, n16, k):
    """Layers large enough for the encoder's long pieces of a row -- five vectors of 256 values, three, four and
    a ragged rest -- and as large with rows of a fraction of one: byte for byte the host route."""
    n = n4 + n8 + n16
    w = _weights(n, k, n + k, torch.float16)
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(n))
    splits = dict(zip(ORDER, (n4, n8, n16)))
    host = pack_layer(quantize_weight(w, perm, splits), None)
    dev = quantize_weight_packed(w.cuda(), perm, splits)
    assert set(host) == set(dev)
    for key in host:
        assert torch.equal(host[key], dev[key].cpu()), key


def _long_piece_rows(k):
    """Rows from which the encoder takes the long pieces: ten vectors of 256 values for every warp of the chip."""
    chunks = -(-(k // 8) // 32)
    return -(-10 * torch.cuda.get_device_properties(0).multi_processor_count * 3 * 8 // chunks)


@pytest.mark.parametrize("k", [16, 512, 528, 1280, 1296, 1552, 2560, 3344])
@pytest.mark.parametrize("share8,share16", [(0.3, 0.01), (1.0, 0.0)])
@pytest.mark.parametrize("fewer", [0, 1])
def test_layer_encoder_pieces_by_size(k, share8, share16, fewer):
    """Layers large enough for the encoder's long pieces of a row, and a row too small for them: rows of up to two
    vectors of 256 values, which keep the short pieces, then two and a rest, five, three and a rest, four and a
    rest, twice five, and 5 + 5 + 4; byte for byte the host route."""
    n = _long_piece_rows(k) - fewer
    n8, n16 = int(share8 * n), int(share16 * n)
    w = _weights(n, k, n + k, torch.float16)
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(n))
    splits = dict(zip(ORDER, (n - n8 - n16, n8, n16)))
    host = pack_layer(quantize_weight(w, perm, splits), None)
    dev = quantize_weight_packed(w.cuda(), perm, splits)
    assert set(host) == set(dev)
    for key in host:
        assert torch.equal(host[key], dev[key].cpu()), key


@pytest.mark.parametrize("m,twice", [(1, False), (8, False), (2, True)])
def test_graphed_step_layers_beside_each_other(m, twice):
    """Layers of very different sizes that run beside each other, inputs changing from step to step; with a
    layer twice in the list (shared scratch) one after another."""
    shapes = [(16, 16, 0, 64), (2048, 1024, 128, 2560), (64, 32, 16, 9728), (4096, 2048, 0, 1024)]
    mods = [FusedMixedLinear.from_layer_data(random_packed_layer(*s, seed=s[3]), dict(zip(ORDER, s[:3])), s[3], "cuda") for s in shapes]
    if twice:
        mods = mods[:2] + mods[1:2]
    step = GraphedDecodeStep(mods, m=m)
    gen = torch.Generator().manual_seed(m)
    for _ in range(12):
        xs = [torch.randn(m, mod.K, generator=gen).half() for mod in mods]
        for buf, x in zip(step.x_host, xs):
            buf.copy_(x)
        out = [y.clone() for y in step.run()]
        for mod, x, y in zip(mods, xs, out):
            assert torch.equal(y, rc.mixed_gemv(x.cuda(), mod._fd()).cpu())


@pytest.mark.parametrize("rows,h", [(1, 8), (33, 2048), (2, 8192), (3, 8200), (200, 16392)])
@pytest.mark.parametrize("with_delta", [False, True])
def test_add_rmsnorm_row_lengths(rows, h, with_delta):
    """Rows shorter than a turn of the block, as long as its registers hold, and longer."""
    gen = torch.Generator().manual_seed(rows + h)
    x, d = (torch.randn(rows, h, generator=gen).half().cuda() for _ in range(2))
    w = (1 + 0.1 * torch.randn(h, generator=gen)).half().cuda()
    xs = x + d if with_delta else x.clone()
    xd = xs.double()
    ref = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    out = torch.empty_like(x)
    rc.add_rmsnorm(x, d if with_delta else None, w, out, 1e-6)
    assert torch.equal(x, xs)
    # two roundings to f16 (2^-11 each; 2^-24 where subnormal) and an FP32 sum far below them
    assert bool(((out.double() - ref).abs() <= 2.1 * 2.0 ** -11 * ref.abs() + 2.0 ** -23).all())


@pytest.mark.parametrize("rows,f", [(1, 8), (32, 9728), (148, 2048), (148, 2056), (295, 4104)])
def test_silu_mul_shares(rows, f):
    """Shares of a CTA of nothing, of one turn, of a turn and one, and of several with rows that end in them."""
    gu = torch.randn(rows, 2 * f, generator=torch.Generator().manual_seed(rows + f)).half().cuda()
    out = torch.empty(rows, f, dtype=torch.float16, device="cuda")
    rc.silu_mul(gu, out)
    g, u = gu[:, :f].double(), gu[:, f:].double()
    ref = g * torch.sigmoid(g) * u
    # silu and product each rounded to f16; a subnormal silu is off by 2^-25, times u
    assert bool(((out.double() - ref).abs() <= 2.1 * 2.0 ** -11 * ref.abs() + 2.0 ** -25 * (u.abs() + 1)).all())


@pytest.mark.parametrize("shape,rows,tiles", [
    ((1280, 896, 128, 1088), 17, "whole"), ((1280, 896, 128, 1088), 64, "whole"), ((300, 130, 20, 576), 100, "whole"),
    ((0, 640, 128, 4096), 129, "whole"), ((0, 0, 256, 8192), 40, "whole"),  # (of one cluster: nobody may leave)
    # cut tiles: up to 64 tokens, shared by up to thirteen CTAs, and more of them, in one and several tiles of tokens
    ((2816, 1280, 128, 8192), 9, "cut"), ((2688, 1280, 128, 8192), 64, "cut"), ((13056, 6144, 256, 2560), 66, "cut"),
    ((4096, 1920, 128, 2560), 193, "cut"), ((3000, 700, 70, 2560), 257, "cut"), ((1280, 640, 128, 4096), 300, "cut"),
    ((2048, 384, 128, 2560), 1280, None), ((600, 303, 100, 336), 700, None),  # the decoded-once GEMM, tiles split along k
])
def test_shared_tiles_do_not_need_their_ctas_at_the_same_time(shape, rows, tiles):
    """CTAs that leave instead of waiting for the others of a tile: the ones that come last do its whole,
    with the same result bit for bit, and nothing is left behind for the next call."""
    layer = random_packed_layer(*shape, seed=rows)
    mod = FusedMixedLinear.from_layer_data(layer, dict(zip(ORDER, shape[:3])), shape[3], "cuda")
    assert streaming_tiles(mod._fd(), rows, torch.float16) == tiles
    x = torch.randn(rows, shape[3], generator=torch.Generator().manual_seed(rows)).half().cuda()
    y = mod(x)
    _lib.lib().rdq_gemm_test_timeout(2)
    try:
        for _ in range(5):
            assert torch.equal(mod(x), y)
    finally:
        _lib.lib().rdq_gemm_test_timeout(0)
    assert torch.equal(mod(x), y)
    rc.check_gemm_status("cuda")


@pytest.mark.parametrize("shape,rows,tiles", [
    ((1280, 896, 128, 1088), 40, "whole"), ((1280, 896, 128, 1088), 120, "whole"),
    ((2816, 1280, 128, 8192), 40, "cut"), ((1280, 640, 128, 4096), 300, "cut"),  # with counting words of the stream, or the capture
])
def test_one_layer_on_several_streams(shape, rows, tiles):
    """Calls of one layer that overlap: three streams at once, and a captured call replayed beside them."""
    k = shape[3]
    layer = random_packed_layer(*shape, seed=21)
    mod = FusedMixedLinear.from_layer_data(layer, dict(zip(ORDER, shape[:3])), k, "cuda")
    assert streaming_tiles(mod._fd(), rows, torch.float16) == tiles
    gen = torch.Generator().manual_seed(rows)
    xs = [torch.randn(rows, k, generator=gen).half().cuda() for _ in range(4)]
    _lib.torch_ext().drop_words()
    refs = [mod(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[3]):
        captured = [mod(xs[3]) for _ in range(3)]
    torch.cuda.synchronize()
    outs = []
    for _ in range(40):
        with torch.cuda.stream(streams[3]):
            graph.replay()
        for s, x in zip(streams[:3], xs):
            with torch.cuda.stream(s):
                outs.append(mod(x))
    torch.cuda.synchronize()
    for i, y in enumerate(outs):
        assert torch.equal(y, refs[i % 3])
    assert all(torch.equal(y, refs[3]) for y in captured)
    rc.check_gemm_status("cuda")
    # (a set of words for the stream of the first calls, the three streams, and the capture until a later call finds it over)
    assert _lib.torch_ext().drop_words() == (4 if tiles == "cut" else 0)


@pytest.mark.parametrize("k", [512, 1040])
@pytest.mark.parametrize("bad", [120, 1 << 40, -121])
def test_layer_encoder_refuses_bad_permutations(k, bad):
    """Entries out of range: refused at once on the host; on the device found without an access out of range,
    reported once, and the inverse holds valid rows."""
    splits = dict(zip(ORDER, (60, 40, 20)))
    w = _weights(120, k, k, torch.float16).cuda()
    perm = torch.randperm(120, generator=torch.Generator().manual_seed(k))
    rc.check_quantize_status("cuda")
    good = quantize_weight_packed(w, perm, splits)
    wrong = perm.clone()
    wrong[77] = bad
    with pytest.raises(IndexError, match="out of range"):
        quantize_weight_packed(w, wrong, splits)
    mod = FusedMixedLinear.from_layer_data(good, splits, k, "cuda")
    for report in (lambda: rc.check_quantize_status("cuda"), lambda: quantize_weight_packed(w, perm, splits),
                   lambda: mod(w[:1])):
        inv = quantize_weight_packed(w, wrong.cuda(), splits)["inv_permutation"]
        assert int(inv.min()) >= 0 and int(inv.max()) < 120
        inv[perm[77]] = 77
        assert torch.equal(inv, good["inv_permutation"]), "the other channels are where they belong"
        with pytest.raises(RuntimeError, match="entry out of range"):
            report()
    rc.check_quantize_status("cuda")
    fromend = quantize_weight_packed(w, (perm - 120).cuda(), splits)
    for key in good:
        assert torch.equal(good[key], fromend[key]), key
    twice = perm.clone()
    twice[5] = twice[6]  # not a permutation, but indices all the same
    inv = quantize_weight_packed(w, twice.cuda(), splits)["inv_permutation"]
    assert int(inv.min()) >= 0 and int(inv.max()) < 120 and int(inv[perm[5]]) == 0
    rc.check_quantize_status("cuda")


@pytest.mark.parametrize("k", [2560, 3344])
def test_layer_encoder_permutations_with_long_pieces(k):
    """The same for layers of long pieces: entries out of range at both ends of the formats, indices from the
    end, an entry twice."""
    n = _long_piece_rows(k)
    n4, n8 = int(0.6 * n), int(0.3 * n)
    splits = dict(zip(ORDER, (n4, n8, n - n4 - n8)))
    w = _weights(n, k, k, torch.float16).cuda()
    perm = torch.randperm(n, generator=torch.Generator().manual_seed(k))
    rc.check_quantize_status("cuda")
    good = quantize_weight_packed(w, perm, splits)
    for at, bad in ((0, n), (n4 - 1, -n - 1), (n4, 1 << 40), (n - 1, -(1 << 40))):
        wrong = perm.clone()
        wrong[at] = bad
        made = quantize_weight_packed(w, wrong.cuda(), splits)
        with pytest.raises(RuntimeError, match="entry out of range"):
            rc.check_quantize_status("cuda")
        inv = made["inv_permutation"]
        assert int(inv.min()) >= 0 and int(inv.max()) < n
        inv[perm[at]] = at
        assert torch.equal(inv, good["inv_permutation"]), "the other channels are where they belong"
        other = torch.arange(n, device="cuda") != at  # the other NVFP4 and FP16 rows are what they were
        assert torch.equal(made["weight_nvfp4"][other[:n4]], good["weight_nvfp4"][other[:n4]])
        assert torch.equal(made["weight_fp16"][other[n4 + n8:]], good["weight_fp16"][other[n4 + n8:]])
    fromend = quantize_weight_packed(w, (perm - n).cuda(), splits)
    for key in good:
        assert torch.equal(good[key], fromend[key]), key
    twice = perm.clone()
    twice[5] = twice[n - 1]
    inv = quantize_weight_packed(w, twice.cuda(), splits)["inv_permutation"]
    assert int(inv.min()) >= 0 and int(inv.max()) < n and int(inv[perm[5]]) == 0
    rc.check_quantize_status("cuda")


def test_layers_with_a_format_group_above_4_gb():
    """Byte offsets beyond 32 bits, decode to prompt: the rows around the border, the first and the last ones."""
    k, n = 65536, 65536 + 128
    gen = torch.Generator(device="cuda").manual_seed(9)
    codes = torch.randint(0, 0x78, (n, k), generator=gen, device="cuda", dtype=torch.uint8)  # up to 2^7
    scale = (torch.rand(n, generator=gen, device="cuda") + 0.5) / 64  # sums of a few hundred: f16 holds them
    perm = torch.randperm(n, generator=gen, device="cuda")
    inv = torch.empty_like(perm)
    inv[perm] = torch.arange(n, device="cuda")
    mod = FusedMixedLinear.from_layer_data({"weight_fp8": codes, "weight_fp8_scale": scale, "inv_permutation": inv},
                                           dict(zip(ORDER, (0, n, 0))), k, "cuda")
    rows = torch.cat([torch.arange(0, 4), torch.arange(65536 - 4, 65536 + 4), torch.arange(n - 4, n)]).cuda()
    w = codes[rows].view(torch.float8_e4m3fn).double() * scale[rows].double()[:, None]
    for m in (1, 40, 300):
        x = torch.randn(m, k, generator=gen, device="cuda").half()
        y = mod(x)[:, perm[rows]].double()
        ref, mags = x.double() @ w.t(), x.double().abs() @ w.abs().t()
        # as in _check_linear
        assert bool(((y - ref).abs() <= (k + 2) * 2.0 ** -24 * mags + 2.0 ** -11 * ref.abs() + 2.0 ** -25).all()), m
    rc.check_linear_status(mod._fd())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_calls_whose_scratch_does_not_fit(dtype):
    """No room for the decoded weights: the kernel that needs none runs instead."""
    splits = dict(zip(ORDER, (6528, 3072, 128)))
    mod = FusedMixedLinear.from_layer_data(random_packed_layer(6528, 3072, 128, 2560, seed=12), splits, 2560, "cuda")
    x = torch.randn(700, 2560, generator=torch.Generator().manual_seed(12)).to(dtype).cuda()
    y = mod(x).float()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # room for the outputs (14 MB each) and converted rows (20 MB), not for 50 MB of scratch
    limit = torch.cuda.memory_reserved() + (52 << 20)
    torch.cuda.set_per_process_memory_fraction(limit / torch.cuda.get_device_properties(0).total_memory)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(60 << 20, dtype=torch.uint8, device="cuda")
        z = mod(x)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert z.dtype == dtype
    # FP32 sums in another order, then a rounding (bf16: to f16 on the way as well)
    step = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
    assert bool(((z.float() - y).abs() <= step * y.abs() + 1e-4 * y.abs().max()).all())


@pytest.mark.parametrize("rows", [1, 40])
def test_silu_mul_of_infinities_and_nan(rows):
    """What a division gives: an infinite gate stays infinite, minus infinity and NaN give NaN, the far ends
    of the range nearly zero and the gate itself."""
    inf, nan = float("inf"), float("nan")
    gate = torch.tensor([inf, -inf, nan, 65504.0, -65504.0, -100.0, -88.0, 88.0, 0.0, -0.0, 1.0, -1.0, 20.0, -20.0, 1e-3, -1e-3])
    gu = torch.cat([gate, torch.ones(16)]).half().cuda().repeat(rows, 1)
    out = torch.empty(rows, 16, dtype=torch.float16, device="cuda")
    rc.silu_mul(gu, out)
    ref = (gu[:, :16].float() / (1 + torch.exp(-gu[:, :16].float()))).half()
    assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out.isinf(), ref.isinf())
    ok = ~ref.isnan()
    assert torch.equal(out.signbit()[ok], ref.signbit()[ok])
    ok &= ~ref.isinf()
    assert bool(((out - ref)[ok].abs() <= 2.0 ** -10 * ref[ok].abs()).all())


def test_single_token_attention_keeps_small_weights():
    """One row of weight 1 before thousands of about 2^-26 whose values are 750 times larger."""
    b, nq, nkv, dh, s = 37, 4, 4, 64, 16384  # as many KV heads as SMs: one split, four warps
    f16 = dict(dtype=torch.float16, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(3)
    k_cache = torch.full((b, nkv, s, dh), -2.25, **f16)
    k_cache[:, :, 0] = 0.0
    v_cache = (500 + 500 * torch.rand(b, nkv, s, dh, generator=gen, device="cuda")).half()
    v_cache[:, :, 0] = 1.0
    qkv = torch.ones(b, (nq + 2 * nkv) * dh, **f16)
    qkv[:, nq * dh:(nq + nkv) * dh] = -2.25
    qkv[:, (nq + nkv) * dh:] = 750.0
    cos, sin = torch.ones(s, dh, **f16), torch.zeros(s, dh, **f16)
    pos = torch.tensor([s - 1], dtype=torch.long, device="cuda")
    out = torch.empty(b, nq * dh, **f16)
    rc.rope_attn_decode(qkv, None, None, cos, sin, pos, k_cache, v_cache, rc.rope_attn_scratch(b, nq, nkv, dh, s, "cuda"), out, nq,
                        0.125, 1e-6)
    w = torch.full((s,), -18.0, dtype=torch.float64, device="cuda").exp()  # scores 0.125 * 64 * -2.25
    w[0] = 1.0
    for i in range(0, b, 9):
        ref = (w[:, None] * v_cache[i].double()).sum(1) / w.sum()
        # the scores are exact; an exponential of -18 is off by 2^-19 of it at most, and so is their sum; then f16
        bound = 2.0 ** -11 * ref + 2.0 ** -18 * (ref - 1.0).abs() + 2.0 ** -20
        assert bool(((out[i].view(nq, dh).double() - ref).abs() <= bound).all())
