"""Prefill GEMM (tcgen05) through the C ABI against the oracle: golden layers, random byte
patterns, the benchmark block shapes, ragged M, bias."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import ORDER, golden_layer_torch, streaming_tiles
from oracle import oracle_np as onp
from rdquant_b200 import _lib, rdquant_cuda
from rdquant_b200.fused_gemv_pack import pack_for_fused_gemv
from rdquant_b200.inference import FusedMixedLinear
from rdquant_b200.synthetic import QWEN3_4B_BLOCK, fixed_splits, random_packed_layer

pytestmark = pytest.mark.gpu
TOL = 2e-3  # max |y - y_ref| / max |y_ref|, FP32-accumulation reference


def _run(layer, splits, k, m, bias=False, seed=0):
    gen = torch.Generator().manual_seed(seed)
    x = torch.randn(m, k, generator=gen).half()
    n = sum(splits.values())
    b = (torch.randn(n, generator=gen) * 0.5).half() if bias else None
    fd = pack_for_fused_gemv(layer, splits, k, "cuda", tiled=False)
    y = rdquant_cuda.mixed_gemm(x.cuda(), fd, b.cuda() if bias else None)
    torch.cuda.synchronize()
    y_ref = onp.mixed_precision_linear(x.numpy(), onp.torch_layer_to_np(layer), splits, k,
                                       b.float().numpy() if bias else None)
    return y.cpu().float().numpy(), y_ref


def test_golden_layers(layers):
    for name, case in layers.items():
        layer, splits, k = golden_layer_torch(case)
        if k % 64:
            with pytest.raises(RuntimeError):
                _run(layer, splits, k, 32)
            continue
        for m in (1, 17, 130):
            y, y_ref = _run(layer, splits, k, m, bias="bias" in layer, seed=m)
            assert onp.rel_err(y, y_ref) < TOL, (name, m)


@pytest.mark.parametrize("m", [16, 100, 128, 300])
@pytest.mark.parametrize("shape", [(128, 128, 128, 256), (64, 32, 16, 512), (256, 0, 0, 1024), (0, 48, 0, 256),
                                   (0, 0, 32, 768), (49, 46, 1, 64), (1664, 768, 128, 4096)])
def test_random_bytes(shape, m):
    n4, n8, n16, k = shape
    layer = random_packed_layer(n4, n8, n16, k, seed=k + m)
    splits = dict(zip(ORDER, (n4, n8, n16)))
    y, y_ref = _run(layer, splits, k, m, bias=(m % 2 == 0), seed=m)
    assert onp.rel_err(y, y_ref) < TOL


@pytest.mark.parametrize("name", list(QWEN3_4B_BLOCK))
def test_block_shapes_m512(name):
    k, n = QWEN3_4B_BLOCK[name]
    splits = fixed_splits(n)
    layer = random_packed_layer(splits["NVFP4"], splits["FP8"], splits["FP16"], k, seed=len(name))
    y, y_ref = _run(layer, splits, k, 512, bias=True, seed=3)
    assert onp.rel_err(y, y_ref) < TOL, name


def test_matches_dequantised_weight_matmul():
    # size-independent property: GEMM == x @ dequant(W)^T with the bit-exact dequantisation kernel
    k, n = 2560, 4096
    splits = fixed_splits(n)
    layer = random_packed_layer(splits["NVFP4"], splits["FP8"], splits["FP16"], k, seed=9)
    fd = pack_for_fused_gemv(layer, splits, k, "cuda", tiled=False)
    dev = {kk: v.cuda() for kk, v in layer.items()}
    w = rdquant_cuda.dequantize_packed(dev, splits, k, inv_perm=dev["inv_permutation"])
    x = torch.randn(2048, k, device="cuda").half()
    y = rdquant_cuda.mixed_gemm(x, fd)
    ref = x.float() @ w.float().T
    err = (y.float() - ref).abs().max() / ref.abs().max()
    assert float(err) < TOL


@pytest.mark.parametrize("m,n,k", [(1024, 9728, 256), (1000, 9800, 192), (4096, 2560, 320)])
def test_large_tiles(m, n, k):
    """Enough tiles to select the 256-token x 256-channel configuration (all tensor-memory
    columns, three 64 KB stages), with ragged M and N, against the oracle and against
    x @ dequant(W)^T."""
    n16 = 128
    n8 = (n // 3) // 128 * 128
    n4 = n - n8 - n16
    layer = random_packed_layer(n4, n8, n16, k, seed=m + k)
    splits = dict(zip(ORDER, (n4, n8, n16)))
    y, y_ref = _run(layer, splits, k, m, bias=True, seed=5)
    assert onp.rel_err(y, y_ref) < TOL


@pytest.mark.parametrize("m", [512, 2048, 8192])
@pytest.mark.parametrize("group", [["q_proj", "k_proj", "v_proj"], ["o_proj"], ["gate_proj", "up_proj"], ["down_proj"]])
def test_benchmark_launches(group, m):
    """The four launches the prefill benchmark times -- q+k+v (2560 -> 6144) and gate+up
    (2560 -> 19456) packed as one layer each by fuse_layers, o and down as they are -- at its three
    token counts.  Every member layer is compared with the oracle on a seeded sample of 64 rows
    (the CPU side stays in seconds at M = 8192), and the whole output with x @ dequant(W)^T, the
    weight coming from the bit-exact dequantisation kernel."""
    from rdquant_b200.fused_gemv_pack import fuse_layers

    members = []
    for i, name in enumerate(group):
        k, n = QWEN3_4B_BLOCK[name]
        splits = fixed_splits(n)
        members.append((random_packed_layer(splits["NVFP4"], splits["FP8"], splits["FP16"], k, seed=51 + i), splits))
    k = QWEN3_4B_BLOCK[group[0]][0]
    data, splits = fuse_layers(members) if len(members) > 1 else members[0]
    fd = pack_for_fused_gemv(data, splits, k, "cuda", tiled=False)
    gen = torch.Generator().manual_seed(m)
    x = torch.randn(m, k, generator=gen).half().cuda()
    y = rdquant_cuda.mixed_gemm(x, fd)
    rdquant_cuda.check_gemm_status(x.device)
    rows = torch.randperm(m, generator=gen)[:64].sort().values
    xs, ys = x[rows.cuda()].cpu().numpy(), y[rows.cuda()].cpu().float().numpy()
    off = 0
    for layer, sp in members:
        n = sum(sp.values())
        y_ref = onp.mixed_precision_linear(xs, onp.torch_layer_to_np(layer), sp, k)
        assert onp.rel_err(ys[:, off:off + n], y_ref) < TOL, (group, m, off)
        off += n
    assert off == y.shape[1]
    dev = {kk: v.cuda() for kk, v in data.items()}
    w = rdquant_cuda.dequantize_packed(dev, splits, k, inv_perm=dev["inv_permutation"])
    worst = 0.0
    for r0 in range(0, m, 2048):  # in panels: the FP32 product of the full problem would take gigabytes
        ref = x[r0:r0 + 2048].float() @ w.float().T
        worst = max(worst, float((y[r0:r0 + 2048].float() - ref).abs().max() / ref.abs().max()))
    assert worst < TOL


@pytest.mark.parametrize("rows,shape,scratch", [(64, (22016, 10624, 128, 1024), False), (250, (22016, 10624, 128, 1024), False),
                                                (600, (22016, 10624, 128, 1024), True), (64, (2560, 1280, 256, 512), True)])
def test_wide_layers_of_few_rows_need_no_decoding(rows, shape, scratch):
    """Which of the two kernels mixed_gemm takes, told by the scratch it asks for; both give the same product."""
    n4, n8, n16, k = shape
    need = ctypes.c_size_t(0)
    assert _lib.lib().rdq_gemm_workspace_size(rows, n4 + n8 + n16, k, ctypes.byref(need)) == 0
    assert (need.value > 0) == scratch
    layer = random_packed_layer(n4, n8, n16, k, seed=rows)
    fd = pack_for_fused_gemv(layer, dict(zip(ORDER, shape[:3])), k, "cuda")
    x = torch.randn(rows, k, generator=torch.Generator().manual_seed(rows)).half()
    y = rdquant_cuda.mixed_gemm(x.cuda(), fd)
    rdquant_cuda.check_gemm_status("cuda")
    some = torch.arange(0, rows, 7)
    ref = onp.mixed_precision_linear(x[some].numpy(), onp.torch_layer_to_np(layer), dict(zip(ORDER, shape[:3])), k)
    assert onp.rel_err(y.cpu()[some].float().numpy(), ref) < TOL


@pytest.mark.parametrize("shape,rows,tiles", [
    # whole tiles, a CTA each: K of less than a chunk, of no whole chunk, groups that end inside a tile
    ((64, 32, 16, 64), 17, "whole"), ((0, 0, 128, 192), 9, "whole"), ((300, 130, 20, 576), 33, "whole"), ((37, 0, 5, 1344), 24, "whole"),
    ((60800, 20480, 5120, 256), 20, "whole"),     # five tiles each
    # clusters of two and four: chunks of k dealt out unevenly, several tiles each (buffers used again)
    ((4096, 2048, 0, 4096), 64, "whole"), ((13056, 6144, 256, 2560), 20, "whole"), ((13056, 6144, 256, 2624), 64, "whole"),
    ((2048, 384, 128, 2560), 20, "whole"), ((640, 384, 0, 9792), 31, "whole"), ((0, 0, 256, 8192), 40, "whole"), ((0, 700, 0, 3008), 48, "whole"),
    ((30000, 4000, 0, 8192), 33, "cut"),          # 170 MB
    # no room for the slots of a cluster of four: cut tiles, clusters of two
    ((2688, 1280, 128, 8192), 64, "cut"), ((2688, 1280, 128, 4096), 64, "whole"),
    # the line to the decode GEMV: rows that it does not keep in shared memory (eight of 2816, seven it does)
    ((2560, 896, 128, 13568), 7, "whole"), ((9600, 4864, 128, 2816), 8, "whole"), ((9600, 4864, 128, 2816), 7, None),
    # block scales copied 8 bytes at a time: whole tiles, one tile of tokens and several
    ((300, 130, 20, 896), 33, "whole"), ((1280, 640, 128, 2176), 100, "whole"), ((1280, 640, 128, 2176), 140, "whole"),
    # whole tiles of more than 64 tokens: clusters of one, two and four; tiles of tokens that are hardly filled
    ((2688, 1280, 128, 1088), 129, "whole"), ((3072, 896, 128, 4096), 128, "whole"), ((640, 384, 0, 2560), 129, "whole"),
    ((300, 130, 20, 2624), 200, "whole"), ((0, 0, 256, 8192), 256, "whole"),
    # cut ones where those are the faster, and beyond 256 rows; there small layers are decoded first
    ((4096, 1920, 128, 2560), 193, "cut"), ((13056, 6144, 256, 2560), 66, "cut"), ((1280, 640, 128, 4096), 300, "cut"),
    ((640, 384, 0, 2560), 257, None),
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_streaming_gemm_tiles(shape, rows, tiles, dtype):
    _check_streaming_gemm(shape, rows, dtype, tiles)


def _check_streaming_gemm(shape, rows, dtype, tiles):
    """The streaming GEMM through the module, with the tiles that are meant, against 64-bit sums over the dequantised weight (test_gpu_dequant.py: bit-exact)."""
    n4, n8, n16, k = shape
    splits = dict(zip(ORDER, shape[:3]))
    layer = random_packed_layer(n4, n8, n16, k, seed=k + rows)
    gen = torch.Generator().manual_seed(rows)
    layer["bias"] = (torch.randn(n4 + n8 + n16, generator=gen) * 0.5).half()
    mod = FusedMixedLinear.from_layer_data(layer, splits, k, "cuda")
    assert streaming_tiles(mod._fd(), rows, dtype) == tiles
    x = torch.randn(rows, k, generator=gen).to(dtype).cuda()
    y = mod(x)
    assert y.dtype == dtype and all(torch.equal(mod(x), y) for _ in range(3))
    rdquant_cuda.check_gemm_status(x.device)
    dev = {key: v.cuda() for key, v in layer.items()}
    w = rdquant_cuda.dequantize_packed(dev, splits, k, inv_perm=dev["inv_permutation"], out_dtype=torch.float32).double()
    ref = x.half().double() @ w.T + dev["bias"].double()
    # the result's rounding is half an ulp of a value (2^-11, 2^-8); FP32 sums of up to 9792 products stay far below
    err = (y.double() - ref).abs()
    half = 2.0 ** (-11 if dtype == torch.float16 else -8)
    assert float((err - 1.01 * half * ref.abs()).max() / ref.abs().max()) < 2e-5


@pytest.mark.parametrize("shape,rows", [
    # clusters of two with tiles FP16, FP16, NVFP4 and FP16, NVFP4, NVFP4 of 32 and 120 rows; FP8 of 48 rows and NVFP4 of 96
    ((4224, 2176, 128, 1536), 134), ((5376, 896, 128, 1536), 134), ((6784, 128, 0, 1408), 177),
    # clusters of four, five tiles each
    ((7936, 1408, 128, 1024), 85), ((8192, 1152, 128, 896), 65),
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_streaming_gemm_clusters_across_token_tiles(shape, rows, dtype):
    """Clusters whose tiles reach from the low ones at the end of a token tile into the high ones of the next: warps without
    rows in one tile have some two tiles later."""
    _check_streaming_gemm(shape, rows, dtype, "whole")


@pytest.mark.parametrize("shape,rows,tiles", [
    # a tile that no cluster of four has room for, of a long K: cut, unless there are more tiles than that
    ((3072, 1408, 128, 13312), 24, "cut"), ((2816, 1280, 128, 8192), 9, "cut"), ((2688, 1280, 128, 12288), 64, "cut"),
    ((2688, 1280, 128, 12288), 48, "whole"), ((5504, 2560, 128, 8192), 33, "whole"), ((12672, 6144, 128, 5120), 9, "cut"),
    # block scales copied 8 bytes at a time, where both cost more, and 4
    ((2816, 1280, 128, 13184), 24, "cut"), ((3456, 1664, 128, 11904), 33, "whole"), ((6656, 3200, 128, 8064), 24, "whole"),
    ((4352, 2048, 128, 6464), 24, "whole"),
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_streaming_gemm_tiles_of_up_to_64_rows(shape, rows, tiles, dtype):
    """Whole tiles and cut ones, each where it is the faster."""
    _check_streaming_gemm(shape, rows, dtype, tiles)


@pytest.mark.parametrize("dtype,tiles", [(torch.float16, "whole"), (torch.bfloat16, None)])
def test_bf16_rows_count_their_rounding(dtype, tiles):
    """A layer near the line between the GEMMs: bf16 rows are rounded ahead of the streaming one, inside the other's first launch."""
    _check_streaming_gemm((6400, 3072, 128, 1152), 230, dtype, tiles)
