"""Calls that follow the kernel that writes what they read: launched while that kernel still runs, they may set
up and ask weights into L2, and read nothing before it is complete."""
import ctypes

import pytest
import torch

from conftest import ORDER
from rdquant_b200 import _lib
from rdquant_b200 import rdquant_cuda as rc
from rdquant_b200.fused_gemv_pack import pack_for_fused_gemv
from rdquant_b200.synthetic import random_packed_layer

pytestmark = pytest.mark.gpu

_READ = ("w_fp4_q", "w_fp4_scales", "w_fp8_q", "w_fp8_scales", "w_fp16", "w_tiled", "perm", "inv_perm", "bias")


def _flat(fd):
    """All tensors that a call reads, in one buffer: (bytes, {name: view})."""
    names = [n for n in _READ if fd.get(n) is not None]
    at, total = {}, 0
    for n in names:
        at[n] = total
        total += (fd[n].numel() * fd[n].element_size() + 255) // 256 * 256
    flat = torch.zeros(total, dtype=torch.uint8, device="cuda")
    views = {}
    for n in names:
        t = fd[n]
        views[n] = flat[at[n]:at[n] + t.numel() * t.element_size()].view(t.dtype).view(t.shape)
        views[n].copy_(t)
    return flat, views


@pytest.mark.parametrize("shape,rows,dtype", [
    ((1280, 896, 128, 2560), 32, torch.float16),   # streaming GEMM, both widths of its token tiles
    ((6144, 3072, 128, 2560), 100, torch.float16),
    ((1280, 896, 128, 2560), 700, torch.float16),  # decoded-once GEMM
    ((1280, 896, 128, 2560), 1, torch.float16),    # tiled GEMV
    ((1280, 896, 128, 2560), 5, torch.bfloat16),
    ((1201, 710, 90, 2064), 3, torch.float16),     # row-major GEMV below 10 MB
    ((1201, 710, 90, 2064), 12, torch.bfloat16),
])
def test_weights_written_by_the_kernel_before(shape, rows, dtype):
    """The copy right before a call lets the call's kernel start at once, reads the host (its blocks end at
    different times) and writes the layer: weights, scales, permutation and bias."""
    n4, n8, n16, k = shape
    n = n4 + n8 + n16
    hosts, fds = [], []
    for seed in (1, 2):
        gen = torch.Generator().manual_seed(seed)
        fd = pack_for_fused_gemv(random_packed_layer(n4, n8, n16, k, seed=seed), dict(zip(ORDER, shape[:3])), k, "cuda")
        fd["bias"] = (torch.randn(n, generator=gen) * 0.5).half().cuda()
        flat, views = _flat(fd)
        hosts.append(flat.cpu().pin_memory())
        fds.append((fd, flat, views))
    fd, live, views = fds[1]
    fd = {**fd, **views}
    assert fd["w_fp4_global_scale"] == fds[0][0]["w_fp4_global_scale"]
    layer = _lib.torch_ext().Layer({key: v for key, v in fd.items() if key != "bias"})
    x = torch.randn(rows, k, generator=torch.Generator().manual_seed(rows)).to(dtype).cuda()
    want = []
    for host in hosts:
        live.copy_(host)
        torch.cuda.synchronize()
        want.append(layer.linear(x, fd["bias"], 0))
        torch.cuda.synchronize()
    assert not torch.equal(*want)
    got = []
    for i in range(40):
        rc.stage_copy(live, hosts[i % 2])
        got.append(layer.linear(x, fd["bias"], 0))
    torch.cuda.synchronize()
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 2]), i
    rc.check_linear_status(fd)


@pytest.mark.parametrize("rows,k", [(32, 2560), (100, 2560), (1, 2560), (8, 2560), (5, 2064)])
def test_weights_written_while_the_call_is_resident(rows, k):
    """The same with a writer that leaves room for the call's blocks on every SM: silu(16) is 16 in f16, so
    that silu_mul of 16 and w / 16 writes the FP16 weights w."""
    n = 2048 if rows < 100 else 8192  # (the streaming GEMM, not the decoded-once one)
    splits = dict(zip(ORDER, (0, 0, n)))
    gen = torch.Generator().manual_seed(rows)
    w = [(torch.randint(-64, 65, (n, k), generator=gen) / 64.0).half() for _ in range(2)]
    inv = torch.randperm(n, generator=gen)
    fds = [pack_for_fused_gemv({"weight_fp16": v, "inv_permutation": inv}, splits, k, "cuda") for v in w]
    fd = fds[1]
    name = "w_tiled" if rows <= rc.MAX_GEMV_M and fd.get("w_tiled") is not None else "w_fp16"
    live = fd[name].view(-1).view(torch.float16)
    cols = 16 * next(c for c in range(1, live.numel() // 16 + 1) if live.numel() % (16 * c) == 0 and live.numel() // (16 * c) <= 4096)
    contents = [f[name].view(-1).view(torch.float16).view(-1, cols).clone() for f in fds]
    gate_up = [torch.cat([torch.full_like(c, 16.0), c / 16], dim=1) for c in contents]
    out = live.view(-1, cols)
    assert out.shape[0] > 8, "up to eight rows the writer would take a place of the decode kernel's"
    layer = _lib.torch_ext().Layer(fd)
    x = torch.randn(rows, k, generator=gen).half().cuda()
    want = []
    for gu, c in zip(gate_up, contents):
        rc.silu_mul(gu, out)
        torch.cuda.synchronize()
        assert torch.equal(out, c)
        want.append(layer.linear(x, None, 0))
        torch.cuda.synchronize()
    got = []
    for i in range(40):
        rc.silu_mul(gate_up[i % 2], out)
        got.append(layer.linear(x, None, 0))
    torch.cuda.synchronize()
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 2]), i
    rc.check_linear_status(fd)


@pytest.mark.parametrize("rows", [1, 16])
def test_gemv_behind_a_gather_that_outlasts_its_waits(rows):
    """The gather of a tensor-parallel step lets the next GEMV start and then waits for the other ranks, here for
    one that never comes: longer than the GEMV's own waits may take, which do not begin before it is done."""
    n4, n8, n16, k = 1280, 896, 128, 2560
    layer = random_packed_layer(n4, n8, n16, k, seed=3)
    fd = pack_for_fused_gemv(layer, dict(zip(ORDER, (n4, n8, n16))), k, "cuda")
    x = torch.randn(rows, k, generator=torch.Generator().manual_seed(rows)).half().cuda()
    want = rc.mixed_gemv(x, fd, None, _lib.RDQ_GEMV_PDL)
    buf, out = torch.zeros(64, dtype=torch.float16, device="cuda"), torch.ones(64, dtype=torch.float16, device="cuda")
    index = torch.arange(64, device="cuda")
    words = torch.tensor([0, 0, 1], dtype=torch.int32, device="cuda")  # the rank's flag, then this rank's state: launch 1
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def gather(wait_ms):
        _lib.check(_lib.lib().rdq_peer_gather(p(buf), p(index), p(out), 64, p(words), 1, p(words[1:]), p(status), wait_ms,
                                              _lib.RDQ_GEMV_PDL, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
                   "rdq_peer_gather")

    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    gather(20)
    a.record()
    gather(20)
    b.record()
    b.synchronize()
    wait_ms = int(20 * 1500.0 / a.elapsed_time(b)) + 1  # 1.5 s
    status.zero_()
    gather(wait_ms)
    got = rc.mixed_gemv(x, fd, None, _lib.RDQ_GEMV_PDL)
    rc.check_status(fd)
    assert int(status) == 10 and int(out.sum()) == 64, "the gather gave up and left its output alone"
    assert torch.equal(got, want)
