"""Calls whose kernel starts while the kernel before still runs."""
import ctypes

import pytest
import torch

from conftest import ORDER
from rdquant_b200 import _lib
from rdquant_b200 import rdquant_cuda as rc
from rdquant_b200.fused_gemv_pack import pack_for_fused_gemv
from rdquant_b200.synthetic import random_packed_layer

pytestmark = pytest.mark.gpu


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
