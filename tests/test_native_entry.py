"""Entry points of the native host path with tensors whose memory cannot be asked for (as tracing makes
them): they answer None or raise, and the process lives.  Each case in a process of its own."""
import subprocess
import sys

import pytest

from conftest import ROOT

_PRELUDE = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from rdquant_b200 import _lib
from rdquant_b200.inference import FusedMixedLinear
ext = _lib.torch_ext()
with FakeTensorMode():
    u8, half = dict(dtype=torch.uint8, device="cuda"), dict(dtype=torch.float16, device="cuda")
    w4, s4 = torch.empty(32, 64, **u8), torch.empty(32, 8, **u8)
    inv = torch.arange(32, dtype=torch.int32, device="cuda")
    fd = {"n_fp4": 32, "n_fp8": 0, "n_fp16": 0, "k": 128, "w_fp4_q": w4, "w_fp4_scales": s4, "inv_perm": inv, "perm": inv}
"""
_CASES = {
    "quantize": """
    perm = torch.arange(32, device="cuda")
    assert ext.quantize_layer(torch.empty(32, 128, **half), perm, 32, 0, 0) is None
""",
    "dequantize": """
    assert ext.dequantize(w4, s4, None, None, None, None, 32, 0, 0, 128) is None
""",
    "layer": """
    try:
        ext.Layer(fd)
    except RuntimeError:
        pass
    else:
        raise SystemExit("a layer without memory was accepted")
""",
    "module": """
    mod = FusedMixedLinear(n_nvfp4=32, n_fp8=0, n_fp16=0, k=128, inv_perm=inv, bias=None, fused_data=fd)
    try:
        mod(torch.empty(2, 128, **half))
    except RuntimeError:
        pass
    else:
        raise SystemExit("a call without memory was accepted")
""",
    "vmap": """
    perm = torch.arange(32, device="cuda")
    seen = []
    def one(w, codes):
        seen.append((ext.quantize_layer(w, perm, 32, 0, 0), ext.dequantize(codes, s4, None, None, None, None, 32, 0, 0, 128)))
        return w
    torch.func.vmap(one)(torch.empty(3, 32, 128, **half), torch.empty(3, 32, 64, **u8))
    assert seen == [(None, None)]
""",
}


@pytest.mark.parametrize("case", list(_CASES))
def test_tensors_without_memory(case):
    res = subprocess.run([sys.executable, "-c", _PRELUDE + _CASES[case]], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, f"exit code {res.returncode}\n{res.stderr[-2000:]}"
