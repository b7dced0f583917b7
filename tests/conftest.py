import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, "tests", "golden")
ORDER = ("NVFP4", "FP8", "FP16")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200) and the built kernels")


def pytest_collection_modifyitems(config, items):
    try:
        import torch

        has_gpu = torch.cuda.is_available()
    except Exception:
        has_gpu = False
    if has_gpu:
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


def golden_layers():
    """{case name: {key: array}} from tests/golden/layers.npz."""
    z = np.load(os.path.join(GOLDEN, "layers.npz"))
    out = {}
    for key in z.files:
        case, rest = key.split("/", 1)
        out.setdefault(case, {})[rest] = z[key]
    return out


def golden_layer_np(case: dict):
    """(layer dict in checkpoint naming with numpy arrays, splits dict, K)."""
    layer = {k[len("saved/"):]: v for k, v in case.items() if k.startswith("saved/")}
    splits = dict(zip(ORDER, (int(v) for v in case["splits"])))
    k = case["weight_f16_bits"].shape[1]
    return layer, splits, k


def golden_layer_torch(case: dict, device="cpu"):
    """Checkpoint-named torch tensors of a golden case (bf16 / f16 restored from bits)."""
    import torch

    layer, splits, k = golden_layer_np(case)
    out = {}
    for key, arr in layer.items():
        t = torch.from_numpy(np.ascontiguousarray(arr))
        if key == "weight_fp16":
            t = t.view(torch.int16).view(torch.bfloat16)
        elif key == "bias":
            t = t.view(torch.int16).view(torch.float16)
        out[key] = t.to(device)
    return out, splits, k


@pytest.fixture(scope="session")
def layers():
    return golden_layers()


def streaming_tiles(fd, rows, dtype):
    """What a linear of so many rows runs on, told by the words and the scratch it asks for: "cut" or "whole" tiles of the
    streaming GEMM, or None for another kernel."""
    import ctypes

    import torch

    from rdquant_b200 import _lib
    from test_capi_symbols import _Layer

    p = lambda key: None if fd.get(key) is None or fd[key].numel() == 0 else fd[key].data_ptr()
    layer = _Layer(n_fp4=fd["n_fp4"], n_fp8=fd["n_fp8"], n_fp16=fd["n_fp16"], K=fd["k"], w_fp4_global_scale=1.0, w_fp4=p("w_fp4_q"),
                   w_fp4_scales=p("w_fp4_scales"), w_fp8=p("w_fp8_q"), w_fp8_scales=p("w_fp8_scales"), w_fp16=p("w_fp16"),
                   w_tiled=p("w_tiled"), perm=p("perm"), inv_perm=p("inv_perm"), gemv_ws=p("workspace"), gemv_counters=p("tile_counters"))
    bf16 = int(dtype == torch.bfloat16)
    if _lib.lib().rdq_linear_uses_words(ctypes.byref(layer), rows, bf16):
        return "cut"
    need = ctypes.c_size_t(0)
    assert _lib.lib().rdq_linear_workspace_size(ctypes.byref(layer), rows, bf16, ctypes.byref(need)) == 0
    rounded = (2 * rows * fd["k"] + 255) // 256 * 256 if bf16 else 0  # bf16 rows as f16
    return "whole" if need.value == rounded + 256 else None
