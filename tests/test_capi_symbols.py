"""The C-ABI library builds for sm_100a without a GPU, loads, and exports every entry point
that include/rdq_b200.h declares.  No compute calls here."""
import ctypes
import os
import re

import pytest

from conftest import ROOT
from rdquant_b200 import _lib


def _declared():
    text = open(os.path.join(ROOT, "include", "rdq_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(rdq_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_header():
    _lib.build()
    handle = ctypes.CDLL(_lib.LIB_PATH)
    names = _declared()
    assert "rdq_gemv_mixed" in names and "rdq_gemm_mixed" in names and "rdq_dequant_packed" in names
    for name in names:
        assert hasattr(handle, name), f"{name} declared in rdq_b200.h but not exported"
    assert sorted(_lib.EXPORTS) == [n for n in names if n in _lib.EXPORTS]
    assert set(names) == set(_lib.EXPORTS)


def test_argument_validation_needs_no_gpu():
    lib = _lib.lib()
    assert lib.rdq_version() >= 100
    # n_fp4 > 0 with K not a multiple of 16 is rejected before anything touches the device
    rc = lib.rdq_dequant_packed(None, None, 1.0, None, None, None, 0, None, None, 0, 16, 0, 0, 24, None)
    assert rc == -1 and b"multiple of 16" in lib.rdq_last_error()
    rc = lib.rdq_gemv_mixed(None, 17, None, None, 1.0, None, None, None, None, None, None, 0, 16, 0, 32, None, None, 0, None)
    assert rc != 0


class _Layer(ctypes.Structure):
    """rdq_layer"""

    _fields_ = ([(name, ctypes.c_int) for name in ("n_fp4", "n_fp8", "n_fp16", "K")] + [("w_fp4_global_scale", ctypes.c_float)]
                + [(name, ctypes.c_void_p) for name in ("w_fp4", "w_fp4_scales", "w_fp8", "w_fp8_scales", "w_fp16", "w_tiled",
                                                        "perm", "inv_perm", "gemv_ws", "gemv_counters")])


@pytest.mark.parametrize("change,text", [
    (dict(K=72), b"multiple of 16"),                        # with an NVFP4 group
    (dict(K=0), b"shape"),
    (dict(n_fp8=-16), b"shape"),
    (dict(w_fp4_scales=None), b"must not be null"),
    (dict(w_fp8_scales=None), b"w_fp8_scales must not be null"),
    (dict(w_fp8_scales=None, w_fp4=None, w_tiled=4096), b"w_fp8_scales must not be null"),
    (dict(w_fp4=4100), b"16-byte aligned"),
    (dict(w_fp4_scales=4098), b"16-byte aligned"),
    (dict(w_fp8=4104), b"16-byte aligned"),
    (dict(w_tiled=4104), b"16-byte aligned"),
    (dict(n_fp4=24, w_tiled=4096), b"no tiled layout"),
    (dict(w_fp4=None), b"neither"),
])
@pytest.mark.parametrize("rows", [1, 40, 3000])
def test_linear_checks_what_its_kernels_rely_on(rows, change, text):
    """Refused before anything touches the device (on a machine without one, and with addresses that are none)."""
    fields = dict(n_fp4=32, n_fp8=16, n_fp16=0, K=128, w_fp4_global_scale=1.0, w_fp4=4096, w_fp4_scales=4096, w_fp8=4096,
                  w_fp8_scales=4096, w_fp16=None, w_tiled=None, perm=4096, inv_perm=4096, gemv_ws=4096, gemv_counters=4096)
    fields.update(change)
    layer = _Layer(**fields)
    lib = _lib.lib()
    need = ctypes.c_size_t(0)
    assert lib.rdq_linear_workspace_size(ctypes.byref(layer), rows, 0, ctypes.byref(need)) < 0 and text in lib.rdq_last_error()
    # no rows' memory either: a call that these checks let through would be refused for that
    for rc in (lib.rdq_linear(ctypes.byref(layer), None, 0, rows, None, None, None, 0, 0, None),
               lib.rdq_linear(ctypes.byref(layer), None, 1, rows, None, None, None, 0, 0, None)):
        assert rc < 0 and text in lib.rdq_last_error()


@pytest.mark.parametrize("n4,n8,k,decode_rows", [(300, 130, 1024, 16), (2001, 900, 4096, 16), (5001, 2503, 4096, 8), (9003, 5007, 8192, 0)])
def test_small_layers_without_tiles_stay_on_the_decode_kernel(n4, n8, k, decode_rows):
    """Which of its kernels a call takes, told by the scratch it asks for: the decode kernel needs none."""
    layer = _Layer(n_fp4=n4, n_fp8=n8, n_fp16=0, K=k, w_fp4_global_scale=1.0, w_fp4=4096, w_fp4_scales=4096, w_fp8=4096,
                   w_fp8_scales=4096, w_fp16=None, w_tiled=None, perm=4096, inv_perm=4096, gemv_ws=4096, gemv_counters=4096)
    need = ctypes.c_size_t(0)
    for x_type in (0, 1):
        for rows in range(1, 20):
            assert _lib.lib().rdq_linear_workspace_size(ctypes.byref(layer), rows, x_type, ctypes.byref(need)) == 0
            assert (need.value == 0) == (rows <= decode_rows), (rows, need.value)


@pytest.mark.parametrize("n4,n8,k,tiled,x_type,first", [
    # row-major layers: f16 and bf16 rows between the lines, K of multiples of 256, 128 and 64, and a short K
    (5001, 2503, 2560, False, 0, 9), (5001, 2503, 2560, False, 1, 17),          # 14 MB
    (2698, 1249, 5504, False, 0, 17), (3600, 1749, 3520, False, 0, 9),          # 15, 13 MB: a wave of the decode kernel, more than one
    (7001, 3503, 4096, False, 0, 1), (7001, 3503, 4096, False, 1, 1),           # 30 MB
    (6001, 3003, 4096, False, 0, 1), (6001, 3003, 3968, False, 1, 1 + 8),       # 26, 25 MB
    (8192, 4035, 2944, False, 0, 1), (8192, 4035, 2944, False, 1, 9),           # 25 MB
    (2451, 1208, 9664, False, 0, 9), (2451, 1208, 9664, False, 1, 9),           # 25 MB
    (22468, 11067, 1472, False, 0, 1), (22468, 11067, 1472, False, 1, 1),       # 35 MB
    # tiled ones whose rows stay out of the decode kernel's shared memory: narrow copies of block scales of a long and a short K
    (2048, 1024, 16000, True, 0, 9), (2048, 1024, 16000, True, 1, 9),           # 35 MB
    (10240, 5120, 2944, True, 0, 8), (4864, 2048, 5760, True, 0, 9),            # 32, 28 MB
])
def test_first_row_of_the_gemm(n4, n8, k, tiled, x_type, first):
    """The fewest rows that leave the decode kernel, told by the scratch beyond that for rounded bf16 rows."""
    layer = _Layer(n_fp4=n4, n_fp8=n8, n_fp16=0, K=k, w_fp4_global_scale=1.0, w_fp4=4096, w_fp4_scales=4096, w_fp8=4096,
                   w_fp8_scales=4096, w_fp16=None, w_tiled=4096 if tiled else None, perm=4096, inv_perm=4096, gemv_ws=4096,
                   gemv_counters=4096)
    need = ctypes.c_size_t(0)
    for rows in range(1, 20):
        assert _lib.lib().rdq_linear_workspace_size(ctypes.byref(layer), rows, x_type, ctypes.byref(need)) == 0
        rounded = (2 * rows * k + 255) // 256 * 256 if x_type else 0
        assert (need.value not in (0, rounded)) == (rows >= first), (rows, need.value)
