"""Build and load ``librdq_b200.so`` -- the C-ABI library holding the sm_100a kernels -- and
``_rdq_torch.so``, the CPython extension with the native per-call host path over it.

Both are built in-tree (``build()``); the library is bound with ``ctypes``, signatures follow
``include/rdq_b200.h``.  There is no fallback: if one is missing or a call fails, a
``RuntimeError`` is raised.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
import subprocess
import sysconfig
import tempfile
import threading
from concurrent.futures import ThreadPoolExecutor

_HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(_HERE, "csrc")
LIB_PATH = os.path.join(CSRC, "librdq_b200.so")
TORCH_EXT_PATH = os.path.join(CSRC, "_rdq_torch.so")
SOURCES = [
    "rdq_api.cu",
    "rdq_dequant.cu",
    "rdq_gemv_generic.cu",
    "rdq_gemv_tiled.cu",
    "rdq_gemm.cu",
    "rdq_gemm_dense.cu",
    "rdq_gemm_stream.cu",
    "rdq_quantize.cu",
    "rdq_stage.cu",
    "rdq_glue.cu",
    "rdq_linear.cu",
]
TORCH_EXT_SOURCE = "rdq_torch.cpp"
HEADERS = ["rdq_common.cuh", "rdq_gemm_common.cuh", "rdq_kernels.cuh", "rdq_gemv_tiled_kernel.inl", "rdq_gemm_kernel.inl",
           os.path.join("..", "..", "include", "rdq_b200.h")]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]

RDQ_GEMV_AUTO = 0
RDQ_GEMV_GENERIC = 1
RDQ_GEMV_PDL = 16
RDQ_GEMV_OPENS = 32
RDQ_GEMV_BESIDE = 128
RDQ_GEMV_TEST_TIMEOUT = 64

RDQ_E_DEVICE = -4

_lock = threading.Lock()
_lib = None


def _older(target: str, files: list) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.exists(p) and os.path.getmtime(p) > t for p in (os.path.join(CSRC, f) for f in files))


def _stale() -> bool:
    return _older(LIB_PATH, SOURCES + HEADERS)


def _run(cmd: list) -> str:
    res = subprocess.run(cmd, cwd=CSRC, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + res.stdout + res.stderr)
    return res.stderr


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the kernels for sm_100a into ``csrc/librdq_b200.so`` and the host path into
    ``csrc/_rdq_torch.so`` (needs nvcc and a C++ compiler, no GPU)."""
    if force or _stale():
        nvcc = os.environ.get("NVCC", "nvcc")
        extra = ["-Xptxas", "-v"] if verbose else []
        with tempfile.TemporaryDirectory() as tmp, ThreadPoolExecutor() as pool:
            objs = [os.path.join(tmp, src + ".o") for src in SOURCES]
            for text in pool.map(lambda so: _run([nvcc, *NVCC_FLAGS, *extra, "-c", so[0], "-o", so[1]]), zip(SOURCES, objs)):
                if verbose:
                    print(text)
            _run([nvcc, "--shared", "-o", LIB_PATH, *objs, "-lcuda"])
    if force or _older(TORCH_EXT_PATH, [TORCH_EXT_SOURCE, HEADERS[-1]]):
        from torch.utils.cpp_extension import include_paths, library_paths

        dirs = include_paths("cuda") + [sysconfig.get_paths()["include"]]
        _run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", TORCH_EXT_SOURCE, "-o", TORCH_EXT_PATH,
              *("-I" + d for d in dirs), *("-L" + d for d in library_paths("cuda")), "-L" + CSRC, "-l:librdq_b200.so",
              "-lc10", "-lc10_cuda", "-lcudart", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-Wl,-rpath,$ORIGIN"])
    return LIB_PATH


def _bind(lib: ctypes.CDLL) -> None:
    vp, i32, f32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    lib.rdq_version.restype = i32
    lib.rdq_version.argtypes = []
    lib.rdq_last_error.restype = ctypes.c_char_p
    lib.rdq_last_error.argtypes = []
    lib.rdq_dequant_packed.restype = i32
    lib.rdq_dequant_packed.argtypes = [vp, vp, f32, vp, vp, vp, i32, vp, vp, i32, i32, i32, i32, i32, vp]
    lib.rdq_gemv_scratch_size.restype = i32
    lib.rdq_gemv_scratch_size.argtypes = [i32, ctypes.POINTER(ctypes.c_size_t), ctypes.POINTER(ctypes.c_size_t)]
    lib.rdq_gemv_mixed.restype = i32
    lib.rdq_gemv_mixed.argtypes = [vp, i32, vp, vp, f32, vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, vp, vp, i32, vp]
    lib.rdq_gemv_tiled_bytes.restype = ctypes.c_size_t
    lib.rdq_gemv_tiled_bytes.argtypes = [i32, i32, i32, i32]
    lib.rdq_gemv_repack.restype = i32
    lib.rdq_gemv_repack.argtypes = [vp, vp, vp, vp, vp, i32, i32, i32, i32, vp]
    lib.rdq_gemv_tiled.restype = i32
    lib.rdq_gemv_tiled.argtypes = [vp, i32, vp, vp, f32, vp, vp, vp, i32, i32, i32, i32, vp, vp, i32, vp]
    lib.rdq_gemv_tiled_stages_x.restype = i32
    lib.rdq_gemv_tiled_stages_x.argtypes = [i32, i32]
    lib.rdq_gemv_tiled_xop.restype = i32
    lib.rdq_gemv_tiled_xop.argtypes = [i32, vp, vp, vp, vp, f32, i32, vp, vp, f32, vp, vp, vp, i32, i32, i32, i32, vp, vp,
                                       i32, vp]
    lib.rdq_gemv_tiled_peer.restype = i32
    lib.rdq_gemv_tiled_peer.argtypes = [vp, i32, vp, vp, f32, vp, vp, vp, vp, i32, vp, i32, i32, i32, i32, vp, vp, i32, vp]
    lib.rdq_peer_gather.restype = i32
    lib.rdq_peer_gather.argtypes = [vp, vp, vp, ctypes.c_longlong, vp, i32, vp, vp, i32, i32, vp]
    lib.rdq_gemv_tiled_noalloc.restype = i32
    lib.rdq_gemv_tiled_noalloc.argtypes = [vp, i32, vp, vp, f32, vp, vp, vp, i32, i32, i32, i32, i32, vp]
    lib.rdq_gemv_tiled_status.restype = i32
    lib.rdq_gemv_tiled_status.argtypes = [vp, vp, i32, vp]
    lib.rdq_gemv_tiled_noalloc_status.restype = i32
    lib.rdq_gemv_tiled_noalloc_status.argtypes = [i32, vp]
    lib.rdq_gemm_status.restype = i32
    lib.rdq_gemm_status.argtypes = [i32, vp]
    lib.rdq_gemm_test_timeout.restype = None
    lib.rdq_gemm_test_timeout.argtypes = [i32]
    lib.rdq_gemm_mixed.restype = i32
    lib.rdq_gemm_mixed.argtypes = [vp, i32, vp, vp, f32, vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, vp]
    lib.rdq_gemm_mixed_ws.restype = i32
    lib.rdq_gemm_mixed_ws.argtypes = [vp, i32, vp, vp, f32, vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, vp, ctypes.c_size_t, vp]
    lib.rdq_gemm_workspace_size.restype = i32
    lib.rdq_gemm_workspace_size.argtypes = [i32, i32, i32, ctypes.POINTER(ctypes.c_size_t)]
    lib.rdq_quantize_nvfp4.restype = i32
    lib.rdq_quantize_nvfp4.argtypes = [vp, i32, i32, i32, vp, vp, vp, vp, vp]
    lib.rdq_quantize_fp8.restype = i32
    lib.rdq_quantize_fp8.argtypes = [vp, i32, i32, i32, vp, vp, vp, vp, vp]
    lib.rdq_quantize_layer.restype = i32
    lib.rdq_quantize_layer.argtypes = [vp, i32, vp, i32, i32, i32, i32, vp, vp, vp, vp, vp, vp, vp, vp, vp]
    lib.rdq_quantize_status.restype = i32
    lib.rdq_quantize_status.argtypes = [vp]
    lib.rdq_add_rmsnorm.restype = i32
    lib.rdq_add_rmsnorm.argtypes = [vp, vp, vp, vp, i32, i32, f32, i32, vp]
    lib.rdq_qk_rope_cache.restype = i32
    lib.rdq_qk_rope_cache.argtypes = [vp, vp, vp, vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, f32, i32, vp]
    lib.rdq_attn_decode_scratch_size.restype = i32
    lib.rdq_attn_decode_scratch_size.argtypes = [i32, i32, i32, i32, ctypes.POINTER(ctypes.c_size_t)]
    lib.rdq_attn_decode.restype = i32
    lib.rdq_attn_decode.argtypes = [vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, f32, i32, vp]
    lib.rdq_rope_attn_decode_scratch_size.restype = i32
    lib.rdq_rope_attn_decode_scratch_size.argtypes = [i32, i32, i32, i32, i32, ctypes.POINTER(ctypes.c_size_t)]
    lib.rdq_rope_attn_decode.restype = i32
    lib.rdq_rope_attn_decode.argtypes = [vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, i32, i32, i32, i32, i32, f32, f32, i32, vp]
    lib.rdq_silu_mul.restype = i32
    lib.rdq_silu_mul.argtypes = [vp, vp, i32, i32, i32, vp]
    lib.rdq_linear_workspace_size.restype = i32
    lib.rdq_linear_workspace_size.argtypes = [vp, i32, i32, ctypes.POINTER(ctypes.c_size_t)]
    lib.rdq_linear.restype = i32
    lib.rdq_linear.argtypes = [vp, vp, i32, i32, vp, vp, vp, ctypes.c_size_t, i32, vp]
    lib.rdq_linear_uses_words.restype = i32
    lib.rdq_linear_uses_words.argtypes = [vp, i32, i32]
    lib.rdq_linear_words.restype = i32
    lib.rdq_linear_words.argtypes = [vp, vp, i32, i32, vp, vp, vp, ctypes.c_size_t, vp, i32, vp]
    lib.rdq_stage_copy.restype = i32
    lib.rdq_stage_copy.argtypes = [vp, vp, ctypes.c_size_t, vp]
    lib.rdq_stage_copy_signal.restype = i32
    lib.rdq_stage_copy_signal.argtypes = [vp, vp, ctypes.c_size_t, vp, vp, vp]


EXPORTS = [
    "rdq_version",
    "rdq_last_error",
    "rdq_dequant_packed",
    "rdq_gemv_scratch_size",
    "rdq_gemv_mixed",
    "rdq_gemv_tiled_bytes",
    "rdq_gemv_repack",
    "rdq_gemv_tiled",
    "rdq_gemv_tiled_noalloc",
    "rdq_gemv_tiled_peer",
    "rdq_gemv_tiled_xop",
    "rdq_gemv_tiled_stages_x",
    "rdq_peer_gather",
    "rdq_gemv_tiled_status",
    "rdq_gemv_tiled_noalloc_status",
    "rdq_gemm_status",
    "rdq_gemm_test_timeout",
    "rdq_gemm_mixed",
    "rdq_gemm_mixed_ws",
    "rdq_gemm_workspace_size",
    "rdq_quantize_nvfp4",
    "rdq_quantize_fp8",
    "rdq_quantize_layer",
    "rdq_quantize_status",
    "rdq_linear",
    "rdq_linear_words",
    "rdq_linear_uses_words",
    "rdq_linear_workspace_size",
    "rdq_stage_copy",
    "rdq_stage_copy_signal",
    "rdq_add_rmsnorm",
    "rdq_qk_rope_cache",
    "rdq_attn_decode_scratch_size",
    "rdq_attn_decode",
    "rdq_rope_attn_decode_scratch_size",
    "rdq_rope_attn_decode",
    "rdq_silu_mul",
]


def available() -> bool:
    return os.path.exists(LIB_PATH) and os.path.exists(TORCH_EXT_PATH)


def lib() -> ctypes.CDLL:
    """Return the loaded library; raise ``RuntimeError`` if it has not been built."""
    global _lib
    if _lib is not None:
        return _lib
    with _lock:
        if _lib is None:
            if not os.path.exists(LIB_PATH):
                raise RuntimeError(
                    f"{LIB_PATH} is missing: the CUDA kernels are not built. "
                    "Run `python -c 'import __graft_entry__ as g; g.build()'` or rdquant_b200._lib.build()."
                )
            handle = ctypes.CDLL(LIB_PATH)
            _bind(handle)
            _lib = handle
    return _lib


_torch_ext = None


def torch_ext():
    """The native host path (module ``_rdq_torch``); raise ``RuntimeError`` if it has not been built."""
    global _torch_ext
    if _torch_ext is None:
        lib()
        with _lock:
            if _torch_ext is None:
                if not os.path.exists(TORCH_EXT_PATH):
                    raise RuntimeError(f"{TORCH_EXT_PATH} is missing: run rdquant_b200._lib.build()")
                loader = importlib.machinery.ExtensionFileLoader("_rdq_torch", TORCH_EXT_PATH)
                spec = importlib.util.spec_from_file_location("_rdq_torch", TORCH_EXT_PATH, loader=loader)
                module = importlib.util.module_from_spec(spec)
                loader.exec_module(module)
                _torch_ext = module
    return _torch_ext


def check(rc: int, what: str) -> None:
    if rc != 0:
        msg = lib().rdq_last_error().decode("utf-8", "replace")
        raise RuntimeError(f"{what} failed (code {rc}): {msg}")
