"""The order of programmatic launches, read from the kernels' sources: a kernel waits for the launch before
it and only then lets the next one start, unless it keeps the shape that bounds how many launches an SM
has places for (the rule at pdl_wait() in rdq_common.cuh)."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "rdquant_b200", "csrc")
# one CTA per SM with the shared memory of a place, in every launch
ALWAYS_ONE_PER_SM = {"stage_copy_kernel", "peer_gather_kernel"}
# launched in stream order: nothing to wait for
STREAM_ORDER = {"decode_rows_kernel", "encode_layer_kernel"}


def _kernels():
    """(name, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.inl"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", text):
            start = text.index("{", m.end())
            name = re.findall(r"(\w+)\s*\(", text[m.end():start])
            depth, i = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            yield next(n for n in name if n.endswith("_kernel")), text[start:i]


def test_kernels_wait_before_they_let_the_next_launch_start():
    seen = set()
    for name, body in _kernels():
        if "pdl_launch_dependents()" not in body:
            continue
        seen.add(name)
        wait = body.find("pdl_wait()")
        if name in STREAM_ORDER:
            assert wait < 0, name
            continue
        assert wait >= 0, name
        for m in re.finditer(r"([^\n]*)pdl_launch_dependents\(\)", body):
            early = m.start() < wait
            assert not early or name in ALWAYS_ONE_PER_SM or "if (first)" in m.group(1), name
    assert {"gemv_tiled_kernel", "gemm_stream_kernel", "gemm_pair_kernel", "gemv_rows_kernel", "rope_attn_kernel"} <= seen


def _function(path, name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, path)).read())
    start = text.index("{", re.search(r"__device__ __forceinline__ \w+ " + name + r"\(", text).end())
    depth, i = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[start:i]


def test_bounded_waits_are_for_the_launch_s_own_work():
    """What waits with a limit may be waiting for the launch before, however long that takes: the limit counts
    from the end of that launch on."""
    for path, name in (("rdq_gemm_common.cuh", "gemm_wait"), ("rdq_common.cuh", "mbar_wait_launch")):
        assert re.search(r"for \(.*pdl_wait\(\)", _function(path, name), re.S), name
    bodies = dict(_kernels())
    # the streaming GEMM: the MMA warp, whose waits are an asm block, needs the activations first
    mma = bodies["gemm_stream_kernel"].split("else if (warp == 2) {")[1].split("else if (warp == 3) {")[0]
    assert 0 <= mma.find("\n    pdl_wait();") < mma.index("wait_bounded(")
    assert not re.search(r"\bmbar_(try|wait)\w*\((?!smem_u32\(&S\.never\))", bodies["gemm_stream_kernel"])
    # the tiled GEMV: all warps but the producer begin with the barrier that stands for the launch before
    tiled = bodies["gemv_tiled_kernel"]
    producer, rest = tiled.split("if (warp > kMmaWarps) {")
    assert 0 <= producer.find("if (!a.beside) pdl_wait();") < producer.index("mbar_wait(")
    for part in rest.split("const int grp = warp / kWarpsPerGroup"):
        waits = re.findall(r"\bmbar_\w*(?:try|wait)\w*\([^,]*", part)
        assert waits[0] == "mbar_wait_launch(smem_u32(&bar_x)" and "bar_x" not in "".join(waits[1:])
    # the decoded-once GEMM waits for it with all threads, ahead of everything
    pair = bodies["gemm_pair_kernel"]
    assert 0 <= pair.find("\n  pdl_wait();") < pair.index("gemm_wait_cluster(")


def test_roles_of_the_streaming_gemm_wait_before_they_read():
    """Without leave to read weights early, each warp of gemm_stream_kernel that reads memory has waited for the
    launch before; ahead of that, addresses are only asked into L2."""
    body = dict(_kernels())["gemm_stream_kernel"]
    setup, *roles = re.split(r"(?:else )?if \(warp (?:== \d|< 8)\) \{", body[:body.index("finish_shared<")])
    roles[-1:] = roles[-1].split("} else {", 1)  # the converters
    assert len(roles) == 6
    read = re.compile(r"load_chunk\(|tma_load_2d\(|row_of\(|cp_async\d+\(|\ba\.(s4|s8|perm|bias)\b")
    waits = re.compile(r"(if \(!a\.early\) )?pdl_wait\(\)")
    reading = 0
    for role in roles:
        first = read.search(role)
        if first:
            reading += 1
            wait = waits.search(role)
            assert wait and wait.start() < first.start(), role[:80]
    assert reading == 4, "weights, activations, block scales, rows of the epilogue"
    assert re.findall(r"if \(a\.early\) (\w+)\(|else (\w+)\(", setup[setup.index("Segment g"):])[:2] == [
        ("load_chunk", ""), ("", "tma_prefetch_2d")]
