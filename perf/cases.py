"""What this framework is asked to do in use, as measurable cases.

A mixed-precision layer (NVFP4 / FP8 / FP16 output channels) serves three situations: decoding,
where a few activation rows meet every weight once and latency and bytes count; prompts, where
hundreds to thousands of rows make it a matrix product; and quantisation, where a weight is encoded
and decoded.  Layers are Qwen3-4B- and Llama-3-70B-shaped, weights ~ N(0, 0.02) with 1 % of the
output channels scaled by 8, activations ~ N(0, 1), channels assigned to the formats at random.

Kinds of cases
  linear   one layer called as a module (``FusedMixedLinear``) or as the functional operator
           (``mixed_precision_linear``), outside a CUDA graph
  block    the linears of one decoder block called as modules, one after another, outside a graph:
           seven projections as a loaded checkpoint has them, or four with siblings fused
  hoststep one decode step over a block whose activations live in pinned host memory
           (``GraphedDecodeStep``)
  decode   decoder blocks with the framework's glue kernels, one token per sequence, as one CUDA
           graph that is replayed per token
  recode   a weight encoded to packed tensors and decoded back (what a quantisation run does per
           layer to know its error)
"""
import torch

from rdquant_b200 import _lib, rdquant_cuda
from rdquant_b200.fused_gemv_pack import fuse_layers, packed_weight_bytes
from rdquant_b200.inference import FusedMixedLinear, GraphedDecodeStep
from rdquant_b200.ops import mixed_precision_linear
from rdquant_b200.quantize import quantize_weight, quantize_weight_packed

# the shapes of one Qwen3-4B decoder block
_QWEN3_4B = {"hidden": 2560, "ffn": 9728, "q_heads": 32, "kv_heads": 8, "head_dim": 128, "fp4": 0.67, "fp16": 0.01}
_GRAPH_BLOCKS = 4  # decoder blocks per graph: 300 MB of weights at the shapes above, more than L2


def listed():
    """The listed cases, from the smallest calls to the largest."""
    return [
        # the smallest call of a decode step: one k or v projection, one token
        {"name": "k_proj, 1 row", "kind": "linear", "call": "module", "k": 2560, "n": 1024, "m": 1, "fp4": 0.67, "fp16": 0.01,
         "dtype": "float16", "bias": False},
        # quantised model evaluated through the functional operator; this K and this many channels have no
        # tiled layout (no multiple of 64 divides it evenly, and the groups are not whole tiles)
        {"name": "odd layer, 5 rows", "kind": "linear", "call": "functional", "k": 4112, "n": 3001, "m": 5, "fp4": 0.67,
         "fp16": 0.01, "dtype": "float16", "bias": True},
        # one token through the projections of a block of a loaded bfloat16 checkpoint, without a graph
        dict(_QWEN3_4B, name="block modules, 1 row", kind="block", m=1, fused=False, dtype="bfloat16"),
        # a caller that holds its activations on the host
        dict(_QWEN3_4B, name="host-to-host step, 1 row", kind="hoststep", m=1),
        # greedy decoding after a 512-token prompt, one sequence and two batch sizes
        dict(_QWEN3_4B, name="decode, batch 1", kind="decode", batch=1, context=512),
        dict(_QWEN3_4B, name="decode, batch 8", kind="decode", batch=8, context=600),
        dict(_QWEN3_4B, name="decode, batch 32", kind="decode", batch=32, context=700),
        # widest layer of a 70B decoder, fused gate + up, at the largest batch of the decode kernel
        {"name": "70B gate+up, 16 rows", "kind": "linear", "call": "module", "k": 8192, "n": 57344, "m": 16, "fp4": 0.85,
         "fp16": 0.0, "dtype": "float16", "bias": False},
        # quantisation of one layer
        {"name": "recode gate_proj", "kind": "recode", "k": 2560, "n": 9728, "fp4": 0.67, "fp16": 0.01},
        # a prompt of 512 tokens through the linears of a block
        dict(_QWEN3_4B, name="prompt of 512, block", kind="block", m=512, fused=True, dtype="float16"),
        # a prompt of no round length through one biased projection of a bfloat16 model
        {"name": "prompt of 1237, q_proj", "kind": "linear", "call": "module", "k": 2560, "n": 4096, "m": 1237, "fp4": 0.67,
         "fp16": 0.01, "dtype": "bfloat16", "bias": True},
        # a long prompt (or a batch of prompts) through the linears of a block
        dict(_QWEN3_4B, name="prompt of 8192, block", kind="block", m=8192, fused=True, dtype="float16"),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _mult(v, unit, least=1):
    return max(least * unit, int(round(v / unit)) * unit)


def _rows(rng, most):
    """Rows of a call: a decode batch or a prompt length, spread over the logarithm of their range."""
    return max(1, min(int(most), int(_log(rng, 1, 9000))))


def _formats(rng):
    return {"fp4": round(rng.uniform(0.5, 0.9), 3), "fp16": rng.choice([0.01, 0.01, 0.0])}


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["linear", "linear", "linear", "block", "block", "decode", "decode", "hoststep", "recode"])
    case = {"kind": kind, **_formats(rng)}
    if kind == "linear":
        odd = rng.random() < 0.2  # a shape without a tiled layout
        k = _mult(_log(rng, 1024, 16384), 16 if odd else 128)
        n = int(_log(rng, 512, 16000)) if odd else _mult(_log(rng, 512, 57344), 128, 4)
        n = min(n, 32_000_000 // k if odd else _mult(480_000_000 // k, 128))
        flops = 2.0 * k * n
        # layers of such shapes are small ones: decode batches and short prompts
        m = _rows(rng, min(200 if odd else 8192, 1.6e12 / flops))
        functional = k * n <= 16_000_000 and rng.random() < 0.4
        case.update(call="functional" if functional else "module", k=k, n=n, m=m, dtype=rng.choice(["float16", "bfloat16"]),
                    bias=rng.random() < 0.3)
        return case
    if kind == "recode":
        k = _mult(_log(rng, 1024, 16384), 16)
        case.update(k=k, n=min(int(_log(rng, 512, 20000)), 60_000_000 // k))
        return case
    head_dim = rng.choice([64, 128, 128])
    kv_heads = rng.choice([2, 4, 8])
    hidden = _mult(rng.uniform(1024, 4096), 128)
    case.update(hidden=hidden, ffn=_mult(hidden * rng.uniform(2.5, 4.0), 128), q_heads=kv_heads * rng.choice([2, 4, 8]),
                kv_heads=kv_heads, head_dim=head_dim)
    if kind == "block":
        per_row = sum(2.0 * k * n for _, k, n in _members(case))
        case.update(m=_rows(rng, min(8192, 1.6e12 / per_row)), fused=rng.random() < 0.5, dtype=rng.choice(["float16", "bfloat16"]))
    elif kind == "hoststep":
        case.update(m=rng.choice([1, 1, 2, 3, 4, 8]))
    else:
        case.update(batch=max(1, int(_log(rng, 1, 65))), context=int(_log(rng, 64, 2000)))
    return case


# ---- shapes

def _members(case):
    """(name, in features, out features) of the seven linears of a block."""
    h, f, d = case["hidden"], case["ffn"], case["head_dim"]
    q, kv = case["q_heads"] * d, case["kv_heads"] * d
    return [("q", h, q), ("k", h, kv), ("v", h, kv), ("o", q, h), ("gate", h, f), ("up", h, f), ("down", f, h)]


_FUSED = (("q", "k", "v"), ("o",), ("gate", "up"), ("down",))


def _splits(n, case):
    """Channels per format: whole groups of 128, at least one FP16 group where the format is used."""
    n16 = 128 if case["fp16"] > 0 and n >= 512 else 0
    n4 = min(int(round(case["fp4"] * n / 128)) * 128, n - n16)
    return {"NVFP4": n4, "FP8": n - n4 - n16, "FP16": n16}


# ---- inputs

def _weight(k, n, gen):
    w = torch.randn(n, k, generator=gen, device="cuda") * 0.02
    w[torch.randperm(n, generator=gen, device="cuda")[: n // 100]] *= 8
    return w.half()


def _permutation(n, splits, gen):
    """Channels assigned to the formats at random, in their original order inside a format."""
    shuffled = torch.randperm(n, generator=gen, device="cuda")
    cuts = [splits["NVFP4"], splits["FP8"], splits["FP16"]]
    return torch.cat([part.sort().values for part in shuffled.split(cuts)])


def _packed(k, n, case, gen, bias=None):
    splits = _splits(n, case)
    return quantize_weight_packed(_weight(k, n, gen), _permutation(n, splits, gen), splits, bias=bias), splits


def _block_modules(case, gen, fused):
    packed = {name: (_packed(k, n, case, gen), k) for name, k, n in _members(case)}
    mods = {}
    for names in (_FUSED if fused else tuple((name,) for name in packed)):
        parts = [packed[name][0] for name in names]
        data, splits = fuse_layers(parts) if len(parts) > 1 else parts[0]
        mods["_".join(names)] = FusedMixedLinear.from_layer_data(data, splits, packed[names[0]][1], "cuda")
    return mods


def _activations(m, k, dtype, gen):
    return torch.randn(m, k, generator=gen, device="cuda").to(getattr(torch, dtype))


@torch.no_grad()
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        k, n = case["k"], case["n"]
        bias = (torch.randn(n, generator=gen, device="cuda") * 0.1).half() if case["bias"] else None
        state = {"x": _activations(case["m"], k, case["dtype"], gen)}
        if case["call"] == "functional":
            splits = _splits(n, case)
            state["qw"] = quantize_weight(_weight(k, n, gen).float(), _permutation(n, splits, gen), splits)
            state["bias"] = bias
            mixed_precision_linear(state["x"][:1], state["qw"].qtensors, state["qw"].splits, state["qw"].inv_permutation, bias)
        else:
            data, splits = _packed(k, n, case, gen, bias)
            state["mod"] = FusedMixedLinear.from_layer_data(data, splits, k, "cuda")
    elif kind == "block":
        mods = list(_block_modules(case, gen, case["fused"]).values())
        state = {"mods": mods, "x": [_activations(case["m"], mod.K, case["dtype"], gen) for mod in mods]}
    elif kind == "hoststep":
        step = GraphedDecodeStep(_block_modules(case, gen, True).values(), m=case["m"])
        for buf in step.x_host:
            buf.copy_(torch.randn(buf.shape, generator=gen, device="cuda"))
        state = {"step": step}
    elif kind == "decode":
        state = _prepare_decode(case, gen)
    else:
        k, n = case["k"], case["n"]
        splits = _splits(n, case)
        state = {"w": _weight(k, n, gen), "perm": _permutation(n, splits, gen), "splits": splits, "k": k}
    state["kind"] = kind
    return state


def _prepare_decode(case, gen):
    b, h, f, dh = case["batch"], case["hidden"], case["ffn"], case["head_dim"]
    nq, nkv, pos = case["q_heads"], case["kv_heads"], case["context"]
    rows = pos + 64  # cache rows allocated: the prompt and room for the tokens to come
    f16 = {"dtype": torch.float16, "device": "cuda"}
    freq = 1.0 / (1.0e6 ** (torch.arange(0, dh, 2, device="cuda").float() / dh))
    angle = torch.arange(rows, device="cuda").float()[:, None] * freq[None, :]
    st = {
        "x": torch.randn(b, h, generator=gen, device="cuda").half(),
        "pos": torch.tensor([pos], dtype=torch.long, device="cuda"),
        "cos": torch.cat([angle.cos(), angle.cos()], -1).half(), "sin": torch.cat([angle.sin(), angle.sin()], -1).half(),
        "scratch": rdquant_cuda.rope_attn_scratch(b, nq, nkv, dh, rows, "cuda"),
        "res": [torch.zeros(b, h, **f16) for _ in range(2)], "hid": torch.zeros(b, h, **f16),
        "att": torch.zeros(b, nq * dh, **f16), "act": torch.zeros(b, f, **f16), "blocks": [],
    }

    def norm_weight(size):
        return (1 + 0.1 * torch.randn(size, generator=gen, device="cuda")).half()

    for _ in range(_GRAPH_BLOCKS):
        mods = _block_modules(case, gen, True)
        for mod in mods.values():
            mod.use_pdl = True
        st["blocks"].append({
            "qkv": mods["q_k_v"], "o": mods["o"], "gate_up": mods["gate_up"], "down": mods["down"],
            "ln1": norm_weight(h), "ln2": norm_weight(h), "qn": norm_weight(dh), "kn": norm_weight(dh),
            "k": torch.randn(b, nkv, rows, dh, generator=gen, device="cuda", dtype=torch.float16),
            "v": torch.randn(b, nkv, rows, dh, generator=gen, device="cuda", dtype=torch.float16) * 0.5,
        })
    st["norm"] = norm_weight(h)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        _decode_step(st, case)  # set-up of the library outside the capture
        stream.synchronize()
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"], stream=stream):
            _decode_step(st, case)
    torch.cuda.current_stream().wait_stream(stream)
    return st


def _decode_step(st, case):
    """One token per sequence through the blocks: the order of calls of the framework's own decoder."""
    rc, eps, flags = rdquant_cuda, 1.0e-6, _lib.RDQ_GEMV_PDL
    b, h, f, dh, nq = case["batch"], case["hidden"], case["ffn"], case["head_dim"], case["q_heads"]
    decode_rows = b <= rc.MAX_GEMV_M
    in_gemv_norm = decode_rows and rc.gemv_stages_x(b, h)
    in_gemv_silu = decode_rows and rc.gemv_stages_x(b, f)
    cur, other = st["res"]
    cur.copy_(st["x"])
    delta = None

    def norm_linear(mod, w):
        nonlocal cur, other
        if in_gemv_norm:
            y = rc.mixed_gemv_norm(cur, delta, w, eps, mod._fd(), residual_out=other, flags=flags)
            cur, other = other, cur
            return y
        rc.add_rmsnorm(cur, delta, w, st["hid"], eps, flags)
        return mod(st["hid"])

    for blk in st["blocks"]:
        qkv = norm_linear(blk["qkv"], blk["ln1"])
        rc.rope_attn_decode(qkv, blk["qn"], blk["kn"], st["cos"], st["sin"], st["pos"], blk["k"], blk["v"], st["scratch"],
                            st["att"], nq, dh ** -0.5, eps, flags)
        delta = blk["o"](st["att"])
        gu = norm_linear(blk["gate_up"], blk["ln2"])
        if in_gemv_silu:
            delta = rc.mixed_gemv_silu(gu, blk["down"]._fd(), flags=flags)
        else:
            rc.silu_mul(gu, st["act"], flags)
            delta = blk["down"](st["act"])
    rc.add_rmsnorm(cur, delta, st["norm"], st["hid"], eps, flags)
    st["out"] = {"hidden": st["hid"], "residual": cur, "k": [blk["k"] for blk in st["blocks"]], "v": [blk["v"] for blk in st["blocks"]]}


# ---- one pass

@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "linear":
        if "mod" in state:
            return state["mod"](state["x"])
        qw = state["qw"]
        return mixed_precision_linear(state["x"], qw.qtensors, qw.splits, qw.inv_permutation, state["bias"])
    if kind == "block":
        return [mod(x) for mod, x in zip(state["mods"], state["x"])]
    if kind == "hoststep":
        return state["step"].run()
    if kind == "decode":
        state["graph"].replay()
        return state["out"]
    data = quantize_weight_packed(state["w"], state["perm"], state["splits"])
    back = rdquant_cuda.dequantize_packed(data, state["splits"], state["k"], inv_perm=data["inv_permutation"])
    return {"back": back, **{key: data[key] for key in sorted(data) if data[key].is_cuda}}


# ---- what a pass cannot do without

def _linear_work(k, n, m, case, act_bytes=2):
    return packed_weight_bytes(_splits(n, case), k) + 4 * n + act_bytes * m * (k + n), 2.0 * m * n * k


def work(case):
    kind = case["kind"]
    if kind == "linear":
        nbytes, flops = _linear_work(case["k"], case["n"], case["m"], case)
    elif kind == "recode":
        k, n = case["k"], case["n"]
        # weight in, packed tensors and index out, packed tensors are then read and the decoded weight written
        nbytes, flops = 2 * n * k + 2 * packed_weight_bytes(_splits(n, case), k) + 2 * n * k + 12 * n, 2.0 * n * k
    else:
        m = case.get("m") or case["batch"]
        parts = [_linear_work(k, n, m, case) for _, k, n in _members(case)]
        nbytes, flops = sum(p[0] for p in parts), sum(p[1] for p in parts)
        if kind == "decode":
            kv = 2 * m * case["kv_heads"] * (case["context"] + 1) * case["head_dim"]
            nbytes = _GRAPH_BLOCKS * (nbytes + 2 * kv)
            flops = _GRAPH_BLOCKS * (flops + 4.0 * m * case["q_heads"] * (case["context"] + 1) * case["head_dim"])
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """float16 outputs of FP32 sums differ by a rounding where the sums' order does (2^-11 of a
    value, so well below 1e-3 over all); bfloat16 outputs by 2^-8 of a value; four decoder blocks
    carry float16 roundings of a dozen stages.  Encoded bytes and decoded weights are exact."""
    if case["kind"] == "recode":
        return "exact"
    if case["kind"] == "decode":
        return {"rel": 1e-2, "max": 0.1}
    return {"rel": 5e-3, "max": 2e-2} if case.get("dtype") == "bfloat16" else {"rel": 1e-3, "max": 5e-3}
