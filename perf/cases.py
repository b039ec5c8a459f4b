"""Performance cases: the calls a program that stores or loads model weights with this package makes.

Every case is a dict of plain values.  ``op`` names the call:

* ``plane_decode`` / ``plane_encode``: one plane payload through the native-extension ABI
  (``ptwm_hardware_backend_v1_dispatch_decode_cuda``, ``ptwm_plane_codec_v1_encode_cuda``), which is how the reference's
  own loader drives the library: chunk by chunk, synchronously, device memory to device memory.
* ``tensor``: one tensor of a container that is already open (``ContainerHandle.decode``, what ``TensorIndex.get_tensor``
  and ``SafeOpen.get_tensor`` call); the compressed bytes are resident on the GPU.
* ``model``: every tensor of an open container in one pass (``ContainerHandle.decode_model``).
* ``load``: a container in pinned host memory to tensors on the GPU: open, parse, copy, plan, decode
  (``ContainerHandle(..., prefetch=True).decode_model_streamed()``).
* ``encode``: CUDA tensors to a container (``compress_model``), fetched as a CUDA tensor, or as host bytes (``to_host``)
  the way ``save_sharded`` does, and put into the program's own buffer.

Weights are synthetic, with the value distributions of trained layers: normal with one sigma (bf16) or with a sigma per
row (the other types), norm vectors close to one, FP8 with a scale per row, MXFP4 and NVFP4 with their block scales.
Shapes are those of the Llama-3-8B layers the package is benchmarked on, smaller models of the same proportions, and
ragged sizes.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import ptwm_b200
from ptwm_b200 import _lib
from ptwm_b200.compressor import HUFFMAN, IDENTITY, RANS, TANS, CompressionConfig, compress_model

_FORCED = {"menu": None, "identity": IDENTITY, "huffman": HUFFMAN, "rans": RANS, "tans": TANS}
_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
# 32-byte canonical ids of the built-in codecs, as the native-extension ABI takes them
_CODEC_IDS = {
    "huffman": bytes.fromhex("614155b5a8c9efb689219bcca3cbf7855e29d3023208ce61cca7a36849248e33"),
    "rans": bytes.fromhex("39c875ef9793a9c5ebe199116debac4c9d5388b8b7cf2fe6b575845f0ca1624e"),
    "tans": bytes.fromhex("e4868545e7b22282695972441494e70569ab27595d19349114e852125d96daa4"),
}
# Compressed share of the raw bytes, for work(): the entropy coders take an exponent plane (a third of its bytes) and leave
# the mantissa planes raw, so it hardly depends on codec or size.
_RATIO = {"bf16": 0.67, "fp16": 0.86, "fp32": 0.83, "fp8": 0.83, "mx": 0.97}


def _model(name, op, weights, codec, chunk, *, d=4096, kv=1024, ffn=14336, layers=1, vocab=0, crc=False, hash=False, **more):
    return dict(name=name, op=op, weights=weights, codec=codec, chunk=chunk, d=d, kv=kv, ffn=ffn, layers=layers, vocab=vocab, crc=crc, hash=hash, **more)


def listed():
    return [
        # The reference's loader decoding one stored chunk of an exponent plane: the smallest unit of work, all latency.
        dict(name="plane_decode_64k_rans", op="plane_decode", codec="rans", n=65536),
        # The same loader's writer handing over one plane, longer than a chunk and of odd length.
        dict(name="plane_encode_200k_huffman", op="plane_encode", codec="huffman", n=200_003),
        # Lazy access by name: a norm vector out of an open model, where launches and host work are all there is.
        dict(name="tensor_norm_4096", op="tensor", weights="bf16", codec="menu", chunk=65536, rows=0, cols=4096, crc=False, hash=False),
        # Lazy access by name: one attention projection, written with the default options (64 KiB chunks, codec by size).
        dict(name="tensor_4096x4096_menu", op="tensor", weights="bf16", codec="menu", chunk=65536, rows=4096, cols=4096, crc=False, hash=False),
        # A large bf16 model in device memory, the recipe of the decode benchmark: six layers with embeddings, 4.7 GB.
        _model("model_bf16_rans", "model", "bf16", "rans", 32768, layers=6, vocab=128256),
        # A model of ragged dimensions written with the default options.
        _model("model_bf16_menu_ragged", "model", "bf16", "menu", 65536, d=3003, kv=751, ffn=10501, layers=2, vocab=5003),
        # A fp32 checkpoint, Huffman coded, whose plane CRCs and payload hashes are written and checked on the way in.
        _model("model_fp32_huffman_verified", "model", "fp32", "huffman", 32768, d=2048, kv=512, ffn=7168, layers=2, vocab=0, crc=True, hash=True),
        # FP8 weights with row scales, default options.
        _model("model_fp8_menu", "model", "fp8", "menu", 65536, layers=1),
        # A microscaling layer set: MXFP4 and NVFP4 weights with their block scales, which are arithmetic coded.
        _model("model_mx_menu", "model", "mx", "menu", 32768, d=4096, kv=1024, ffn=14336, layers=1),
        # A whole load of a two-layer bf16 model from pinned host memory, with plane CRCs checked.
        _model("load_bf16_rans", "load", "bf16", "rans", 32768, layers=2, crc=True),
        # Writing a bf16 model, the benchmark's recipe.
        _model("encode_bf16_rans", "encode", "bf16", "rans", 32768, layers=4, to_host=False),
        # Writing a small fp16 model of ragged dimensions with the default options and every check, to host bytes.
        _model("encode_fp16_menu_ragged", "encode", "fp16", "menu", 65536, d=765, kv=191, ffn=2677, layers=2, vocab=1001, crc=True, hash=True, to_host=True),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi], odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("plane_decode", "plane_encode", "tensor", "tensor", "model", "model", "model", "load", "encode", "encode"))
    if op.startswith("plane"):
        return dict(op=op, codec=rng.choice(("rans", "huffman", "tans")), n=_log_int(rng, 1000, 600_000))
    chunk = rng.choice((32768, 65536, 65536, _log_int(rng, 8192, 524288)))
    codec = rng.choice(("menu", "menu", "rans", "huffman", "tans", "identity"))
    crc, hash_ = rng.random() < 0.4, rng.random() < 0.25
    if op == "tensor":
        if rng.random() < 0.1:  # an unchunked plane (chunk 0): a handful of serial streams, so small
            return dict(op=op, weights=rng.choice(("bf16", "fp16", "fp32")), codec=codec, chunk=0, rows=_log_int(rng, 8, 600), cols=_log_int(rng, 8, 600), crc=crc, hash=hash_)
        return dict(op=op, weights=rng.choice(("bf16", "bf16", "fp16", "fp32")), codec=codec, chunk=chunk, rows=rng.choice((0, _log_int(rng, 64, 8192))),
                    cols=_log_int(rng, 64, 8192), crc=crc, hash=hash_)
    weights = rng.choice(("bf16", "bf16", "bf16", "fp16", "fp32", "fp8", "mx"))
    d = _log_int(rng, 200, 4096)
    if weights == "mx":
        d = max(256, d // 64 * 64)  # whole scale blocks
    case = dict(op=op, weights=weights, codec=codec if weights != "mx" else "menu", chunk=chunk, d=d, kv=max(64, d // 4 // 64 * 64), ffn=max(256, int(d * rng.uniform(2.5, 3.6)) // 64 * 64),
                layers=rng.randint(1, 3), vocab=rng.choice((0, _log_int(rng, 500, 30000))), crc=crc, hash=hash_)
    if op == "encode":
        case["to_host"] = rng.random() < 0.3
    return case


# ---- inputs -----------------------------------------------------------------------------------------
def _weights(rows, cols, g, per_row):
    w = torch.randn(rows, cols, generator=g, device="cuda")
    if not per_row:
        return w.mul_(0.02)
    lo, hi = math.log(0.005), math.log(0.05)
    return w.mul_(torch.exp(torch.rand(rows, 1, generator=g, device="cuda") * (hi - lo) + lo))


def _norm(n, g):
    return 1 + 0.01 * torch.randn(n, generator=g, device="cuda")


def _fp4(x):
    """E2M1 codes of x (nearest of 0, 0.5, 1, 1.5, 2, 3, 4, 6), two to a byte."""
    edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=x.device)
    c = torch.bucketize(x.abs(), edges).to(torch.uint8) | ((x < 0).to(torch.uint8) << 3)
    return c[..., 0::2] | (c[..., 1::2] << 4)


def _shapes(case):
    """(name, rows, cols) of the matrices of a model, and the length of its norm vectors."""
    d, kv, ffn, out = case["d"], case["kv"], case["ffn"], []
    for i in range(case["layers"]):
        out += [(f"l{i}.{n}", r, c) for n, r, c in (("q", d, d), ("k", kv, d), ("v", kv, d), ("o", d, d), ("gate", ffn, d), ("up", ffn, d), ("down", d, ffn))]
    return out


def _model_tensors(case, g):
    tensors, usage, weights = {}, {}, case["weights"]
    vocab, d = case["vocab"], case["d"]
    dt = _DTYPES.get(weights, torch.bfloat16)
    if vocab:
        tensors["embed"] = _weights(vocab, d, g, False).to(dt)
    for name, rows, cols in _shapes(case):
        if weights == "mx" and not (name.endswith("gate") or name.endswith("up") or name.endswith("down")):
            tensors[name] = _weights(rows, cols, g, False).to(torch.bfloat16)  # attention stays bf16 in such models
            continue
        w = _weights(rows, cols, g, weights != "bf16")
        if weights == "fp8":
            scale = w.abs().amax(1, keepdim=True) / 448.0
            tensors[name] = (w / scale).to(torch.float8_e4m3fn)
            tensors[name + "_scale"] = scale.reshape(-1)
        elif weights == "mx" and name.endswith("down"):  # MXFP4: E8M0 scales per 32
            b = w.reshape(rows, cols // 32, 32)
            e = (127 + torch.ceil(torch.log2(b.abs().amax(-1).clamp_min(1e-30) / 6.0))).clamp(0, 254)
            tensors[name] = _fp4((b / torch.exp2(e - 127).unsqueeze(-1)).reshape(rows, cols))
            tensors[name + "_scale"] = e.to(torch.uint8)
            usage[name], usage[name + "_scale"] = "fp4", "scale"
        elif weights == "mx":  # NVFP4: E4M3 scales per 16 and one fp32 scale
            top = w.abs().amax() / (448.0 * 6.0)
            b = w.reshape(rows, cols // 16, 16)
            s8 = (b.abs().amax(-1) / 6.0 / top).to(torch.float8_e4m3fn)
            s = s8.float() * top
            tensors[name] = _fp4((b / torch.where(s == 0, torch.ones_like(s), s).unsqueeze(-1)).reshape(rows, cols))
            tensors[name + "_scale"], tensors[name + "_scale_2"] = s8, top.reshape(1)
            usage[name], usage[name + "_scale"], usage[name + "_scale_2"] = "fp4", "scale", "global_scale"
        else:
            tensors[name] = w.to(dt)
    for i in range(case["layers"]):
        for n in ("attn_norm", "ffn_norm"):
            tensors[f"l{i}.{n}"] = _norm(d, g).to(dt)
    if vocab:
        tensors["norm"] = _norm(d, g).to(dt)
        tensors["lm_head"] = _weights(vocab, d, g, False).to(dt)
    return tensors, usage


def _config(case):
    return CompressionConfig(streaming_chunk=case["chunk"] or None, forced_codec=_FORCED[case["codec"]], emit_plane_crc=case["crc"], emit_payload_hash=case["hash"])


def _exponent_plane(n, g):
    """n bytes of the exponent plane of normal bf16 weights."""
    w = (torch.randn(n, generator=g, device="cuda") * 0.02).to(torch.bfloat16).view(torch.int16)
    return ((w >> 7) & 0xFF).to(torch.uint8)


def _encode_plane(state):
    device = state["in"].device.index or 0
    n = _lib.lib().ptwm_plane_codec_v1_encode_cuda(0, None, 0, state["codec"], 32, state["in"].data_ptr(), state["in"].numel(), state["out"].data_ptr(),
                                                   state["out"].numel(), ctypes.byref(state["needed"]), device)
    if n < 0:
        raise RuntimeError(_lib.last_error())
    return n


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    op = case["op"]
    if op.startswith("plane"):
        plane = _exponent_plane(case["n"], g)
        state = {"op": "plane_encode", "codec": _CODEC_IDS[case["codec"]], "in": plane, "out": torch.zeros(case["n"] + 16, dtype=torch.uint8, device="cuda"),
                 "needed": ctypes.c_uint64()}
        if op == "plane_encode":
            torch.cuda.synchronize()  # the library reads the plane on a stream of its own
            return state
        torch.cuda.synchronize()
        size = _encode_plane(state)
        return {"op": op, "codec": state["codec"], "in": state["out"][:size].clone(), "out": torch.zeros_like(plane)}
    if op == "tensor":
        dt = _DTYPES[case["weights"]]
        rows, cols = case["rows"], case["cols"]
        tensors = {"before": _weights(67, 129, g, False).to(dt), "w": _norm(cols, g).to(dt) if not rows else _weights(rows, cols, g, case["weights"] != "bf16").to(dt),
                   "after": _norm(1000, g).to(dt)}
        usage = {}
    else:
        tensors, usage = _model_tensors(case, g)
    if op == "encode":
        # the buffer the container goes to (a file's mapping, a staging buffer): no coder makes a plane longer than raw, give or take its records
        cap = sum(t.numel() * t.element_size() for t in tensors.values()) * 33 // 32 + (1 << 20)
        out = np.zeros(cap, dtype=np.uint8) if case["to_host"] else torch.zeros(cap, dtype=torch.uint8, device="cuda")
        return {"op": op, "tensors": tensors, "usage": usage, "config": _config(case), "to_host": case["to_host"], "out": out}
    blob = compress_model(tensors, _config(case), usage=usage).to_tensor()
    if op == "load":
        host = torch.empty(blob.numel(), dtype=torch.uint8, pin_memory=True)
        host.copy_(blob)
        return {"op": op, "host": host}
    return {"op": op, "handle": ptwm_b200.ContainerHandle(blob)}


# ---- one pass ---------------------------------------------------------------------------------------
def _plain(t):
    """Sub-byte and 8-bit floating tensors as their bytes, which can be compared everywhere."""
    return t if t.dtype in (torch.bfloat16, torch.float16, torch.float32, torch.uint8) else t.view(torch.uint8)


def run(state):
    op = state["op"]
    if op == "plane_decode":
        device = state["in"].device.index or 0
        n = _lib.lib().ptwm_hardware_backend_v1_dispatch_decode_cuda(0, None, 0, state["codec"], 32, state["in"].data_ptr(), state["in"].numel(), state["out"].data_ptr(),
                                                                     state["out"].numel(), device)
        if n < 0:
            raise RuntimeError(_lib.last_error())
        return state["out"]
    if op == "plane_encode":
        return [_encode_plane(state), state["out"]]
    if op == "tensor":
        return _plain(state["handle"].decode("w"))
    if op == "model":
        return [_plain(t) for _, t in state["handle"].decode_model()]
    if op == "load":
        return [_plain(t) for _, t in ptwm_b200.ContainerHandle(state["host"], prefetch=True).decode_model_streamed()]
    enc = compress_model(state["tensors"], state["config"], usage=state["usage"])
    state["out"][:enc.size] = np.frombuffer(enc.to_bytes(), dtype=np.uint8) if state["to_host"] else enc.to_tensor()
    return [enc.size, state["out"]]


# ---- what a pass cannot do without --------------------------------------------------------------------
def _raw_bytes(case):
    eb = {"bf16": 2, "fp16": 2, "fp32": 4, "fp8": 1}
    if case["op"] == "tensor":
        return max(case["rows"], 1) * case["cols"] * eb[case["weights"]]
    d, vocab, w = case["d"], case["vocab"], case["weights"]
    total = 2 * vocab * d * eb.get(w, 2) if w in ("bf16", "fp16", "fp32") else 2 * vocab * d * 2
    for name, rows, cols in _shapes(case):
        if w != "mx":
            total += rows * cols * eb[w] + (4 * rows if w == "fp8" else 0)
        elif name.endswith("down"):
            total += rows * cols // 2 + rows * cols // 32
        elif name.endswith("gate") or name.endswith("up"):
            total += rows * cols // 2 + rows * cols // 16
        else:
            total += rows * cols * 2
    return total


def work(case):
    """Bytes of one pass: the compressed form once and the decoded form once, whichever is read and whichever written.  The
    coders do integer work on bytes; no floating-point operations."""
    if case["op"].startswith("plane"):
        return {"bytes": case["n"] * 1.33, "flops": 0}
    ratio = 1.0 if case["codec"] == "identity" else _RATIO[case["weights"]]
    return {"bytes": _raw_bytes(case) * (1 + ratio), "flops": 0}


def tolerance(case):
    """A lossless format: decoded tensors and written containers are the same bytes whoever makes them."""
    return "exact"
