"""Damaged payloads must end in an error code (or different bytes), never in a
fault: every decode loop is bounded by the symbol count and every read is
clamped to the resident blob.  Mirrors the reference's accepted outcomes
(tests/ptwm/core/test_decompressor_errors.py:35-77)."""
import time

import numpy as np
import pytest
import torch

import oracle
import ptwm_b200
from ptwm_b200 import _lib
from _data import spec_bf16, specs_fp8

pytestmark = pytest.mark.gpu


def _raw(t):
    return t.contiguous().view(torch.uint8).cpu().numpy().tobytes()


@pytest.mark.parametrize("codec", [oracle.HUFFMAN, oracle.RANS, oracle.TANS])
def test_mutated_payload_bytes(codec):
    specs = [spec_bf16("w", 64, 512, 3)] + specs_fp8("f", 32, 256, 4)
    blob = oracle.write_container(specs, forced_codec=codec, chunk_size=4096)
    base = ptwm_b200.ContainerHandle(blob, device=0, verify=False)
    infos = base.tensor_infos()
    rng = np.random.default_rng(5)
    outcomes = {"error": 0, "different": 0, "same": 0}
    for trial in range(40):
        t = infos[int(rng.integers(0, len(infos)))]
        pos = int(rng.integers(t["first_byte"], t["end_byte"]))
        m = bytearray(blob)
        m[pos] ^= int(rng.integers(1, 256))
        try:
            h = ptwm_b200.ContainerHandle(bytes(m), device=0, verify=False)
            got = dict(h.decode_model())
        except (ptwm_b200.PtwmError, ValueError):
            outcomes["error"] += 1
            continue
        same = all(_raw(got[s.name]) == s.raw for s in specs)
        outcomes["same" if same else "different"] += 1
    assert outcomes["error"] + outcomes["different"] > 0
    # the context is still usable afterwards
    assert _raw(dict(base.decode_model())["w"]) == specs[0].raw


def test_mutated_payload_bytes_with_a_lane_per_stream():
    # 4300 tANS chunks: the kernel with 32 chunks per block
    raw = np.minimum(np.random.default_rng(8).geometric(0.4, 1029 * 4300), 40).astype(np.uint8).tobytes()
    blob = oracle.write_container([oracle.TensorSpec("p", oracle.DT_U8, [len(raw)], raw)], forced_codec=oracle.TANS, chunk_size=1029)
    base = ptwm_b200.ContainerHandle(blob, device=0, verify=False)
    info = base.tensor_infos()[0]
    rng = np.random.default_rng(9)
    for trial in range(8):
        m = bytearray(blob)
        for pos in rng.integers(info["first_byte"] + (info["end_byte"] - info["first_byte"]) // 50, info["end_byte"], 1 << trial):
            m[pos] ^= int(rng.integers(1, 256))
        try:
            assert _raw(ptwm_b200.ContainerHandle(bytes(m), device=0, verify=False).decode("p")) != raw
        except (ptwm_b200.PtwmError, ValueError):
            pass
    assert _raw(base.decode("p")) == raw


def _decode_damaged(blob, edits):
    """The whole container's bytes out of a plan made from the sound one, and whether the run was refused; ``edits`` are (place, bytes)."""
    handle = ptwm_b200.ContainerHandle(blob, device=0, verify=False)
    plan, dev = handle.plan(None), handle.blob_on_device().clone()
    for at, raw in edits:
        dev[at:at + len(raw)] = torch.frombuffer(bytearray(raw), dtype=torch.uint8).cuda()
    out = torch.full((plan.out_bytes,), 0xCD, dtype=torch.uint8, device="cuda")
    scratch = torch.zeros(max(plan.scratch_bytes, 1), dtype=torch.uint8, device="cuda")
    plan.run(dev, out, scratch, flags=ptwm_b200.NO_SYNC)
    try:
        plan.finish(0)
        refused = False
    except ptwm_b200.PtwmError:
        refused = True
    return out.cpu().numpy(), refused


@pytest.mark.parametrize("n", [2048, 1997])
@pytest.mark.parametrize("dtype", ["u8", "bf16"])
def test_damaged_rans_chunks_among_thousands(dtype, n):
    # more chunks than the kernels with a table entry per slot take, eight to a warp, which reads tables of pairs where all eight allow it
    rng = np.random.default_rng(n)
    chunks, width = 3600, 2 if dtype == "bf16" else 1
    raw = np.minimum(rng.geometric(0.4, chunks * n), 30).astype(np.uint8) + 100
    raw[::n] = 130  # the same highest symbol everywhere
    low = rng.integers(0, 256, len(raw)).astype(np.uint16)
    full = ((low & 0x80) << 8 | raw.astype(np.uint16) << 7 | low & 0x7F).astype(np.uint16) if width == 2 else raw
    spec = oracle.TensorSpec("p", oracle.DT_BF16 if width == 2 else oracle.DT_U8, [len(raw)], full.tobytes())
    blob = oracle.write_container([spec], forced_codec=oracle.RANS, chunk_size=n)
    want = np.frombuffer(full.tobytes(), np.uint8)
    piece = lambda k: raw[k * n:(k + 1) * n].tobytes()
    payload = lambda k: oracle.plane_encode(oracle.RANS, piece(k))[2]
    header = 5 + 1 + 2 * (payload(0)[5] + 1)  # tag, length, highest symbol, frequencies; then four lengths and the streams

    def damaged(k, at, new):
        was = payload(k)
        place = blob.index(was)
        assert was[0] == 1 and was[5] == payload(0)[5]
        new = new(was[at:at + 4]) if callable(new) else new
        try:
            decoded = oracle.plane_decode(oracle.RANS, was[:at] + new + was[at + len(new):], n)
        except oracle.OracleError:
            decoded = None
        return k, (place + at, new), decoded

    flip = lambda v: bytes([v[0] ^ 0x5A])
    word = lambda f: lambda v: (f(int.from_bytes(v, "little")) & 0xFFFFFFFF).to_bytes(4, "little")
    streams = header + 16
    one = 5 + 1 + 2 * 103  # the frequency of a symbol that is there
    cases = [damaged(3, streams + 100, flip), damaged(20, streams, word(lambda x: 5)), damaged(37, streams, word(lambda x: x | 1 << 31)), damaged(60, streams, word(lambda x: x >> 8)),
             damaged(81, one, lambda v: bytes([v[0] ^ 1])), damaged(100, header, word(lambda x: x + 1)), damaged(133, 5, b"\xff"), damaged(150, 5, b"\x00"), damaged(3599, streams + 7, flip)]
    assert sum(c[2] is None for c in cases) >= 4 and cases[2][2] is not None and cases[2][2] != piece(37)
    got, refused = _decode_damaged(blob, [c[1] for c in cases])
    assert refused
    hit = {c[0] for c in cases}
    same = (got[:len(want)] == want).reshape(chunks, n * width).all(1)
    assert same[[k for k in range(chunks) if k not in hit]].all()
    # what the oracle decodes all the same is decoded alike, alone among sound chunks
    sound = [c for c in cases if c[2] is not None]
    got, refused = _decode_damaged(blob, [c[1] for c in sound])
    assert not refused
    symbols = got[:len(want)] if width == 1 else (got[:len(want)].view(np.uint16) >> 7 & 0xFF).astype(np.uint8)
    for k, _, decoded in sound:
        assert symbols[k * n:(k + 1) * n].tobytes() == decoded, k
    assert (got[:len(want)] == want).reshape(chunks, n * width).all(1).sum() == chunks - sum(c[2] != piece(c[0]) for c in sound)


def test_mutated_bytes_of_thousands_of_rans_chunks():
    raw = np.minimum(np.random.default_rng(8).geometric(0.4, 1029 * 3700), 30).astype(np.uint8).tobytes()
    blob = oracle.write_container([oracle.TensorSpec("p", oracle.DT_U8, [len(raw)], raw)], forced_codec=oracle.RANS, chunk_size=1029)
    info = ptwm_b200.ContainerHandle(blob, device=0, verify=False).tensor_infos()[0]
    rng = np.random.default_rng(9)
    for trial in range(12):
        places = rng.integers(info["first_byte"], info["end_byte"], 1 << trial)
        got, refused = _decode_damaged(blob, [(int(p), bytes([blob[p] ^ int(rng.integers(1, 256))])) for p in places])
        assert trial < 3 or refused or got[:len(raw)].tobytes() != raw
    got, refused = _decode_damaged(blob, [])
    assert not refused and got[:len(raw)].tobytes() == raw


@pytest.mark.parametrize("chunk", [0, 2, 5])
def test_damaged_order1_scale_ac_chunk_in_a_block_of_four(chunk):
    # six chunks beside another codec: two blocks, the second not full; the warps beside the one with the damaged chunk go on
    n, chunks = 4096, 6
    rng = np.random.default_rng(chunk)
    raw = ((np.cumsum(rng.random(n * chunks) < 0.05) * 7) % 3).astype(np.uint8).tobytes()
    skewed = np.minimum(rng.geometric(0.5, 3000), 9).astype(np.uint8).tobytes()
    blob = oracle.write_container([oracle.TensorSpec("s", oracle.DT_U8, [1, len(raw)], raw, usage="scale"), oracle.TensorSpec("p", oracle.DT_U8, [len(skewed)], skewed)],
                                  chunk_size=n, menu=(oracle.HUFFMAN, oracle.O1SAC))
    state, version, payload = oracle.plane_encode(oracle.O1SAC, raw[chunk * n:(chunk + 1) * n])
    place = blob.index(state + payload)
    assert version == 1
    more = bytes([state[31] | 0x80])  # a context without a row
    pair = (int.from_bytes(state[32:34], "little") + 1).to_bytes(2, "little")  # shares that do not add up
    for at, new, refuses in ((31, more, True), (32, pair, True), (len(state) + 8, bytes(20), False), (len(state), b"\xff" * len(payload), False)):
        got, refused = _decode_damaged(blob, [(place + at, new)])
        assert refused == refuses
        same = [got[k * n:(k + 1) * n].tobytes() == raw[k * n:(k + 1) * n] for k in range(chunks)]
        assert all(same[:chunk] + same[chunk + 1:]) and not same[chunk]
        assert got[-(-len(raw) // 256) * 256:][:len(skewed)].tobytes() == skewed


def test_truncated_container_is_refused():
    specs = [spec_bf16("w", 32, 256, 6)]
    blob = oracle.write_container(specs, chunk_size=2048)
    for cut in (10, len(blob) // 2, len(blob) - 1):
        with pytest.raises((ptwm_b200.PtwmError, ValueError)):
            ptwm_b200.ContainerHandle(blob[:cut], device=0)


def test_tans_stream_of_more_than_2_32_bits_for_few_symbols_is_refused():
    # as the right stream modulo 2^32 bits: its symbols at the bottom, the first state at the top, 512 MiB of nothing between them
    plane = bytes(7 if i % 9 == 0 else 200 for i in range(400))
    _, _, payload = oracle.plane_encode(oracle.TANS, plane)
    assert payload[0] == 1 and payload[5] == 11
    at = 5 + 3 + 3 * int.from_bytes(payload[6:8], "little")
    bits = int.from_bytes(payload[at:at + 8], "little")
    stream = int.from_bytes(payload[at + 8:], "little")
    state, top = stream >> (bits - 11), 2**32 + bits - 11
    src = torch.zeros(at + 8 + (2**32 + bits + 7) // 8, dtype=torch.uint8, device="cuda")
    put = lambda pos, raw: src[pos:pos + len(raw)].copy_(torch.frombuffer(bytearray(raw), dtype=torch.uint8))
    put(0, payload[:at] + (2**32 + bits).to_bytes(8, "little"))
    low = stream & ((1 << (bits - 11)) - 1)
    put(at + 8, low.to_bytes((bits + 7) // 8, "little"))
    high = (state << (top % 8)).to_bytes(3, "little")
    put(at + 8 + top // 8, high[:src.numel() - at - 8 - top // 8])
    assert _plane_decode_tans(src, len(plane)) == -8


def _plane_decode_tans(src, n):
    out = torch.zeros(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return _lib.lib().ptwm_hardware_backend_v1_dispatch_decode_cuda(0, None, 0, bytes.fromhex("e4868545e7b22282695972441494e70569ab27595d19349114e852125d96daa4"), 32,
                                                                    src.data_ptr(), src.numel(), out.data_ptr(), n, 0)


def test_tans_stream_with_far_more_symbols_than_declared_is_refused_in_the_time_of_a_few_chunks():
    # a stream of ones under this table: runs of some 56,000 symbols each that never fall in with one another; one lane walks 64 Ki
    # symbols in 3 ms at most
    n, bits = 1 << 16, 312557
    table = b"".join(bytes([sym]) + freq.to_bytes(2, "little") for sym, freq in enumerate((2039, 3, 2, 4)))
    blob = bytes([11]) + (4).to_bytes(2, "little") + table + bits.to_bytes(8, "little") + b"\xff" * ((bits + 7) // 8)
    src = torch.frombuffer(bytearray(b"\x01" + n.to_bytes(4, "little") + blob), dtype=torch.uint8).cuda()
    took = []
    for _ in range(3):
        began = time.perf_counter()
        assert _plane_decode_tans(src, n) == -8
        took.append(time.perf_counter() - began)
    assert min(took) < 0.03, took
