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
