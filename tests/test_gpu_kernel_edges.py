"""The decoders and encoders at the sizes where their work splits: remainders of lanes, warps, runs and blocks, launches on
either side of a choice of kernel, and planes that leave the usual alphabet.  Everything is exact: decoded bytes against the
source, written containers against the oracle's."""
import time

import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import oracle
import ptwm_b200
from ptwm_b200 import _lib
from ptwm_b200.compressor import CompressionConfig, HUFFMAN, IDENTITY, RANS, TANS, compress_model
from _data import mixed_model, weights
from test_gpu_decode import IDS

pytestmark = pytest.mark.gpu


def plane(kind: str, n: int, seed: int = 0) -> bytes:
    rng = np.random.default_rng((n, seed))
    if kind == "exponent":
        w = weights(1, n, seed + n, False).to(torch.bfloat16).view(torch.int16).numpy().reshape(-1)
        return ((w.astype(np.uint16) >> 7) & 0xFF).astype(np.uint8).tobytes()
    if kind == "rare":  # one symbol with nearly all of the table
        return np.where(rng.random(n) < 1 / 3000, 7, 200).astype(np.uint8).tobytes()
    if kind == "nibble":
        return rng.integers(0, 16, n, dtype=np.uint8).tobytes()
    return np.minimum(rng.geometric(0.03, n), 255).astype(np.uint8).tobytes()  # "wide": an alphabet of 200 and more


def check(specs, **kw):
    blob = oracle.write_container(specs, **kw)
    got = ptwm_b200.ContainerHandle(blob, device=0, verify=True).decode_model()
    for (name, t), s in zip(got, specs):
        assert t.contiguous().view(torch.uint8).cpu().numpy().tobytes() == s.raw, name


def u8(name, raw, cols=None):
    return oracle.TensorSpec(name, oracle.DT_U8, [len(raw)] if cols is None else [len(raw) // cols, cols], raw, usage="standard" if cols is None else "scale")


@pytest.mark.parametrize("kind", ["exponent", "rare", "nibble", "wide"])
@pytest.mark.parametrize("codec", [HUFFMAN, RANS, TANS])
def test_decode_chunk_lengths(kind, codec):
    # lanes with nothing to do, groups of eight and their remainders, runs of 256 symbols: 1, 31, 32, 127, 128 and more than that
    lengths = (1, 2, 3, 5, 31, 33, 63, 64, 65, 255, 256, 257, 511, 513, 1029, 8191, 8193, 127 * 256 + 9, 128 * 256, 128 * 256 + 1, 70001)
    check([u8(f"p{n}", plane(kind, n)) for n in lengths], chunk_size=1 << 20, forced_codec=codec, emit_crc=True)


@pytest.mark.parametrize("codec,chunks", [(RANS, 1), (RANS, 591), (RANS, 592), (RANS, 593), (RANS, 595), (RANS, 3552), (RANS, 3553),
                                          (TANS, 295), (TANS, 296), (TANS, 297), (HUFFMAN, 593)])
@pytest.mark.parametrize("dtype", ["u8", "bf16", "fp32"])
def test_decode_launch_sizes(codec, chunks, dtype):
    n = 67 * (chunks - 1) + 5  # a last chunk of five
    if dtype == "u8":
        specs = [u8("p", plane("exponent", n))]
    else:
        t = weights(1, n, chunks, False).to(torch.bfloat16 if dtype == "bf16" else torch.float32)
        specs = [oracle.TensorSpec("p", oracle.DT_BF16 if dtype == "bf16" else oracle.DT_F32, [n], t.view(torch.uint8).numpy().tobytes())]
    check(specs, chunk_size=67, forced_codec=codec)


@pytest.mark.parametrize("n", [200_000, 233_000, 300_000, 600_001])
@pytest.mark.parametrize("chunks", [1, 149, 445])
def test_rans_decode_streams_in_shared_memory(n, chunks):
    # streams that fit beside the table of a block, of two and of four blocks to an SM, and streams that go through the rings
    n //= {1: 1, 149: 3, 445: 8}[chunks]
    raw = plane("wide", n)
    low = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8).astype(np.uint16)
    wide = ((low & 0x80) << 8 | np.frombuffer(raw, np.uint8).astype(np.uint16) << 7 | low & 0x7F).astype(np.uint16)
    check([u8("p", raw)] + [u8(f"q{k}", plane("wide", 100, k)) for k in range(chunks - 1)], chunk_size=1 << 20, forced_codec=RANS)
    check([oracle.TensorSpec("p", oracle.DT_BF16, [n], wide.tobytes())], chunk_size=1 << 20, forced_codec=RANS, emit_crc=True)


def launched(call):
    """The kernels that `call` launches, by name."""
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
        call()
        torch.cuda.synchronize()
    names = [e.key for e in p.key_averages() if "_kernel" in e.key]
    if not names:
        pytest.skip("no kernels seen: the profiler has no access to the device here")
    return names


@pytest.mark.parametrize("n, chunks, kernel", [(1499, 1, 3), (1499, 592, 3), (1500, 1, 2), (1500, 592, 2), (1499, 593, 4), (50_000, 592, 1)])
def test_rans_decode_kernel_of_a_small_launch(n, chunks, kernel):
    # short chunks: the table that is quickly built; then the one that is quickly read, with streams in shared memory where four blocks' fit
    raw = plane("nibble", n * chunks)
    blob = oracle.write_container([u8("p", raw)], chunk_size=n, forced_codec=RANS)
    handle = ptwm_b200.ContainerHandle(blob, device=0)
    assert any(f"rans_decode_kernel_t<false, {kernel}>" in k for k in launched(lambda: handle.decode("p")))
    assert handle.decode("p").cpu().numpy().tobytes() == raw


@pytest.mark.parametrize("codec, others, chunks, kernel", [(TANS, 100, 592, 1), (TANS, 592, 340, 2), (TANS, 592, 341, 1), (TANS, 592, 444, 1), (TANS, 592, 445, 4), (TANS, 592, 593, 4),
                                                           (HUFFMAN, 8000, 340, 2), (HUFFMAN, 8000, 341, 1), (HUFFMAN, 8000, 445, 4), (HUFFMAN, 19_000, 296, 2), (HUFFMAN, 19_000, 297, 4)])
def test_rans_decode_kernel_beside_other_codecs(codec, others, chunks, kernel):
    # a launch that would take most of an SM's shared memory takes less of it where other decoders want theirs
    g, n = torch.Generator(device="cuda").manual_seed(chunks), 2048
    skewed = (torch.rand(n * chunks, generator=g, device="cuda").clamp_min(1e-9).log() / -0.18).to(torch.int32).remainder(32).to(torch.uint8)
    rest = (torch.randn(n * others, generator=g, device="cuda") * 0.02).bfloat16() if codec == TANS else torch.randint(0, 16, (n * others,), generator=g, device="cuda", dtype=torch.uint8)
    enc = compress_model({"p": skewed, "q": rest}, CompressionConfig(streaming_chunk=n, codec_menu=(IDENTITY, RANS, codec)))
    assert enc.plane_codecs["p"] == [RANS] and enc.plane_codecs["q"][-1] == codec
    handle = ptwm_b200.ContainerHandle(enc.to_tensor())
    assert any(f"rans_decode_kernel_t<false, {kernel}>" in k for k in launched(handle.decode_model))
    got = dict(handle.decode_model())
    assert torch.equal(got["p"], skewed) and torch.equal(got["q"].view(torch.uint8), rest.view(torch.uint8))


def counted(counts, rng, cluster=0):
    """2048 symbols with exactly these counts, which are then the table's frequencies; the last `cluster` symbols put side by side."""
    syms = np.repeat(np.arange(100, 100 + len(counts)), counts)
    rng.shuffle(syms)
    if cluster:
        rare = np.flatnonzero(syms >= 100 + len(counts) - cluster)
        rest = np.delete(syms, rare)
        syms = np.concatenate([rest[:700], syms[rare], rest[700:]])
    return syms.astype(np.uint8)


@pytest.mark.parametrize("mix", ["fit", "mixed"])
@pytest.mark.parametrize("dtype", ["u8", "bf16", "fp8"])
def test_rans_decode_tables_of_pairs(dtype, mix):
    # first slots of symbols on either side of where the parts of the table meet (64, 2032) and of 32 slots, one and two symbols, the longest
    # list, rare symbols side by side (more than eight bytes to eight symbols); "mixed": eight chunks of which some have three symbols to 32 slots
    rng = np.random.default_rng(5)
    fit = [[1024, 1024], [1, 2047], [2047, 1], [63, 1969, 16], [64, 1968, 16], [65, 1966, 17], [64, 31, 1, 1952], [64, 32, 1, 1951], [1] * 35 + [30, 1967, 16],
           [64, 1967] + [1] * 17, [32, 32, 31, 1, 31, 1, 32, 32, 1856], [2] * 32 + [1952, 8, 8, 8, 8], [4, 8, 16, 36, 70, 140, 300, 500, 700, 270, 3, 1]]
    other = [[2048], [100, 5, 5, 1938], [70, 1, 1, 1976], [1000, 2, 2, 2, 1042], [2000, 20, 2, 2, 24], [54] * 36 + [104]]
    chunks = []
    for k in range(3600):
        pick = other if mix == "mixed" and rng.random() < 0.05 else fit
        counts = pick[rng.integers(len(pick))]
        chunks.append(counted(counts, rng, 24 if len(counts) == 19 else 0))
    raw = np.concatenate(chunks)[:-300]
    if dtype == "u8":
        spec = u8("p", raw.tobytes())
    elif dtype == "bf16":
        low = rng.integers(0, 256, len(raw)).astype(np.uint16)
        spec = oracle.TensorSpec("p", oracle.DT_BF16, [len(raw)], ((low & 0x80) << 8 | raw.astype(np.uint16) << 7 | low & 0x7F).astype(np.uint16).tobytes())
    else:
        spec = oracle.TensorSpec("p", oracle.DT_E4M3, [len(raw)], (raw * 37 & 0xFF).astype(np.uint8).tobytes())
    check([spec], chunk_size=2048, forced_codec=RANS)


@pytest.mark.parametrize("alphabet", [2, 31, 33, 64, 256])
@pytest.mark.parametrize("cols", [1, 5, 8, 9, 37, 0])
def test_order1_scale_ac_shares_and_rows(alphabet, cols):
    # more than 32 symbols after one another leave the shares that are searched first; rows end inside and between groups of eight
    rng = np.random.default_rng(alphabet)
    specs = []
    for k, n in enumerate((37 * 8, 37 * 80, 37 * 400)):
        raw = ((np.cumsum(rng.integers(0, 2, n)) * 7 + rng.integers(0, alphabet, n)) % alphabet).astype(np.uint8).tobytes()
        raw = raw[:n // cols * cols] if cols else raw
        specs.append(u8(f"s{k}", raw, cols or None))
    check(specs, chunk_size=None if cols else 1500, forced_codec=oracle.O1SAC)


@pytest.mark.parametrize("alphabet, chunks", [(3, 1), (3, 3), (3, 4), (3, 5), (3, 296), (3, 297), (200, 296)])
def test_order1_scale_ac_beside_other_codecs(alphabet, chunks):
    # four chunks to a block that has an SM to itself, a last block that is not full, one chunk too many for that, and tables too large for four
    rng = np.random.default_rng(alphabet + chunks)
    n = 30000 * (chunks - 1) + 27001
    raw = ((np.cumsum(rng.random(n) < 0.05) * 7) % alphabet).astype(np.uint8).tobytes()  # runs: only the symbol before predicts them
    specs, menu = [u8("s", raw, n), u8("p", plane("exponent", 3000))], (oracle.HUFFMAN, oracle.O1SAC)
    assert oracle.write_container(specs[:1], chunk_size=30000, menu=menu) == oracle.write_container(specs[:1], chunk_size=30000, forced_codec=oracle.O1SAC)
    check(specs, chunk_size=30000, menu=menu, emit_crc=True)
    names = launched(ptwm_b200.ContainerHandle(oracle.write_container(specs, chunk_size=30000, menu=menu), device=0).decode_model)
    alone = alphabet == 3 and chunks <= 296  # the others wait a moment for that only then
    assert any("head_start" in k for k in names) == alone and any(f"o1sac_decode_kernel<{4 if alone else 1}>" in k for k in names)


@pytest.mark.parametrize("dtype, n, chunks, lanes", [("fp16", 12, 2368, 32), ("fp16", 12, 2371, 32), ("fp16", 12, 2372, 64), ("fp16", 12, 3552, 64), ("fp16", 12, 3553, 32),
                                                     ("fp16", 12, 4737, 32), ("fp16", 12, 4799, 32), ("fp16", 12, 4800, 64), ("fp16", 64, 2900, 64), ("fp16", 64, 3100, 32), ("fp8", 20, 2371, 32),
                                                     ("fp8", 20, 2372, 64), ("fp8", 20, 4737, 64), ("bytes", 16, 3000, 32), ("bytes", 24, 2399, 32), ("bytes", 24, 2400, 64)])
def test_tans_decode_lanes_where_both_take_as_many_rounds(dtype, n, chunks, lanes):
    g, n = torch.Generator(device="cuda").manual_seed(chunks), 1024 * n
    w = torch.randn(n * chunks, generator=g, device="cuda")
    t = (w * 0.02).half() if dtype == "fp16" else (w * 40).to(torch.float8_e4m3fn) if dtype == "fp8" else (w * 20).round().clamp(-127, 127).to(torch.int8).view(torch.uint8)
    handle = ptwm_b200.ContainerHandle(compress_model({"t": t}, CompressionConfig(streaming_chunk=n, forced_codec=TANS)).to_tensor())
    names = launched(lambda: handle.decode("t"))  # (the first of two coded planes of fp8 takes 64 whatever the second does)
    assert {k for k in (32, 64) if any(f"tans_decode_kernel<{k}>" in name for name in names)} == ({lanes, 64} if dtype == "fp8" else {lanes})
    assert torch.equal(handle.decode("t").view(torch.uint8), t.view(torch.uint8))


@pytest.mark.parametrize("chunks", [1, 31, 33, 4735, 4736, 4737])
@pytest.mark.parametrize("dtype", ["u8", "bf16", "fp32", "fp8"])
def test_tans_decode_with_a_lane_per_stream(dtype, chunks):
    # chunks of 1029 symbols: from some 4000 on they go to the kernel with 32 chunks per block, and one more than fills the GPU goes back
    n = 1029 * (chunks - 1) + 7 if chunks > 4000 else 1029 * 4200 + 1029 * (chunks - 1) + 515  # a last chunk of 7, or blocks with 1, 31 and 1 chunks
    if dtype == "u8":
        specs = [u8("p", plane("exponent", n))]
    elif dtype == "fp8":
        t = weights(1, n, chunks, False).mul(40).to(torch.float8_e4m3fn)
        specs = [oracle.TensorSpec("p", oracle.DT_E4M3, [n], t.view(torch.uint8).numpy().tobytes())]
    else:
        t = weights(1, n, chunks, False).to(torch.bfloat16 if dtype == "bf16" else torch.float32)
        specs = [oracle.TensorSpec("p", oracle.DT_BF16 if dtype == "bf16" else oracle.DT_F32, [n], t.view(torch.uint8).numpy().tobytes())]
    check(specs, chunk_size=1029, forced_codec=TANS)


@pytest.mark.parametrize("dtype", ["u8", "bf16", "fp32", "fp8"])
@pytest.mark.parametrize("chunk, chunks", [(63, 3), (255, 3), (257, 3), (513, 600), (2999, 3), (3000, 297), (4097, 149), (16385, 2), (70001, 2), (3001, 889), (8193, 889), (3001, 1777)])
def test_tans_decode_with_many_lanes_per_chunk(dtype, chunk, chunks):
    # every number of lanes, with runs that fill them, fewer runs than lanes and a single one, odd lengths, and a short last chunk
    n = chunk * chunks - chunk // 3
    specs = [u8("p", plane("exponent", n))]
    if dtype == "fp8":
        t = weights(1, n, chunks, False).mul(40).to(torch.float8_e4m3fn)
        specs = [oracle.TensorSpec("p", oracle.DT_E4M3, [n], t.view(torch.uint8).numpy().tobytes())]
    elif dtype != "u8":
        t = weights(1, n, chunks, False).to(torch.bfloat16 if dtype == "bf16" else torch.float32)
        specs = [oracle.TensorSpec("p", oracle.DT_BF16 if dtype == "bf16" else oracle.DT_F32, [n], t.view(torch.uint8).numpy().tobytes())]
    check(specs, chunk_size=chunk, forced_codec=TANS)


@pytest.mark.parametrize("dtype", ["u8", "bf16", "fp32", "fp8"])
@pytest.mark.parametrize("chunk, chunks", [(2047, 600), (2999, 2369), (3999, 889), (4000, 889), (5499, 1777), (5500, 1777), (10239, 889), (10240, 889), (10240, 1777)])
def test_tans_decode_runs_of_a_chunk(dtype, chunk, chunks):
    # on either side of where a chunk gets fewer runs than lanes, with one round of blocks and one chunk more
    test_tans_decode_with_many_lanes_per_chunk(dtype, chunk, chunks)


@pytest.mark.parametrize("chunks", [1, 400, 1200])
def test_tans_decode_of_uneven_streams(chunks):
    # nearly all of the symbols in a small part of the bits: walks that meet late or never, and paths that are followed by one lane alone
    rng = np.random.default_rng(chunks)
    specs = []
    for k, n in enumerate((3500, 20000, 65536) if chunks == 1 else (3500,)):
        zeros = np.zeros(n * chunks, dtype=np.uint8)
        half = zeros.copy(); half[::2 * n] = 1
        for at in range(0, n * chunks, n): half[at + n // 2:at + n // 2 + n // 4] = rng.integers(0, 200, n // 4)
        rare = (rng.random(n * chunks) < 0.001).astype(np.uint8)
        period = np.resize(np.array([0, 0, 1, 0, 2], dtype=np.uint8), n * chunks)
        specs += [u8(f"half{k}", half.tobytes()), u8(f"rare{k}", rare.tobytes()), u8(f"period{k}", period.tobytes())]
    check(specs, chunk_size=len(specs[-1].raw) // chunks if chunks > 1 else None, forced_codec=TANS)


def uneven(kind: str, n: int, rng) -> np.ndarray:
    """A chunk whose rarer symbols lie together or far apart: a walk that starts wrong meets more symbols than the chunk holds."""
    p = np.zeros(n, dtype=np.uint8)
    k = max(2, int(n * rng.uniform(0.002, 0.05)))
    if kind == "sparse":
        return (rng.random(n) < rng.uniform(0.005, 0.05)).astype(np.uint8)
    if kind == "front":  # followed by two symbols in turn
        p[:k], p[k + 1::2] = rng.integers(1, 6, k), 250
    else:  # exponents of normal weights, or bytes of any value, at both ends
        e = rng.normal(0, 0.02, 2 * k).astype(np.float32).view(np.uint32) >> 23 & 0xFF if kind == "ends" else rng.integers(1, 256, 2 * k)
        p[:k], p[n - k:] = e[:k], e[k:]
    return p


@pytest.mark.parametrize("kind", ["sparse", "front", "ends", "noise"])
@pytest.mark.parametrize("chunk, chunks", [(1225, 1), (2000, 400), (2000, 1800), (3000, 120), (3000, 400), (4096, 200), (9000, 1000), (16384, 100), (70001, 4)])
def test_tans_decode_where_wrong_starts_meet_more_symbols(kind, chunk, chunks):
    rng = np.random.default_rng(chunk + chunks)
    raw = np.concatenate([uneven(kind, chunk, rng) for _ in range(chunks)])
    wide = raw.astype(np.uint16) << 7  # bf16 with these exponents
    check([u8("p", raw.tobytes())], chunk_size=chunk, forced_codec=TANS)
    check([oracle.TensorSpec("p", oracle.DT_BF16, [len(raw)], wide.tobytes())], chunk_size=chunk, forced_codec=TANS)


def test_decode_of_mostly_zero_weights():
    # nonzero at both ends of a vector, or in the first and last row of a matrix: tANS has the smallest payload
    specs = []
    for k in range(40):
        v, m = torch.zeros(4096), torch.zeros(64 << k % 2, 64 << k % 2)
        v[:20], v[-20:] = weights(1, 20, k, False), weights(1, 20, k + 99, False)
        m[0], m[-1] = weights(1, m.shape[1], k, False), weights(1, m.shape[1], k + 99, False)
        for name, t in (("v", v), ("m", m)):
            specs.append(oracle.TensorSpec(f"{name}{k}", oracle.DT_BF16, list(t.shape), t.to(torch.bfloat16).view(torch.uint8).numpy().tobytes()))
    for chunk in (4096, 65536):
        check(specs, chunk_size=chunk, menu=(oracle.IDENTITY, oracle.HUFFMAN, oracle.RANS, oracle.TANS, oracle.O1SAC), emit_crc=True)
        check(specs, chunk_size=chunk, forced_codec=TANS)


def test_decode_two_coded_planes_in_many_chunks():
    # more chunks than are spread over scratch: the second plane's lanes merge with the first one, every codec on its own stream
    for menu in ((oracle.HUFFMAN, oracle.RANS, oracle.O1SAC), (oracle.TANS, oracle.O1SAC), (oracle.IDENTITY, oracle.HUFFMAN, oracle.RANS, oracle.TANS, oracle.O1SAC)):
        check(mixed_model(2), chunk_size=501, menu=menu, emit_crc=True, emit_hash=True)


@pytest.mark.parametrize("codec", [HUFFMAN, TANS, RANS])
def test_decode_small_tensors_beside_a_large_one(codec):
    # more chunks than are spread over scratch: small tensors with two and more coded planes join the launch of the large one (not with rANS)
    specs = []
    for k, n in enumerate((501 * 620 + 7, 1, 37, 500, 501, 502, 1500, 30000, 70000)):
        for name, dt, code in (("b", torch.bfloat16, oracle.DT_BF16), ("f", torch.float32, oracle.DT_F32), ("e", torch.float8_e4m3fn, oracle.DT_E4M3)):
            t = (1 + 0.01 * weights(1, n, k, False)) if dt == torch.bfloat16 else weights(1, n, k, False).mul(8)
            specs.append(oracle.TensorSpec(f"{name}{k}", code, [n], t.to(dt).view(torch.uint8).numpy().tobytes()))
    check(specs, chunk_size=501, forced_codec=codec, emit_crc=True)


@pytest.mark.parametrize("shift", [0, 1, 2, 8])
def test_payload_hash_blocks_and_alignment(shift):
    lengths = (0, 1, 31, 32, 33, 8191, 8192, 8193, 8192 + 32, 2 * 8192, 3 * 8192 + 45)
    specs, tensors = [], {}
    for n in lengths:
        raw = np.random.default_rng(n).integers(0, 256, n + shift, dtype=np.uint8)
        tensors[f"t{n}"] = torch.from_numpy(raw).cuda()[shift:]
        specs.append(u8(f"t{n}", raw[shift:].tobytes()))
    enc = compress_model(tensors, CompressionConfig(streaming_chunk=4096, forced_codec=IDENTITY, emit_payload_hash=True))
    assert enc.to_bytes() == oracle.write_container(specs, chunk_size=4096, forced_codec=IDENTITY, emit_hash=True)
    check(specs, chunk_size=4096, forced_codec=IDENTITY, emit_hash=True)


@pytest.mark.parametrize("kind", ["exponent", "rare", "nibble", "wide"])
@pytest.mark.parametrize("codec", [HUFFMAN, RANS, TANS])
def test_encode_chunk_lengths(kind, codec):
    lengths = (1, 2, 3, 4, 5, 7, 31, 32, 33, 255, 257, 511, 512, 513, 1023, 1025, 4099, 16385, 40000)
    specs = [u8(f"p{n}", plane(kind, n)) for n in lengths]
    tensors = {s.name: torch.frombuffer(bytearray(s.raw), dtype=torch.uint8).cuda() for s in specs}
    for chunk in (None, 1021):
        got = compress_model(tensors, CompressionConfig(streaming_chunk=chunk, forced_codec=codec)).to_bytes()
        assert got == oracle.write_container(specs, chunk_size=chunk, forced_codec=codec), chunk


def encode_check(planes, chunk, codec):
    specs = [u8(f"p{k}", raw) for k, raw in enumerate(planes)]
    tensors = {s.name: torch.frombuffer(bytearray(s.raw), dtype=torch.uint8).cuda() for s in specs}
    assert compress_model(tensors, CompressionConfig(streaming_chunk=chunk, forced_codec=codec)).to_bytes() == oracle.write_container(specs, chunk_size=chunk, forced_codec=codec)


@pytest.mark.parametrize("kind", ["exponent", "rare", "nibble", "wide"])
def test_huffman_encode_shares_of_a_stream(kind):
    # eight warps to a stream: shares without a round, of one, with words that two or more shares meet in; more chunks than take them
    lengths = [4 * 512 * k + d for k in (1, 7, 8, 9, 17) for d in (-5, 0, 1, 6)]
    encode_check([plane(kind, n) for n in lengths], None, HUFFMAN)
    encode_check([plane(kind, 600 * 149)], 600, HUFFMAN)


@pytest.mark.parametrize("shift", [0, 1, 8, 16])
def test_encode_split_of_a_view(shift):
    # 16-bit elements from an address that is a multiple of 2, 16 and 32 bytes: single elements, two 128-bit loads, one of 256 bits
    for n in (31, 32, 33, 5000, 70001):
        w = weights(1, n + shift, n, False).to(torch.bfloat16).reshape(-1)
        spec = oracle.TensorSpec("t", oracle.DT_BF16, [n], w[shift:].clone().view(torch.uint8).numpy().tobytes())
        got = compress_model({"t": w.cuda()[shift:]}, CompressionConfig(streaming_chunk=4096, forced_codec=RANS)).to_bytes()
        assert got == oracle.write_container([spec], chunk_size=4096, forced_codec=RANS), n


@pytest.mark.parametrize("chunks", [1, 18, 19, 37, 38, 74, 75])
@pytest.mark.parametrize("kind", ["exponent", "rare", "wide"])
def test_huffman_encode_blocks_of_a_cluster(kind, chunks):
    # eight, four, two blocks to a chunk and one: shares of all of them without a round, with one and with two, and streams of a few bits
    for length in (5, 1029, 4 * 512 * 64 + 2051, 4 * 512 * 65 + 6):
        encode_check([plane(kind, length * (chunks - 1) + length // 2 + 1)], length, HUFFMAN)


def test_huffman_encode_of_a_short_plane_takes_no_longer_than_of_a_long_one():
    # streams of one round where a cluster has 64 warps to each: 25.4 us of the kernel instead of 8.5 when every warp without a round was asked
    lib, needed, best = _lib.lib(), _lib.C.c_uint64(), {}
    for n in (1000, 20_000):
        src = torch.frombuffer(bytearray(plane("exponent", n)), dtype=torch.uint8).cuda()
        out = torch.empty(n + 16, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        for _ in range(60):
            began = time.perf_counter()
            assert 0 < lib.ptwm_plane_codec_v1_encode_cuda(1, None, 0, bytes.fromhex(IDS[HUFFMAN]), 32, src.data_ptr(), n, out.data_ptr(), n + 16, _lib.C.byref(needed), 0) < n
            best[n] = min(best.get(n, 1), time.perf_counter() - began)
    assert best[1000] < 1.1 * best[20_000], best


@pytest.mark.parametrize("codec", [HUFFMAN, RANS, TANS])
@pytest.mark.parametrize("n", [1, 16384, 16385, 70001, 600001])
def test_plane_encode_gathers_where_it_fits(codec, n):
    # several blocks put the payload together, coded or raw; a buffer one byte short stays as it is
    for raw in (plane("exponent", n), np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8).tobytes()):
        want = oracle.plane_encode(codec, raw)[2]
        src, out = torch.frombuffer(bytearray(raw), dtype=torch.uint8).cuda(), torch.full((len(want) + 32,), 0xCD, dtype=torch.uint8, device="cuda")
        needed, ident = _lib.C.c_uint64(), bytes.fromhex(IDS[codec])
        torch.cuda.synchronize()
        for cap, rc in ((len(want) - 1, -2), (len(want), len(want))):
            assert _lib.lib().ptwm_plane_codec_v1_encode_cuda(1, None, 0, ident, 32, src.data_ptr(), n, out.data_ptr(), cap, _lib.C.byref(needed), 0) == rc
            assert out.cpu().numpy().tobytes() == (b"\xcd" * (len(want) + 32) if rc < 0 else want + b"\xcd" * 32)
        assert needed.value == len(want)


@pytest.mark.parametrize("span", [1, 2, 46, 47, 48, 63, 64, 127, 128, 200])
@pytest.mark.parametrize("far", [False, True])
def test_rans_encode_rows_of_an_alphabet(span, far):
    # symbols 50 .. 50 + span - 1 on either side of a list's rows, with and without one that lies far below, which some chunks do not hold
    rng = np.random.default_rng(span)
    p = (50 + np.minimum(rng.geometric(0.08, 40000) - 1, span - 1)).astype(np.uint8)
    p[7], p[20000] = 50 + span - 1, 50
    if far: p[rng.integers(0, 20000, 3)] = 3
    encode_check([p.tobytes(), plane("exponent", 9001), plane("wide", 3000)], 1500, RANS)


def test_plan_run_in_a_captured_graph():
    specs = mixed_model()
    handle = ptwm_b200.ContainerHandle(oracle.write_container(specs, chunk_size=1000, menu=(oracle.HUFFMAN, oracle.RANS, oracle.O1SAC)), device=0)
    plan, blob = handle.plan(None), handle.blob_on_device()
    out = torch.zeros(plan.out_bytes, dtype=torch.uint8, device="cuda")
    scratch = torch.empty(max(plan.scratch_bytes, 1), dtype=torch.uint8, device="cuda")
    plan.run(blob, out, scratch)
    want = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run(blob, out, scratch, flags=ptwm_b200.NO_SYNC)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for k, s in enumerate(specs):
            a = plan.out_offsets[k]
            assert torch.equal(out[a:a + len(s.raw)], want[a:a + len(s.raw)]), s.name
