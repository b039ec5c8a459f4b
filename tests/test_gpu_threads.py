"""Calls from several threads and on several streams of one process: no call waits for another's copy, and every one gets its
own bytes and its own verdict."""
import threading
import time

import pytest
import torch

import oracle
import ptwm_b200
from ptwm_b200 import _lib
from ptwm_b200.compressor import CompressionConfig, IDENTITY, compress_model
from _data import mixed_model

pytestmark = pytest.mark.gpu


def test_plans_reach_the_device_while_a_container_is_copied_to_the_host():
    big = torch.randint(0, 256, (768 << 20,), dtype=torch.uint8, device="cuda")
    enc = compress_model({"w": big}, CompressionConfig(streaming_chunk=None, forced_codec=IDENTITY))
    enc.to_bytes()  # staging memory and threads are there
    handle = ptwm_b200.ContainerHandle(oracle.write_container(mixed_model(), chunk_size=4096), device=0)
    ptwm_b200.DecodePlan(handle).prepare(0)
    data, span = [], []

    def copy():
        span.append(time.perf_counter())
        data.append(enc.to_bytes())
        span.append(time.perf_counter())

    done = []
    t = threading.Thread(target=copy)
    t.start()
    while t.is_alive():
        began = time.perf_counter()
        ptwm_b200.DecodePlan(handle).prepare(0)
        done.append((began, time.perf_counter()))
    t.join()
    # a plan takes well under a millisecond, the copy some fifty
    assert sum(span[0] <= a and b <= span[1] for a, b in done) >= 10
    assert torch.equal(torch.frombuffer(bytearray(data[0]), dtype=torch.uint8)[-(1 << 20):], enc.to_tensor()[-(1 << 20):].cpu())
    raw = ptwm_b200.ContainerHandle(data[0], device=0).decode("w")
    assert torch.equal(raw, big)


def test_plans_reach_the_device_while_another_thread_hashes():
    # the hash of one tensor is a serial chain, here of some 100 ms
    big = torch.randint(0, 256, (256 << 20,), dtype=torch.uint8, device="cuda")
    config = CompressionConfig(streaming_chunk=None, forced_codec=IDENTITY, emit_payload_hash=True)
    compress_model({"w": big}, config)  # its memory is in the pool
    handle = ptwm_b200.ContainerHandle(oracle.write_container(mixed_model(), chunk_size=4096), device=0)
    ptwm_b200.DecodePlan(handle).prepare(0)
    torch.cuda.synchronize()
    span, blob = [], []

    def encode():
        span.append(time.perf_counter())
        blob.append(compress_model({"w": big}, config))
        span.append(time.perf_counter())

    done = []
    t = threading.Thread(target=encode)
    t.start()
    while t.is_alive():
        began = time.perf_counter()
        ptwm_b200.DecodePlan(handle).prepare(0)
        done.append((began, time.perf_counter()))
    t.join()
    assert sum(a >= span[0] + 0.3 * (span[1] - span[0]) and b <= span[1] for a, b in done) >= 3  # begun and done in the midst of the hash
    assert torch.equal(ptwm_b200.ContainerHandle(blob[0].to_tensor(), verify=True).decode("w"), big)


def test_a_plan_dropped_in_flight_does_not_answer_for_the_next_one():
    blob = oracle.write_container(mixed_model(), chunk_size=4096, forced_codec=oracle.RANS)
    handle = ptwm_b200.ContainerHandle(blob, device=0)
    handle.decode_model()  # every kernel is loaded: a load waits for the device
    resident = handle.blob_on_device()
    damaged = torch.zeros_like(resident)  # no valid header in it
    first, second = ptwm_b200.DecodePlan(handle), ptwm_b200.DecodePlan(handle)
    out, out2 = (torch.empty(first.out_bytes, dtype=torch.uint8, device="cuda") for _ in range(2))
    scratch, scratch2 = (torch.empty(max(first.scratch_bytes, 1), dtype=torch.uint8, device="cuda") for _ in range(2))
    first.prepare(0)
    memory = first._dev_mem  # of the runs, kept until they are over
    slow, fast = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    with torch.cuda.stream(slow):
        torch.cuda._sleep(1_000_000_000)  # half a second
        first.run(resident, out, scratch, flags=ptwm_b200.NO_SYNC)
    del first
    second.prepare(0)
    with torch.cuda.stream(fast):
        second.run(damaged, out2, scratch2, flags=ptwm_b200.NO_SYNC)
    slow.synchronize()
    with torch.cuda.stream(fast), pytest.raises(ptwm_b200.PtwmError):
        second.finish(0)
    del memory


def test_a_container_whose_address_was_taken_outlives_the_work_that_reads_it():
    tensors = {"w": torch.randint(0, 256, (1 << 20,), dtype=torch.uint8, device="cuda")}
    enc = compress_model(tensors, CompressionConfig(streaming_chunk=65536, forced_codec=IDENTITY))
    size = enc.size
    plan = ptwm_b200.DecodePlan(ptwm_b200.ContainerHandle(enc.to_bytes(), device=0))
    out = torch.empty(plan.out_bytes, dtype=torch.uint8, device="cuda")
    slow, L = torch.cuda.Stream(), _lib.lib()
    plan.prepare(0)
    where = L.ptwm_b200_encoded_device_ptr(enc._e)
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    with torch.cuda.stream(slow):
        torch.cuda._sleep(500_000_000)
        assert L.ptwm_b200_plan_run(plan._p, where, 0, size, out.data_ptr(), out.numel(), 0, 0, ptwm_b200.NO_SYNC, 0, slow.cuda_stream) == 0
    del enc
    recycled = [torch.full((size,), 255, dtype=torch.uint8, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    assert torch.equal(out[:1 << 20], tensors["w"])
    del recycled


@pytest.mark.parametrize("priority", [0, -1])
def test_threads_decode_plans_of_several_codecs_at_once(priority):
    specs = mixed_model(2)
    blobs = [oracle.write_container(specs, chunk_size=chunk, menu=(oracle.HUFFMAN, oracle.RANS, oracle.TANS, oracle.O1SAC)) for chunk in (501, 4096, 65536)]
    wrong, raised = [], []

    def decode(blob):
        try:
            with torch.cuda.stream(torch.cuda.Stream(priority=priority)):
                handle = ptwm_b200.ContainerHandle(blob, device=0)
                for _ in range(8):
                    wrong.extend(s.name for (name, t), s in zip(handle.decode_model(), specs) if t.contiguous().view(torch.uint8).cpu().numpy().tobytes() != s.raw)
        except Exception as e:
            raised.append(e)

    threads = [threading.Thread(target=decode, args=(blob,)) for blob in blobs + blobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not raised and not wrong
