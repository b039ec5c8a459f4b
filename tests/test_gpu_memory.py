"""Device memory when the program's allocator holds nearly all of it: what the library allocates for itself comes from there then."""
import numpy as np
import pytest
import torch

import oracle
import ptwm_b200
from ptwm_b200 import _lib
from ptwm_b200.compressor import CompressionConfig, compress_model
from _data import mixed_model

pytestmark = pytest.mark.gpu


def test_calls_that_allocate_when_torch_holds_the_memory_free():
    L = _lib.lib()
    compress_model({"w": torch.zeros(4096, dtype=torch.bfloat16, device="cuda")}, CompressionConfig())  # registers torch's allocator
    raw = np.random.default_rng(0).integers(0, 256, 48 << 20, dtype=np.uint8)
    out = np.empty(raw.size + 64, dtype=np.uint8)
    specs = mixed_model()
    handle = ptwm_b200.ContainerHandle(oracle.write_container(specs, chunk_size=4096), device=0)
    handle.decode_model()
    assert L.ptwm_plane_codec_v1_encode(raw.ctypes.data, 1 << 16, out.ctypes.data, out.size) > 0  # kernels are loaded, streams are there
    torch.cuda.empty_cache()
    held = [torch.empty(torch.cuda.mem_get_info()[0] - (256 << 20), dtype=torch.uint8, device="cuda")]
    try:
        for _ in range(16):
            held.append(torch.empty(24 << 20, dtype=torch.uint8, device="cuda"))
    except torch.OutOfMemoryError:
        pass
    held.clear()  # free for torch, not for the driver
    try:
        assert L.ptwm_plane_codec_v1_encode(raw.ctypes.data, raw.size, out.ctypes.data, out.size) == raw.size + 1, _lib.last_error()
        assert out[0] == 0 and np.array_equal(out[1:raw.size + 1], raw)
        plan = ptwm_b200.DecodePlan(handle)
        tensors = torch.empty(plan.out_bytes, dtype=torch.uint8, device="cuda")
        scratch = torch.empty(max(plan.scratch_bytes, 1), dtype=torch.uint8, device="cuda")
        plan.run(handle.blob_on_device(), tensors, scratch)
        for k, s in enumerate(specs):
            a = plan.out_offsets[k]
            assert tensors[a:a + len(s.raw)].cpu().numpy().tobytes() == s.raw, s.name
    finally:
        torch.cuda.empty_cache()
