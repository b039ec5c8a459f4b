// Helpers shared by the translation units of libptwm_b200.so: error string,
// CUDA error macro, device guard and the per-device persistent state.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/ptwm_b200.h"
#include "kernels.cuh"

namespace ptwm {

// Last error of the calling thread (returned by ptwm_b200_last_error).
std::string& last_error_ref();
inline int64_t fail(int64_t rc, const std::string& m) { last_error_ref() = m; return rc; }

#define CUDA_TRY(expr)                                                                                        \
    do {                                                                                                      \
        cudaError_t e_ = (expr);                                                                              \
        if (e_ != cudaSuccess) return ::ptwm::fail(PTWM_RC_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// Makes `dev` current for the scope and restores the previous device.
struct DeviceGuard {
    int prev = -1;
    cudaError_t err;
    explicit DeviceGuard(int dev) { err = cudaGetDevice(&prev); if (err == cudaSuccess && prev != dev) err = cudaSetDevice(dev); }
    ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};

// Device memory.  An encode's comes from the allocator the program registered (ptwm_b200_set_allocator), else from cudaMalloc: it
// takes work memory several times the size of the tensors; handed out and taken back by the driver that was 55 of the 64 ms
// of a 1.7 GB model.  The blocks belong to the stream the encode runs on, which is all an allocator that recycles memory in
// stream order has to know.  Everything else is small and asks cudaMalloc, and the program's allocator where the driver has no
// more: that one may be holding gigabytes free, the encoder's work memory among them.
struct Allocator { ptwm_b200_alloc_fn alloc = nullptr; ptwm_b200_free_fn free = nullptr; };
Allocator current_allocator();
void set_allocator(Allocator a);

struct DeviceBuf {
    void* p = nullptr;
    Allocator from;
    int device = 0;
    cudaStream_t stream = nullptr;
    DeviceBuf() = default;
    DeviceBuf(const DeviceBuf&) = delete;
    DeviceBuf& operator=(const DeviceBuf&) = delete;
    ~DeviceBuf() {
        if (!p) return;
        if (from.free) from.free(uint64_t(reinterpret_cast<uintptr_t>(p)), uint32_t(device), uint64_t(reinterpret_cast<uintptr_t>(stream)));
        else { DeviceGuard g{device}; cudaFree(p); }
    }
    template <class T> T* as() const { return static_cast<T*>(p); }
    cudaError_t alloc(size_t n, cudaStream_t st, bool registered = true) {
        stream = st;
        if (!n) n = 1;
        cudaError_t e = cudaGetDevice(&device);
        if (e != cudaSuccess) return e;
        const Allocator a = current_allocator();
        if (!registered || !a.alloc) {
            e = cudaMalloc(&p, n);
            if (e != cudaErrorMemoryAllocation || !a.alloc) return e;
            cudaGetLastError();  // answered here: not the next launch's
        }
        p = reinterpret_cast<void*>(uintptr_t(a.alloc(n, uint32_t(device), uint64_t(reinterpret_cast<uintptr_t>(st)))));
        if (!p) return cudaErrorMemoryAllocation;
        from = a;
        return cudaSuccess;
    }
};

struct DeviceState {
    cudaStream_t stream = nullptr;   // the library's process-persistent stream for the device
    CrcTables* d_tabs = nullptr;     // CRC byte table and x^(2^k) powers
    bool attrs = false;
    cudaStream_t side[4] = {nullptr, nullptr, nullptr, nullptr};  // independent decoders of one pass run side by side
    std::vector<cudaStream_t> spare; // streams of encodes that have ended (their payload hashes ran there)
    std::vector<uint32_t*> words;    // free words of pinned memory, one for every plan that has run (its status summary)
    void* stage = nullptr;           // pinned host buffer the plan work lists pass through on their way to the device
    size_t stage_cap = 0;
    std::mutex copy_mu;              // for the two below: containers on their way to host memory (copy_to_host)
    uint8_t* copy_stage = nullptr;
    cudaStream_t copy_stream = nullptr;
};

// Caller holds a DeviceGuard for `dev`.
int64_t device_state(int dev, DeviceState** out);
const CrcTables& crc_tables();

// A stream that nobody else uses until it is given back, idle by then.
int64_t take_stream(DeviceState& ds, cudaStream_t* s);
void give_stream(DeviceState& ds, cudaStream_t s);

// Device bytes into ordinary host memory; what writes them has completed.
int64_t copy_to_host(uint8_t* dst, const uint8_t* src, size_t n, DeviceState& ds);

inline uint64_t align_up(uint64_t v, uint64_t a) { return (v + a - 1) / a * a; }

// One plane into one payload on the device (encoder.cu); body of ptwm_plane_codec_v1_encode_cuda.
int64_t encode_plane_cuda(int codec, const uint8_t* state, size_t state_len, uint8_t state_version, uint64_t in_dev, size_t n, uint64_t out_dev, size_t out_cap,
                          uint64_t* needed, cudaStream_t st);

}  // namespace ptwm
