// gpe_internal.h — shared host/device helpers of the engine (not part of the C ABI).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <string>

#include "../../include/gpe.h"

namespace gpe {

// ----- error plumbing (thread-local, like the reference's last_error in cuda-render.cu:20-27) -----
void set_error(int32_t status, const char* fmt, ...);
void set_cuda_error(cudaError_t e, const char* what);
void clear_error();

#define GPE_TRY_CUDA(expr)                                                                                 \
    do {                                                                                                   \
        cudaError_t e_ = (expr);                                                                           \
        if (e_ != cudaSuccess) {                                                                           \
            ::gpe::set_cuda_error(e_, #expr);                                                              \
            return GPE_ERR_CUDA;                                                                           \
        }                                                                                                  \
    } while (0)

#define GPE_CHECK_LAUNCH(name)                                                                             \
    do {                                                                                                   \
        cudaError_t e_ = cudaGetLastError();                                                               \
        if (e_ != cudaSuccess) {                                                                           \
            ::gpe::set_cuda_error(e_, name);                                                               \
            return GPE_ERR_CUDA;                                                                           \
        }                                                                                                  \
    } while (0)

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) & ~(a - 1); }

// Bump allocator over one device allocation (the reference carves each arena out of one cudaMalloc at
// 128 B alignment, cuda-engine.cpp:14-29; 256 B here so every array can be a TMA or vector base).
struct Carver {
    size_t off = 0;
    template <class T>
    size_t take(size_t count)
    {
        const size_t o = off;
        off            = align_up(off + sizeof(T) * (count ? count : 1), 256);
        return o;
    }
};

// Where a kernel goes: its stream, and whether its launch may overlap the end of the kernel before it there.
struct Place {
    cudaStream_t st;
    bool follows;
};

// The launches of a graph that the engine captures itself, on one stream: every kernel but the first (or one behind a
// memset) may be launched while the one before it ends. What a caller captures, or launches stage by stage, keeps full
// dependencies.
struct Sequence {
    bool own    = false; // the engine's own capture is running
    bool behind = false; // a kernel precedes
    void begin()
    {
        own    = true;
        behind = false;
    }
    void end() { own = false; }
    void cut() { behind = false; }
    Place at(cudaStream_t st)
    {
        const Place p = {st, own && behind};
        behind        = true;
        return p;
    }
};

// Whether a caller (or the engine itself) is capturing st.
bool capturing(cudaStream_t st);
// For a kernel right behind another of the same call on st: full dependencies where a caller is capturing.
Place behind(cudaStream_t st);

#if defined(__CUDACC__)
// First statement of every kernel that may be launched so: the rest of it waits until the kernel before it is complete
// and its writes are visible, so that only the launch overlaps and no pass sees another order. Short passes gain most:
// one step of 16,384 atoms with its state in and out 51.2 -> 47.1 us, 20 substeps of them 675 -> 616, 16 MLS-MPM steps
// of 65,536 particles 126 -> 115, a published and drawn frame of 1M 40.3 -> 32.9, a step of 1M 307.6 -> 304.4. The
// kernel before gives no earlier signal than its blocks' ends: with one at its start the waiting blocks took the room of those still to
// come (1M particles 304 -> 317 us a step, 256 batched scenes 1353 -> 1405).
__device__ __forceinline__ void follow() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t launch(const Place& at, dim3 grid, unsigned block, void (*kernel)(P...), const A&... args)
{
    cudaLaunchAttribute attr{};
    attr.id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim  = grid;
    c.blockDim = dim3(block);
    c.stream   = at.st;
    c.attrs    = &attr;
    c.numAttrs = at.follows ? 1u : 0u;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
#endif

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

int32_t current_device(int* dev);
int32_t sm_count();
// Whether a kernel on the current device may read or write the caller's array at p: device (or managed) memory of this
// device, aligned to `align` bytes. What fails this (another device's memory, an odd offset into an array) goes through
// cudaMemcpyAsync, which takes any. Null arrays pass.
bool kernel_can_use(const void* p, size_t align);

// ----- counting sort of 32-bit keys (shared by PBF and the MPM spatial sort) -----
// Workspace sizes for a sort of up to n_max items into n_keys buckets.
size_t scan_blocks(uint32_t n_keys);
constexpr int SCAN_TILE = 2048; // cells of one tile of the scan
// count[n_keys] -> start[n_keys+1] exclusive scan; zeroes count (and zero_bytes[n_keys] when given). bsum
// needs scan_blocks(n_keys) entries; with have_sums it holds the tiles' totals on entry.
int32_t launch_exclusive_scan(uint32_t* count, uint32_t n_keys, uint32_t* bsum, uint32_t* start,
                              Place at, uint8_t* zero_bytes = nullptr, bool have_sums = false);
// kernel launches of launch_exclusive_scan for n_keys buckets
int32_t scan_launches(uint32_t n_keys, bool have_sums = false);
// bucket[start[key] + rank] = i for every (key, rank) pair. n sizes the launch; with n_dev the kernel takes
// the live count from the device (which must not exceed n).
int32_t launch_scatter(const uint2* keyrank, int64_t n, const uint32_t* start, uint32_t* bucket, uint32_t ncells,
                       Place at, const int32_t* n_dev = nullptr);


// ----- warm-start network (mlp.cu) as the PBF engine sees it -----
struct MlpDev;
// Pair set of a network: features [cap][12] and targets [cap]; idx = the particle's sorted index when the
// pair was taken; cnt[0] = pairs written (appended with atomics), cnt[1] = pairs whose target is written.
struct MlpData {
    float* X;
    float* T;
    int32_t* idx;
    int32_t* cnt;
    int64_t cap;
};
const MlpDev* mlp_device(const gpe_mlp* m);
MlpData mlp_data(gpe_mlp* m);
// iterations per step of the plain solve whose pairs the network learned (20 unless collected otherwise)
int32_t mlp_pair_iters(const gpe_mlp* m);
void mlp_set_pair_iters(gpe_mlp* m, int32_t iters);

#if defined(__CUDACC__)
// Packed FP32 pairs (sm_100 and later): two IEEE round-to-nearest operations in one instruction, with the
// same results as the scalar forms component by component.
__device__ __forceinline__ float2 sub2(const float2 a, const float2 b)
{
    float2 d;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "sub.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 fma2(const float2 a, const float2 b, const float2 c)
{
    float2 d;
    asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

__device__ __forceinline__ float2 add2(const float2 a, const float2 b)
{
    float2 d;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "add.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 mul2(const float2 a, const float2 b)
{
    float2 d;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "mul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
#endif

} // namespace gpe
