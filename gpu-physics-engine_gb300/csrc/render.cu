// render.cu — headless particle splat rasteriser: the reference's render path without D3D12
// (backgroundKernel and drawKernel, libs/render/source/cuda-render.cu:214-310, launched by launchFill
// :189-213), drawing a published view into a pitched RGBA8 device image.
//
// The reference blends every splat into the image with an unsynchronised read-modify-write per pixel
// (drawKernel, :296-307), so overlapping splats of concurrent threads can overwrite each other and the
// image depends on scheduling. Every splat has the same colour and alpha, so the sequential result depends
// only on how many splats cover a pixel: blending k times is f^k(background) with f the reference's
// alpha() (:244-258). Here a first pass counts, with one atomic per particle, the splats centred on each
// pixel; a second pass sums those counts over the footprint around each pixel (integer sums, exact) and
// shades the pixel by applying f that many times, so the image is the sequential one, bit for bit and
// independent of scheduling.
#include <cuda_runtime.h>

#include <algorithm>

#include "gpe_internal.h"

namespace gpe {
namespace {

constexpr int SPLAT_R = 2; // the 5 x 5 footprint without its corners (:293-307)
constexpr uint8_t SPLAT_R8 = 140u, SPLAT_G8 = 210u, SPLAT_B8 = 255u;
constexpr uint8_t SPLAT_A      = 100u;

// alpha(over, under) of the reference for one channel, in its operation order without contraction
__device__ __forceinline__ uint8_t blend(uint8_t over, uint8_t under, float a, float ia)
{
    const float s = __fadd_rn(__fadd_rn(__fmul_rn((float)over, a), __fmul_rn((float)under, ia)), 0.5f);
    return (uint8_t)s;
}

// Applications of f after which every channel sits at its fixed point, from any start byte: at most 11 for
// the splat colour (140, 210, 255) at alpha 100 (every start 0..255 iterated on the host); the table keeps
// 16 entries and f^k = f^15 for k >= 15.
constexpr int32_t BLEND_K = 16;
// The gradient background of a row is (255 - t, 160 - t, 80) with t = (uint8)(100 y / height) in 0..100;
// row BLEND_BLACK of the table starts from the grid lines' black.
constexpr int32_t BLEND_ROWS = 102, BLEND_BLACK = 101;

// f^k of every background, k = 0..15: the same for every frame and image size. Rebuilt by every frame's
// splat pass (identical bytes), so a frame never reads it before it exists.
__device__ uchar4 g_blend[BLEND_ROWS][BLEND_K];

__device__ __forceinline__ void build_blend_row(int32_t row)
{
    const float a  = __fmul_rn((float)SPLAT_A, 1.f / 255.f);
    const float ia = __fsub_rn(1.f, a);
    const uint8_t t = (uint8_t)min(row, 100);
    uchar4 c = row == BLEND_BLACK ? make_uchar4(0u, 0u, 0u, 255u)
                                  : make_uchar4((uint8_t)(255u - t), (uint8_t)(160u - t), 80u, 255u);
    g_blend[row][0] = c;
    for (int32_t k = 1; k < BLEND_K; ++k) {
        c.x             = blend(SPLAT_R8, c.x, a, ia);
        c.y             = blend(SPLAT_G8, c.y, a, ia);
        c.z             = blend(SPLAT_B8, c.z, a, ia);
        g_blend[row][k] = c;
    }
}

// One atomic per particle: the number of particles whose splat is centred on each pixel. Particles whose
// centre pixel lies outside the image draw nothing (the reference's early continue, :286-287). Block (0, 0)
// also writes the blend table.
__global__ void k_splat_point(const gpe_view* __restrict__ vp, gpe_view vv, int32_t* __restrict__ centres,
                              int32_t width, int32_t height, float scale)
{
    follow();
    if (blockIdx.x == 0 && blockIdx.y == 0) {
        for (int32_t row = threadIdx.x; row < BLEND_ROWS; row += blockDim.x) { build_blend_row(row); }
    }
    const gpe_view view = vp ? *vp : vv;
    const int32_t chunks = view.chunks_x * view.chunks_y;
    for (int32_t chunk = blockIdx.y; chunk < chunks; chunk += gridDim.y) {
        const int32_t n                = min(view.counts[chunk], view.chunk_capacity);
        const float2* __restrict__ pos = reinterpret_cast<const float2*>(view.pos) + (size_t)chunk * view.chunk_capacity;
        for (int32_t a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
            const float2 p   = pos[a];
            const int32_t px = (int32_t)(p.x * scale); // truncation, as (int32_t)(p.x * kSimScale) at :284
            const int32_t py = (int32_t)(p.y * scale);
            if (px < 0 || py < 0 || px >= width || py >= height) { continue; }
            atomicAdd(&centres[(size_t)py * width + px], 1);
        }
    }
}

// the centre counts start from zero (n of them; a memset between the kernels costs about 2 us more of stream time)
__global__ void __launch_bounds__(256) k_clear_centres(int32_t* __restrict__ centres, int64_t n, bool vec)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (!vec) {
        if (i < n) { centres[i] = 0; }
    } else if (4 * i + 3 < n) {
        reinterpret_cast<int4*>(centres)[i] = make_int4(0, 0, 0, 0);
    } else {
        for (int64_t q = 4 * i; q < n; ++q) { centres[q] = 0; }
    }
}

// One thread shades 4 x 4 pixels, a block of 256 threads 128 x 32.
constexpr int32_t SH_PX = 4, SH_ROWS = 4, SH_THREADS = 256;
constexpr int32_t SH_TW = 32 * SH_PX, SH_TH = SH_ROWS * SH_THREADS / 32;

// The coverage of a pixel is the sum of the centre counts over the footprint around it: rows +-2 over
// columns +-1, rows -1..1 over columns +-2 (the 21 pixels of the 5 x 5 square without its corners). A thread walks
// down the 8 rows that its 4 x 4 pixels see; each row's 8 counts (neighbouring threads share them in L1) give 3- and
// 5-wide sums, which it adds to the pixels of the up to five rows they belong to. A pixel covered k times gets
// f^k(background) with f the reference's blend: the table row of its background (the chunk grid lines' black, or the
// row's gradient value, :224-242) at min(k, 15).
// VEC: rows of counts and of the image start on 16-byte boundaries and the width is a multiple of 4, so a row's counts
// are three 16-byte loads and four pixels one store. Bound by memory: 32 MB at 2048 x 2048. A 32 x 64 tile of counts in
// shared memory, one column of 8 pixels a thread (60 shared loads and 8 four-byte stores): 13.8 us; this 9.2 (10.3 without the bound of 8
// blocks an SM, whose 1,024 blocks then take two waves).
template <bool VEC>
__global__ void __launch_bounds__(SH_THREADS, 8)
    k_shade(uint8_t* __restrict__ rgba, int64_t pitch, const int32_t* __restrict__ centres, int32_t width,
            int32_t height, int32_t line_every)
{
    follow();
    const uint32_t across = ((uint32_t)width + SH_TW - 1u) / SH_TW; // blocks a row of tiles
    const int64_t x64     = (int64_t)(blockIdx.x % across) * SH_TW + (threadIdx.x & 31u) * SH_PX;
    const int64_t y64     = (int64_t)(blockIdx.x / across) * SH_TH + (threadIdx.x >> 5) * SH_ROWS;
    if (x64 >= width || y64 >= height) { return; }
    const int32_t x = (int32_t)x64, y = (int32_t)y64;
    int32_t sum[SH_ROWS][SH_PX] = {};
#pragma unroll
    for (int32_t r = -SPLAT_R; r < SH_ROWS + SPLAT_R; ++r) {
        const int32_t gy = y + r;
        if (gy < 0 || gy >= height) { continue; }
        const int32_t* row = centres + (size_t)gy * (size_t)width;
        int32_t v[SH_PX + 2 * SPLAT_R]; // columns x - 2 .. x + 5
        if constexpr (VEC) {
            const int4 z = make_int4(0, 0, 0, 0);
            const int4 b = *reinterpret_cast<const int4*>(row + x);
            const int4 a = x > 0 ? *reinterpret_cast<const int4*>(row + x - 4) : z;
            const int4 c = x + 4 < width ? *reinterpret_cast<const int4*>(row + x + 4) : z;
            v[0] = a.z, v[1] = a.w, v[2] = b.x, v[3] = b.y, v[4] = b.z, v[5] = b.w, v[6] = c.x, v[7] = c.y;
        } else {
#pragma unroll
            for (int32_t q = 0; q < SH_PX + 2 * SPLAT_R; ++q) {
                const int32_t gx = x + q - SPLAT_R;
                v[q]             = gx >= 0 && gx < width ? row[gx] : 0;
            }
        }
#pragma unroll
        for (int32_t q = 0; q < SH_PX; ++q) {
            const int32_t h3 = v[q + 1] + v[q + 2] + v[q + 3];
            const int32_t h5 = h3 + v[q] + v[q + 4];
#pragma unroll
            for (int32_t j = 0; j < SH_ROWS; ++j) {
                if (r - j == 2 || r - j == -2) { sum[j][q] += h3; }
                if (r - j >= -1 && r - j <= 1) { sum[j][q] += h5; }
            }
        }
    }
    bool xline[SH_PX];
#pragma unroll
    for (int32_t q = 0; q < SH_PX; ++q) { xline[q] = (x + q) % line_every == 0; }
#pragma unroll
    for (int32_t j = 0; j < SH_ROWS; ++j) {
        const int32_t gy = y + j;
        if (gy >= height) { break; }
        const int32_t sel = gy % line_every == 0
                                ? BLEND_BLACK
                                : (int32_t)(uint8_t)__fmul_rn(100.f, __fdiv_rn((float)gy, (float)height));
        uint32_t px[SH_PX];
#pragma unroll
        for (int32_t q = 0; q < SH_PX; ++q) {
            px[q] = reinterpret_cast<const uint32_t*>(g_blend[xline[q] ? BLEND_BLACK : sel])[min(sum[j][q], BLEND_K - 1)];
        }
        uint8_t* out = rgba + (size_t)gy * (size_t)pitch + 4 * (size_t)x;
        if constexpr (VEC) {
            *reinterpret_cast<uint4*>(out) = make_uint4(px[0], px[1], px[2], px[3]);
        } else {
#pragma unroll
            for (int32_t q = 0; q < SH_PX; ++q) {
                if (x + q < width) { reinterpret_cast<uint32_t*>(out)[q] = px[q]; }
            }
        }
    }
}

} // namespace
} // namespace gpe

using namespace gpe;

extern "C" int32_t gpe_render_frame(const gpe_raster* r, const gpe_view* view, int32_t view_mem, void* stream)
{
    gpe::clear_error();
    if (!r || !view || !r->rgba || !r->coverage || r->width <= 0 || r->height <= 0 ||
        r->pitch < 4 * (int64_t)r->width || !(r->scale > 0.f) || !(r->chunk_dim > 0.f) ||
        (view_mem != GPE_MEM_HOST && view_mem != GPE_MEM_DEVICE)) {
        return GPE_ERR_BAD_ARG;
    }
    const int32_t line_every = (int32_t)(r->chunk_dim * r->scale); // (int32_t)(kChunkDim * kSimScale), :228
    if (line_every <= 0) { return GPE_ERR_BAD_ARG; }
    cudaStream_t st     = as_stream(stream);
    const gpe_view* vp  = view_mem == GPE_MEM_DEVICE ? view : nullptr;
    gpe_view vv{};
    // grid rows walk the chunks: one row a chunk for a host view; a device view is read only by the kernel
    // (its chunk count may change between replays of a captured frame), so a fixed 64 rows stride over them
    int32_t rows = 64;
    if (view_mem == GPE_MEM_HOST) {
        vv = *view;
        if (!vv.pos || !vv.counts || vv.chunks_x <= 0 || vv.chunks_y <= 0 || vv.chunk_capacity <= 0) {
            return GPE_ERR_BAD_ARG;
        }
        rows = (int32_t)std::min<int64_t>((int64_t)vv.chunks_x * vv.chunks_y, 65535);
    }
    {
        const int64_t n = (int64_t)r->width * r->height;
        const bool vec  = reinterpret_cast<uintptr_t>(r->coverage) % 16 == 0;
        k_clear_centres<<<(unsigned)(((vec ? (n + 3) / 4 : n) + 255) / 256), 256, 0, st>>>(r->coverage, n, vec);
        GPE_CHECK_LAUNCH("k_clear_centres");
    }
    {
        // about 32 blocks of 256 per SM: one particle a thread for a million particles
        const int32_t cols = max(1, (int32_t)std::min<int64_t>((32 * sm_count() + rows - 1) / rows, 65535));
        GPE_TRY_CUDA(launch(behind(st), dim3((unsigned)cols, (unsigned)rows), 256, k_splat_point, vp, vv, r->coverage,
                            r->width, r->height, r->scale));
    }
    const bool vec = r->width % 4 == 0 && reinterpret_cast<uintptr_t>(r->coverage) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(r->rgba) % 16 == 0 && r->pitch % 16 == 0;
    const unsigned grid = (unsigned)(((int64_t)r->width + SH_TW - 1) / SH_TW * (((int64_t)r->height + SH_TH - 1) / SH_TH));
    GPE_TRY_CUDA(launch(behind(st), grid, SH_THREADS, vec ? k_shade<true> : k_shade<false>, r->rgba, r->pitch,
                        r->coverage, r->width, r->height, line_every));
    return GPE_OK;
}
