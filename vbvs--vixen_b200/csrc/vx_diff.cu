// vx_diff.cu - differentiable form: a forward render that records each
// pixel's hit, and the adjoint kernel that scatters dL/d(colour) into the
// brick attribute pool.  No reference counterpart.
//
// The traversal is discrete and is not differentiated: the forward pass
// records (hit flags, brick, voxel) per pixel and the backward pass replays
// those indices.  Pixel colour of a hit = c * k with the Lambert factor
// k = 0.3 + max(n . L, 0) * 0.7 of shaders/Lighting.glsl:19-28 (L =
// normalize(1,1,-1), n the entry-face normal); a miss shows the sky colour,
// which does not depend on the attributes.
//   kind 0 (per-voxel colour): c = attr[(brick*512 + voxel)*3 + ch]
//   kind 1 (DXT1 endpoints held in FP32 before quantisation): the voxel's
//     block b = brick*32 + (voxel >> 4) has endpoints e0 = attr[b*6 + 0..2],
//     e1 = attr[b*6 + 3..5] and the fixed 2-bit selector s of texel
//     (voxel & 15) in idx[b]; c = w0*e0 + w1*e1 with (w0, w1) = (1, 0),
//     (0, 1), (2/3, 1/3), (1/3, 2/3) for s = 0..3, the interpolation of
//     DXT1ColorCompressor::decodeColorHead (DXT1Compressor.cpp:34-35).
// Loss = sum over pixels and channels of (pixel - target)^2; the adjoint of a
// hit pixel is g = 2 (pixel - target) k, added to dL/dc (kind 0) or w0 g,
// w1 g to dL/de0, dL/de1 (kind 1).  Runs of pixels that hit the same voxel /
// block are combined first, so each costs one reduction per channel (or pair).

#include <algorithm>

#include "vx_cast.cuh"
#include "vx_regular.cuh"

namespace vx {
namespace {

constexpr int DBLOCK = 256;

// 0.3 + max(n . L, 0) * 0.7 with n on one axis: n . L is +-L[axis] (the other
// products are zeros), L = (a, a, -a).
__device__ __forceinline__ float lambert_k(uint32_t flags) {
    const float Ld = (1.0f * 1.0f + 1.0f * 1.0f) + (-1.0f) * (-1.0f);
    const float Linv = 1.0f / sqrtf(Ld);
    const bool neg = flags & F_NEG, z = ((flags >> 1) & 3u) == 2u;
    return 0.3f + (neg == z ? 1.0f * Linv : 0.0f) * 0.7f;
}

__device__ __forceinline__ void dxt_weights(uint32_t sel, float& w0, float& w1) {
    w0 = (sel == 0) ? 1.0f : (sel == 1) ? 0.0f : (sel == 2) ? (2.0f / 3.0f) : (1.0f / 3.0f);
    w1 = (sel == 0) ? 0.0f : (sel == 1) ? 1.0f : (sel == 2) ? (1.0f / 3.0f) : (2.0f / 3.0f);
}

// The cameras of one launch: VX_DIFF_MAX_VIEWS views at most, passed by value
// (kernel parameter space), so a multi-view launch needs no device copy.
struct Views {
    CameraDev cam[VX_DIFF_MAX_VIEWS];
};

// One pixel of the forward pass: cast, record, shade.  GENERAL: the scene is
// not DevScene::ordinary (as in vx_kernels.cu).
template <bool GENERAL>
__device__ __forceinline__ void forward_pixel(const DevScene& s, const CameraDev& cam, uint32_t px, uint32_t py,
                                              uint32_t w, uint32_t hgt, uint32_t i, int kind,
                                              const float* __restrict__ attr, const uint32_t* __restrict__ idx,
                                              float* __restrict__ image, vx_hit* __restrict__ record,
                                              uint32_t* stkN, float* stkT, uint32_t* cyc, uint32_t stride) {
    vx_ray r;
    float uv_y;
    camera_ray(cam, px, py, w, hgt, r, &uv_y);
    Hit h;
    if constexpr (GENERAL)
        cast_ray(s, r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, 0.0f, FLT_MAX_, stkN, stkT, cyc, stride, h);
    else
        cast_plain(s, r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, 0.0f, FLT_MAX_, stkN, stkT, cyc, stride, MAX_ITER + 1, h);
    store_hit(record, i, h);
    float c[3];
    if (h.flags & F_HIT) {
        const float k = lambert_k(h.flags);
        if (kind == 0) {
            const float* a = attr + (size_t(h.brick) * 512 + h.voxel) * 3;
            c[0] = __ldg(a) * k; c[1] = __ldg(a + 1) * k; c[2] = __ldg(a + 2) * k;
        } else {
            const size_t b = size_t(h.brick) * 32 + (h.voxel >> 4);
            const uint32_t sel = (__ldg(idx + b) >> ((h.voxel & 15u) * 2u)) & 3u;
            float w0, w1;
            dxt_weights(sel, w0, w1);
            const float* e = attr + b * 6;
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) c[ch] = (w0 * __ldg(e + ch) + w1 * __ldg(e + 3 + ch)) * k;
        }
    } else {
        const float k = 1.0f - uv_y * 0.5f;
        c[0] = 0.5f * k; c[1] = 0.7f * k; c[2] = 1.0f * k;
    }
    float* o = image + size_t(i) * 3;
    o[0] = c[0]; o[1] = c[1]; o[2] = c[2];
}

// Images and records are view-major: pixel p of view v is entry v * w * hgt + p.
// The work is split into warp tasks of 8 x 4 pixels (the
// eight pieces of a 32 x 8 tile are consecutive tasks), so a warp's rays are
// neighbours in both image directions.  A block holds FWD_WARPS warps, one task
// each: small blocks free their slot as soon as their warps finish, where one
// block per 32 x 8 tile would hold its slot until the slowest of its eight
// warps finished (the orbit views mix rays that hit near with rays that miss far).
#ifndef VX_DIFF_FWD_WARPS
#define VX_DIFF_FWD_WARPS 2
#endif
constexpr int FWD_WARPS = VX_DIFF_FWD_WARPS;
constexpr int FWD_THREADS = FWD_WARPS * 32;

template <bool GENERAL>
__global__ void __launch_bounds__(FWD_THREADS, (GENERAL ? 768 : 1024) / FWD_THREADS) diff_forward_kernel(
    const __grid_constant__ DevScene s, Views views, uint32_t nviews, uint32_t w, uint32_t hgt, int kind, const float* __restrict__ attr,
    const uint32_t* __restrict__ idx, float* __restrict__ image, vx_hit* __restrict__ record) {
    extern __shared__ uint32_t smem[];
    uint32_t* stkN = smem + threadIdx.x;
    float* stkT = reinterpret_cast<float*>(smem + s.max_levels * FWD_THREADS) + threadIdx.x;
    uint32_t* cyc = smem + 2 * s.max_levels * FWD_THREADS + threadIdx.x;
    const uint32_t per_view = w * hgt;
    const uint32_t tw = (w + 31) / 32, tiles = tw * ((hgt + 7) / 8);
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t t = uint64_t(blockIdx.x) * FWD_WARPS + (threadIdx.x >> 5);
    if (t >= uint64_t(nviews) * tiles * 8) return;
    const uint32_t piece = uint32_t(t & 7u), tt = uint32_t(t >> 3);
    const uint32_t v = tt / tiles, tl = tt - v * tiles;
    const uint32_t px = (tl % tw) * 32 + (piece & 3u) * 8 + (lane & 7u);
    const uint32_t py = (tl / tw) * 8 + (piece >> 2) * 4 + (lane >> 3);
    if (px >= w || py >= hgt) return;
    forward_pixel<GENERAL>(s, views.cam[v], px, py, w, hgt, v * per_view + py * w + px, kind, attr, idx, image, record,
                           stkN, stkT, cyc, FWD_THREADS);
}

// grad[0 .. 1] += (x, y) in one reduction (8-byte aligned).
__device__ __forceinline__ void add_pair(float* at, float x, float y) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" :: "l"(at), "f"(x), "f"(y) : "memory");
}

// The adjoint.  A warp takes 32 consecutive pixels; neighbours that hit the same
// voxel / block form runs, whose sums go up by shuffles (a step only while some
// run of the warp is longer) and are added by the run's first lane.  PAIRS: the
// gradient is 8-byte aligned, two channels per reduction.  The loss is kept per
// thread over all its pixels and reduced once per block.
// Bound: the latency of its loads (record 16, image 12 and target 12 bytes a
// pixel; DRAM 46 % busy, three quarters of the stalls) and the reductions at L2.  Measured (B200, 16 views of 512 x 512, per-voxel colours)
// against groups of equal keys anywhere in the warp (__match_any_sync on 64
// bits, a shuffle per lane and channel) with a block reduction per 256 pixels:
// 154 -> 53 us; 4.2 M pixels of a closed surface 93 -> 33 us, with DXT1 endpoints
// 166 -> 38 us.  8 / 16 / 32 blocks per SM 50 / 48 / 48 us (10.5 us with 32 for
// 0.4 M pixels, 13 with 8), a block per 256 pixels 76 us.
//
// Records need not be an image's: shuffled pixels of a few voxels, or two voxels in
// turn, make 32 runs of few places, whose reductions then queue at a few addresses
// of L2 (4 M pixels of two voxels in turn, 8 in all: 4.40 ms; random ones of 8
// voxels 2.28 ms, of 64 DXT1 blocks 4.54 ms).  So a warp with MERGE_RUNS runs or more
// bounds the number of its places from below by the bits of a hash, and where that is
// half the runs or less, adds up the runs of one place first, in pairs and pairs of
// pairs: 0.28, 0.53 and 0.78 ms (groups of equal keys anywhere in the warp: 0.44,
// 0.78, 1.53).  The test costs a surface in runs of nine 31.3 -> 33.2 us and the 16
// views 52.5 -> 52.9; merging without it where all places differ 10.3 -> 13.0 us, and
// from 4 runs on instead of 8 runs of nine in DXT1 blocks 37.8 -> 38.8.
constexpr uint32_t MERGE_RUNS = 8;
template <int KIND, bool PAIRS>
__global__ void __launch_bounds__(DBLOCK) diff_backward_kernel(uint32_t n, const uint32_t* __restrict__ idx,
                                                               const vx_hit* __restrict__ record,
                                                               const float* __restrict__ image,
                                                               const float* __restrict__ target,
                                                               float* __restrict__ grad, float* __restrict__ loss) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    constexpr int CH = KIND == 0 ? 3 : 6;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t step = uint64_t(gridDim.x) * DBLOCK;
    float lsum = 0.0f;
    for (uint64_t base = uint64_t(blockIdx.x) * DBLOCK + (threadIdx.x & ~31u); base < n; base += step) {
        const uint64_t i = base + lane;
        uint4 rec = make_uint4(0u, NONE, 0u, 0u);
        float d[3] = {0.0f, 0.0f, 0.0f};
        if (i < n) {
            rec = __ldg(reinterpret_cast<const uint4*>(record) + i);
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) d[ch] = __ldg(image + i * 3 + ch) - __ldg(target + i * 3 + ch);
        }
        lsum += (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2];
        const uint32_t flags = (rec.w >> 16) & 0xFFu, voxel = rec.w & 0xFFFFu;
        const bool hit = flags & F_HIT;
        // the pixel's place: voxel or 16-voxel block of the brick; misses differ from every hit
        const uint32_t part = hit ? (KIND == 0 ? voxel : voxel >> 4) : 0xFFFFFFFFu;
        const uint64_t key = uint64_t(rec.y) * (KIND == 0 ? 512u : 32u) + part;
        float v[CH];
        {
            const float k = lambert_k(flags);
            float w0 = 1.0f, w1 = 0.0f;
            if constexpr (KIND == 1)
                if (hit) dxt_weights((__ldg(idx + key) >> ((voxel & 15u) * 2u)) & 3u, w0, w1);
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                const float g = 2.0f * d[ch] * k;
                if constexpr (KIND == 0) {
                    v[ch] = g;
                } else {
                    v[ch] = w0 * g;
                    v[3 + ch] = w1 * g;
                }
            }
        }
        // runs: `first` marks their first lanes, `same` the lanes that continue one
        const uint32_t brick_before = __shfl_up_sync(FULL, rec.y, 1), part_before = __shfl_up_sync(FULL, part, 1);
        const bool first = lane == 0 || rec.y != brick_before || part != part_before;
        const uint32_t same = ~__ballot_sync(FULL, first);
        // lanes of the run behind this one
        const uint32_t after = same >> lane >> 1;
        const uint32_t left = after == FULL ? 32u : uint32_t(__ffs(int(~after))) - 1u;
        uint32_t longer = same;  // bit l: lanes l, l + 1, .. l + reach - 1 all continue runs
        for (uint32_t reach = 1; longer; reach <<= 1) {
#pragma unroll
            for (int ch = 0; ch < CH; ++ch) {
                const float u = __shfl_down_sync(FULL, v[ch], reach);
                if (reach <= left) v[ch] += u;
            }
            longer &= longer >> reach;
        }
        bool adds = hit && first;
        const uint32_t heads = __ballot_sync(FULL, adds), runs = __popc(heads);
        const uint32_t bit = adds ? 1u << ((uint32_t(key) * 0x9E3779B1u) >> 27) : 0u;
        if (runs >= MERGE_RUNS && 2u * uint32_t(__popc(__reduce_or_sync(FULL, bit))) <= runs) {
            const uint32_t peers = __match_any_sync(FULL, key) & heads;  // the runs of this place
            const bool head = adds;
            uint32_t rank = __popc(peers & ((1u << lane) - 1u));
            uint32_t rest = head ? peers & ~((2u << lane) - 1u) : 0u;  // those behind this one
            adds = head && rank == 0u;
            while (__any_sync(FULL, rest != 0u)) {
                const int from = rest ? __ffs(int(rest)) - 1 : int(lane);
#pragma unroll
                for (int ch = 0; ch < CH; ++ch) {
                    const float u = __shfl_sync(FULL, v[ch], from);
                    if (rest) v[ch] += u;
                }
                rest &= ~__ballot_sync(FULL, head && (rank & 1u));  // odd ranks are in the sums before them now
                rank >>= 1;
            }
        }
        if (adds) {
            float* dst = grad + key * CH;
            if constexpr (KIND == 1) {
#pragma unroll
                for (int j = 0; j < 6; j += 2) {
                    if constexpr (PAIRS) {
                        add_pair(dst + j, v[j], v[j + 1]);
                    } else {
                        atomicAdd(dst + j, v[j]);
                        atomicAdd(dst + j + 1, v[j + 1]);
                    }
                }
            } else if constexpr (PAIRS) {
                const bool odd = key & 1u;  // 12 bytes a voxel: the pair starts at its second channel
                add_pair(dst + (odd ? 1 : 0), odd ? v[1] : v[0], odd ? v[2] : v[1]);
                atomicAdd(dst + (odd ? 0 : 2), odd ? v[0] : v[2]);
            } else {
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) atomicAdd(dst + ch, v[ch]);
            }
        }
    }
    if (loss) {
        for (int off = 16; off > 0; off >>= 1) lsum += __shfl_down_sync(FULL, lsum, off);
        __shared__ float sums[DBLOCK / 32];
        if (lane == 0) sums[threadIdx.x >> 5] = lsum;
        __syncthreads();
        if (threadIdx.x < 32) {
            float t = threadIdx.x < DBLOCK / 32 ? sums[threadIdx.x] : 0.0f;
            for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(FULL, t, off);
            if (threadIdx.x == 0) atomicAdd(loss, t);
        }
    }
}

}  // namespace
}  // namespace vx

extern "C" int vx_diff_forward_views(const vx_scene* scene, const vx_camera_pc* pcs, uint32_t views, uint32_t w,
                                     uint32_t h, int32_t kind, const float* attr, const uint32_t* dxt_idx,
                                     float* image, vx_hit* record, void* stream) {
    using namespace vx;
    if (!scene || !pcs || !attr || !image || !record || (kind == 1 && !dxt_idx) || (kind != 0 && kind != 1))
        return fail(VX_EINVAL, "vx_diff_forward: bad argument");
    if (views > VX_DIFF_MAX_VIEWS)
        return fail(VX_EOVERFLOW, "vx_diff_forward_views: more than VX_DIFF_MAX_VIEWS views in one call");
    const uint64_t n = uint64_t(w) * h * views;
    if (n > 0xFFFFFFFFull) return fail(VX_EOVERFLOW, "vx_diff_forward: views * width * height exceeds 2^32");
    if (reinterpret_cast<uintptr_t>(record) % 16 || reinterpret_cast<uintptr_t>(image) % 4)
        return fail(VX_EINVAL, "vx_diff_forward: misaligned output");
    if (n == 0) return VX_OK;
    const DevScene& s = scene_dev(scene);
    Views v{};
    for (uint32_t k = 0; k < views; ++k) v.cam[k] = camera_from_pc(pcs[k]);
    const size_t smem = (size_t(2) * size_t(s.max_levels) + CYC_WORDS) * FWD_THREADS * sizeof(uint32_t);
    auto* kernel = s.ordinary ? diff_forward_kernel<false> : diff_forward_kernel<true>;
    // stacks of scenes deeper than 15 levels need more than 48 KiB per 256 threads
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return fail(VX_ECUDA, std::string("vx_diff_forward: ") + cudaGetErrorString(e));
    }
    const uint64_t tasks = uint64_t(views) * ((w + 31) / 32) * ((h + 7) / 8) * 8;
    const uint64_t blocks = (tasks + FWD_WARPS - 1) / FWD_WARPS;
    if (blocks > 0x7FFFFFFFull) return fail(VX_EOVERFLOW, "vx_diff_forward: too many pixels for one launch");
    kernel<<<uint32_t(blocks), FWD_THREADS, smem, static_cast<cudaStream_t>(stream)>>>(s, v, views, w, h, kind, attr,
                                                                                      dxt_idx, image, record);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VX_OK : fail(VX_ECUDA, std::string("vx_diff_forward: ") + cudaGetErrorString(e));
}

extern "C" int vx_diff_forward(const vx_scene* scene, const vx_camera_pc* pc, uint32_t w, uint32_t h, int32_t kind,
                               const float* attr, const uint32_t* dxt_idx, float* image, vx_hit* record,
                               void* stream) {
    if (!pc) return vx::fail(VX_EINVAL, "vx_diff_forward: bad argument");
    return vx_diff_forward_views(scene, pc, 1, w, h, kind, attr, dxt_idx, image, record, stream);
}

extern "C" int vx_diff_backward(uint32_t n, int32_t kind, const uint32_t* dxt_idx, const vx_hit* record,
                                const float* image, const float* target, float* grad, float* loss, void* stream) {
    using namespace vx;
    if ((n && (!record || !image || !target || !grad)) || (kind == 1 && !dxt_idx) || (kind != 0 && kind != 1))
        return fail(VX_EINVAL, "vx_diff_backward: bad argument");
    if (n == 0) return VX_OK;
    const bool pairs = reinterpret_cast<uintptr_t>(grad) % 8 == 0;
    auto* kernel = kind == 0 ? (pairs ? diff_backward_kernel<0, true> : diff_backward_kernel<0, false>)
                             : (pairs ? diff_backward_kernel<1, true> : diff_backward_kernel<1, false>);
    const uint32_t blocks = uint32_t(std::min<uint64_t>((uint64_t(n) + DBLOCK - 1) / DBLOCK, 148 * 32));
    kernel<<<blocks, DBLOCK, 0, static_cast<cudaStream_t>(stream)>>>(n, dxt_idx, record, image, target, grad, loss);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VX_OK : fail(VX_ECUDA, std::string("vx_diff_backward: ") + cudaGetErrorString(e));
}

namespace vx {
VX_VIOLATION_READER(violations_diff)
}  // namespace vx
