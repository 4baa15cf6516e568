// vx_kernels.cu - plain (one launch per scene) cast and render kernels.
#include <algorithm>

#include "vx_cast.cuh"
#include "vx_regular.cuh"
#include "vx_palette.h"

namespace vx {
namespace {

// Threads per block of the cast kernel, and warps per block of the render
// kernel (each warp one 8 x 4 piece of a 32 x 8 tile).
#ifndef VX_CAST_BLOCK
#define VX_CAST_BLOCK 64
#endif
#ifndef VX_RENDER_WARPS
#define VX_RENDER_WARPS 2
#endif
constexpr int BLOCK = VX_CAST_BLOCK;
constexpr int RENDER_WARPS = VX_RENDER_WARPS;
constexpr int RENDER_THREADS = RENDER_WARPS * 32;
// Threads per SM the kernels are compiled for.  Plain form: 1,024 leave 64
// registers a thread.  At 768 / 896 / 1,024 / 1,152 / 1,280 threads the 1080p cave
// frame takes 123 / 119 / 116 / 123 / 139 us, the 4K city frame with shadow rays 1.10
// / 1.04 / 1.01 / 1.04 / 1.21 ms, incoherent rays with LOD 217 / 213 / 214 / 233 /
// 244 us, a 1279 x 717 render 53.7 / 53.0 / 52.1 / 54.8 / 58.6 us (more warps to issue
// from, until spills cost more); only 512 x 512 rays in pixel rows, two waves of
// blocks, are faster at 768 (53.6 against 54.8 us).  General form, which carries more
// state: 896 for the cast (72 registers; at 64 it spills: 0.1249 against 0.1188 ms for
// the cave frame), 768 for the others.
constexpr int CAST_THREADS = 1024;
constexpr int GENERAL_CAST_THREADS = 896, GENERAL_THREADS = 768;

// Which form a launch takes: the general one (vx_cast.cuh) when counters are
// wanted, and for a scene that is not DevScene::ordinary, none of whose rays the
// plain form takes itself: sent through the plain kernels they would all go out of
// line there, on 64 registers (256^3 scene moved by 2^17, 1024 x 768 rays: cast 237
// us, this way 194; render 217 and 177, forward pass 226 and 178, incoherent rays
// 224 and 187).
template <bool LOD, bool GENERAL>
__global__ void __launch_bounds__(BLOCK, (GENERAL ? GENERAL_CAST_THREADS : CAST_THREADS) / BLOCK) cast_kernel(const __grid_constant__ DevScene s, const vx_ray* __restrict__ rays, uint32_t n,
                                                      float tmin, float tmax, vx_hit* __restrict__ hits,
                                                      void* __restrict__ color,
                                                      vx_ray_counters* __restrict__ counters, LodCone lod) {
    extern __shared__ uint32_t smem[];
    uint32_t* stkN = smem + threadIdx.x;
    float* stkT = reinterpret_cast<float*>(smem + s.max_levels * BLOCK) + threadIdx.x;
    uint32_t* cyc = smem + 2 * s.max_levels * BLOCK + threadIdx.x;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2* r2 = reinterpret_cast<const float2*>(rays + i);
    const float2 a = __ldg(r2), b = __ldg(r2 + 1), c = __ldg(r2 + 2);
    Hit h;
    if constexpr (GENERAL) cast_ray<LOD>(s, a.x, a.y, b.x, b.y, c.x, c.y, tmin, tmax, stkN, stkT, cyc, BLOCK, h, lod);
    else cast_plain<LOD>(s, a.x, a.y, b.x, b.y, c.x, c.y, tmin, tmax, stkN, stkT, cyc, BLOCK, MAX_ITER + 1, h, lod);
    store_hit(hits, i, h);
    if (color) store_color(s, color, i, h);
    if (GENERAL && counters) {
        uint4 rc;
        rc.x = (h.iters & 0xFFFFu) | (h.grid_reads << 16);
        rc.y = h.dda_steps;
        rc.z = (h.run_iters & 0xFFFFu) | (h.run_grid_reads << 16);
        rc.w = h.run_dda_steps;
        reinterpret_cast<uint4*>(counters)[i] = rc;
    }
}

// The cast of rays compacted on the device: `count` (device) rays of at most
// n_max, the hit record of ray i going to slot map[i].  The per-ray work is
// cast_kernel's (castRay, no colour or counters).
template <bool GENERAL>
__global__ void __launch_bounds__(BLOCK, (GENERAL ? GENERAL_THREADS : CAST_THREADS) / BLOCK) cast_mapped_kernel(
    const __grid_constant__ DevScene s, const vx_ray* __restrict__ rays, uint32_t n_max,
    const uint32_t* __restrict__ count, const uint32_t* __restrict__ map, float tmin, float tmax,
    vx_hit* __restrict__ hits) {
    extern __shared__ uint32_t smem[];
    uint32_t* stkN = smem + threadIdx.x;
    float* stkT = reinterpret_cast<float*>(smem + s.max_levels * BLOCK) + threadIdx.x;
    uint32_t* cyc = smem + 2 * s.max_levels * BLOCK + threadIdx.x;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= min(n_max, __ldg(count))) return;
    const float2* r2 = reinterpret_cast<const float2*>(rays + i);
    const float2 a = __ldg(r2), b = __ldg(r2 + 1), c = __ldg(r2 + 2);
    Hit h;
    if constexpr (GENERAL) cast_ray(s, a.x, a.y, b.x, b.y, c.x, c.y, tmin, tmax, stkN, stkT, cyc, BLOCK, h);
    else cast_plain(s, a.x, a.y, b.x, b.y, c.x, c.y, tmin, tmax, stkN, stkT, cyc, BLOCK, MAX_ITER + 1, h);
    store_hit(hits, __ldg(map + i), h);
}

// Pixels go to warps in 8 x 4 pieces of 32 x 8 tiles (the reference dispatches
// 8 x 8 workgroups, ComputeDispatchNode.cpp:272-301): a warp's rays are
// neighbours in both image directions, so their traversals diverge less than
// along a row.  Warp task t is piece t & 7 of tile t >> 3; a block holds
// RENDER_WARPS consecutive tasks.  Outputs are indexed by pixel (y * w + x).
template <bool GENERAL>
__global__ void __launch_bounds__(RENDER_THREADS, (GENERAL ? GENERAL_THREADS : CAST_THREADS) / RENDER_THREADS) render_kernel(
    const __grid_constant__ DevScene s, CameraDev cam, uint32_t w, uint32_t hgt, uint32_t* __restrict__ image, vx_hit* __restrict__ hits,
    void* __restrict__ color) {
    extern __shared__ uint32_t smem[];
    uint32_t* stkN = smem + threadIdx.x;
    float* stkT = reinterpret_cast<float*>(smem + s.max_levels * RENDER_THREADS) + threadIdx.x;
    uint32_t* cyc = smem + 2 * s.max_levels * RENDER_THREADS + threadIdx.x;
    const uint32_t tw = (w + 31) / 32;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t t = uint64_t(blockIdx.x) * RENDER_WARPS + (threadIdx.x >> 5);
    const uint32_t piece = uint32_t(t & 7u), tile = uint32_t(t >> 3);
    const uint32_t px = (tile % tw) * 32 + (piece & 3u) * 8 + (lane & 7u);
    const uint32_t py = (tile / tw) * 8 + (piece >> 2) * 4 + (lane >> 3);
    if (px >= w || py >= hgt) return;
    const uint32_t i = py * w + px;
    vx_ray r;
    float uv_y;
    camera_ray(cam, px, py, w, hgt, r, &uv_y);
    Hit h;
    if constexpr (GENERAL)
        cast_ray(s, r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, 0.0f, FLT_MAX_, stkN, stkT, cyc, RENDER_THREADS, h);
    else
        cast_plain(s, r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, 0.0f, FLT_MAX_, stkN, stkT, cyc, RENDER_THREADS,
                   MAX_ITER + 1, h);
    if (hits) store_hit(hits, i, h);
    if (color) store_color(s, color, i, h);
    if (image) {
        // computeLighting (Lighting.glsl:19-28) or the sky gradient
        // (VoxelRayMarch.comp:493-499), stored as RGBA8.
        float cr, cg, cb;
        if (h.flags & F_HIT) {
            float br = 1.0f, bg = 1.0f, bb = 1.0f;
            if (s.color_kind == VX_COLOR_RGBA8) {
                const uint32_t c = __ldg(s.rgba + size_t(h.brick) * 512 + h.voxel);
                br = float(c & 0xFFu) / 255.0f;
                bg = float((c >> 8) & 0xFFu) / 255.0f;
                bb = float((c >> 16) & 0xFFu) / 255.0f;
            } else if (s.color_kind == VX_COLOR_DXT1) {
                dxt_texel(s.dxt, h.brick, h.voxel, br, bg, bb);
            } else if (s.color_kind == VX_COLOR_MATERIAL) {
                // getMaterialColor(voxelData & 0xFF) (VoxelRayMarch.comp:188-192)
                const Rgb m = material_color_shader(__ldg(s.rgba + size_t(h.brick) * 512 + h.voxel) & 0xFFu);
                br = m.r; bg = m.g; bb = m.b;
            }
            const float Ld = (1.0f * 1.0f + 1.0f * 1.0f) + (-1.0f) * (-1.0f);
            const float Linv = 1.0f / sqrtf(Ld);
            const float L[3] = {1.0f * Linv, 1.0f * Linv, -1.0f * Linv};
            float nrm[3] = {0.0f, 0.0f, 0.0f};
            const int axis = (h.flags >> 1) & 3;
            nrm[axis] = (h.flags & F_NEG) ? -1.0f : 1.0f;
            if (s.nrm) {
                // Compressed shading (VoxelRayMarch_Compressed.comp:242-256): the
                // decoded normal blended with the entry-face normal,
                // normalize(n_dxt + face * 0.5).
                float dx, dy, dz;
                dxt_normal(s, h.brick, h.voxel, dx, dy, dz);
                const dxtn::F3 b = dxtn::unit(dxtn::F3{dx, dy, dz} + dxtn::F3{nrm[0], nrm[1], nrm[2]} * 0.5f);
                nrm[0] = b.x; nrm[1] = b.y; nrm[2] = b.z;
            }
            const float nd = (nrm[0] * L[0] + nrm[1] * L[1]) + nrm[2] * L[2];
            const float diffuse = gmax(nd, 0.0f) * 0.7f;
            const float k = 0.3f + diffuse;
            cr = br * k; cg = bg * k; cb = bb * k;
        } else {
            const float k = 1.0f - uv_y * 0.5f;
            cr = 0.5f * k; cg = 0.7f * k; cb = 1.0f * k;
        }
        auto u8 = [](float v) -> uint32_t { return uint32_t(fclamp(v, 0.0f, 1.0f) * 255.0f + 0.5f); };
        image[i] = u8(cr) | (u8(cg) << 8) | (u8(cb) << 16) | (255u << 24);
    }
}

__global__ void __launch_bounds__(256) ordinary_check_kernel(DevScene s, uint32_t* __restrict__ mismatch) {
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    const uint32_t bpa = uint32_t(s.bpa), slots = bpa * bpa * bpa;
    for (uint32_t i = first; i < slots; i += step) {
        const uint32_t b = __ldg(s.grid + i);
        if (b != NONE && __ldg(s.coord + b) != (i % bpa | (i / bpa % bpa) << 10 | (i / (bpa * bpa)) << 20)) *mismatch = 1u;
    }
    for (uint64_t i = first; i < s.node_count; i += step) {
        const uint2 nd = __ldg(s.nodes + i);
        const uint32_t inner = ~(nd.y >> 8) & nd.y & 0xFFu;  // children that PUSH may enter
        if (inner && uint64_t(nd.x) + uint32_t(__popc(inner)) > s.node_count) *mismatch = 1u;
    }
}

__global__ void camera_rays_kernel(CameraDev cam, uint32_t w, uint32_t hgt, vx_ray* __restrict__ rays) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w * hgt) return;
    vx_ray r;
    camera_ray(cam, i % w, i / w, w, hgt, r, nullptr);
    rays[i] = r;
}

size_t stack_bytes(const DevScene& s, int threads) {
    return (size_t(2) * size_t(s.max_levels) + CYC_WORDS) * size_t(threads) * sizeof(uint32_t);
}

// Stacks of scenes deeper than 15 levels take more than the 48 KiB of dynamic
// shared memory a launch gets without opting in (64 KiB at 23 levels).
template <class K>
cudaError_t allow_smem(K kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
}

}  // namespace

int launch_cast(const DevScene& s, const vx_ray* rays, uint32_t n, float tmin, float tmax, vx_hit* hits,
                void* color, vx_ray_counters* counters, void* stream, const vx_lod_params* lod) {
    if (n == 0) return int(cudaSuccess);
    const uint32_t grid = (n + BLOCK - 1) / BLOCK;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t smem = stack_bytes(s, BLOCK);
    const bool cone = lod && lod->ray_dir_size > 0.0f;
    const LodCone lc = cone ? LodCone{lod->ray_orig_size, lod->ray_dir_size} : LodCone{0.0f, 0.0f};
    const bool general = counters || !s.ordinary;
    auto* kernel = cone ? (general ? cast_kernel<true, true> : cast_kernel<true, false>)
                        : (general ? cast_kernel<false, true> : cast_kernel<false, false>);
    if (cudaError_t e = allow_smem(kernel, smem)) return int(e);
    kernel<<<grid, BLOCK, smem, st>>>(s, rays, n, tmin, tmax, hits, color, counters, lc);
    return int(cudaGetLastError());
}

int launch_cast_mapped(const DevScene& s, const vx_ray* rays, uint32_t n_max, const uint32_t* count,
                       const uint32_t* map, float tmin, float tmax, vx_hit* hits, void* stream) {
    if (n_max == 0) return int(cudaSuccess);
    const size_t smem = stack_bytes(s, BLOCK);
    auto* kernel = s.ordinary ? cast_mapped_kernel<false> : cast_mapped_kernel<true>;
    if (cudaError_t e = allow_smem(kernel, smem)) return int(e);
    kernel<<<(n_max + BLOCK - 1) / BLOCK, BLOCK, smem, static_cast<cudaStream_t>(stream)>>>(
        s, rays, n_max, count, map, tmin, tmax, hits);
    return int(cudaGetLastError());
}

int launch_render(const DevScene& s, const CameraDev& cam, uint32_t w, uint32_t h, uint32_t* image, vx_hit* hits,
                  void* color, void* stream) {
    const uint64_t n = uint64_t(w) * h;
    if (n == 0) return int(cudaSuccess);
    static_assert(8 % RENDER_WARPS == 0, "a block covers whole 8 x 4 pieces of one 32 x 8 tile");
    const uint64_t grid = uint64_t((w + 31) / 32) * ((h + 7) / 8) * (8 / RENDER_WARPS);
    if (grid > 0x7FFFFFFFull) return int(cudaErrorInvalidValue);
    const size_t smem = stack_bytes(s, RENDER_THREADS);
    auto* kernel = s.ordinary ? render_kernel<false> : render_kernel<true>;
    if (cudaError_t e = allow_smem(kernel, smem)) return int(e);
    kernel<<<uint32_t(grid), RENDER_THREADS, smem, static_cast<cudaStream_t>(stream)>>>(s, cam, w, h, image, hits, color);
    return int(cudaGetLastError());
}

int launch_ordinary_check(const DevScene& s, uint32_t* mismatch, void* stream) {
    const uint64_t slots = uint64_t(s.bpa) * uint64_t(s.bpa) * uint64_t(s.bpa);
    const uint64_t items = std::max<uint64_t>(slots, s.node_count);
    ordinary_check_kernel<<<uint32_t(std::min<uint64_t>((items + 255) / 256, 148 * 8)), 256, 0,
                            static_cast<cudaStream_t>(stream)>>>(s, mismatch);
    return int(cudaGetLastError());
}

int launch_camera_rays(const CameraDev& cam, uint32_t w, uint32_t h, vx_ray* rays, void* stream) {
    const uint64_t n = uint64_t(w) * h;
    if (n == 0) return int(cudaSuccess);
    camera_rays_kernel<<<uint32_t((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(cam, w, h, rays);
    return int(cudaGetLastError());
}

}  // namespace vx

namespace vx {
VX_VIOLATION_READER(violations_kernels)
}  // namespace vx
