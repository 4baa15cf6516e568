// vx_payload.cu - the compressed brick payloads the rebuild writes
// (SVORebuild.cpp:615-722): DXT normal blocks from geometric normals and DXT1
// colour blocks from per-voxel colours, each built on the GPU (one thread per
// 16-voxel block) or on the host from the same code; and the per-hit normal
// decode of the compressed shader (getCompressedVoxelNormal,
// VoxelRayMarch_Compressed.comp:160-165).
#include <algorithm>
#include <thread>
#include <vector>

#include "vx_cast.cuh"
#include "vx_dxt1.h"
#include "vx_dxtn.h"
#include "vx_pairs.cuh"
#include "vx_palette.h"

namespace vx {
namespace {

constexpr uint32_t SMS = 148;  // of a B200; only shapes the grids

// MaterialIdToColor of every material word.  The colour is a function of the
// id below 256 and of id % 256 above, so a block puts both tables into shared
// memory, a plane per channel (ids of neighbouring voxels then fall in different
// banks), and a thread writes float `f` of the output from word f / 3: four
// consecutive floats as one 16-byte store, from the output's first 16-byte
// boundary (`head` floats in) on; the floats before it and behind the last tile go
// one by one.  Bound: DRAM, 16 bytes a word.  Measured (B200, 76.8 M words):
// evaluating the palette's branches per word and storing channels one by one 0.531
// ms, tables and 16-byte stores 0.205 ms (6.0 TB/s); 16 / 32 / 64 blocks per SM
// 0.221 / 0.215 / 0.205 ms.  15.4 M words to an output off 16 bytes: single
// stores 128 us, from the boundary on 52 us; aligned 50 us.
constexpr uint32_t PALETTE = 512;  // ids 0..255, then the wheel of ids 256 and up
constexpr uint32_t RGB_TILE = 768;  // 16-byte stores of a tile (1024 words), three a thread

__global__ void __launch_bounds__(256) material_rgb_kernel(const uint32_t* __restrict__ words, uint64_t n,
                                                           uint32_t head, float* __restrict__ rgb) {
    static_assert(PALETTE % 256 == 0, "filled by whole blocks");
    __shared__ float plane[3][PALETTE];
    for (uint32_t i = threadIdx.x; i < PALETTE; i += blockDim.x) {
        const Rgb c = material_color_payload(i);
        plane[0][i] = c.r;
        plane[1][i] = c.g;
        plane[2][i] = c.b;
    }
    __syncthreads();
    auto entry = [](uint32_t id) { return id < 256u ? id : 256u + (id & 255u); };
    const uint64_t tiles = (3 * n - head) / (4 * RGB_TILE);  // head <= 3 n
    const float* p = &plane[0][0];
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t* src = words + tile * 1024;
        float4* dst = reinterpret_cast<float4*>(rgb + head) + tile * RGB_TILE;
#pragma unroll
        for (uint32_t k = 0; k < 3; ++k) {
            const uint32_t q = k * 256 + threadIdx.x, f = head + 4 * q, w = f / 3;
            const uint32_t ch = f - 3 * w;  // 0, 1 or 2: the first float's channel; the fourth has it too, a word on
            const uint32_t a = entry(__ldg(src + w)), b = entry(__ldg(src + w + 1));
            const uint32_t c1 = ch == 2u ? 0u : ch + 1u, c2 = ch == 0u ? 2u : ch - 1u;
            dst[q] = make_float4(p[ch * PALETTE + a], p[c1 * PALETTE + (ch == 2u ? b : a)],
                                 p[c2 * PALETTE + (ch == 0u ? a : b)], p[ch * PALETTE + b]);
        }
    }
    const uint64_t done = 4 * RGB_TILE * tiles;
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < 3 * n - done;
         i += uint64_t(gridDim.x) * blockDim.x) {
        const uint64_t f = i < head ? i : i + done;
        rgb[f] = plane[f % 3][entry(__ldg(words + f / 3))];
    }
}

// A warp takes a run of consecutive bricks, lane k block k of each.  A block's
// encoding is a function of its 64-bit key (dxtn::block_key), and keys repeat:
// of a million occupied blocks of a 512^3 noise scene 37,000 differ, and the 100
// commonest make two thirds.  So a call keeps the results it has: each warp the
// last ones in a direct-mapped table of its own (NRM_WAYS keys and blocks in
// shared memory), all warps together in a table in device memory (NRM_SLOTS
// entries, cleared when the call begins).  Blocks found there are written at
// once; the keys of the others are queued, and when 32 are queued the whole warp
// encodes them, one per lane.  The encoder (about 3,400 instructions) then runs
// for some 5 % of the blocks, with all lanes busy.  Measured (B200, 150,001
// bricks): every block encoded 0.693 ms (513 M warp instructions), the warps'
// own tables alone 0.45 ms, with the device table 0.229 ms (81 M), and 0.235 ms
// with the warps' tables written and read in an order that the memory model
// promises; 64 to 512 ways per warp, before that order, 0.237 / 0.234 / 0.229 /
// 0.278 ms.  Bound: latency, at 36 % issue: of
// fetching the encoder's instructions (the largest stall), of the tables' loads and of
// the encoder's serial chain.
// Blocks that do not repeat pay for the tables and for the fewer warps they leave
// room for: bricks of random voxels at 50 % fill (no two blocks equal) 0.802 -> 0.946 ms
// for 150,001 and 58 -> 74 us for 10,000, at 25 % (40 % equal) 0.681 -> 0.700 ms.  Tried
// against it and slower on noise than it gains there: 5, 6 or 8 blocks per SM with 64
// to 256 ways (noise 0.243 -> 0.275 .. 0.316 ms), and leaving the tables alone for six
// bricks of eight where few blocks were found (0.930, noise 0.256 .. 0.295 ms; with an
// encoder of its own for them 1.06, the code no longer fits the instruction cache).
//
// The device table is one per device and nothing orders its readers and
// writers, warps of this call and of calls on other streams.  So an entry
// carries a 64-bit check of its key and block: whatever mixture of entries a
// lane may read, it takes it only with its own key and the check that belongs
// to all of it (and a key's block is the same whoever encoded it); anything else
// reads as a miss.  The reads go through L1: the commonest keys would otherwise
// be read from the same few lines of L2 by every warp (0.47 against 0.21 ms for
// 150,000 bricks).
constexpr int NRM_SLOT_BITS = 16;
constexpr uint32_t NRM_SLOTS = 1u << NRM_SLOT_BITS;
__device__ ulonglong2 g_normal_table[NRM_SLOTS * 2];  // {key, check}, {block}

__device__ __forceinline__ unsigned long long normal_check(unsigned long long key, unsigned long long a,
                                                           unsigned long long b) {
    unsigned long long x = (key ^ (a * 0x9E3779B97F4A7C15ull)) + (b ^ 0xD6E8FEB86659FD93ull) * 0xC2B2AE3D27D4EB4Full;
    x ^= x >> 29;
    return x * 0xBF58476D1CE4E5B9ull;
}
__device__ __forceinline__ bool read_entry(const ulonglong2* e, unsigned long long key, unsigned long long& a,
                                           unsigned long long& b) {
    unsigned long long k, c;
    asm volatile("ld.global.ca.v2.u64 {%0, %1}, [%2];" : "=l"(k), "=l"(c) : "l"(e) : "memory");
    asm volatile("ld.global.ca.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(e + 1) : "memory");
    return k == key && c == normal_check(key, a, b);
}

__global__ void __launch_bounds__(256) clear_normal_table_kernel() {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < NRM_SLOTS * 2; i += gridDim.x * blockDim.x)
        g_normal_table[i] = make_ulonglong2(0ull, 0ull);
}

constexpr int NRM_WARPS = 4;
constexpr int NRM_BLOCKS = 4;  // per SM: 3 / 4 / 5 / 6 take 0.242 / 0.228 / 0.264 / 0.274 ms for 150,001 bricks
constexpr int NRM_WAY_BITS = 8;
constexpr uint32_t NRM_WAYS = 1u << NRM_WAY_BITS;

struct NormalWarp {
    uint4 block[NRM_WAYS];
    uint2 key[NRM_WAYS];      // 0: empty (no occupied block has key 0)
    uint2 queue_key[64];
    uint32_t queue_at[64];    // block's place in the warp's run
};

__global__ void __launch_bounds__(NRM_WARPS * 32, NRM_BLOCKS) build_normals_kernel(const uint32_t* __restrict__ occ,
                                                                       uint32_t bricks, uint32_t per_warp,
                                                                       uint4* __restrict__ out) {
    extern __shared__ uint4 dyn[];
    __shared__ float4 tab[dxtn::NUM_CODES];
    const uint32_t lane = threadIdx.x & 31u;
    NormalWarp& w = reinterpret_cast<NormalWarp*>(dyn)[threadIdx.x >> 5];
    if (threadIdx.x < dxtn::NUM_CODES) tab[threadIdx.x] = dxtn::code_entry(int(threadIdx.x));
    for (uint32_t i = lane; i < NRM_WAYS; i += 32) w.key[i] = make_uint2(0u, 0u);
    __syncthreads();
    const dxtn::CodeTable lookup{tab};
    const uint64_t first = (uint64_t(blockIdx.x) * NRM_WARPS + (threadIdx.x >> 5)) * per_warp;  // the warp's bricks
    // only the top bits of a product depend on all bits of the key, whose bytes are mostly 0 or 255
    auto hash = [](uint2 k) {
        const uint32_t h = (k.x * 0x9E3779B1u) ^ (k.y * 0x85EBCA77u);
        return (h ^ (h >> 15)) * 0x2C1B3C6Du;
    };
    // a multiplier per warp: two common keys that share a way do so in few warps, not in all of
    // them (which would then all read the same lines of the device table)
    const uint32_t mult = ((blockIdx.x * NRM_WARPS + (threadIdx.x >> 5)) * 0x9E3779B2u) | 1u;
    auto way = [&](uint32_t h) { return (h * mult) >> (32 - NRM_WAY_BITS); };
    auto slot = [](uint32_t h) { return g_normal_table + 2 * size_t(h >> (32 - NRM_SLOT_BITS)); };
    // Keeps a result of each of `lanes`, the lanes that call it, in the warp's table:
    // one of the lanes that share a way writes its key and block.  The mask comes from a
    // vote of the whole warp (or is a queue's length), never from who happens to arrive
    // together: two parties of one branch would each elect a writer for a way, and the
    // key of one could end up with the block of the other.
    auto keep = [&](uint32_t lanes, uint2 k, uint32_t h, uint4 v) {
        const uint32_t group = __match_any_sync(lanes, way(h));
        if (uint32_t(__ffs(int(group)) - 1) == lane) {
            w.key[way(h)] = k;
            w.block[way(h)] = v;
        }
    };
    uint32_t queued = 0;  // warp-uniform
    // encodes the queue's last n <= 32 keys, one per lane; the queue's and the table's
    // writes before it are ordered by the caller's __syncwarp, its own by the one at its end
    auto drain = [&](uint32_t n) {
        queued -= n;
        if (lane < n) {
            const uint2 k = w.queue_key[queued + lane];
            uint8_t code[16];
            dxtn::key_codes(uint64_t(k.x) | (uint64_t(k.y) << 32), code);
            uint64_t a, b;
            dxtn::encode_coded(code, lookup, a, b);
            const uint4 v = make_uint4(uint32_t(a), uint32_t(a >> 32), uint32_t(b), uint32_t(b >> 32));
            out[first * 32 + w.queue_at[queued + lane]] = v;
            const uint32_t h = hash(k);
            keep(0xFFFFFFFFu >> (32u - n), k, h, v);
            const unsigned long long key = (unsigned long long)(k.x) | ((unsigned long long)(k.y) << 32);
            slot(h)[0] = make_ulonglong2(key, normal_check(key, a, b));
            slot(h)[1] = make_ulonglong2(a, b);
        }
        __syncwarp();
    };
    const uint32_t end = uint32_t(min(first + per_warp, uint64_t(bricks)));
    for (uint32_t brick = uint32_t(min(first, uint64_t(bricks))); brick < end; ++brick) {
        const uint64_t key = dxtn::block_key(occ + uint64_t(brick) * 16, int(lane));
        const uint2 k = make_uint2(uint32_t(key), uint32_t(key >> 32));
        const uint32_t h = hash(k), at = way(h);
        const uint2 have = w.key[at];
        bool found = have.x == k.x && have.y == k.y;
        const uint64_t i = uint64_t(brick) * 32 + lane;
        if (!key) out[i] = make_uint4(0u, 0u, 0u, 0u);
        else if (found) out[i] = w.block[at];
        unsigned long long a = 0, b = 0;
        const bool known = key && !found && read_entry(slot(h), key, a, b);
        __syncwarp();  // every lane has read the warp's table, which now changes
        const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, known);
        if (known) {
            const uint4 v = make_uint4(uint32_t(a), uint32_t(a >> 32), uint32_t(b), uint32_t(b >> 32));
            out[i] = v;
            keep(lanes, k, h, v);
            found = true;
        }
        const uint32_t miss = __ballot_sync(0xFFFFFFFFu, key && !found);
        if (key && !found) {
            const uint32_t q = queued + __popc(miss & ((1u << lane) - 1u));
            w.queue_key[q] = k;
            w.queue_at[q] = uint32_t(i - first * 32);
        }
        queued += __popc(miss);
        __syncwarp();  // votes order no memory: the table and the queue are read by other lanes next
        if (queued >= 32) drain(32);
    }
    if (queued) drain(queued);
}

// Few bricks: a thread per block, no tables.  The tables pay once a brick finds
// most of its blocks there; below that the queue's serial encodings cost more than
// they save.  This way and with the tables in runs of two: 3,000 bricks 21 and 28 us;
// 8,192 of 512^3 / 256^3 / 192^3 / 128^3 noise 40 and 40 / 42 and 47 / 42 and 48 / 44 and
// 44; 12,000 of them 57 and 50 / 60 and 57 / 60 and 60 / 62 and 53.  Runs of one wave
// are longer, find more in their warp's table and keep fewer warps busy: 20,000 bricks
// of 512^3 / 256^3 noise 72 / 95 us with them and 74 / 80 in runs of two, 45,000 bricks
// 116 / 142 and 140 / 149.
constexpr uint32_t NRM_DIRECT = 8192;
__global__ void __launch_bounds__(128) build_normals_direct_kernel(const uint32_t* __restrict__ occ, uint32_t blocks,
                                                                   uint4* __restrict__ out) {
    __shared__ float4 tab[dxtn::NUM_CODES];
    if (threadIdx.x < dxtn::NUM_CODES) tab[threadIdx.x] = dxtn::code_entry(int(threadIdx.x));
    __syncthreads();
    const uint32_t i = blockIdx.x * 128 + threadIdx.x;
    if (i >= blocks) return;
    uint64_t a, b;
    dxtn::brick_block(occ + (i >> 5) * 16, int(i & 31), dxtn::CodeTable{tab}, a, b);
    out[i] = make_uint4(uint32_t(a), uint32_t(a >> 32), uint32_t(b), uint32_t(b >> 32));
}

// One warp per brick: the brick's 512 RGB texels (6 KiB) are copied to shared
// memory (16-byte asynchronous copies when the colours are 16-byte aligned)
// with a 52-word stride per 16-texel block, so that the lanes' 16-byte texel
// reads (lane k = block k) fall in different banks; lane k then encodes block k
// and the warp writes its 256 output bytes contiguously.  Bound: the FMA pipe, whose
// packed operations take two cycles (68 % busy, issue 56 %).  Measured (B200, 150,001 bricks of materials): scalar searches with
// indices 0.465 ms (445 M warp instructions), pairs 0.363 ms, empty texels
// cleared in registers instead of shared memory 0.337 ms; a second buffer per
// warp, the next brick arriving during the encoding, 0.347 ms (fewer warps fit);
// 3 / 4 / 5 / 6 blocks per SM 0.343 / 0.337 / 0.335 / 0.339 ms.
constexpr int DXT1_WARPS = 4;
constexpr int DXT1_BLOCKS = 4;  // per SM
constexpr int DXT1_STRIDE = 52;

// dxt1::encode16 with the texels in pairs (dxt1::dist2 of two texels in packed
// operations, each half rounded as the scalar one), the same block:
//  - the farthest pair: first the greatest distance, by maxima without indices,
//    then the first i whose row holds it and the first j > i in that row.  Row i
//    also takes the distance of texel i to itself, +0 (or NaN, which a maximum
//    ignores): no distance is below +0, so it changes no maximum of a row with a
//    later texel at a finite distance, and where the greatest distance is 0 the
//    first row with a finite texel has one;
//  - the nearest reference: the first smallest of four.
__device__ __forceinline__ float2 dist2_pair(float2 ar, float2 ag, float2 ab, float2 br, float2 bg, float2 bb,
                                             float nz) {
    const float2 x = sub2(ar, br), y = sub2(ag, bg), z = sub2(ab, bb);
    return __fadd2_rn(__fadd2_rn(mul2(x, x, nz), mul2(y, y, nz)), mul2(z, z, nz));
}

__device__ __forceinline__ uint64_t encode_block_pairs(const float* p, uint32_t occupied, float nz) {
    float2 r[8], g[8], b[8];  // texels 2k, 2k + 1
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // 4 texels = 12 floats = 3 16-byte words
        const float4 u = reinterpret_cast<const float4*>(p)[3 * q], v = reinterpret_cast<const float4*>(p)[3 * q + 1],
                     w = reinterpret_cast<const float4*>(p)[3 * q + 2];
        r[2 * q] = make_float2(u.x, u.w);
        g[2 * q] = make_float2(u.y, v.x);
        b[2 * q] = make_float2(u.z, v.y);
        r[2 * q + 1] = make_float2(v.z, w.y);
        g[2 * q + 1] = make_float2(v.w, w.z);
        b[2 * q + 1] = make_float2(w.x, w.w);
    }
    // empty texels are (0, 0, 0) (the rebuild's input for them)
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (!((occupied >> (2 * k)) & 1u)) r[k].x = g[k].x = b[k].x = 0.0f;
        if (!((occupied >> (2 * k + 1)) & 1u)) r[k].y = g[k].y = b[k].y = 0.0f;
    }
    auto texel = [&](int t) {
        return (occupied >> t) & 1u ? dxt1::texel(p, t) : dxt1::C3{0.0f, 0.0f, 0.0f};
    };
    auto part = [](const float2* v, int i) { return i & 1 ? v[i >> 1].y : v[i >> 1].x; };
    const float LOWEST = -3.402823466e+38f;
    float row[15], best = LOWEST;
#pragma unroll
    for (int i = 0; i < 15; ++i) {
        const float2 ir = dup2(part(r, i)), ig = dup2(part(g, i)), ib = dup2(part(b, i));
        row[i] = LOWEST;
#pragma unroll
        for (int k = (i + (i & 1)) / 2; k < 8; ++k) {  // odd i: pairs from i + 1 on; even i: pair (i, i + 1) too
            const float2 d = dist2_pair(ir, ig, ib, r[k], g[k], b[k], nz);
            row[i] = fmaxf(fmaxf(row[i], d.x), d.y);
        }
        best = fmaxf(best, row[i]);
    }
    int i0 = 15;
#pragma unroll
    for (int i = 14; i >= 0; --i)
        if (row[i] == best) i0 = i;
    // the first j > i0 at that distance; none (all distances NaN): texels (0, 0)
    int i1 = 16;
    {
        const dxt1::C3 c = texel(i0);
        const float2 ir = dup2(c.r), ig = dup2(c.g), ib = dup2(c.b);
#pragma unroll
        for (int k = 7; k >= 0; --k) {
            const float2 d = dist2_pair(ir, ig, ib, r[k], g[k], b[k], nz);
            if (d.y == best && 2 * k + 1 > i0) i1 = 2 * k + 1;
            if (d.x == best && 2 * k > i0) i1 = 2 * k;
        }
    }
    if (i1 == 16) i0 = i1 = 0;
    const uint32_t head = dxt1::encode_head(texel(i0), texel(i1));
    dxt1::C3 ref[4];
    dxt1::decode_head(head, ref);
    uint32_t bits = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float2 d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) d[j] = dist2_pair(r[k], g[k], b[k], dup2(ref[j].r), dup2(ref[j].g), dup2(ref[j].b),
                                                         nz);
        auto nearest = [](float d0, float d1, float d2, float d3) {
            uint32_t bi = d1 < d0 ? 1u : 0u;
            float bd = fminf(d0, d1);
            if (d2 < bd) bi = 2u;
            bd = fminf(bd, d2);
            return d3 < bd ? 3u : bi;
        };
        bits |= nearest(d[0].x, d[1].x, d[2].x, d[3].x) << (4 * k);
        bits |= nearest(d[0].y, d[1].y, d[2].y, d[3].y) << (4 * k + 2);
    }
    return uint64_t(head) | (uint64_t(bits) << 32);
}

template <bool VEC>
__global__ void __launch_bounds__(DXT1_WARPS * 32, DXT1_BLOCKS) build_dxt1_kernel(const float* __restrict__ rgb,
                                                                     const uint32_t* __restrict__ occ,
                                                                     uint64_t bricks, float neg_zero,
                                                                     uint64_t* __restrict__ out) {
    extern __shared__ float4 stage4[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* stage = reinterpret_cast<float*>(stage4) + warp * (32 * DXT1_STRIDE);
    for (uint64_t brick = uint64_t(blockIdx.x) * DXT1_WARPS + warp; brick < bricks;
         brick += uint64_t(gridDim.x) * DXT1_WARPS) {
        const uint32_t o = __ldg(occ + brick * 16 + (lane >> 1));
        const float* src = rgb + brick * 1536;
        if constexpr (VEC) {
#pragma unroll
            for (int k = 0; k < 12; ++k) {  // 12 16-byte words per block
                const int q = lane + 32 * k;
                const uint32_t at = uint32_t(__cvta_generic_to_shared(stage + (q / 12) * DXT1_STRIDE + (q % 12) * 4));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(at), "l"(src + 4 * q) : "memory");
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        } else {
            for (int f = lane; f < 1536; f += 32) stage[(f / 48) * DXT1_STRIDE + f % 48] = __ldg(src + f);
        }
        __syncwarp();
        const uint32_t mask = (o >> ((lane & 1) * 16)) & 0xFFFFu;
        out[brick * 32 + lane] = mask ? encode_block_pairs(stage + lane * DXT1_STRIDE, mask, neg_zero) : 0ull;
        __syncwarp();  // the stage is free for the next brick
    }
}

// normalize(decode) of each hit voxel's texel; zeros on a miss or an LOD hit.
__global__ void __launch_bounds__(256) hit_normals_kernel(DevScene s, const uint4* __restrict__ hits, uint32_t n,
                                                          float* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint4 h = __ldg(hits + i);
    float x = 0.0f, y = 0.0f, z = 0.0f;
    const uint32_t flags = (h.w >> 16) & 0xFFu;
    if ((flags & F_HIT) && h.y != NONE) dxt_normal(s, h.y, h.w & 0xFFFFu, x, y, z);
    out[size_t(i) * 3] = x;
    out[size_t(i) * 3 + 1] = y;
    out[size_t(i) * 3 + 2] = z;
}

int cuda_err(cudaError_t e, const char* what) {
    return fail(VX_ECUDA, std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")");
}

}  // namespace
}  // namespace vx

extern "C" int vx_build_normals_dev(const uint32_t* occ_dev, uint32_t brick_count, uint64_t* out_dev, void* stream) {
    using namespace vx;
    if (brick_count && (!occ_dev || !out_dev)) return fail(VX_EINVAL, "vx_build_normals_dev: null argument");
    if (reinterpret_cast<uintptr_t>(occ_dev) % 16 || reinterpret_cast<uintptr_t>(out_dev) % 16)
        return fail(VX_EINVAL, "vx_build_normals_dev: buffers need 16-byte alignment");
    if (brick_count == 0) return VX_OK;
    const size_t smem = NRM_WARPS * sizeof(NormalWarp);
    static_assert(NRM_WARPS * sizeof(NormalWarp) <= 48 * 1024, "within a launch's default shared memory");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint4* out = reinterpret_cast<uint4*>(out_dev);
    if (brick_count < NRM_DIRECT) {
        build_normals_direct_kernel<<<brick_count / 4 + 1, 128, 0, st>>>(occ_dev, brick_count * 32, out);
    } else {
        // one wave of warps, each with a run of bricks; two waves of short runs while the runs would be short anyway
        const uint64_t warps = uint64_t(SMS) * NRM_BLOCKS * NRM_WARPS;
        const uint32_t per_warp = brick_count < 2 * NRM_DIRECT ? 2u : uint32_t((brick_count + warps - 1) / warps);
        const uint64_t run = uint64_t(per_warp) * NRM_WARPS;
        clear_normal_table_kernel<<<SMS, 256, 0, st>>>();
        build_normals_kernel<<<uint32_t((brick_count + run - 1) / run), NRM_WARPS * 32, smem, st>>>(occ_dev, brick_count,
                                                                                                   per_warp, out);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VX_OK : cuda_err(e, "vx_build_normals_dev");
}

static int vx_build_normals_body(const uint32_t* occ, uint32_t brick_count, uint64_t* out) {
    using namespace vx;
    if (brick_count && (!occ || !out)) return fail(VX_EINVAL, "vx_build_normals: null argument");
    const unsigned T = std::max(1u, std::min(64u, std::thread::hardware_concurrency()));
    float4 tab[dxtn::NUM_CODES];
    for (int c = 0; c < dxtn::NUM_CODES; ++c) tab[c] = dxtn::code_entry(c);
    const dxtn::CodeTable lookup{tab};
    auto work = [&](uint64_t b0, uint64_t b1) {
        for (uint64_t b = b0; b < b1; ++b)
            for (int k = 0; k < 32; ++k)
                dxtn::brick_block(occ + 16 * b, k, lookup, out[(b * 32 + k) * 2], out[(b * 32 + k) * 2 + 1]);
    };
    if (T == 1 || brick_count < 256) {
        work(0, brick_count);
        return VX_OK;
    }
    std::vector<std::thread> th;
    const uint64_t chunk = (uint64_t(brick_count) + T - 1) / T;
    for (unsigned t = 0; t < T; ++t) {
        const uint64_t b0 = uint64_t(t) * chunk, b1 = std::min<uint64_t>(brick_count, b0 + chunk);
        if (b0 >= b1) break;
        th.emplace_back(work, b0, b1);
    }
    for (auto& x : th) x.join();
    return VX_OK;
}

extern "C" int vx_build_normals(const uint32_t* occ, uint32_t brick_count, uint64_t* out) {
    return vx::guarded("vx_build_normals", [&] { return vx_build_normals_body(occ, brick_count, out); });
}

extern "C" int vx_build_dxt1_dev(const float* rgb_dev, const uint32_t* occ_dev, uint32_t brick_count,
                                 uint64_t* out_dev, void* stream) {
    using namespace vx;
    if (brick_count && (!rgb_dev || !occ_dev || !out_dev)) return fail(VX_EINVAL, "vx_build_dxt1_dev: null argument");
    if (reinterpret_cast<uintptr_t>(occ_dev) % 16 || reinterpret_cast<uintptr_t>(out_dev) % 8 ||
        reinterpret_cast<uintptr_t>(rgb_dev) % 4)
        return fail(VX_EINVAL, "vx_build_dxt1_dev: misaligned buffer");
    if (brick_count == 0) return VX_OK;
    const size_t smem = size_t(DXT1_WARPS) * 32 * DXT1_STRIDE * sizeof(float);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto* kernel = reinterpret_cast<uintptr_t>(rgb_dev) % 16 == 0 ? build_dxt1_kernel<true> : build_dxt1_kernel<false>;
    static_assert(DXT1_WARPS * 32 * DXT1_STRIDE * sizeof(float) <= 48 * 1024, "within a launch's default shared memory");
    const uint32_t grid = uint32_t(std::min<uint64_t>((uint64_t(brick_count) + DXT1_WARPS - 1) / DXT1_WARPS,
                                                      uint64_t(SMS) * DXT1_BLOCKS));
    kernel<<<grid, DXT1_WARPS * 32, smem, st>>>(rgb_dev, occ_dev, brick_count, -0.0f, out_dev);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VX_OK : cuda_err(e, "vx_build_dxt1_dev");
}

static int vx_build_dxt1_body(const float* rgb, const uint32_t* occ, uint32_t brick_count, uint64_t* out) {
    using namespace vx;
    if (brick_count && (!rgb || !occ || !out)) return fail(VX_EINVAL, "vx_build_dxt1: null argument");
    const unsigned T = std::max(1u, std::min(64u, std::thread::hardware_concurrency()));
    auto work = [&](uint64_t b0, uint64_t b1) {
        for (uint64_t b = b0; b < b1; ++b)
            for (int k = 0; k < 32; ++k) out[b * 32 + k] = dxt1::brick_block(rgb + b * 512 * 3, occ + 16 * b, k);
    };
    if (T == 1 || brick_count < 256) {
        work(0, brick_count);
        return VX_OK;
    }
    std::vector<std::thread> th;
    const uint64_t chunk = (uint64_t(brick_count) + T - 1) / T;
    for (unsigned t = 0; t < T; ++t) {
        const uint64_t b0 = uint64_t(t) * chunk, b1 = std::min<uint64_t>(brick_count, b0 + chunk);
        if (b0 >= b1) break;
        th.emplace_back(work, b0, b1);
    }
    for (auto& x : th) x.join();
    return VX_OK;
}

extern "C" int vx_build_dxt1(const float* rgb, const uint32_t* occ, uint32_t brick_count, uint64_t* out) {
    return vx::guarded("vx_build_dxt1", [&] { return vx_build_dxt1_body(rgb, occ, brick_count, out); });
}

static int vx_material_rgb_body(const uint32_t* words, uint64_t n, float* rgb) {
    if (n && (!words || !rgb)) return vx::fail(VX_EINVAL, "vx_material_rgb: null argument");
    const unsigned T = std::max(1u, std::min(64u, std::thread::hardware_concurrency()));
    auto work = [&](uint64_t a, uint64_t b) {
        for (uint64_t i = a; i < b; ++i) {
            const vx::Rgb c = vx::material_color_payload(words[i]);
            rgb[3 * i] = c.r;
            rgb[3 * i + 1] = c.g;
            rgb[3 * i + 2] = c.b;
        }
    };
    if (T == 1 || n < (uint64_t(1) << 16)) {
        work(0, n);
        return VX_OK;
    }
    std::vector<std::thread> th;
    const uint64_t chunk = (n + T - 1) / T;
    for (unsigned t = 0; t < T; ++t) {
        const uint64_t a = uint64_t(t) * chunk, b = std::min(n, a + chunk);
        if (a >= b) break;
        th.emplace_back(work, a, b);
    }
    for (auto& x : th) x.join();
    return VX_OK;
}

extern "C" int vx_material_rgb(const uint32_t* words, uint64_t n, float* rgb) {
    return vx::guarded("vx_material_rgb", [&] { return vx_material_rgb_body(words, n, rgb); });
}

extern "C" int vx_material_rgb_dev(const uint32_t* words, uint64_t n, float* rgb, void* stream) {
    using namespace vx;
    if (n && (!words || !rgb)) return fail(VX_EINVAL, "vx_material_rgb_dev: null argument");
    if (reinterpret_cast<uintptr_t>(words) % 4 || reinterpret_cast<uintptr_t>(rgb) % 4)
        return fail(VX_EINVAL, "vx_material_rgb_dev: misaligned buffer");
    if (n == 0) return VX_OK;
    // one wave of blocks (each fills its tables first); more once a block has four tiles all the same
    const uint64_t tiles = (n + 1023) / 1024;
    const unsigned blocks = unsigned(std::max(std::min<uint64_t>(tiles, SMS * 8), std::min<uint64_t>(tiles / 4, SMS * 64)));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t head = uint32_t(16 - reinterpret_cast<uintptr_t>(rgb) % 16) % 16 / 4;  // floats: at most 3 <= 3 n
    material_rgb_kernel<<<blocks, 256, 0, st>>>(words, n, head, rgb);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VX_OK : cuda_err(e, "vx_material_rgb_dev");
}

extern "C" int vx_hit_normals(const vx_scene* scene, const vx_hit* hits_dev, uint32_t n, float* normals_dev,
                              void* stream) {
    using namespace vx;
    if (!scene || (n && (!hits_dev || !normals_dev))) return fail(VX_EINVAL, "vx_hit_normals: null argument");
    const DevScene& s = scene_dev(scene);
    if (!s.nrm) return fail(VX_EINVAL, "vx_hit_normals: the scene has no normal payload");
    if (reinterpret_cast<uintptr_t>(hits_dev) % 16 || reinterpret_cast<uintptr_t>(normals_dev) % 4)
        return fail(VX_EINVAL, "vx_hit_normals: misaligned buffer");
    if (n == 0) return VX_OK;
    hit_normals_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        s, reinterpret_cast<const uint4*>(hits_dev), n, normals_dev);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VX_OK : cuda_err(e, "vx_hit_normals");
}

namespace vx {
VX_VIOLATION_READER(violations_payload)
}  // namespace vx
