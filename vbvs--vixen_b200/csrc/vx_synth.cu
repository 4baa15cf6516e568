// vx_synth.cu - the value-noise occupancy generator on the device.
//
// Produces exactly the bits of vx_synth_noise (vx_build.cpp): the same lattice
// hash, the same binary32 operation order per voxel (the kernels are built
// with --fmad=false), and the same threshold, the value of ascending rank
// N - round(fill * N), found by a radix select over the values' bit patterns.
//
// The field is not stored: it is computed twice, once for a histogram of the
// values' top 16 bits and once for the occupancy bits, where only the values in
// the threshold's bin (1 to 2 % of a noise field) have to wait for the exact
// threshold as candidates.  What a value costs decides: interpolating the
// lattice along z and y is the same for a whole row, so a block does it once
// per lattice cell of 8 rows (tile) and each voxel is left with one
// interpolation along x per octave, four rows at a time in packed pairs.  Bound:
// instruction issue (70 %).  Measured (B200, 512^3, 3 octaves) against a thread
// per voxel with a stored field, three histogram passes over it and a pack pass:
// field 2.49 + histograms 0.68 + pack 0.48 ms -> histogram 0.21 + bits 0.29 ms and
// 0.05 ms for the select; the whole call, allocations included, 5.78 -> 1.27 ms,
// and 33 MiB of scratch instead of 512.
#include <algorithm>
#include <cstdint>
#include <vector>

#include "vx_hash.h"
#include "vx_internal.h"
#include "vx_pairs.cuh"

namespace vx {
namespace {

constexpr uint32_t MAX_OCT = 16;
constexpr uint32_t THREADS = 256;
constexpr uint32_t TILE_ROWS = 8;      // rows (consecutive y, one z) per tile; R is a multiple of 64
constexpr uint32_t QUADS = TILE_ROWS / 4;
// Values are in [0, 2): bit patterns below 0x40000000.  The first histogram is
// over the top 16 bits from 2^-15 up (its bin 0 takes everything below), so
// that it needs 8 KiB per block and five blocks fit on an SM; a refining one
// has a bin for each 14-bit digit.
constexpr uint32_t FIRST_BASE = 0x3800, FIRST_BINS = 0x4000 - FIRST_BASE;
constexpr uint32_t HIST_BINS = 16384;
constexpr uint32_t CAND_BUFFER = 2048;  // candidates a block gathers before it writes them out
constexpr uint32_t LOW_BINS = 65536;
// Dynamic shared memory the kernels may be launched with.  The rows of the octaves
// have 4,131 cells at most (R = 2048, 16 octaves of spacings 32768 down to 1): a
// refining histogram of 64 KiB and 8 * 4 * 4,131 bytes of cells make 197,728.  One
// value for every call: the attribute belongs to the kernel, not to a launch, and a
// call on another thread must find it no smaller than it needs.
constexpr uint32_t NOISE_SMEM = 200 * 1024;

struct OctDev {
    uint32_t s, cells;
    uint32_t first;  // of the octave's cells in a row of all octaves' cells
    float amp;
    const float* lat;
};
struct NoiseParams {
    uint32_t R, octaves, row_cells;  // row_cells: cells of all octaves
    float neg_zero;       // -0 (vx_pairs.cuh)
    const uint2* column;  // [octave][x]: place in a row's cells, weight along x
    OctDev oct[MAX_OCT];
};

// What the select kernels leave for the next steps.
struct Selected {
    unsigned long long rank;   // rank of the threshold among the values of the chosen bin
    unsigned long long count;  // values in it
    uint32_t bin;
    uint32_t candidates;       // written so far
};

// Cell and smooth weight of coordinate v at lattice spacing s, as the host row
// loop computes them.
__device__ __forceinline__ void cell_of(uint32_t v, uint32_t s, uint32_t& cell, float& w) {
    const float p = (float(v) + 0.5f) / float(s);
    const float c = floorf(p);
    const float f = p - c;
    w = f * f * (3.0f - 2.0f * f);
    cell = uint32_t(c);
}

// The lattices of all octaves and the column table.
__global__ void lattice_kernel(NoiseParams p, float* lat, uint64_t total, uint2* column, uint64_t seed) {
    const uint64_t first = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x, step = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t t = first; t < total; t += step) {
        uint32_t o = 0;
        while (o + 1 < p.octaves && lat + t >= p.oct[o + 1].lat) ++o;
        const uint64_t u = uint64_t(lat + t - p.oct[o].lat), c = p.oct[o].cells;
        if (u >= c * c * c) continue;  // between two octaves
        const uint32_t i = uint32_t(u % c), j = uint32_t((u / c) % c), k = uint32_t(u / (c * c));
        lat[t] = float(hash4(seed, o, i, j, k) >> 40) * (1.0f / 16777216.0f);
    }
    for (uint64_t t = first; t < uint64_t(p.octaves) * p.R; t += step) {
        const uint32_t o = uint32_t(t / p.R);
        uint32_t cell;
        float w;
        cell_of(uint32_t(t % p.R), p.oct[o].s, cell, w);
        column[t] = make_uint2(p.oct[o].first + cell, __float_as_uint(w));
    }
}

// The values of all voxels, tile by tile (TILE_ROWS rows of one z slice, all
// columns).  use(bits, x, y, z, word) gets the bit patterns of four rows y ..
// y + 3 at column x, called by whole warps whose lanes hold 32 consecutive x;
// word: the 32-voxel word of the first row.  after_tile() runs with the block
// in step after every tile.
// OCT: octaves the registers hold (p.octaves at most).
template <uint32_t OCT, class Use, class After>
__device__ __forceinline__ void for_each_value(const NoiseParams& p, float4* cells, Use use, After after_tile) {
    __shared__ uint32_t row_j[MAX_OCT][TILE_ROWS], slice_k[MAX_OCT];
    __shared__ float row_w[MAX_OCT][TILE_ROWS], slice_w[MAX_OCT];
    const uint32_t R = p.R, C = p.row_cells;
    const uint32_t tiles_y = R / TILE_ROWS;
    const uint32_t width = min(R, THREADS), groups = THREADS / width;  // R < 256: several quads side by side
    const uint32_t col = threadIdx.x % width, group = threadIdx.x / width;
    // cells and weights of a tile's rows and slice, read by the step along z and y only
    auto rows_of = [&](uint32_t tile) {
        const uint32_t z = tile / tiles_y, y0 = (tile - z * tiles_y) * TILE_ROWS;
        if (threadIdx.x < p.octaves * TILE_ROWS) {
            const uint32_t o = threadIdx.x / TILE_ROWS, y = threadIdx.x % TILE_ROWS;
            cell_of(y0 + y, p.oct[o].s, row_j[o][y], row_w[o][y]);
        } else if (threadIdx.x - p.octaves * TILE_ROWS < p.octaves) {
            const uint32_t o = threadIdx.x - p.octaves * TILE_ROWS;
            cell_of(z, p.oct[o].s, slice_k[o], slice_w[o]);
        }
    };
    if (blockIdx.x < tiles_y * R) rows_of(blockIdx.x);
    __syncthreads();
    for (uint32_t tile = blockIdx.x; tile < tiles_y * R; tile += gridDim.x) {
        const uint32_t z = tile / tiles_y, y0 = (tile - z * tiles_y) * TILE_ROWS;
        // Along z and y, once per lattice cell and row: a thread takes a cell for
        // four rows and reads the lattice when the row's cell changes.
        // cells[c * QUADS + q] holds rows 4q .. 4q + 3 of cell c.
        for (uint32_t e = threadIdx.x; e < QUADS * C; e += THREADS) {
            const uint32_t c = e < C ? e : e - C, q = e < C ? 0u : 1u;
            uint32_t o = 0;
            while (o + 1 < p.octaves && c >= p.oct[o + 1].first) ++o;
            const uint32_t i = c - p.oct[o].first, n = p.oct[o].cells;
            const float* lo = p.oct[o].lat + size_t(slice_k[o]) * n * n + i;
            const float* hi = lo + size_t(n) * n;
            const float wz = slice_w[o];
            float a0 = 0.0f, b0 = 0.0f, a1 = 0.0f, b1 = 0.0f, lz[4];
            uint32_t j_read = 0xFFFFFFFFu;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                const uint32_t j = row_j[o][q * 4 + k];
                if (j != j_read) {
                    a0 = __ldg(lo + size_t(j) * n);
                    b0 = __ldg(lo + size_t(j + 1) * n);
                    a1 = __ldg(hi + size_t(j) * n);
                    b1 = __ldg(hi + size_t(j + 1) * n);
                    j_read = j;
                }
                const float wy = row_w[o][q * 4 + k];
                const float ly0 = a0 + wy * (b0 - a0);
                const float ly1 = a1 + wy * (b1 - a1);
                lz[k] = ly0 + wz * (ly1 - ly0);
            }
            cells[c * QUADS + q] = make_float4(lz[0], lz[1], lz[2], lz[3]);
        }
        __syncthreads();
        for (uint32_t x0 = 0; x0 < R; x0 += width) {
            const uint32_t x = x0 + col;
            if (x < R && group < groups) {
                const float4* at[OCT];
                float2 wx[OCT];
#pragma unroll
                for (uint32_t o = 0; o < OCT; ++o)
                    if (o < p.octaves) {
                        const uint2 t = __ldg(p.column + o * R + x);
                        at[o] = cells + t.x * QUADS;
                        wx[o] = make_float2(__uint_as_float(t.y), __uint_as_float(t.y));
                    }
#pragma unroll 2
                for (uint32_t q = group; q < QUADS; q += groups) {
                    float2 out[2];
#pragma unroll
                    for (uint32_t o = 0; o < OCT; ++o)
                        if (o < p.octaves) {
                            const float4 a = at[o][q], b = at[o][QUADS + q];
                            const float2 a2[2] = {make_float2(a.x, a.y), make_float2(a.z, a.w)};
                            const float2 b2[2] = {make_float2(b.x, b.y), make_float2(b.z, b.w)};
                            const float2 amp = make_float2(p.oct[o].amp, p.oct[o].amp);
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                const float2 v = __fadd2_rn(a2[k], mul2(wx[o], sub2(b2[k], a2[k]), p.neg_zero));
                                // octave 0 has amplitude 1: 0 + 1 * v is v (no value is -0)
                                out[k] = o == 0 ? v : __fadd2_rn(out[k], mul2(amp, v, p.neg_zero));
                            }
                        }
                    const uint32_t bits[4] = {__float_as_uint(out[0].x), __float_as_uint(out[0].y),
                                              __float_as_uint(out[1].x), __float_as_uint(out[1].y)};
                    const uint32_t y = y0 + q * 4;
                    use(bits, x, y, z, (z * R + y) * (R / 32) + x / 32);  // R <= 2048: the word index is below 2^28
                }
            }
        }
        if (tile + gridDim.x < tiles_y * R) rows_of(tile + gridDim.x);
        __syncthreads();
        after_tile();
    }
}

// FIRST: histogram of the values' top 16 bits, FIRST_BASE and below in bin 0;
// else of (bits >> shift) & (HIST_BINS - 1) over the values whose bits match
// prefix under mask.  One shared-memory histogram per persistent block.
template <uint32_t OCT, bool FIRST>
__global__ void __launch_bounds__(THREADS) noise_histogram_kernel(const __grid_constant__ NoiseParams p, uint32_t mask,
                                                                  uint32_t prefix, int shift,
                                                                  unsigned long long* __restrict__ out) {
    extern __shared__ uint4 dyn[];
    constexpr uint32_t BINS = FIRST ? FIRST_BINS : HIST_BINS;
    uint32_t* hist = reinterpret_cast<uint32_t*>(dyn);
    float4* cells = reinterpret_cast<float4*>(hist + BINS);
    for (uint32_t b = threadIdx.x; b < BINS; b += THREADS) hist[b] = 0u;
    __syncthreads();
    for_each_value<OCT>(
        p, cells,
        [&](const uint32_t (&bits)[4], uint32_t, uint32_t, uint32_t, uint32_t) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if constexpr (FIRST)
                    atomicAdd(&hist[min(max(bits[k] >> 16, FIRST_BASE) - FIRST_BASE, FIRST_BINS - 1u)], 1u);
                else if ((bits[k] & mask) == prefix)
                    atomicAdd(&hist[(bits[k] >> shift) & (HIST_BINS - 1u)], 1u);
            }
        },
        [] {});
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < BINS; b += THREADS)
        if (hist[b]) atomicAdd(out + b, (unsigned long long)hist[b]);
}

// Occupancy bits: values from solid_from up are solid, values in
// [lo, solid_from) become candidates {bit index << 16 | low 16 bits}, gathered
// per block and written out when the buffer is half full (a tile with more
// than it holds writes the rest one by one).
template <uint32_t OCT>
__global__ void __launch_bounds__(THREADS) noise_bits_kernel(const __grid_constant__ NoiseParams p, uint32_t lo,
                                                             uint32_t solid_from, int shell,
                                                             uint32_t* __restrict__ out, Selected* __restrict__ sel,
                                                             unsigned long long* __restrict__ candidates) {
    extern __shared__ uint4 dyn[];
    unsigned long long* buffer = reinterpret_cast<unsigned long long*>(dyn);
    float4* cells = reinterpret_cast<float4*>(buffer + CAND_BUFFER);
    __shared__ uint32_t held, base;
    const uint32_t lane = threadIdx.x & 31u, row_words = p.R / 32, last = p.R - 1u, range = solid_from - lo;
    if (threadIdx.x == 0) held = 0u;
    __syncthreads();
    auto flush = [&] {
        const uint32_t n = min(held, CAND_BUFFER);
        __syncthreads();
        if (threadIdx.x == 0) {
            base = atomicAdd(&sel->candidates, n);
            held = 0u;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += THREADS) candidates[base + i] = buffer[i];
        __syncthreads();
    };
    for_each_value<OCT>(
        p, cells,
        [&](const uint32_t (&bits)[4], uint32_t x, uint32_t y, uint32_t z, uint32_t at) {
            uint32_t mine = 0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t word = __ballot_sync(0xFFFFFFFFu, bits[k] >= solid_from);
                if (lane == uint32_t(k)) mine = word;
            }
            if (shell) {  // lane k < 4 holds the word of row y + k
                if (z == 0u || z == last || y + lane == 0u || y + lane == last) mine = 0xFFFFFFFFu;
                if (x < 32u) mine |= 1u;
                if (x + 32u > last) mine |= 0x80000000u;
            }
            if (lane < 4) out[at + lane * row_words] = mine;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (bits[k] - lo < range) {
                    const unsigned long long c =
                        (((unsigned long long)(at + k * row_words) * 32 + lane) << 16) | (bits[k] & 0xFFFFu);
                    const uint32_t i = atomicAdd(&held, 1u);
                    if (i < CAND_BUFFER) buffer[i] = c;
                    else candidates[atomicAdd(&sel->candidates, 1u)] = c;
                }
        },
        [&] {
            if (held > CAND_BUFFER / 2) flush();
        });
    __syncthreads();
    if (held) flush();
}

// One block: the bin that holds rank `rank` of the histogram (2048, 16384 or
// 65536 bins), the rank within it and its count.  Groups of 32 bins are
// summed with coalesced loads, the group totals scanned, then the group's bins.
constexpr uint32_t SELECT_GROUPS = LOW_BINS / 32;
template <class T>
__global__ void __launch_bounds__(1024) select_kernel(const T* __restrict__ hist, uint32_t bins, Selected* __restrict__ sel) {
    __shared__ unsigned long long total[SELECT_GROUPS], warp_sum[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, groups = bins / 32;
    const unsigned long long rank = sel->rank;
    auto scan32 = [&](unsigned long long v) {  // inclusive, over the warp
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xFFFFFFFFu, v, d);
            if (lane >= uint32_t(d)) v += u;
        }
        return v;
    };
#pragma unroll 8
    for (uint32_t g = warp; g < groups; g += 32) {
        unsigned long long v = hist[g * 32 + lane];
        for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
        if (lane == 0) total[g] = v;
    }
    __syncthreads();
    const uint32_t per = groups / 1024 ? groups / 1024 : 1, first = threadIdx.x * per;  // 2 or 1 groups a thread
    unsigned long long mine = 0;
    for (uint32_t i = 0; i < per; ++i) mine += first + i < groups ? total[first + i] : 0ull;
    const unsigned long long incl = scan32(mine);
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    if (warp == 0) warp_sum[lane] = scan32(warp_sum[lane]);
    __syncthreads();
    const unsigned long long before = (warp ? warp_sum[warp - 1] : 0ull) + incl - mine;
    const uint32_t found = __ballot_sync(0xFFFFFFFFu, rank >= before && rank < before + mine);
    if (!found) return;  // the rank lies in another warp's groups
    const int src = __ffs(int(found)) - 1;
    unsigned long long run = __shfl_sync(0xFFFFFFFFu, before, src);
    uint32_t g = __shfl_sync(0xFFFFFFFFu, first, src);
    while (rank >= run + total[g]) run += total[g++];
    const unsigned long long h = hist[g * 32 + lane], end = run + scan32(h);
    if (rank >= end - h && rank < end) {
        sel->bin = g * 32 + lane;
        sel->count = h;
        sel->rank = rank - (end - h);
    }
}

__global__ void candidate_histogram_kernel(const unsigned long long* __restrict__ candidates,
                                           const Selected* __restrict__ sel, uint32_t* __restrict__ hist) {
    const uint32_t n = sel->candidates;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(hist + (uint32_t(candidates[i]) & 0xFFFFu), 1u);
}

// Candidates from the threshold up (sel->bin: its low 16 bits) are solid.
__global__ void candidate_bits_kernel(const unsigned long long* __restrict__ candidates,
                                      const Selected* __restrict__ sel, uint32_t* __restrict__ out) {
    const uint32_t n = sel->candidates, low = sel->bin;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long c = candidates[i], at = c >> 16;
        if ((uint32_t(c) & 0xFFFFu) >= low) atomicOr(out + (at >> 5), 1u << (at & 31u));
    }
}

struct DevBuf {
    void* p = nullptr;
    ~DevBuf() { if (p) cudaFree(p); }
};

// The kernels for the octave count: registers for 4, 8 or 16 octaves.
struct NoiseKernels {
    void (*first)(NoiseParams, uint32_t, uint32_t, int, unsigned long long*);
    void (*refine)(NoiseParams, uint32_t, uint32_t, int, unsigned long long*);
    void (*bits)(NoiseParams, uint32_t, uint32_t, int, uint32_t*, Selected*, unsigned long long*);
};
NoiseKernels kernels_for(uint32_t octaves) {
    if (octaves <= 4) return {noise_histogram_kernel<4, true>, noise_histogram_kernel<4, false>, noise_bits_kernel<4>};
    if (octaves <= 8) return {noise_histogram_kernel<8, true>, noise_histogram_kernel<8, false>, noise_bits_kernel<8>};
    return {noise_histogram_kernel<16, true>, noise_histogram_kernel<16, false>, noise_bits_kernel<16>};
}

}  // namespace
}  // namespace vx

static int vx_synth_noise_dev_body(uint32_t R, uint32_t spacing, uint32_t octaves, float fill, uint64_t seed,
                                  int32_t shell, uint64_t* out_bits_dev, void* stream) {
    using namespace vx;
    if (!out_bits_dev || R < 64 || R % 64 != 0 || R > 2048 || octaves < 1 || octaves > 16 || spacing < 1 ||
        (spacing >> (octaves - 1)) < 1 || !(fill >= 0.0f && fill <= 1.0f))
        return fail(VX_EINVAL, "vx_synth_noise_dev: bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint64_t N = uint64_t(R) * R * R;
    auto cerr = [](cudaError_t e, const char* w) {
        return fail(VX_ECUDA, std::string("vx_synth_noise_dev: ") + w + ": " + cudaGetErrorString(e));
    };
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    NoiseParams p{};
    p.R = R;
    p.octaves = octaves;
    p.neg_zero = -0.0f;
    // one allocation: histograms, the select's state, the lattices (each at a
    // multiple of 64 floats), the candidates
    const uint64_t o_low = HIST_BINS * sizeof(unsigned long long), o_sel = o_low + LOW_BINS * 4;
    const uint64_t o_col = o_sel + 256, o_lat = o_col + uint64_t(octaves) * R * sizeof(uint2);
    std::vector<uint64_t> at(octaves + 1, 0);
    float amp = 1.0f;
    for (uint32_t o = 0; o < octaves; ++o) {
        OctDev& q = p.oct[o];
        q.s = spacing >> o;
        q.amp = amp;
        amp *= 0.5f;
        q.cells = (R + q.s - 1) / q.s + 2;
        q.first = p.row_cells;
        p.row_cells += q.cells;
        at[o + 1] = at[o] + ((uint64_t(q.cells) * q.cells * q.cells + 63) & ~uint64_t(63));
    }
    const uint64_t o_cand = o_lat + at[octaves] * 4;
    const uint64_t cap = std::max<uint64_t>(N / 32, 4096);
    DevBuf mem;
    cudaError_t e = cudaMalloc(&mem.p, o_cand + cap * 8);
    if (e != cudaSuccess) return cerr(e, "cudaMalloc");
    char* base = static_cast<char*>(mem.p);
    auto* hist = reinterpret_cast<unsigned long long*>(base);
    auto* low = reinterpret_cast<uint32_t*>(base + o_low);
    auto* sel = reinterpret_cast<Selected*>(base + o_sel);
    auto* lat = reinterpret_cast<float*>(base + o_lat);
    auto* cand = reinterpret_cast<unsigned long long*>(base + o_cand);
    for (uint32_t o = 0; o < octaves; ++o) p.oct[o].lat = lat + at[o];
    p.column = reinterpret_cast<const uint2*>(base + o_col);
    lattice_kernel<<<uint32_t(std::min<uint64_t>((at[octaves] + 255) / 256, uint64_t(sms) * 8)), 256, 0, st>>>(
        p, lat, at[octaves], reinterpret_cast<uint2*>(base + o_col), seed);
    const size_t row_bytes = size_t(p.row_cells) * 4;
    const uint64_t tiles = uint64_t(R / TILE_ROWS) * R;
    const NoiseKernels k = kernels_for(octaves);
    // shared memory and persistent grid of a kernel with `side` bytes beside its cells
    struct Shape {
        size_t smem;
        uint32_t grid;
    };
    auto shape = [&](auto* kernel, size_t side, Shape& out) {
        out.smem = side + TILE_ROWS * row_bytes;
        cudaError_t r = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(NOISE_SMEM));
        int per_sm = 1;
        if (r == cudaSuccess) r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, THREADS, out.smem);
        out.grid = uint32_t(std::min<uint64_t>(tiles, uint64_t(sms) * uint64_t(std::max(1, per_sm))));
        return r;
    };
    Shape first{}, refine{}, bits{};
    e = shape(k.first, FIRST_BINS * 4, first);
    if (e == cudaSuccess) e = shape(k.refine, HIST_BINS * 4, refine);
    if (e == cudaSuccess) e = shape(k.bits, CAND_BUFFER * 8, bits);
    if (e != cudaSuccess) return cerr(e, "launch shape");
    auto* out32 = reinterpret_cast<uint32_t*>(out_bits_dev);
    const uint64_t n_solid = uint64_t(double(fill) * double(N) + 0.5);
    if (n_solid == 0) {
        k.bits<<<bits.grid, THREADS, bits.smem, st>>>(p, 0xFFFFFFFFu, 0xFFFFFFFFu, shell, out32, sel, cand);  // no value
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        return e == cudaSuccess ? VX_OK : cerr(e, "noise_bits_kernel");
    }
    // One level of the select: the bin of the threshold in the first histogram
    // (mask 0, shift < 0) or among the values whose bits match prefix under mask.
    Selected s{};
    s.rank = N - n_solid;
    auto level = [&](uint32_t mask, uint32_t prefix, int shift) -> int {
        s.candidates = 0;
        cudaError_t r = cudaMemsetAsync(hist, 0, HIST_BINS * sizeof(unsigned long long), st);
        if (r == cudaSuccess) r = cudaMemcpyAsync(sel, &s, sizeof(s), cudaMemcpyHostToDevice, st);
        if (r != cudaSuccess) return cerr(r, "select state");
        const Shape& sh = shift < 0 ? first : refine;
        (shift < 0 ? k.first : k.refine)<<<sh.grid, THREADS, sh.smem, st>>>(p, mask, prefix, shift, hist);
        select_kernel<<<1, 1024, 0, st>>>(hist, shift < 0 ? FIRST_BINS : HIST_BINS, sel);
        r = cudaGetLastError();
        if (r == cudaSuccess) r = cudaMemcpyAsync(&s, sel, sizeof(s), cudaMemcpyDeviceToHost, st);
        if (r == cudaSuccess) r = cudaStreamSynchronize(st);
        return r == cudaSuccess ? VX_OK : cerr(r, "noise_histogram_kernel");
    };
    if (int r = level(0u, 0u, -1)) return r;
    if (s.bin != 0 && s.count <= cap) {
        const uint32_t lo = (FIRST_BASE + s.bin) << 16;
        e = cudaMemsetAsync(low, 0, LOW_BINS * 4, st);
        if (e != cudaSuccess) return cerr(e, "candidate histogram");
        k.bits<<<bits.grid, THREADS, bits.smem, st>>>(p, lo, lo + 0x10000u, shell, out32, sel, cand);
        candidate_histogram_kernel<<<sms * 4, 256, 0, st>>>(cand, sel, low);
        select_kernel<<<1, 1024, 0, st>>>(low, LOW_BINS, sel);
        candidate_bits_kernel<<<sms * 4, 256, 0, st>>>(cand, sel, out32);
    } else {
        // nearly all values alike, or a threshold below 2^-15: 14, 14 and 2 bits one after the other
        s.rank = N - n_solid;
        if (int r = level(0u, 0u, 16)) return r;
        const uint32_t top = s.bin << 16;
        if (int r = level(0xFFFF0000u, top, 2)) return r;
        const uint32_t mid = top | (s.bin << 2);
        if (int r = level(0xFFFFFFFCu, mid, 0)) return r;
        const uint32_t thr = mid | (s.bin & 3u);
        k.bits<<<bits.grid, THREADS, bits.smem, st>>>(p, thr, thr, shell, out32, sel, cand);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cerr(e, "noise_bits_kernel");
    return VX_OK;
}

extern "C" int vx_synth_noise_dev(uint32_t R, uint32_t spacing, uint32_t octaves, float fill, uint64_t seed,
                                  int32_t shell, uint64_t* out_bits_dev, void* stream) {
    return vx::guarded("vx_synth_noise_dev", [&] { return vx_synth_noise_dev_body(R, spacing, octaves, fill, seed, shell, out_bits_dev, stream); });
}
