// vx_regular.cuh - the cast of regular rays: castRay (and castRayWithLOD) for
// callers that want no work counters.
//
// A ray is plain when the scene's world box and tree (DevScene::ordinary), its direction
// and its origin (ORD_LO) have ordinary sizes, so that no value is NaN; other
// rays take cast_general, the iteration of vx_cast.cuh (and launches over scenes
// that are not ordinary take kernels made of it).  A plain ray is regular
// when every |1 / d| is at most REG_RCP; then the octree loop needs none of the
// reference's special cases for rays nearly parallel to an axis: every corner
// t value is below the 1000 limit of its corrected minimum (|px - n| < 1.6
// with px in [0.5, 2.5) and the entry position n in [0.9, 2.1], times 550),
// every axis steps, and no conversion leaves the int range.  A warp takes the
// regular form (REG) when all its rays are regular, else the form with those
// cases (one of the two, never both: mixed warps of incoherent rays would pay
// for each).  All forms compute castRayImpl's results bit for bit; every
// floating-point result below is the reference's operation on its operands, or
// one of these exact replacements:
//  - fma(half, c, t) for half * c + t: half is a power of two, so the product
//    is exact and the sum is rounded once in both forms;
//  - the quantiser of executePopPhase, trunc(clamp(px - 1) * 2^22), read off
//    px's bits: for px in [1, 2) it is the mantissa's top 22 bits, outside it
//    saturates, so clamping the bits to [1, 2) gives the same integer;
//  - quotients a / d by an axis direction whose reciprocal is known: Markstein's
//    theorem (IBM J. R&D 34(1), 1990), see div_known;
//  - clamp then truncate for clamp(int(floor(x)), 0, 7).
// Every child that PUSH may enter is a node of an ordinary scene (checked when the
// scene is made), so no bound is tested there; where a child lies beyond the nodes
// the reference's loop stands still up to its cap, which the general iteration
// proves after two rounds and this one, which looks for repeats at POPs, would run
// through (256^3 noise cut to a tenth of its nodes: 84 us there, 370 here).
// Without counters three more things need not be done:
//  - a child descriptor that reads as "not fetched" is read again only when the
//    parent changes (it would read the same);
//  - the brick of a ray's entry point (the second lookup) is marched once: its
//    march has the same operands at every leaf, so a second one misses too;
//  - a proven repeat ends the ray at once.  Repeats are looked for at POPs only:
//    pushes lower the scale and steps inside a parent lower the position, so
//    every cycle holds a POP, and after a POP idx = 0 and h = 0 (the masked bits
//    the reference takes idx from are zero).  What lies between two POPs does
//    not read the stack.  If the states of two successive POPs are equal, each
//    later stretch repeats the one between them: it writes the stack slots it
//    wrote before with the same values, so the slot its POP reads holds what it
//    held.  Cycles with several POPs are found against checkpoints (POP number
//    8, 16, 32, ...) of state and stack.  (A step that moves no axis, which only
//    a ray that is not regular can take, leaves everything but t_min as it was:
//    when t_min stays too, the state repeats.)
//
// Bound: instruction issue, and in launches of few warps the dependent steps of
// the longest one (descriptor, slot, voxels; then one voxel after the other).
// Measured against the general iteration (B200): 1024^3 cave, 1920 x 1080 primary
// rays 239 -> 116 us; 512 x 512 rays in pixel rows through a 256^3 scene
// 123 -> 54 us; 2048^3 city at 4K with shadow rays 1.65 -> 1.00 ms; 1,000,003
// incoherent rays with LOD 308 -> 218 us; 24-scene batched frame, primary pass
// 1.24 -> 0.68 ms, bounce pass 1.77 -> 1.04 ms.
// Of this the branch-free march over bricks whose coordinates come from their
// slot took 86 -> 55 us, 139 -> 120 us and 2.72 -> 2.46 ms per frame; one place
// for the hit record and the rare quotients out of line (the bounce pass waits
// for instructions: its lanes are all over the loop) 2.46 -> 2.26 ms per frame.
// Tried and slower: the second form per lane instead of per warp (55.5 -> 56.8,
// 119 -> 122 us), out of line (119 -> 124 us), or for all rays (119 -> 145 us,
// frame 2.26 -> 2.46 ms).
#pragma once
#include "vx_cast.cuh"

namespace vx {
namespace {

constexpr float REG_RCP = 550.0f;
constexpr float ORD_LO = 1.0e5f;
constexpr int REG_CYC_WORDS = 7;          // words of the last POP's state per thread
constexpr uint32_t ENTRY_UNREAD = 0xFFFFFFFEu, ENTRY_MISSED = 0xFFFFFFFDu;
constexpr uint32_t REG_CK_FIRST = 8;      // POP number of the first checkpoint
constexpr int REG_CK_WORDS = 8 + 2 * 23;  // state, pushed mask, stack

// RN(a / d) from y = RN(1 / d).  After the first correction q is within one
// unit in the last place of a / d (its error is that of r alone, 2^-22 of the
// first q's), so by Markstein's theorem the second one rounds correctly: the
// remainder of a faithful q is exact, and q + r * y rounded once is RN(a / d).
// Needs |a| >= TINY_NUM (with |d| >= 1e-8) or a remainder may fall below the denormals.
constexpr float TINY_NUM = 8.470329e-22f;  // 2^-70
__device__ __forceinline__ float div_known(float a, float d, float y) {
    float q = a * y;
    q = __fmaf_rn(__fmaf_rn(-q, d, a), y, q);
    return __fmaf_rn(__fmaf_rn(-q, d, a), y, q);
}

// The integer part of x in [0, 7] as 0x4B000000 | int: adding 2^23 rounded
// toward zero leaves it in the low bits.
__device__ __forceinline__ uint32_t trunc_bits(float x) { return __float_as_uint(__fadd_rz(x, 8388608.0f)); }
// float(v) for v < 2^23.
__device__ __forceinline__ float small_float(uint32_t v) { return __uint_as_float(v | 0x4B000000u) - 8388608.0f; }

// Rays that are not plain, out of line: the general iteration with its stack
// in local memory.  Scenes none of whose rays are plain do not come here (their
// launches take the general kernels); what does is rays from farther than ORD_LO,
// the odd extreme direction and the odd scene of a batch.  Rays that are all so
// far away (256^3 scene seen from 2e5) take 76 us this way and 59 in the general
// kernel; with the caller's stack instead of local memory 77 to 79 us, and the
// plain rays 1 to 2 % more.
template <bool LOD>
__device__ __noinline__ void cast_general(const DevScene& s, float ox, float oy, float oz, float ddx, float ddy,
                                          float ddz, float tMinArg, float tMaxArg, Hit& h, LodCone lod) {
    uint32_t node[23], cyc[CYC_WORDS];
    float tmax[23];
    cast_ray<LOD, true>(s, ox, oy, oz, ddx, ddy, ddz, tMinArg, tMaxArg, node, tmax, cyc, 1, h, lod);
}

// The quotients as they stand, for numerators below TINY_NUM: out of line, the
// march hardly ever needs it.
__device__ __noinline__ float3 tiny_quotients(float ax, float ay, float az, float dx, float dy, float dz) {
    return make_float3(ax / dx, ay / dy, az / dz);
}

struct RegRay {
    float lo[3], d[3], rcp[3];  // grid-local origin, direction, 1 / direction (+-1e8 where |d| < 1e-8)
    float tEntry;
};
// An axis the brick march cannot step along (SVOBrickDDA.cpp:202-209, 424-430).
template <bool REG>
__device__ __forceinline__ bool still(float d) { return !REG && fabsf(d) < 1e-8f; }

// The exact hit t and axis at voxel corner vmn (traverseBrickView,
// SVOBrickDDA.cpp:472-505).
template <bool REG>
__device__ __forceinline__ void regular_hit(const RegRay& r, const float vmn[3], uint32_t voxel, Hit& h) {
    float a[3], tn[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) a[i] = (r.d[i] > 0.0f ? vmn[i] : vmn[i] + 1.0f) - r.lo[i];
    float hitT;
    if (nmin3(fabsf(a[0]), fabsf(a[1]), fabsf(a[2])) >= TINY_NUM) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            tn[i] = still<REG>(r.d[i]) ? -__int_as_float(0x7f800000) : div_known(a[i], r.d[i], r.rcp[i]);
        hitT = nmax(nmax3(tn[0], tn[1], tn[2]), 0.0f);  // no zero among tn: no sign of zero to keep
    } else {
        const float3 q = tiny_quotients(a[0], a[1], a[2], r.d[0], r.d[1], r.d[2]);
        const float qa[3] = {q.x, q.y, q.z};
#pragma unroll
        for (int i = 0; i < 3; ++i) tn[i] = still<REG>(r.d[i]) ? -__int_as_float(0x7f800000) : qa[i];
        hitT = gmax(gmax(gmax(tn[0], tn[1]), tn[2]), 0.0f);
    }
    const bool ax = tn[0] >= tn[1] && tn[0] >= tn[2], ay = tn[1] >= tn[2];
    const float da = ax ? r.d[0] : (ay ? r.d[1] : r.d[2]);
    h.t = hitT;
    h.voxel = voxel;
    h.flags = F_HIT | (ax ? 0u : (ay ? 2u : 4u)) | (da > 0.0f ? F_NEG : 0u);
}

// traverseBrickAndReturnHit (SVOBrickDDA.cpp:187-225) and traverseBrickView
// (:390-533).  The first voxel is tested before the march is set up: most hits
// are its.  The cell is kept as 4-bit fields x | y << 4 | z << 8 (a step out
// of the brick sets bit 3 of its field); one 8-byte load gives the 64 voxels
// of a slice, read again when z steps.
template <bool REG>
__device__ __forceinline__ bool regular_brick(const DevScene& s, uint32_t brick, const uint32_t slot[3],
                                              const RegRay& r, Hit& h) {
    const float bmn[3] = {small_float(slot[0] * 8u), small_float(slot[1] * 8u), small_float(slot[2] * 8u)};
    float tn[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) tn[i] = ((r.rcp[i] > 0.0f ? bmn[i] : bmn[i] + 8.0f) - r.lo[i]) * r.rcp[i];
    const float tMin = nmax(nmax3(tn[0], tn[1], tn[2]), r.tEntry);
    float ep[3];
    uint32_t c[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        ep[i] = r.lo[i] + r.d[i] * tMin;
        if constexpr (REG) c[i] = trunc_bits(nclamp(ep[i] - bmn[i], 0.0f, 7.0f)) & 7u;
        else c[i] = uint32_t(iclamp(f2i(floorf(ep[i] - bmn[i])), 0, 7));
    }
    const uint2* occ = reinterpret_cast<const uint2*>(s.occ) + size_t(bounded(brick, s.brick_count, V_BRICK)) * 8;
    uint2 w = __ldg(occ + c[2]);
    uint32_t bit = c[1] * 8u + c[0];
    float vmn[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) vmn[i] = bmn[i] + small_float(c[i]);
    uint32_t voxel = c[2] * 64u + bit;
    if (!(((bit & 32u ? w.y : w.x) >> (bit & 31u)) & 1u)) {
        float tNext[3], a[3], tf[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] = (r.d[i] > 0.0f ? vmn[i] + 1.0f : vmn[i]) - ep[i];
            tf[i] = ((r.rcp[i] > 0.0f ? bmn[i] + 8.0f : bmn[i]) - r.lo[i]) * r.rcp[i];
        }
        const float tMax = nmin3(tf[0], tf[1], tf[2]);
        if (nmin3(fabsf(a[0]), fabsf(a[1]), fabsf(a[2])) >= TINY_NUM) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
                tNext[i] = still<REG>(r.d[i]) ? FLT_MAX_ : tMin + div_known(a[i], r.d[i], r.rcp[i]);
        } else {
            const float3 q = tiny_quotients(a[0], a[1], a[2], r.d[0], r.d[1], r.d[2]);
            const float qa[3] = {q.x, q.y, q.z};
#pragma unroll
            for (int i = 0; i < 3; ++i) tNext[i] = still<REG>(r.d[i]) ? FLT_MAX_ : tMin + qa[i];
        }
        uint32_t p = c[0] | (c[1] << 4) | (c[2] << 8);
        const uint32_t sx = r.d[0] > 0.0f ? 1u : ~0u, sy = r.d[1] > 0.0f ? 16u : ~15u, sz = r.d[2] > 0.0f ? 256u : ~255u;
        // Branch-free over the axes: the smallest tNext is the one the reference's
        // comparisons pick (ties go to z, then y), and lanes that step along
        // different axes stay together.
        for (;;) {
            if (nmin3(tNext[0], tNext[1], tNext[2]) > tMax) return false;
            const bool ax = tNext[0] < tNext[1] && tNext[0] < tNext[2];
            const bool ay = !ax && tNext[1] < tNext[2];
            const bool az = !ax && !ay;
            p += ax ? sx : (ay ? sy : sz);
            if (ax) tNext[0] += fabsf(r.rcp[0]);
            if (ay) tNext[1] += fabsf(r.rcp[1]);
            if (az) tNext[2] += fabsf(r.rcp[2]);
            if (p & 0x888u) return false;
            if (az) w = __ldg(occ + (p >> 8));
            if (((p & 0x40u ? w.y : w.x) >> ((p & 7u) | ((p >> 1) & 0x18u))) & 1u) break;
        }
        vmn[0] = bmn[0] + small_float(p & 7u);
        vmn[1] = bmn[1] + small_float((p >> 4) & 7u);
        vmn[2] = bmn[2] + small_float(p >> 8);
        voxel = (p & 7u) | ((p >> 1) & 0x38u) | ((p >> 2) & 0x1C0u);
    }
    regular_hit<REG>(r, vmn, voxel, h);
    return true;
}

// The brick slot at slot position x >= 0 (a lookup of handleLeafHit), truncated.
// The clamps of the lookups that cannot bind are left out: positions are at
// most 0.999 of a side or a side - 0.001, sides are at least 4 (0.999 w <= w -
// 0.001) and at most 8 * bpa (so the slot is below bpa).  Returns the slot's
// brick; DevScene::ordinary says that it has the slot's coordinates, so they
// need not be loaded.
__device__ __forceinline__ uint32_t regular_lookup(const DevScene& s, const float x[3], uint32_t slot[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) slot[i] = trunc_bits(x[i]) & 0x7FFFFFu;
    return grid_lookup(s, int(slot[0]), int(slot[1]), int(slot[2]));
}

// Long cycles: checkpoints of the POP state (w[0..6]), the pushed mask and the
// pushed stack slots in per-thread local memory.
__device__ __forceinline__ void regular_checkpoint(const uint32_t* w, uint32_t pushed, const uint32_t* stkN,
                                                   const float* stkT, int stride, uint32_t* ck) {
    for (int k = 0; k < REG_CYC_WORDS; ++k) ck[k] = w[k];
    ck[7] = pushed;
    for (uint32_t m = pushed; m; m &= m - 1u) {
        const int j = __ffs(int(m)) - 1;
        ck[8 + 2 * j] = stkN[j * stride];
        ck[9 + 2 * j] = __float_as_uint(stkT[j * stride]);
    }
}
__device__ __forceinline__ bool regular_repeats(const uint32_t* w, uint32_t pushed, const uint32_t* stkN,
                                                const float* stkT, int stride, const uint32_t* ck) {
    bool eq = pushed == ck[7];
    for (int k = 0; k < REG_CYC_WORDS; ++k) eq = eq && w[k] == ck[k];
    for (uint32_t m = pushed; eq && m; m &= m - 1u) {
        const int j = __ffs(int(m)) - 1;
        eq = stkN[j * stride] == ck[8 + 2 * j] && __float_as_uint(stkT[j * stride]) == ck[9 + 2 * j];
    }
    return eq;
}

// A plain ray: setup (cast_init) and loop.  r holds lo, d and 1 / d.
template <bool LOD, bool REG>
__device__ __forceinline__ bool cast_body(const DevScene& s, const float o[3], RegRay& r, float tMinArg,
                                          float tMaxArg, uint32_t* stkN, float* stkT, uint32_t* cyc, int stride,
                                          int budget, Hit& h, LodCone lod) {
    // intersectAABB (SVOTraversal.cpp:117-149) and the entry (:540-560)
    float n[3];
    float tRayStart, t_min, t_max;
    float cf[3], bs[3];
    uint32_t flip = 0u;  // ~octant_mask & 7: axes with d > 0
    // axes the octree steps along (computeRayCoefficients' 1e-5)
    const bool cs[3] = {REG || fabsf(r.d[0]) >= 1e-5f, REG || fabsf(r.d[1]) >= 1e-5f, REG || fabsf(r.d[2]) >= 1e-5f};
    {
        bool inside = true;
        float tnear[3], tfar[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            inside = inside && o[i] >= s.wmin[i] && o[i] <= s.wmax[i];
            float inv = r.rcp[i];
            if (still<REG>(r.d[i])) {
                if (o[i] < s.wmin[i] || o[i] > s.wmax[i]) return true;
                inv = r.d[i] >= 0.0f ? 1e20f : -1e20f;
            }
            const bool pos = inv > 0.0f;
            tnear[i] = ((pos ? s.wmin[i] : s.wmax[i]) - o[i]) * inv;
            tfar[i] = ((pos ? s.wmax[i] : s.wmin[i]) - o[i]) * inv;
        }
        float tEntry = nmax3(tnear[0], tnear[1], tnear[2]);
        float tExit = nmin3(tfar[0], tfar[1], tfar[2]);
        if (!(tEntry <= tExit && tExit >= 0.0f)) return true;
        tEntry = nmax(tEntry, tMinArg);
        tExit = nmin(tExit, tMaxArg);
        if (tEntry >= tExit || tExit < 0.0f) return true;
        r.tEntry = tEntry;
        tRayStart = inside ? 0.0f : nmax(0.0f, tEntry);
        // computeRayCoefficients (:699-728)
        float side[3], first[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float x = o[i] + r.d[i] * tRayStart - s.wmin[i];
            n[i] = (s.wsinv[i] != 0.0f ? x * s.wsinv[i] : x / s.wsize[i]) + 1.0f;
            cf[i] = cs[i] ? -fabsf(r.rcp[i]) : 1.0f / -1e-5f;
            bs[i] = cf[i] * n[i];
            if (r.d[i] > 0.0f) {
                flip |= 1u << i;
                bs[i] = 3.0f * cf[i] - bs[i];
            }
            side[i] = cf[i] - bs[i];
            first[i] = 2.0f * cf[i] - bs[i];
            if (still<REG>(r.d[i])) r.rcp[i] = r.d[i] >= 0.0f ? 1e8f : -1e8f;  // from here on the brick march's
        }
        t_max = nmin(nmin3(side[0], side[1], side[2]), 1.0f);
        t_min = inside ? 0.0f : nmax(nmax3(first[0], first[1], first[2]), 0.0f);
    }
    const float t_root = t_max;
    // selectInitialOctant (:730-766); idxw is the octant idx in world order
    // (idx ^ flip), the bit it has in the stored masks
    float px[3];
    uint32_t idxw = flip;
    {
        const bool usePos = t_min < 0.01f;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float m = (flip >> i) & 1u ? 3.0f - n[i] : n[i];
            const bool upper = (usePos || !cs[i]) ? m >= 1.5f : 1.5f * cf[i] - bs[i] > t_min;
            px[i] = upper ? 1.5f : 1.0f;
            if (upper) idxw ^= 1u << i;
        }
    }
    // the corrected minimum of computeCorrectedTcMax (:768-784)
    auto limited = [&](float t, int i, float t_max_now) {
        return REG || (cs[i] && fabsf(t) < 1000.0f) ? t : t_max_now;
    };
    int scale = ESVO_MAX_SCALE, iter = 0;
    const int limit = imin(budget, MAX_ITER);
    const int leaf_scale = s.min_scale + s.brick_user_scale;
    uint32_t parent = 0u, pushed = 0u, entry_brick = ENTRY_UNREAD, npop = 0u, sig_pop = 0u, sig_ck = 0u;
    float exp2 = 0.5f, hh = t_max;
    uint32_t ck[REG_CK_WORDS];
    bool refetch = true;
    uint2 nd = make_uint2(0u, 0u);
    for (;;) {
        ++iter;
        if (refetch) nd = __ldg(s.nodes + bounded(parent, s.node_count, V_NODE));
        refetch = false;
        // checkChildValidity (:295-326)
        const float t0 = px[0] * cf[0] - bs[0], t1 = px[1] * cf[1] - bs[1], t2 = px[2] * cf[2] - bs[2];
        const float tc = nmin3(limited(t0, 0, t_max), limited(t1, 1, t_max), limited(t2, 2, t_max));
        const float tv = nmin(t_max, tc);
        const uint32_t child = nd.y >> idxw;
        const bool in_range = (child & 1u) && t_min <= tv;
        if constexpr (LOD) {
            if (in_range) {  // as in cast_step
                const float wd = tRayStart + t_min * s.wrl;
                const float vs = __int_as_float((scale - ESVO_MAX_SCALE - 1 + 127) << 23) * s.wsize[0];
                if (wd * lod.dir + lod.orig >= vs) {
                    h.t = wd;
                    h.node = parent;
                    h.flags = F_HIT | (1u << 1) | (iter >= MAX_ITER ? F_ITER_CAP : 0u);
                    h.scale = uint32_t(scale - s.min_scale);
                    return true;
                }
            }
        }
        const bool is_leaf = (child & 0x100u) || scale == leaf_scale;
        if (in_range && !is_leaf) {
            // executePushPhase (:328-378)
            const float half = exp2 * 0.5f;
            const float tc_raw = REG ? tc : nmin3(t0, t1, t2);
            if (tc_raw < hh) {
                const uint32_t k = bounded(uint32_t(scale - s.min_scale), uint32_t(s.max_levels), V_STACK);
                stkN[k * stride] = parent;
                stkT[k * stride] = t_max;
                pushed |= 1u << (scale - s.min_scale);
            }
            hh = tc_raw;
            const uint32_t inner = ~(nd.y >> 8) & nd.y & ((1u << idxw) - 1u);
            parent = nd.x + __popc(inner);  // a node: DevScene::ordinary
            refetch = true;
            --scale;
            exp2 = half;
            t_max = tv;
            idxw = flip;
            if (__fmaf_rn(half, cf[0], t0) > t_min) { idxw ^= 1u; px[0] += half; }
            if (__fmaf_rn(half, cf[1], t1) > t_min) { idxw ^= 2u; px[1] += half; }
            if (__fmaf_rn(half, cf[2], t2) > t_min) { idxw ^= 4u; px[2] += half; }
            if (scale < s.min_scale) break;
        } else {
            if (in_range) {
                // handleLeafHit (SVOBrickDDA.cpp:65-181)
                float x[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const float l = (flip >> i) & 1u ? 3.0f - exp2 - px[i] : px[i];
                    float b = (l - 1.0f) + (r.d[i] > 0.0f ? 0.001f : -0.001f);
                    if (!cs[i]) {
                        // the ray's clamped entry position (:98-121)
                        const float e = (o[i] + r.d[i] * nmax(r.tEntry, 0.0f)) - s.wmin[i];
                        b = s.wsinv[i] != 0.0f ? e * s.wsinv[i] : e / s.wsize[i];
                    }
                    x[i] = nclamp(b, 0.001f, 0.999f) * s.wslots[i];  // (b * wsize) / 8: the same rounding
                }
                uint32_t slot[3];
                uint32_t brick = regular_lookup(s, x, slot);
                uint32_t method = 1u << 4;
                if (brick == NONE) {
                    method = 2u << 4;
                    if (entry_brick == ENTRY_UNREAD) {
                        const float te0 = nmax(r.tEntry, 0.0f);
#pragma unroll
                        for (int i = 0; i < 3; ++i)
                            x[i] = nclamp(((o[i] + r.d[i] * te0) - s.wmin[i]) + r.d[i] * 0.01f, 0.0f, s.wsm[i]) * 0.125f;
                        entry_brick = regular_lookup(s, x, slot);
                    }
                    brick = entry_brick;
                    if (brick == NONE) {
                        // leaf child of the parent at the local octant (leafToBrickView, SVORebuild.cpp:569-574)
                        method = 3u << 4;
                        const uint32_t valid = nd.y & 0xFFu, leafs = valid & (nd.y >> 8);
                        if ((leafs >> idxw) & 1u) {
                            const uint32_t ci = nd.x + __popc(valid & ~leafs) + __popc(leafs & ((1u << idxw) - 1u));
                            if (ci < s.node_count) {
                                const uint32_t b = __ldg(s.node_brick + ci);
                                if (b < s.brick_count) {
                                    brick = b;
                                    const uint32_t bc = __ldg(s.coord + b);
                                    slot[0] = bc & 0x3FFu;
                                    slot[1] = (bc >> 10) & 0x3FFu;
                                    slot[2] = (bc >> 20) & 0x3FFu;
                                }
                            }
                        }
                    }
                }
                if (brick < ENTRY_MISSED) {
                    if (regular_brick<REG>(s, brick, slot, r, h)) {
                        h.brick = brick;
                        h.node = parent;
                        h.flags |= method;
                        h.scale = uint32_t(s.max_levels - 1);
                        return true;
                    }
                    if (method == (2u << 4)) entry_brick = ENTRY_MISSED;
                }
            }
            // executeAdvancePhase (:380-416); it sets t_min whether or not a leaf was missed
            uint32_t step = 0u;
            if (cs[0] && t0 <= tc) { step |= 1u; px[0] -= exp2; }
            if (cs[1] && t1 <= tc) { step |= 2u; px[1] -= exp2; }
            if (cs[2] && t2 <= tc) { step |= 4u; px[2] -= exp2; }
            const float t_before = t_min;
            t_min = nmax(tc, 0.0f);
            idxw ^= step;
            if (!REG && step == 0u && t_min == t_before) {
                h.flags = F_ITER_CAP;
                return true;
            }
            if ((idxw ^ flip) & step) {
                // executePopPhase (:418-510), step mask recomputed at the new position (:672-681)
                if (scale == ESVO_MAX_SCALE) {
                    if (t_min > t_max || px[0] < 1.0f || px[0] >= 2.0f || px[1] < 1.0f || px[1] >= 2.0f ||
                        px[2] < 1.0f || px[2] >= 2.0f)
                        break;
                } else {
                    float u[3];
                    int q[3];
                    uint32_t diff = 0u;
#pragma unroll
                    for (int i = 0; i < 3; ++i) u[i] = px[i] * cf[i] - bs[i];
                    const float uc = nmin3(limited(u[0], 0, t_max), limited(u[1], 1, t_max), limited(u[2], 2, t_max));
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        q[i] = iclamp(__float_as_int(px[i]), 0x3F800000, 0x3FFFFFFF);
                        const int up = iclamp(__float_as_int(px[i] + exp2), 0x3F800000, 0x3FFFFFFF);
                        if (cs[i] && u[i] <= uc) diff |= uint32_t(q[i] ^ up);
                    }
                    if (diff < 2u) break;  // the same quantised position
                    scale = 30 - __clz(diff);
                    if (scale < s.min_scale) break;
                    exp2 = __int_as_float((scale - ESVO_MAX_SCALE + 127) << 23);
                    parent = 0u;
                    t_max = t_root;
                    if ((pushed >> (scale - s.min_scale)) & 1u) {
                        const uint32_t k = bounded(uint32_t(scale - s.min_scale), uint32_t(s.max_levels), V_STACK);
                        parent = stkN[k * stride];
                        t_max = stkT[k * stride];
                    }
                    refetch = true;
                    const int keep = -(2 << (ESVO_MAX_SCALE - scale));
#pragma unroll
                    for (int i = 0; i < 3; ++i) px[i] = __int_as_float(q[i] & keep);
                    idxw = flip;
                    hh = 0.0f;
                    // the search for repeats
                    const uint32_t w[REG_CYC_WORDS] = {uint32_t(scale), parent, __float_as_uint(px[0]),
                                                       __float_as_uint(px[1]), __float_as_uint(px[2]),
                                                       __float_as_uint(t_min), __float_as_uint(t_max)};
                    const uint32_t sig = ((w[0] + w[1] + w[2]) + (w[3] + w[4] + w[5])) + w[6];
                    ++npop;
                    bool repeat = false;
                    if (sig == sig_pop && npop > 1u) {
                        repeat = true;
#pragma unroll
                        for (int k = 0; k < REG_CYC_WORDS; ++k) repeat = repeat && w[k] == cyc[k * stride];
                    }
                    if (npop >= REG_CK_FIRST) {
                        if ((npop & (npop - 1u)) == 0u) {
                            regular_checkpoint(w, pushed, stkN, stkT, stride, ck);
                            sig_ck = sig;
                        } else if (sig == sig_ck) {
                            repeat = repeat || regular_repeats(w, pushed, stkN, stkT, stride, ck);
                        }
                    }
                    if (repeat) {
                        h.flags = F_ITER_CAP;
                        return true;
                    }
                    sig_pop = sig;
#pragma unroll
                    for (int k = 0; k < REG_CYC_WORDS; ++k) cyc[k * stride] = w[k];
                }
            }
        }
        if (iter >= limit) {
            if (limit < MAX_ITER) return false;
            break;
        }
    }
    if (iter >= MAX_ITER) h.flags = F_ITER_CAP;
    return true;
}

// The cast of one ray without counters.  Writes h.t, brick, node, voxel, flags
// and scale.  stkN / stkT: max_levels slots, cyc: REG_CYC_WORDS, each `stride`
// apart.  False (h unset) when `budget` iterations have not ended the ray
// (rays that are not plain have no budget).
template <bool LOD = false>
__device__ __forceinline__ bool cast_plain(const DevScene& s, float ox, float oy, float oz, float ddx, float ddy,
                                           float ddz, float tMinArg, float tMaxArg, uint32_t* stkN, float* stkT,
                                           uint32_t* cyc, int stride, int budget, Hit& h,
                                           LodCone lod = LodCone{0.0f, 0.0f}) {
    // validateRayInput's normalisation and the reciprocals, as in cast_init
    const float dd = (ddx * ddx + ddy * ddy) + ddz * ddz;
    const float dinv = 1.0f / sqrtf(dd);
    RegRay r;
    r.d[0] = ddx * dinv;
    r.d[1] = ddy * dinv;
    r.d[2] = ddz * dinv;
    const float o[3] = {ox, oy, oz};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        r.rcp[i] = 1.0f / r.d[i];
        r.lo[i] = o[i] + (0.0f - s.wmin[i]);
    }
    if (!(s.ordinary && dd >= 1e-30f && dd <= 1e30f &&
          fabsf(r.lo[0]) + fabsf(r.lo[1]) + fabsf(r.lo[2]) <= ORD_LO)) {
        cast_general<LOD>(s, ox, oy, oz, ddx, ddy, ddz, tMinArg, tMaxArg, h, lod);
        return true;
    }
    h.t = 0.0f;
    h.brick = NONE;
    h.node = NONE;
    h.voxel = 0xFFFFu;
    h.flags = 0u;
    h.scale = 0u;
    const bool reg = nmax3(fabsf(r.rcp[0]), fabsf(r.rcp[1]), fabsf(r.rcp[2])) <= REG_RCP;
    if (__any_sync(__activemask(), !reg))
        return cast_body<LOD, false>(s, o, r, tMinArg, tMaxArg, stkN, stkT, cyc, stride, budget, h, lod);
    return cast_body<LOD, true>(s, o, r, tMinArg, tMaxArg, stkN, stkT, cyc, stride, budget, h, lod);
}

}  // namespace
}  // namespace vx
