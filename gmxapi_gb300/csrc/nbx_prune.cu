// Dynamic / rolling pair-list pruning on the GPU.
//
// Same masks as the reference's prune-only kernel
// (src/gromacs/nbnxm/cuda/nbnxm_cuda_kernel_pruneonly.cuh:104-279):
//  - fresh list: every set (j-cluster, i-cluster, warp-half) bit is re-tested;
//    it stays in the outer mask if any of its 8x4 atom pairs is within
//    rlistOuter, and is set in the inner mask (used by the force kernel) if
//    any pair is within rlistInner;
//  - rolling pass: only bits in (outer XOR inner) are re-tested and may be
//    added to the inner mask.
// Fresh pass: one warp per list entry, lane = one cluster pair of the cj4 group
// in hand; minima of packed squared distances decide, and the few that lie
// within rounding of a radius are recomputed exactly.
// Rolling pass: one warp per list entry; the few bits to re-test are numbered
// over the warp and each lane tests whole bits (32 atom pairs).  Compiled with
// --fmad=false; r^2 = fma(dz, dz, fma(dy, dy, dx dx)) is written out with
// explicit multiply-adds, so it rounds exactly like the CPU restatement.
#include "nbx_internal.cuh"

#include <algorithm>

namespace nbx
{
namespace
{

// warps per block (a warp per list entry in both passes)
constexpr int kPruneWarpsRolling = 4;
constexpr int kPruneWarpsFresh   = 4;

// Packed FP32 arithmetic without contraction (this unit is compiled with --fmad=false, and the
// intrinsics round each operation): r^2 = (dx dx + dy dy) + dz dz exactly as the scalar form.
__device__ __forceinline__ float2 p_sub(float2 a, float2 b)
{
    unsigned long long ra = *reinterpret_cast<unsigned long long*>(&a);
    unsigned long long rb = *reinterpret_cast<unsigned long long*>(&b);
    unsigned long long rd;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
    return *reinterpret_cast<float2*>(&rd);
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Squared distance with the rounding of the reference's norm2 in its prune kernel.
__device__ __forceinline__ float exact_r2(float dx, float dy, float dz)
{
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// The smallest squared distance between the 8 atoms at xi (shifted by s*) and the 4 at xj, each
// rounded as the CPU restatement rounds it.
__device__ __noinline__ float exact_min_r2(const float4* xi, const float4* xj, float sx,
                                           float sy, float sz)
{
    unsigned m = 0xffffffffu;
    for (int b = 0; b < kCl / kSplit; b++)
    {
        const float4 q = xj[b];
        for (int a = 0; a < kCl; a++)
        {
            const float4 p = xi[a];
            m = min(m, __float_as_uint(exact_r2((p.x + sx) - q.x, (p.y + sy) - q.y, (p.z + sz) - q.z)));
        }
    }
    return __uint_as_float(m);
}

// Per-warp shared memory of the fresh pass: x, y and z of three groups' four packed records.
constexpr int kFreshDepth = 3;
struct FreshSmem
{
    float4 x[kFreshDepth][kJg][6];
};

// Lanes (jm, part), part < 6, copy the coordinates (96 of the record's 160 bytes) of j-cluster cj into
// buffer b, if there is one, and close the copy group.
__device__ __forceinline__ void fresh_copy(FreshSmem& sm, int b, int cj, bool any, const float* xqp, int lane)
{
    if (any && (lane & 7) < 6)
    {
        const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(&sm.x[b][lane >> 3][lane & 7]));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                     "l"(xqp + (size_t)cj * kPackWords + 4 * (lane & 7))
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// Fresh prune of one list entry by one warp.  Lane (c, jm) = (lane & 7, lane >> 3) takes the cluster
// pair of i-cluster c and j-cluster jm of each cj4 group, so its flags sit at the mask bit of the
// lane's own number and four ballots make the group's masks.  The pass is bound by the FMA pipe
// (64 squared distances per cluster pair), so they are formed as |x_j|^2 - 2 x_i.x_j + |x_i|^2 about
// the entry's first atom: three packed multiply-adds per two pairs (the two halves' atoms a, a + 4
// in one operation, from the cluster-packed records) instead of six operations, and three-input
// minima.  That form rounds differently: with coordinates up to A from the origin and a radius R
// its error is below 10 2^-24 (3 A + R)^2 (three coordinate roundings, the two norms and four
// additions, each of terms below (|x_i| + |x_j|)^2).  A minimum within 16 2^-24 (3 A + R)^2 of a
// radius, about one in 10^4, is therefore recomputed by exact_min_r2, and the masks equal the
// exact ones bit for bit.  Fillers: an i-filler's norm is 1e9 (never in range), a j-filler is far
// away by itself, and two fillers are as far apart as their shift (ff_in, ff_out).
// 960k-atom water list (523k groups, cold caches): 330 us with the exact form on all 64 pairs and a
// block per entry, 247 us now (FMA pipe 49 %; the rest is latency at 16 warps of 128 registers per SM --
// the i-atoms read from shared memory instead, at 24 warps, took 272 us).
__device__ void prune_entry_fresh(const Sci& s, const Cj4* cj4, unsigned* imask_outer, const float4* xq,
                                  const float* xqp, const float* shiftvec, float outer2, float inner2, FreshSmem& sm)
{
    const int      lane = threadIdx.x & 31;
    const int      c    = lane & 7;
    const int      jm   = lane >> 3;
    const unsigned full = 0xffffffffu;
    if (s.cj4_start >= s.cj4_end)
    {
        return;
    }
    // three groups' coordinates in shared memory, one computed and two groups' copies in flight; the
    // lane's j-cluster indices are loaded one group further ahead
    Cj4*       g   = const_cast<Cj4*>(cj4) + s.cj4_start;
    Cj4* const end = const_cast<Cj4*>(cj4) + s.cj4_end;
    unsigned*  om  = imask_outer + 2 * (size_t)s.cj4_start;
    int        cj0 = g->cj[jm], cj1 = 0, cj2 = 0;
    int4       imn = *reinterpret_cast<const int4*>(&g->imei[0]);
    if (g + 1 < end)
    {
        cj1 = g[1].cj[jm];
    }
    if (g + 2 < end)
    {
        cj2 = g[2].cj[jm];
    }
    __syncwarp();  // the readers of the last entry's shared memory are done
    fresh_copy(sm, 0, cj0, g < end, xqp, lane);
    fresh_copy(sm, 1, cj1, g + 1 < end, xqp, lane);
    const float sx = shiftvec[3 * s.shift], sy = shiftvec[3 * s.shift + 1], sz = shiftvec[3 * s.shift + 2];
    const float4* const xi = xq + (size_t)s.sci * kSc + c * kCl;
    const float4        o4 = xq[(size_t)s.sci * kSc];
    const float         ox = o4.x + sx, oy = o4.y + sy, oz = o4.z + sz;
    float2              xm[kCl], ym[kCl], zm[kCl], ni[kCl];  // {-2 x, -2 x}, ..., {|x|^2, |x|^2}
    float               amax     = 0.0f;
    bool                has_fill = false;
#pragma unroll
    for (int a = 0; a < kCl; a++)
    {
        const float4 p    = xi[a];
        const bool   fill = p.x == kFarAway;
        const float  x = (p.x + sx) - ox, y = (p.y + sy) - oy, z = (p.z + sz) - oz;
        const float  n = exact_r2(x, y, z);
        const float  m = fill ? 0.0f : -2.0f, nf = fill ? 1.0e9f : n;
        amax           = fmaxf(amax, fill ? 0.0f : n);
        has_fill |= fill;
        ni[a] = make_float2(nf, nf);
        xm[a] = make_float2(m * x, m * x);
        ym[a] = make_float2(m * y, m * y);
        zm[a] = make_float2(m * z, m * z);
    }
    amax              = __uint_as_float(__reduce_max_sync(full, __float_as_uint(amax)));
    const float reach = 3.0f * sqrtf(amax) + sqrtf(outer2);
    const float eps   = 9.5367432e-7f * reach * reach;
    // two fillers of this shift: the exact arithmetic on their coordinates
    const float  ff = exact_r2((kFarAway + sx) - kFarAway, (kFarAway + sy) - kFarAway, (kFarAway + sz) - kFarAway);
    const bool   any_ff = ff < outer2 && __any_sync(full, has_fill);
    const float2 ox2 = make_float2(ox, ox), oy2 = make_float2(oy, oy), oz2 = make_float2(oz, oz);
    int          b   = 0;
    for (; g < end; g++, om += 2, b = (b == kFreshDepth - 1) ? 0 : b + 1)
    {
        const unsigned check0 = (unsigned)imn.x, check1 = (unsigned)imn.z;
        const int      cj_own = cj0;
        __syncwarp();  // the readers of the buffer two ahead (the group before this one) are done
        fresh_copy(sm, (b == 0) ? kFreshDepth - 1 : b - 1, cj2, g + 2 < end, xqp, lane);
        cj0 = cj1;
        cj1 = cj2;
        if (g + 1 < end)
        {
            imn = *reinterpret_cast<const int4*>(&g[1].imei[0]);
        }
        if (g + 3 < end)
        {
            cj2 = g[3].cj[jm];
        }
        asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncwarp();
        if (!(check0 | check1))
        {
            continue;
        }
        const float4* const rec = sm.x[b][jm];
        float2              xj[4], yj[4], zj[4], m[4];
#pragma unroll
        for (int h = 0; h < 2; h++)
        {
            const float4 x = rec[h], y = rec[2 + h], z = rec[4 + h];
            xj[2 * h]     = p_sub(make_float2(x.x, x.y), ox2);
            xj[2 * h + 1] = p_sub(make_float2(x.z, x.w), ox2);
            yj[2 * h]     = p_sub(make_float2(y.x, y.y), oy2);
            yj[2 * h + 1] = p_sub(make_float2(y.z, y.w), oy2);
            zj[2 * h]     = p_sub(make_float2(z.x, z.y), oz2);
            zj[2 * h + 1] = p_sub(make_float2(z.z, z.w), oz2);
            m[2 * h] = m[2 * h + 1] = make_float2(3.0e38f, 3.0e38f);
        }
#pragma unroll
        for (int a = 0; a < kCl; a += 2)
        {
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                const float2 t = __ffma2_rn(xm[a], xj[q], __ffma2_rn(ym[a], yj[q], __ffma2_rn(zm[a], zj[q], ni[a])));
                const float2 u = __ffma2_rn(
                        xm[a + 1], xj[q], __ffma2_rn(ym[a + 1], yj[q], __ffma2_rn(zm[a + 1], zj[q], ni[a + 1])));
                m[q] = make_float2(min3(m[q].x, t.x, u.x), min3(m[q].y, t.y, u.y));
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            m[q] = __fadd2_rn(m[q], __ffma2_rn(zj[q], zj[q], __ffma2_rn(yj[q], yj[q], __fmul2_rn(xj[q], xj[q]))));
        }
        float m0 = fminf(min3(m[0].x, m[1].x, m[2].x), m[3].x);
        float m1 = fminf(min3(m[0].y, m[1].y, m[2].y), m[3].y);
        // distances of the minima from the radii (of unset bits too: one vote for all)
        const float d0 = fminf(fabsf(m0 - inner2), fabsf(m0 - outer2));
        const float d1 = fminf(fabsf(m1 - inner2), fabsf(m1 - outer2));
        if (__any_sync(full, fminf(d0, d1) <= eps))
        {
            if (d0 <= eps)
            {
                m0 = exact_min_r2(xi, xq + (size_t)cj_own * kCl, sx, sy, sz);
            }
            if (d1 <= eps)
            {
                m1 = exact_min_r2(xi, xq + (size_t)cj_own * kCl + kCl / kSplit, sx, sy, sz);
            }
        }
        if (any_ff)
        {
            const float4 xa = rec[0], xb = rec[1];
            if (has_fill && (xa.x == kFarAway || xa.z == kFarAway || xb.x == kFarAway || xb.z == kFarAway))
            {
                m0 = fminf(m0, ff);
            }
            if (has_fill && (xa.y == kFarAway || xa.w == kFarAway || xb.y == kFarAway || xb.w == kFarAway))
            {
                m1 = fminf(m1, ff);
            }
        }
        const unsigned nw0 = check0 & __ballot_sync(full, m0 < inner2);
        const unsigned nw1 = check1 & __ballot_sync(full, m1 < inner2);
        const unsigned ou0 = check0 & __ballot_sync(full, m0 < outer2);
        const unsigned ou1 = check1 & __ballot_sync(full, m1 < outer2);
        if (lane == 0)
        {
            *reinterpret_cast<uint2*>(om) = make_uint2(ou0, ou1);
            g->imei[0].imask              = nw0;
            g->imei[1].imask              = nw1;
        }
    }
}

// Position of the k-th (from 0) set bit of m, which has more than k set bits: a binary search on
// the population counts of the lower halves of shrinking windows.
__device__ __forceinline__ int nth_set_bit(unsigned m, int k)
{
    int pos = 0;
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1)
    {
        const int c = __popc((m >> pos) & ((1u << w) - 1u));
        if (k >= c)
        {
            k -= c;
            pos += w;
        }
    }
    return pos;
}

// Per-warp shared memory of the rolling pass: the j-clusters of the 32 groups in hand and the
// inner-mask bits found in range, per half.
struct RollSmem
{
    int      cj[32][kJg];
    unsigned add[kSplit][32];
};

// The rolling prune of one list entry by one warp: only bits in (outer XOR inner) are tested, a few
// per group.  The lanes take the entry's groups 32 at a time (one record per lane), a warp scan of
// the per-lane bit counts numbers the bits, and lane l tests bits l, l + 32, ...: all 32 atom pairs
// of the bit's (i-cluster, j-cluster half), the i-atom pairs {a, a + 4} against each j-atom in
// packed FP32x2 arithmetic.  Bits with a pair within the inner radius are ORed into the inner masks
// through shared memory.  Each warp waits on three dependent loads: the entry, its records, the
// atoms.
__device__ void prune_entry_rolling(const Sci& s, const Cj4* cj4, const unsigned* imask_outer, const float4* xq,
                                    const float* shiftvec, float inner2, RollSmem& sm)
{
    const int      lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const float sx = shiftvec[3 * s.shift], sy = shiftvec[3 * s.shift + 1], sz = shiftvec[3 * s.shift + 2];
    const float4* const xi = xq + (size_t)s.sci * kSc;
    for (int g0 = s.cj4_start; g0 < s.cj4_end; g0 += 32)
    {
        const int g  = g0 + lane;
        unsigned  m0 = 0u, m1 = 0u, c0 = 0u, c1 = 0u;
        if (g < s.cj4_end)
        {
            const Cj4   c = cj4[g];
            const uint2 o = reinterpret_cast<const uint2*>(imask_outer)[g];
            m0            = c.imei[0].imask;
            m1            = c.imei[1].imask;
            c0            = m0 ^ o.x;
            c1            = m1 ^ o.y;
#pragma unroll
            for (int jm = 0; jm < kJg; jm++)
            {
                sm.cj[lane][jm] = c.cj[jm];
            }
        }
        sm.add[0][lane] = 0u;
        sm.add[1][lane] = 0u;
        const int n0    = __popc(c0);
        const int n     = n0 + __popc(c1);
        int       incl  = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int t = __shfl_up_sync(full, incl, o);
            if (lane >= o)
            {
                incl += t;
            }
        }
        const int total = __shfl_sync(full, incl, 31);
        __syncwarp();
        for (int t0 = 0; t0 < total; t0 += 32)
        {
            const int t = t0 + lane;
            // the lane holding bit t: the first lane whose inclusive count exceeds t
            int owner = 0;
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1)
            {
                if (__shfl_sync(full, incl, owner + step - 1) <= t)
                {
                    owner += step;
                }
            }
            const int      o_excl = __shfl_sync(full, incl - n, min(owner, 31));
            const int      o_n0   = __shfl_sync(full, n0, min(owner, 31));
            const unsigned o_c0   = __shfl_sync(full, c0, min(owner, 31));
            const unsigned o_c1   = __shfl_sync(full, c1, min(owner, 31));
            if (t >= total)
            {
                continue;
            }
            const int  k    = t - o_excl;
            const int  half = k < o_n0 ? 0 : 1;
            const int  bit  = half == 0 ? nth_set_bit(o_c0, k) : nth_set_bit(o_c1, k - o_n0);
            const int  cj   = sm.cj[owner][bit / kNcl];
            const int  ic   = bit % kNcl;
            float2     xa[kCl / 2], ya[kCl / 2], za[kCl / 2];
            float4     xb[kCl / kSplit];
#pragma unroll
            for (int a = 0; a < kCl / 2; a++)
            {
                const float4 p = xi[ic * kCl + a];
                const float4 q = xi[ic * kCl + a + kCl / 2];
                xa[a]          = make_float2(p.x + sx, q.x + sx);
                ya[a]          = make_float2(p.y + sy, q.y + sy);
                za[a]          = make_float2(p.z + sz, q.z + sz);
            }
#pragma unroll
            for (int b = 0; b < kCl / kSplit; b++)
            {
                xb[b] = xq[cj * kCl + half * (kCl / kSplit) + b];
            }
            unsigned m = 0xffffffffu;
#pragma unroll
            for (int b = 0; b < kCl / kSplit; b++)
            {
                const float2 xj = make_float2(xb[b].x, xb[b].x);
                const float2 yj = make_float2(xb[b].y, xb[b].y);
                const float2 zj = make_float2(xb[b].z, xb[b].z);
#pragma unroll
                for (int a = 0; a < kCl / 2; a++)
                {
                    const float2 dx = p_sub(xa[a], xj);
                    const float2 dy = p_sub(ya[a], yj);
                    const float2 dz = p_sub(za[a], zj);
                    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                    m = min(m, min(__float_as_uint(r2.x), __float_as_uint(r2.y)));
                }
            }
            // r^2 and the squared cut-off are non-negative floats: r^2 < c^2 exactly when the bit
            // pattern of r^2 is the smaller one
            if (m < __float_as_uint(inner2))
            {
                atomicOr(&sm.add[half][owner], 1u << bit);
            }
        }
        __syncwarp();
        if (g < s.cj4_end)
        {
            const unsigned a0 = sm.add[0][lane], a1 = sm.add[1][lane];
            if (a0 | a1)
            {
                Imei* const im = const_cast<Cj4*>(cj4)[g].imei;
                im[0].imask    = m0 | a0;
                im[1].imask    = m1 | a1;
            }
        }
        __syncwarp();
    }
}

// A warp per list entry in both passes.
template<int kPruneWarps, bool kFresh>
__global__ void __launch_bounds__(32 * kPruneWarps, kFresh ? 4 : 6) k_prune(DeviceView v, int part, int nparts)
{
    pdl_begin();
    __shared__ RollSmem  rsm[kFresh ? 1 : kPruneWarps];
    __shared__ FreshSmem fsm[kFresh ? kPruneWarps : 1];
    const int           numSci = v.hdr->num_sci;
    if (v.hdr->status & (kStatusListOverflow | kStatusExclOverflow))
    {
        return;
    }
    if constexpr (kFresh)
    {
        // the next entry's record is loaded while the current entry is pruned
        const int stride = gridDim.x * kPruneWarps;
        int       e      = blockIdx.x * kPruneWarps + (threadIdx.x >> 5);
        Sci       sn{};
        if (e < numSci)
        {
            sn = v.sci[e];
        }
        for (; e < numSci; e += stride)
        {
            const Sci s = sn;
            if (e + stride < numSci)
            {
                sn = v.sci[e + stride];
            }
            prune_entry_fresh(s, v.cj4, v.imask_outer, v.xq, v.xqp, v.shiftvec, v.rlist2, v.rlist_inner2,
                              fsm[threadIdx.x >> 5]);
        }
    }
    else
    {
        // entries part, part + nparts, ...
        const int warp = threadIdx.x >> 5;
        for (int e = part + (blockIdx.x * kPruneWarps + warp) * nparts; e < numSci;
             e += gridDim.x * kPruneWarps * nparts)
        {
            prune_entry_rolling(v.sci[e], v.cj4, v.imask_outer, v.xq, v.shiftvec, v.rlist_inner2, rsm[warp]);
        }
    }
}

// The system of global entry e in a batch: a search of the entry prefix sums.
__device__ __forceinline__ int batch_system_of(const int* entry_prefix, int nsys, int e)
{
    int lo = 0, hi = nsys - 1;
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        if (entry_prefix[mid] <= e)
        {
            lo = mid;
        }
        else
        {
            hi = mid - 1;
        }
    }
    return lo;
}

// The same prune over a batch of systems: global entry index -> system by a
// search of the entry prefix sums; entries whose index within their system is
// part (mod nparts) are pruned.
template<int kPruneWarps, bool kFresh>
__global__ void __launch_bounds__(32 * kPruneWarps)
        k_batch_prune(const BatchSys* sys, const int* entry_prefix, int nsys, float outer2, float inner2, int part,
                      int nparts)
{
    pdl_begin();
    __shared__ RollSmem  rsm[kFresh ? 1 : kPruneWarps];
    __shared__ FreshSmem fsm[kFresh ? kPruneWarps : 1];
    const int           total = entry_prefix[nsys];
    if constexpr (kFresh)
    {
        for (int e = blockIdx.x * kPruneWarps + (threadIdx.x >> 5); e < total; e += gridDim.x * kPruneWarps)
        {
            const int       k = batch_system_of(entry_prefix, nsys, e);
            const BatchSys& b = sys[k];
            prune_entry_fresh(b.sci[e - entry_prefix[k]], b.cj4, b.imask_outer, b.xq, b.xqp, b.shiftvec, outer2,
                              inner2, fsm[threadIdx.x >> 5]);
        }
    }
    else
    {
        const int warp = threadIdx.x >> 5;
        for (int e = blockIdx.x * kPruneWarps + warp; e < total; e += gridDim.x * kPruneWarps)
        {
            const int k     = batch_system_of(entry_prefix, nsys, e);
            const int local = e - entry_prefix[k];
            if ((local % nparts) != part)
            {
                continue;
            }
            const BatchSys& b = sys[k];
            prune_entry_rolling(b.sci[local], b.cj4, b.imask_outer, b.xq, b.shiftvec, inner2, rsm[warp]);
        }
    }
}

// One wave of resident blocks of a prune kernel (SM count x blocks per SM at its register and
// shared-memory use), computed once: entries are spread over the blocks by the grid-stride loops,
// so a second partial wave would only add a tail.
template<auto kKernel, int kThreads>
int resident_grid()
{
    static int blocks = 0;
    if (blocks == 0)
    {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kKernel, kThreads, 0);
        blocks = std::max(sms, 1) * std::max(per_sm, 1);
    }
    return blocks;
}

} // namespace

cudaError_t launch_batch_prune(const BatchSys* sys, const int* entry_prefix, int nsys, float outer2, float inner2,
                               int fresh, int part, int nparts, cudaStream_t s)
{
    if (fresh)
    {
        constexpr auto kKernel = k_batch_prune<kPruneWarpsFresh, true>;
        launch_pdl(kKernel, resident_grid<kKernel, 32 * kPruneWarpsFresh>(), 32 * kPruneWarpsFresh, 0, s, sys,
                   entry_prefix, nsys, outer2, inner2, part, 1);
    }
    else
    {
        constexpr auto kKernel = k_batch_prune<kPruneWarpsRolling, false>;
        launch_pdl(kKernel, resident_grid<kKernel, 32 * kPruneWarpsRolling>(), 32 * kPruneWarpsRolling, 0, s, sys,
                   entry_prefix, nsys, outer2, inner2, part, nparts);
    }
    return cudaGetLastError();
}

cudaError_t launch_prune(const DeviceView& v, int fresh, int part, int nparts, cudaStream_t s)
{
    if (fresh)
    {
        constexpr auto kKernel = k_prune<kPruneWarpsFresh, true>;
        launch_pdl(kKernel, resident_grid<kKernel, 32 * kPruneWarpsFresh>(), 32 * kPruneWarpsFresh, 0, s, v, 0, 1);
    }
    else
    {
        constexpr auto kKernel = k_prune<kPruneWarpsRolling, false>;
        launch_pdl(kKernel, resident_grid<kKernel, 32 * kPruneWarpsRolling>(), 32 * kPruneWarpsRolling, 0, s, v,
                   part, nparts);
    }
    return cudaGetLastError();
}

} // namespace nbx
