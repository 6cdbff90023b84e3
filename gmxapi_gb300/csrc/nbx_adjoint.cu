// Adjoint of the cluster-pair force / energy kernel.
//
// There is no counterpart in the reference (it only computes forces).  Given
// upstream gradients G_i = dL/dF_i on the forces and gE = dL/dE on the LJ and
// Coulomb energies, one pass over the same pair list recomputes every pair
// term (nothing from the forward pass is stored) and accumulates
//   dL/dx  (a Hessian-vector product with G, plus -gE times the forces),
//   dL/dq  per atom,
//   dL/d(6 C6), dL/d(12 C12) per type pair (FP64 sums).
// For a pair with r = x_i - x_j (+ shift), s = r^2, force on i f = phi(s) r and
// g = G_i - G_j:
//   dL/dr = phi g + (2 phi'(s) (g.r) - gE_lj phi_lj - gE_c qq psi) r,
// with phi = phi_lj + qq psi, phi_lj = (12C12 r^-12 - 6C6 r^-6) / r^2 and, for
// Ewald, psi = erfc(br)/r^3 + (2b/sqrt(pi)) e^{-b^2 r^2}/r^2 (minus 1/r^3 for an
// excluded pair), whose derivative is psi' = -(1.5 psi + (2b/sqrt(pi)) b^2
// e^{-b^2 r^2}) / r^2 for normal and excluded pairs alike.
//
// Layout: persistent warps, one list entry per warp, an 8x8 cluster pair per step: lane (j, ip) =
// (lane >> 2, lane & 3) computes j-atom j against the i-atoms ip and ip + 4 in one FP32x2 instruction
// stream.  The entry's i-atoms and their upstream gradients sit in shared memory as packed pairs, the
// lane's i-side sums beside them (one slot per lane and i-cluster: no conflicts); the j-side sums stay in
// registers and end in one add per lane.
//
// Type-pair gradients.  The terms d6 and d12 of a step are 8x8 matrices G over (j-atom, i-atom), and the
// table gradient is sum_steps P_j^T G P_i with one-hot type matrices P: a contraction, so it runs on the
// tensor cores.  The lane mapping above is the A fragment of mma.m16n8k8 (rows: the j-atoms of d6, then
// those of d12; k = i-atom) and P_i its B fragment.  A float is split into two tf32 parts of 11 bits; a
// one-hot factor keeps their products exact, and the two are summed in accumulators of their own over the at
// most 8 steps of a j-cluster.  The products D = G P_i then turn through shared memory into the B fragment
// of P_j^T D, which is added in FP32 over the entry and in FP64 beyond it.  (Float atomics on per-warp
// tables in shared memory, which this replaces, are compare-and-swap loops.)  Against 64 bits the sigma and
// epsilon gradients are off by 0.1-2e-7 (1 to 15 types), with those tables by 3-5.6e-7.
// The kernel is bound by the latency of dependent arithmetic at 16 warps per SM (issue 53 %, FMA pipe 44 %, L1 72 %).
// 24,000-atom 8-type liquid: 91.5 us with one pair per lane and table atomics, 52.4 us now; a gradient step of 16
// liquids of 2,000 to 50,000 atoms 1276 and 923 us.
#include "nbx_internal.cuh"
#include "nbx_pair_x2.cuh"

#include <algorithm>

namespace nbx
{
namespace
{

constexpr int kAdjThreads     = 256;
constexpr int kAdjBlocksPerSm = 2;  // 16 warps per SM
constexpr int kAdjWarps       = kAdjThreads / 32;
constexpr int kAdjMaxTypes1   = 16;
constexpr int kAdjRow         = 16;  // type-pair rows of 16 entries in shared memory

// Constants of the pair loop; gE_*: upstream energy gradients (0 in the flavours without them).
struct AdjConsts
{
    float rc2, pbeta, nbeta2l2, c2b, nb2c2b2, sh_ewald, nk_rf2, k_rf, c_rf, epsfac, cpot6, cpot12;
    float gE_lj, gE_c;
    int   filler;  // the type of empty slots
};

__device__ __forceinline__ AdjConsts adj_consts(const DeviceView& v)
{
    AdjConsts k;
    k.rc2      = v.rc2;
    k.pbeta    = v.pbeta;
    k.nbeta2l2 = -v.beta2l2;
    k.c2b      = v.c2b;
    k.nb2c2b2  = -2.0f * v.beta * v.beta * v.c2b;
    k.sh_ewald = v.sh_ewald;
    k.nk_rf2   = -2.0f * v.k_rf;
    k.k_rf     = v.k_rf;
    k.c_rf     = v.c_rf;
    k.epsfac   = v.epsfac;
    k.cpot6    = v.cpot6 * (1.0f / 6.0f);
    k.cpot12   = v.cpot12 * (1.0f / 12.0f);
    k.gE_lj    = 0.0f;
    k.gE_c     = 0.0f;
    k.filler   = v.ntypes1 - 1;
    return k;
}

// The per-system arrays one list entry of the adjoint touches.
struct AdjPtrs
{
    const float4* xq;
    const Cj4*    cj4;
    const Excl*   excl;
    const float*  shiftvec;
    const float4* gnb;  // upstream gradient and type (int bits) per slot
    float4*       dnb;
};

// Shared memory of one warp.
struct AdjWarp
{
    // per i-cluster and ip: {x, x', y, y'}, {z, z', q, q'}, {gx, gx', gy, gy'}, {gz, gz', type, type'} of
    // the atoms ip and ip + 4
    float4 irec[kNcl][4][4];
    // per i-cluster and lane: {x, x', y, y'}, {z, z', q, q'} sums (rows padded by four entries: the
    // reduction reads eight lanes' sums of two clusters at a time)
    float4 acc[kNcl][2 * 32 + 4];
    float4 jx[32], jg[32];
    float4 turn[32];  // the type products between the two tensor-core passes
};

__device__ __forceinline__ void mma_tf32(float (&d)[4], const float (&a)[4], float b0, float b1)
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
                 "{%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])),
                   "r"(__float_as_uint(a[3])), "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}

// x as two tf32 operands: its leading 11 significant bits, and the rest rounded to 11 bits (the tensor cores
// read the upper 19 bits of an operand, so half a unit of the last of them is added; cvt.rna takes three
// instructions for the same).
__device__ __forceinline__ void tf32_split(float x, float& head, float& rest)
{
    head = __uint_as_float(__float_as_uint(x) & 0xffffe000u);
    rest = __uint_as_float(__float_as_uint(x - head) + 0x1000u);
}

// j-side sums of the lane's j-atom over its two i-atoms' slots, and the j-cluster's products D of type tile n
// (columns 2 ip + {0, 1}): {d6, d6', d12, d12'} of the heads and of the rests.
template<bool kBig>
struct AdjJ
{
    float2 x, y, z, q;
    float  hi[kBig ? 2 : 1][4], lo[kBig ? 2 : 1][4];
};

__device__ __forceinline__ float2 pick2(bool a, bool b, float2 v)
{
    return make_float2(a ? v.x : 0.0f, b ? v.y : 0.0f);
}

// One step: i-cluster c against the lane's j-atom.  okA / okB: the pair's mask bit (and, on the diagonal,
// j > i); intA / intB: its exclusion bit as 0 / 1.
template<bool kEwald, bool kGE, bool kBig, bool kExcl>
__device__ __forceinline__ void adj_step(const AdjConsts& k, const char* __restrict__ nbfp_b, AdjWarp& w, int c,
                                         int lane, const float4 xj, const float4 gj, float qje, int tjb, bool okA,
                                         bool okB, float intA, float intB, AdjJ<kBig>& dj)
{
    const int     ip = lane & 3;
    const float4  i0 = w.irec[c][0][ip], i1 = w.irec[c][1][ip], i2 = w.irec[c][2][ip], i3 = w.irec[c][3][ip];
    const int     tA = __float_as_int(i3.z), tB = __float_as_int(i3.w);
    const float2  dx = sub2(make_float2(i0.x, i0.y), f2(xj.x));
    const float2  dy = sub2(make_float2(i0.z, i0.w), f2(xj.y));
    const float2  dz = sub2(make_float2(i1.x, i1.y), f2(xj.z));
    float2        r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
    const bool    inA = okA && r2.x < k.rc2, inB = okB && r2.y < k.rc2;
    r2                = make_float2(fmaxf(r2.x, kMinDist2), fmaxf(r2.y, kMinDist2));
    float2       rinv = make_float2(fast_rsqrt(r2.x), fast_rsqrt(r2.y));
    rinv              = fma2(rinv, fma2(mul2(r2, f2(-0.5f)), mul2(rinv, rinv), f2(0.5f)), rinv);
    // pairs out of range add zeros: 1/r = 0, and no upstream gradient (0 times one that is not finite is not 0)
    rinv               = pick2(inA, inB, rinv);
    const float2 rinv2 = mul2(rinv, rinv);
    const float2 ljA   = *reinterpret_cast<const float2*>(nbfp_b + (tA << 7) + tjb);
    const float2 ljB   = *reinterpret_cast<const float2*>(nbfp_b + (tB << 7) + tjb);
    float2       rinv6 = mul2(mul2(rinv2, rinv2), rinv2);
    if (kExcl)
    {
        rinv6 = mul2(rinv6, make_float2(intA, intB));
    }
    // C / r^n as products that stay finite down to the smallest distance where C is 0 (r^-14 alone overflows
    // below 1.8 pm), and rounded once where the two terms cancel
    const float2 vdisp  = make_float2(ljA.x * rinv6.x, ljB.x * rinv6.y);
    const float2 vrep   = mul2(make_float2(ljA.y * rinv6.x, ljB.y * rinv6.y), rinv6);
    const float2 phi_lj = mul2(sub2(vrep, vdisp), rinv2);
    float2       psi, dpsi, hq = f2(0.0f);  // Coulomb phi / qq, 2 r^2 times its s-derivative, energy / qq
    if (kEwald)
    {
        const float2 tt   = fma2(f2(k.pbeta), mul2(r2, rinv), f2(1.0f));
        const float2 t    = make_float2(fast_rcp(tt.x), fast_rcp(tt.y));
        const float2 earg = mul2(f2(k.nbeta2l2), r2);
        const float2 expm = make_float2(fast_ex2(earg.x), fast_ex2(earg.y));
        const float2 tp   = mul2(t, erfc_poly2(t));  // erfc(beta r) = tp expm
        psi               = mul2(mul2(expm, fma2(tp, rinv, f2(k.c2b))), rinv2);
        if (kGE)
        {
            hq = fma2(mul2(tp, expm), rinv, make_float2(-intA * k.sh_ewald, -intB * k.sh_ewald));
        }
        if (kExcl)
        {
            const float2 ex = mul2(make_float2(intA - 1.0f, intB - 1.0f), rinv);  // -(1 - int) / r
            psi             = fma2(ex, rinv2, psi);
            if (kGE)
            {
                hq = add2(hq, ex);
            }
        }
        dpsi = fma2(f2(-3.0f), psi, mul2(f2(k.nb2c2b2), expm));
    }
    else
    {
        const float2 r3 = kExcl ? mul2(mul2(rinv, rinv2), make_float2(intA, intB)) : mul2(rinv, rinv2);
        psi             = add2(r3, f2(k.nk_rf2));
        dpsi            = mul2(f2(-3.0f), r3);
        if (kGE)
        {
            hq = fma2(f2(k.k_rf), r2, sub2(mul2(rinv, make_float2(intA, intB)), f2(k.c_rf)));
        }
    }
    const float2 qi   = make_float2(i1.z, i1.w);
    const float2 qq   = mul2(qi, f2(qje));
    const float2 phi  = fma2(qq, psi, phi_lj);
    const float2 gx   = pick2(inA, inB, sub2(make_float2(i2.x, i2.y), f2(gj.x)));
    const float2 gy   = pick2(inA, inB, sub2(make_float2(i2.z, i2.w), f2(gj.y)));
    const float2 gz   = pick2(inA, inB, sub2(make_float2(i3.x, i3.y), f2(gj.z)));
    const float2 gr   = fma2(gz, dz, fma2(gy, dy, mul2(gx, dx)));
    // 2 phi' (g.r), phi' = (qq dpsi + (8 vdisp - 14 vrep) / r^2) / (2 r^2)
    const float2 dphi = fma2(qq, dpsi, mul2(fma2(f2(-14.0f), vrep, mul2(f2(8.0f), vdisp)), rinv2));
    float2       coef = mul2(mul2(dphi, rinv2), gr);
    float2       wq   = mul2(psi, gr);  // dL/d(q_i q_j) / epsfac
    if (kGE)
    {
        coef = sub2(coef, pick2(inA, inB, fma2(f2(k.gE_c), mul2(qq, psi), mul2(f2(k.gE_lj), phi_lj))));
        wq   = add2(wq, pick2(inA, inB, mul2(f2(k.gE_c), hq)));
    }
    const float2 ux = fma2(phi, gx, mul2(coef, dx));
    const float2 uy = fma2(phi, gy, mul2(coef, dy));
    const float2 uz = fma2(phi, gz, mul2(coef, dz));
    float4* const pa = &w.acc[c][lane];
    float4 a0 = pa[0], a1 = pa[32];
    const float2 sx = add2(make_float2(a0.x, a0.y), ux), sy = add2(make_float2(a0.z, a0.w), uy);
    const float2 sz = add2(make_float2(a1.x, a1.y), uz), sq = fma2(wq, f2(qje), make_float2(a1.z, a1.w));
    pa[0]  = make_float4(sx.x, sx.y, sy.x, sy.y);
    pa[32] = make_float4(sz.x, sz.y, sq.x, sq.y);
    dj.x   = add2(dj.x, ux);
    dj.y   = add2(dj.y, uy);
    dj.z   = add2(dj.z, uz);
    dj.q   = fma2(wq, qi, dj.q);
    // dL/d(6C6) and dL/d(12C12) of the pairs, by i type
    const float2 gr6 = mul2(gr, rinv6);
    float2       d6  = mul2(gr6, rinv2);
    float2       d12 = mul2(gr6, mul2(rinv6, rinv2));
    if (kGE)
    {
        d6  = fma2(f2(k.gE_lj), fma2(rinv6, f2(1.0f / 6.0f), f2(k.cpot6)), d6);
        d12 = fma2(f2(k.gE_lj), fma2(mul2(rinv6, rinv6), f2(1.0f / 12.0f), f2(k.cpot12)), d12);
    }
    if (kGE || kExcl)
    {
        const bool cA = inA && (!kExcl || intA != 0.0f), cB = inB && (!kExcl || intB != 0.0f);
        d6            = pick2(cA, cB, d6);
        d12           = pick2(cA, cB, d12);
    }
    const int row = lane >> 2;
    float     h[4], r[4];
    tf32_split(d6.x, h[0], r[0]);
    tf32_split(d12.x, h[1], r[1]);
    tf32_split(d6.y, h[2], r[2]);
    tf32_split(d12.y, h[3], r[3]);
#pragma unroll
    for (int n = 0; n < (kBig ? 2 : 1); n++)
    {
        const float b0 = tA == row + 8 * n ? 1.0f : 0.0f, b1 = tB == row + 8 * n ? 1.0f : 0.0f;
        mma_tf32(dj.hi[n], h, b0, b1);
        mma_tf32(dj.lo[n], r, b0, b1);
    }
}

// Type-pair sums of an entry: C fragments of P_j^T D (rows: j types lane >> 2 (+ 8), columns: i types
// 2 (lane & 3) + {0, 1} of tile n) of dL/d(6C6) (negated) and dL/d(12C12).
template<bool kBig>
struct AdjTypes
{
    float s6[kBig ? 2 : 1][4], s12[kBig ? 2 : 1][4];
};

// All set cluster pairs of one cj4 group.  m: the mask of the lane's half; u: both halves' masks; wA / wB:
// the lane's exclusion words (i-atoms ip and ip + 4).
template<bool kEwald, bool kGE, bool kBig, bool kExcl>
__device__ __forceinline__ void adj_group(const AdjConsts& k, const char* __restrict__ nbfp_b, AdjWarp& w,
                                          float4* dnb, int cj_lane, unsigned m, unsigned u, unsigned wA,
                                          unsigned wB, int sci, bool central, int lane, AdjTypes<kBig>& types)
{
    const unsigned full = 0xffffffffu;
    const int      j = lane >> 2, ip = lane & 3;
#pragma unroll 1
    for (int jm = 0; jm < kJg; jm++)
    {
        unsigned  rem = (u >> (jm * kNcl)) & 0xffu;
        const int cj  = __shfl_sync(full, cj_lane, jm);
        if (!rem)
        {
            continue;
        }
        const float4   xj   = w.jx[jm * kCl + j], gj = w.jg[jm * kCl + j];
        const int      tj   = __float_as_int(gj.w);
        const float    qje  = xj.w * k.epsfac;
        // an empty slot has no pairs (two empty slots coincide)
        const unsigned mj   = tj == k.filler ? 0u : m >> (jm * kNcl);
        const unsigned xA   = wA >> (jm * kNcl), xB = wB >> (jm * kNcl);
        const int      diag = kExcl && central ? cj - sci * kNcl : -1;  // the diagonal i-cluster, if in 0 .. 7
        AdjJ<kBig>     dj;
        dj.x = dj.y = dj.z = dj.q = f2(0.0f);
#pragma unroll
        for (int n = 0; n < (kBig ? 2 : 1); n++)
        {
#pragma unroll
            for (int i = 0; i < 4; i++)
            {
                dj.hi[n][i] = dj.lo[n][i] = 0.0f;
            }
        }
        auto step = [&](int c) {
            bool  okA = (mj >> c) & 1u, okB = okA;
            float intA = 1.0f, intB = 1.0f;
            if (kExcl)
            {
                // the diagonal cluster pair counts j > i only
                okA  = okA && !(c == diag && j <= ip);
                okB  = okB && !(c == diag && j <= ip + 4);
                intA = ((xA >> c) & 1u) ? 1.0f : 0.0f;
                intB = ((xB >> c) & 1u) ? 1.0f : 0.0f;
            }
            adj_step<kEwald, kGE, kBig, kExcl>(k, nbfp_b, w, c, lane, xj, gj, qje, tj * 8, okA, okB, intA, intB, dj);
        };
#pragma unroll 1
        while (rem)
        {
            const int ca = __ffs(rem) - 1;
            rem &= rem - 1;
            if (rem)
            {
                // two independent steps share a basic block
                const int cb = __ffs(rem) - 1;
                rem &= rem - 1;
                step(ca);
                step(cb);
            }
            else
            {
                step(ca);
            }
        }
        // j side: the two slots, then the four ip lanes reduce-scattered to one component each
        float2      xy = make_float2(dj.x.x + dj.x.y, dj.y.x + dj.y.y);
        float2      zq = make_float2(dj.z.x + dj.z.y, -k.epsfac * (dj.q.x + dj.q.y));
        const bool  o1 = lane & 1, o2 = lane & 2;
        float2      keep = o2 ? zq : xy, send = o2 ? xy : zq;
        keep.x += __shfl_xor_sync(full, send.x, 2);
        keep.y += __shfl_xor_sync(full, send.y, 2);
        float one = (o1 ? keep.y : keep.x) + __shfl_xor_sync(full, o1 ? keep.x : keep.y, 1);
        atomicAdd(reinterpret_cast<float*>(&dnb[cj * kCl + j]) + ip, -one);
        // type pairs: D of row j turns into the B fragment (k = j-atoms ip and ip + 4, n = i type lane >> 2)
        // of the product with the one-hot j types
        const int   t0 = __shfl_sync(full, tj, 4 * ip), t1 = __shfl_sync(full, tj, 16 + 4 * ip);
        const float p[4] = { t0 == j ? 1.0f : 0.0f, kBig && t0 == j + 8 ? 1.0f : 0.0f, t1 == j ? 1.0f : 0.0f,
                             kBig && t1 == j + 8 ? 1.0f : 0.0f };
#pragma unroll
        for (int n = 0; n < (kBig ? 2 : 1); n++)
        {
            __syncwarp();  // the readers of the last product are done
            w.turn[lane] = make_float4(dj.hi[n][0] + dj.lo[n][0], dj.hi[n][1] + dj.lo[n][1], dj.hi[n][2] + dj.lo[n][2],
                                       dj.hi[n][3] + dj.lo[n][3]);
            __syncwarp();
            // element (j, type a) of d6 sits in lane 4 j + a / 2, component a & 1 (d12: + 2)
            const float* d = reinterpret_cast<const float*>(w.turn) + 16 * ip + 4 * (j >> 1) + (j & 1);
#pragma unroll
            for (int q = 0; q < 2; q++)
            {
                float h0, r0, h1, r1, hs[4] = { 0, 0, 0, 0 }, rs[4] = { 0, 0, 0, 0 };
                tf32_split(d[2 * q], h0, r0);
                tf32_split(d[64 + 2 * q], h1, r1);
                mma_tf32(hs, p, h0, h1);
                mma_tf32(rs, p, r0, r1);
                float(&sum)[4] = q == 0 ? types.s6[n] : types.s12[n];
#pragma unroll
                for (int i = 0; i < (kBig ? 4 : 2); i++)
                {
                    sum[i] += hs[i] + rs[i];
                }
            }
        }
    }
}

// FP64 sums per lane: (column tile, C fragment element, {6C6, 12C12})
template<bool kBig>
__host__ __device__ constexpr int adj_lane_sums()
{
    return kBig ? 16 : 4;
}

// Copies of the lanes' sums in a block: one per warp, or with 16 values a lane (32 KB for 8 warps, which
// would leave room for one block per SM) one that the warps add to atomically.
template<bool kBig>
__host__ __device__ constexpr int adj_sum_copies()
{
    return kBig ? 1 : kAdjWarps;
}

// The type terms of one list entry pair by pair: what the products with one-hot matrices cannot sum, since a term that
// is not finite (an upstream gradient that is not, or atoms so close that r^-14 overflows) times their zeros reaches
// every type pair.  Such a term goes to its own type pair here, as every other of the entry.  Lane (j, ip) as in
// adj_step; sums: the warp's FP64 type-pair sums (element 0 of lane 0).  (Arguments by value: an address taken of the
// caller's variables would put them, and through the shift vectors the whole DeviceView, into local memory.)
template<bool kGE>
__device__ __noinline__ void adj_types_by_pair(const AdjWarp* w, double* sums, const Cj4* cj4, const Excl* excl,
                                               const float4* xq, const float4* gnb, int sci, int shift, int cj4_start,
                                               int cj4_end, float rc2, float gE_lj, float cpot6, float cpot12, int filler)
{
    const int lane = threadIdx.x & 31, j = lane >> 2, ip = lane & 3;
    for (int g = cj4_start; g < cj4_end; g++)
    {
        const Imei     im = cj4[g].imei[j >> 2];
        const unsigned wA = excl[im.excl_ind].pair[(j & 3) * kCl + ip], wB = excl[im.excl_ind].pair[(j & 3) * kCl + ip + 4];
        for (int b = 0; b < 32; b++)
        {
            const int cj = cj4[g].cj[b / kNcl], c = b % kNcl, at = cj * kCl + j;
            if (!((im.imask >> b) & 1u))
            {
                continue;
            }
            const float4 xj = xq[at], gj = gnb[at];
            const int    tj = __float_as_int(gj.w);
            const bool   diag = shift == kCentral && cj == sci * kNcl + c;
            const float4 i0 = w->irec[c][0][ip], i1 = w->irec[c][1][ip], i2 = w->irec[c][2][ip], i3 = w->irec[c][3][ip];
            for (int h = 0; h < 2; h++)
            {
                const float dx = (h ? i0.y : i0.x) - xj.x, dy = (h ? i0.w : i0.z) - xj.y, dz = (h ? i1.y : i1.x) - xj.z;
                float       r2 = fmaf(dz, dz, fmaf(dy, dy, __fmul_rn(dx, dx)));
                // (the diagonal cluster pair counts j > i only)
                if (tj == filler || !(r2 < rc2) || !(((h ? wB : wA) >> b) & 1u) || (diag && j <= ip + 4 * h))
                {
                    continue;
                }
                r2                = fmaxf(r2, kMinDist2);
                float rinv        = fast_rsqrt(r2);
                rinv              = fmaf(rinv, fmaf(-0.5f * r2, rinv * rinv, 0.5f), rinv);
                const float rinv2 = rinv * rinv, rinv6 = rinv2 * rinv2 * rinv2;
                const float gx = (h ? i2.y : i2.x) - gj.x, gy = (h ? i2.w : i2.z) - gj.y, gz = (h ? i3.y : i3.x) - gj.z;
                const float gr6 = (gx * dx + gy * dy + gz * dz) * rinv6;
                float       d6 = gr6 * rinv2, d12 = gr6 * (rinv6 * rinv2);
                if (kGE)
                {
                    d6  = fmaf(gE_lj, fmaf(rinv6, 1.0f / 6.0f, cpot6), d6);
                    d12 = fmaf(gE_lj, fmaf(rinv6 * rinv6, 1.0f / 12.0f, cpot12), d12);
                }
                // the element of adj_flush that is (i type a, j type tj)
                const int a = __float_as_int(h ? i3.w : i3.z);
                double*   e = sums + 64 * (4 * (a >> 3) + (a & 1) + 2 * (tj >> 3)) + 4 * (tj & 7) + ((a & 7) >> 1);
                atomicAdd(e, -(double)d6);
                atomicAdd(e + 32, (double)d12);
            }
        }
    }
}

// One list entry.  gsum: the lane's FP64 type-pair sums (shared memory, stride 32).
template<bool kEwald, bool kGE, bool kBig>
__device__ __forceinline__ void adj_entry(const AdjConsts& k, const AdjPtrs& p, const Sci& s,
                                          const char* __restrict__ nbfp_b, AdjWarp& w, double* gsum, int lane)
{
    const unsigned full    = 0xffffffffu;
    const float    sx = p.shiftvec[3 * s.shift], sy = p.shiftvec[3 * s.shift + 1], sz = p.shiftvec[3 * s.shift + 2];
    const bool     central = (s.shift == kCentral);
    __syncwarp();
    // lane (c, ip) fills the records of the i-atoms ip and ip + 4 of i-cluster c
    {
        const int    c = lane >> 2, ip = lane & 3;
        const int    a = s.sci * kSc + c * kCl + ip;
        const float4 x0 = p.xq[a], x1 = p.xq[a + 4], g0 = p.gnb[a], g1 = p.gnb[a + 4];
        w.irec[c][0][ip] = make_float4(x0.x + sx, x1.x + sx, x0.y + sy, x1.y + sy);
        w.irec[c][1][ip] = make_float4(x0.z + sz, x1.z + sz, x0.w, x1.w);
        w.irec[c][2][ip] = make_float4(g0.x, g1.x, g0.y, g1.y);
        w.irec[c][3][ip] = make_float4(g0.z, g1.z, g0.w, g1.w);
    }
#pragma unroll
    for (int c = 0; c < kNcl; c++)
    {
        w.acc[c][lane]      = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        w.acc[c][32 + lane] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    AdjTypes<kBig> types;
#pragma unroll
    for (int n = 0; n < (kBig ? 2 : 1); n++)
    {
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            types.s6[n][i] = types.s12[n][i] = 0.0f;
        }
    }
    // the next group's record and j-atoms are loaded while a group is computed
    int4   rec_ime{};
    int    rec_cj = 0;
    float4 xr{}, gr{};
    auto load_record = [&](int g) {
        rec_ime = *reinterpret_cast<const int4*>(&p.cj4[g].imei[0]);
        rec_cj  = (lane < kJg) ? p.cj4[g].cj[lane] : 0;
    };
    auto load_atoms = [&]() {
        const int a = __shfl_sync(full, rec_cj, lane >> 3) * kCl + (lane & (kCl - 1));
        xr          = p.xq[a];
        gr          = p.gnb[a];
    };
    if (s.cj4_start < s.cj4_end)
    {
        load_record(s.cj4_start);
        load_atoms();
    }
    for (int j4 = s.cj4_start; j4 < s.cj4_end; j4++)
    {
        const int4 ime     = rec_ime;
        const int  cj_lane = rec_cj;
        __syncwarp();
        w.jx[lane] = xr;
        w.jg[lane] = gr;
        __syncwarp();
        if (j4 + 1 < s.cj4_end)
        {
            load_record(j4 + 1);
            load_atoms();
        }
        const unsigned m0 = (unsigned)ime.x, m1 = (unsigned)ime.z;
        const unsigned m  = lane < 16 ? m0 : m1;
        if ((ime.y | ime.w) == 0)
        {
            adj_group<kEwald, kGE, kBig, false>(k, nbfp_b, w, p.dnb, cj_lane, m, m0 | m1, ~0u, ~0u, s.sci, central,
                                                lane, types);
        }
        else
        {
            const unsigned* pair = p.excl[lane < 16 ? ime.y : ime.w].pair;
            const int       at   = ((lane >> 2) & 3) * kCl + (lane & 3);
            adj_group<kEwald, kGE, kBig, true>(k, nbfp_b, w, p.dnb, cj_lane, m, m0 | m1, pair[at], pair[at + 4], s.sci,
                                               central, lane, types);
        }
    }
    // the i-side sums: lane (c, ip) adds the eight j-lanes' slots of the atoms ip and ip + 4
    __syncwarp();
    {
        const int c = lane >> 2, ip = lane & 3;
        float4    t0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), t1 = t0;
#pragma unroll
        for (int j = 0; j < kCl; j++)
        {
            const float4 a = w.acc[c][4 * j + ip], b = w.acc[c][32 + 4 * j + ip];
            t0.x += a.x;
            t0.y += a.y;
            t0.z += a.z;
            t0.w += a.w;
            t1.x += b.x;
            t1.y += b.y;
            t1.z += b.z;
            t1.w += b.w;
        }
        const int at = s.sci * kSc + c * kCl + ip;
        red_add_v4(&p.dnb[at], t0.x, t0.z, t1.x, t1.z);
        red_add_v4(&p.dnb[at + 4], t0.y, t0.w, t1.y, t1.w);
    }
    float total = 0.0f;
#pragma unroll
    for (int n = 0; n < (kBig ? 2 : 1); n++)
    {
#pragma unroll
        for (int i = 0; i < (kBig ? 4 : 2); i++)
        {
            total += types.s6[n][i] + types.s12[n][i];
        }
    }
    if (__any_sync(full, !isfinite(total)))
    {
        adj_types_by_pair<kGE>(&w, gsum - lane, p.cj4, p.excl, p.xq, p.gnb, s.sci, s.shift, s.cj4_start, s.cj4_end, k.rc2,
                               k.gE_lj, k.cpot6, k.cpot12, k.filler);
        return;
    }
#pragma unroll
    for (int n = 0; n < (kBig ? 2 : 1); n++)
    {
#pragma unroll
        for (int i = 0; i < (kBig ? 4 : 2); i++)
        {
            const int v = n * 4 + i;
            if (kBig)
            {
                atomicAdd(&gsum[32 * (2 * v)], -(double)types.s6[n][i]);
                atomicAdd(&gsum[32 * (2 * v + 1)], (double)types.s12[n][i]);
            }
            else
            {
                gsum[32 * (2 * v)] -= (double)types.s6[n][i];
                gsum[32 * (2 * v + 1)] += (double)types.s12[n][i];
            }
        }
    }
}

// Dynamic shared memory: the type table, the warps' FP64 type-pair sums, the warps' slots.
template<bool kBig>
constexpr size_t adj_smem()
{
    return sizeof(float2) * kAdjRow * kAdjRow + sizeof(double) * adj_sum_copies<kBig>() * 32 * adj_lane_sums<kBig>()
           + sizeof(AdjWarp) * kAdjWarps;
}

// Type table in rows of 16, cleared sums.
template<bool kBig>
__device__ __forceinline__ void adj_setup(const DeviceView& v, float2* nbfp_s, double* gsum_s)
{
    const int nt1 = v.ntypes1;
    for (int m = threadIdx.x; m < nt1 * nt1; m += blockDim.x)
    {
        nbfp_s[(m / nt1) * kAdjRow + m % nt1] = v.nbfp[m];
    }
    for (int m = threadIdx.x; m < adj_sum_copies<kBig>() * 32 * adj_lane_sums<kBig>(); m += blockDim.x)
    {
        gsum_s[m] = 0.0;
    }
    __syncthreads();
}

// The block's type-pair sums into the global padded table: thread (value, lane) adds the warps' sums, one
// FP64 atomic per non-zero element and block.
template<bool kBig>
__device__ __forceinline__ void adj_flush(const DeviceView& v, const double* gsum_s, double* gnbfp)
{
    __syncthreads();
    constexpr int per = 32 * adj_lane_sums<kBig>();
    for (int m = threadIdx.x; m < per; m += blockDim.x)
    {
        double t = 0.0;
        for (int w = 0; w < adj_sum_copies<kBig>(); w++)
        {
            t += gsum_s[w * per + m];
        }
        const int val = m >> 5, lane = m & 31, i = (val >> 1) & 3, n = val >> 3;
        const int b = (lane >> 2) + 8 * (i >> 1), a = 2 * (lane & 3) + (i & 1) + 8 * n;  // j type, i type
        if (t != 0.0 && a < v.ntypes1 && b < v.ntypes1)
        {
            atomicAdd(&gnbfp[2 * (a * v.ntypes1 + b) + (val & 1)], t);
        }
    }
}

template<bool kEwald, bool kGE, bool kBig>
__global__ void __launch_bounds__(kAdjThreads, kAdjBlocksPerSm)
        k_backward(DeviceView v, const float4* gnb, float4* dnb, double* gnbfp, int* work_counter,
                   const double* gE)
{
    pdl_begin();
    extern __shared__ float4 adj_dyn[];
    float2* const  nbfp_s = reinterpret_cast<float2*>(adj_dyn);
    double* const  gsum_s = reinterpret_cast<double*>(nbfp_s + kAdjRow * kAdjRow);
    AdjWarp* const warps  = reinterpret_cast<AdjWarp*>(gsum_s + adj_sum_copies<kBig>() * 32 * adj_lane_sums<kBig>());
    adj_setup<kBig>(v, nbfp_s, gsum_s);
    if (v.hdr->status & (kStatusListOverflow | kStatusExclOverflow | kStatusGridOverflow))
    {
        return;
    }
    AdjConsts k = adj_consts(v);
    if (kGE)
    {
        k.gE_lj = (float)gE[0];
        k.gE_c  = (float)gE[1];
    }
    const int     warp   = threadIdx.x >> 5;
    const int     lane   = threadIdx.x & 31;
    const int     numSci = v.hdr->num_sci;
    const AdjPtrs p      = { v.xq, v.cj4, v.excl, v.shiftvec, gnb, dnb };
    for (;;)
    {
        int e = 0;
        if (lane == 0)
        {
            e = atomicAdd(work_counter, 1);
        }
        e = __shfl_sync(0xffffffffu, e, 0);
        if (e >= numSci)
        {
            break;
        }
        adj_entry<kEwald, kGE, kBig>(k, p, v.sci[e], reinterpret_cast<const char*>(nbfp_s), warps[warp],
                                     gsum_s + (kBig ? 0 : warp) * 32 * adj_lane_sums<kBig>() + lane, lane);
    }
    adj_flush<kBig>(v, gsum_s, gnbfp);
}

// The adjoint over all systems of a batch (shared type table and type-pair
// gradient sums; per-system upstream energy gradients gE[2 s], gE[2 s + 1]).
template<bool kEwald, bool kGE, bool kBig>
__global__ void __launch_bounds__(kAdjThreads, kAdjBlocksPerSm)
        k_batch_backward(DeviceView cv, const BatchSys* __restrict__ sys, const int* prefix, int nsys,
                         double* gnbfp, int* work_counter, const double* gE)
{
    pdl_begin();
    extern __shared__ float4 adj_dyn[];
    float2* const  nbfp_s = reinterpret_cast<float2*>(adj_dyn);
    double* const  gsum_s = reinterpret_cast<double*>(nbfp_s + kAdjRow * kAdjRow);
    AdjWarp* const warps  = reinterpret_cast<AdjWarp*>(gsum_s + adj_sum_copies<kBig>() * 32 * adj_lane_sums<kBig>());
    adj_setup<kBig>(cv, nbfp_s, gsum_s);
    AdjConsts k     = adj_consts(cv);
    const int warp  = threadIdx.x >> 5;
    const int lane  = threadIdx.x & 31;
    const int total = prefix[nsys];
    for (;;)
    {
        int e = 0;
        if (lane == 0)
        {
            e = atomicAdd(work_counter, 1);
        }
        e = __shfl_sync(0xffffffffu, e, 0);
        if (e >= total)
        {
            break;
        }
        const int       sidx = find_system(prefix, nsys, e);
        const BatchSys& b    = sys[sidx];
        if (kGE)
        {
            k.gE_lj = (float)gE[2 * sidx];
            k.gE_c  = (float)gE[2 * sidx + 1];
        }
        const AdjPtrs p = { b.xq, b.cj4, b.excl, b.shiftvec, b.gnb, b.dnb };
        adj_entry<kEwald, kGE, kBig>(k, p, b.sci[e - prefix[sidx]], reinterpret_cast<const char*>(nbfp_s), warps[warp],
                                     gsum_s + (kBig ? 0 : warp) * 32 * adj_lane_sums<kBig>() + lane, lane);
    }
    adj_flush<kBig>(cv, gsum_s, gnbfp);
}

// Batched upstream gradients to grid order, outputs cleared.
__global__ void k_batch_adj_prepare(const BatchSys* __restrict__ sys, BatchMap map, const float* gF,
                                    int* counter,
                                    double* gnbfp, int n_gnbfp)
{
    pdl_begin();
    // block 0 also clears the work queue and the FP64 type-pair gradient table
    if (blockIdx.x == 0)
    {
        for (int i = threadIdx.x; i < n_gnbfp; i += blockDim.x)
        {
            gnbfp[i] = 0.0;
        }
        if (threadIdx.x == 0)
        {
            *counter = 0;
        }
    }
    const int2      part = map.slots[blockIdx.x];
    const BatchSys& b    = sys[part.x];
    const int       k    = part.y + threadIdx.x;
    if (k >= b.hdr->num_cells * kSc)
    {
        return;
    }
    const int     a = b.atom_indices[k];
    const float*  g = gF + 3 * (size_t)(b.atom_base + (a >= 0 ? a : 0));
    const float   t = __int_as_float(b.tgrid[k]);
    const_cast<float4*>(b.gnb)[k] = (a >= 0) ? make_float4(g[0], g[1], g[2], t) : make_float4(0.0f, 0.0f, 0.0f, t);
    b.dnb[k]                      = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// Batched atom-order outputs, dL/dq with the self-energy term.
__global__ void k_batch_adj_finish(DeviceView cv, const BatchSys* __restrict__ sys, BatchMap map,
                                   const double* gE,
                                   float* gx, float* gq)
{
    pdl_begin();
    const int2      part = map.atoms[blockIdx.x];
    const BatchSys& b    = sys[part.x];
    const int       a    = part.y + threadIdx.x;
    if (a >= b.n)
    {
        return;
    }
    const int    k = b.cells[a];
    const float4 d = b.dnb[k];
    const size_t o = (size_t)b.atom_base + a;
    if (gx)
    {
        gx[3 * o]     = d.x;
        gx[3 * o + 1] = d.y;
        gx[3 * o + 2] = d.z;
    }
    if (gq)
    {
        const float q    = b.xq[k].w;
        const float self = (cv.coulomb == 0) ? -2.0f * cv.epsfac * cv.beta * 0.5641895835477563f * q
                                             : -cv.epsfac * cv.c_rf * q;
        gq[o]            = gE ? d.w + (float)gE[2 * part.x + 1] * self : d.w;
    }
}

// Charges of all systems (concatenated atom order) into xq.w and each system's q.
__global__ void k_batch_set_q(const BatchSys* __restrict__ sys, BatchMap map, const float* q)
{
    pdl_begin();
    const int2      part = map.slots[blockIdx.x];
    const BatchSys& b    = sys[part.x];
    const int       k    = part.y + threadIdx.x;
    if (k >= b.hdr->num_cells * kSc)
    {
        return;
    }
    const int a = b.atom_indices[k];
    if (a >= 0)
    {
        const float qa                  = q[(size_t)b.atom_base + a];
        const_cast<float4*>(b.xq)[k].w  = qa;
        b.q[a]                          = qa;
    }
}

constexpr int kLossThreads = 256;

// Loss sum |F - F_target|^2 (FP64) and its gradient 2 (F - F_target) per coordinate.
__global__ void k_match_loss(const float* f, const float* ft, size_t n3, float* gF,
                             double* loss)
{
    pdl_begin();
    __shared__ double sum[kLossThreads / 32];
    double            acc = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += (size_t)gridDim.x * blockDim.x)
    {
        const float d = f[i] - ft[i];
        gF[i]         = 2.0f * d;
        acc += (double)d * (double)d;
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    }
    if ((threadIdx.x & 31) == 0)
    {
        sum[threadIdx.x >> 5] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (int w = 1; w < kLossThreads / 32; w++)
        {
            acc += sum[w];
        }
        if (acc != 0.0)
        {
            atomicAdd(loss, acc);
        }
    }
}

// Upstream force gradients to grid order; clears the output accumulators.
// Per grid slot: the coordinates of this evaluation into xq and xqp (as k_convert_x, with the box shifts of
// the last search) when x is given, the upstream force gradient (and the type) in grid order, a cleared dL/dx
// accumulator; block 0 also clears the work queue and the FP64 type-pair gradient table (in place
// of separate memsets).
__global__ void k_adj_prepare(DeviceView v, const float* x, const float* gF, float4* gnb,
                              float4* dnb, int* counter, double* gnbfp, int n_gnbfp)
{
    pdl_begin();
    if (blockIdx.x == 0)
    {
        for (int i = threadIdx.x; i < n_gnbfp; i += blockDim.x)
        {
            gnbfp[i] = 0.0;
        }
        if (threadIdx.x == 0)
        {
            *counter = 0;
        }
    }
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= v.hdr->num_cells * kSc)
    {
        return;
    }
    const int   a = v.atom_indices[k];
    const int   t = v.tgrid[k];
    float       g[3] = { 0.0f, 0.0f, 0.0f };
    if (a >= 0)
    {
        for (int d = 0; d < 3; d++)
        {
            g[d] = gF[3 * a + d];
        }
    }
    if (x && a >= 0)
    {
        const float q    = v.xq[k].w;
        const int   code = v.image[a];
        float       c[3];
        for (int d = 0; d < 3; d++)
        {
            const int sh = (int)(signed char)((code >> (8 * d)) & 0xff);
            c[d]         = (sh == 0) ? x[3 * a + d] : x[3 * a + d] + (float)sh * v.g.box[d];
        }
        v.xq[k] = make_float4(c[0], c[1], c[2], q);
        // the cluster-packed copy follows: a full prune tests the atoms of xq against those of xqp
        write_packed_slot(v.xqp, k, c[0], c[1], c[2], q, t);
    }
    gnb[k] = make_float4(g[0], g[1], g[2], __int_as_float(t));
    dnb[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// Atom-order outputs; dL/dq also gets the self-energy term.  Block 0 also copies the type-pair
// gradients out of the padded (nt+1)^2 table into the caller's nt^2 one when gout is given (the
// adjoint kernel has finished: no separate launch).
__global__ void k_adj_finish(DeviceView v, const float4* dnb, const double* gE, float* gx,
                             float* gq, const double* gpad, double* gout)
{
    pdl_begin();
    if (gout && blockIdx.x == 0)
    {
        const int nt = v.ntypes1 - 1;
        for (int m = threadIdx.x; m < nt * nt; m += blockDim.x)
        {
            const int i = m / nt, j = m % nt;
            gout[2 * m]     = gpad[2 * (i * (nt + 1) + j)];
            gout[2 * m + 1] = gpad[2 * (i * (nt + 1) + j) + 1];
        }
    }
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= v.n)
    {
        return;
    }
    const int    k = v.cells[a];
    const float4 d = dnb[k];
    if (gx)
    {
        gx[3 * a]     = d.x;
        gx[3 * a + 1] = d.y;
        gx[3 * a + 2] = d.z;
    }
    if (gq)
    {
        const float q    = v.xq[k].w;
        // d/dq of -epsfac beta/sqrt(pi) q^2 (Ewald) or -epsfac c_rf q^2 / 2 (RF)
        const float self = (v.coulomb == 0) ? -2.0f * v.epsfac * v.beta * 0.5641895835477563f * q
                                            : -v.epsfac * v.c_rf * q;
        gq[a]            = gE ? d.w + (float)gE[1] * self : d.w;
    }
}

// Lorentz-Berthelot type table {6 C6, 12 C12} from per-type sigma and epsilon (one block):
// sigma_ij = (sigma_i + sigma_j) / 2, epsilon_ij = sqrt(epsilon_i epsilon_j), C6 = 4 eps s^6,
// C12 = 4 eps s^12 (the combination nblib applies, api/nblib/gmxsetup.cpp:143-166).
__global__ void k_lb_table(const double* sig, const double* eps, int nt, double* table)
{
    pdl_begin();
    for (int m = threadIdx.x; m < nt * nt; m += blockDim.x)
    {
        const int    i = m / nt, j = m - (m / nt) * nt;
        const double s  = 0.5 * (sig[i] + sig[j]);
        const double e  = sqrt(eps[i] * eps[j]);
        const double s2 = s * s;
        const double s6 = s2 * s2 * s2;
        const double c6 = 4.0 * e * s6;
        table[2 * m]     = 6.0 * c6;
        table[2 * m + 1] = 12.0 * (c6 * s6);
    }
}

constexpr int kLbThreads = 256;
constexpr int kLbTerms   = 12;  // 55 types, what two tables in 48 KB allow

// Its adjoint: d L / d sigma_k and d L / d epsilon_k from d L / d table (one block; every type's
// sums run over its row and column in a fixed order).  d epsilon_ij / d epsilon_i is written
// epsilon_j / (2 epsilon_ij), as the derivative of the square root of the product.
__global__ void k_lb_table_backward(const double* sig, const double* eps, int nt,
                                    const double* gt, double* gsig, double* geps)
{
    pdl_begin();
    extern __shared__ double lbs[];  // [2][nt * nt]: d L / d sigma_ij, d L / d epsilon_ij
    double* gs = lbs;
    double* ge = lbs + nt * nt;
    for (int m = threadIdx.x; m < nt * nt; m += blockDim.x)
    {
        const int    i = m / nt, j = m - (m / nt) * nt;
        const double s  = 0.5 * (sig[i] + sig[j]);
        const double e  = sqrt(eps[i] * eps[j]);
        const double s2 = s * s;
        const double s5 = s2 * s2 * s;
        const double s6 = s5 * s;
        const double g6 = gt[2 * m], g12 = gt[2 * m + 1];
        // 6 C6 = 24 e s^6, 12 C12 = 48 e s^12
        gs[m] = g6 * 144.0 * e * s5 + g12 * 576.0 * e * s5 * s6;
        ge[m] = g6 * 24.0 * s6 + g12 * 48.0 * s6 * s6;
    }
    __syncthreads();
    // the terms of row k (sigma_k, epsilon_k as the first index) and column k (as the second) in place of the
    // derivatives, a thread each: square roots and quotients in FP64 one after the other took most of 10.8 us
    double ts[kLbTerms], te[kLbTerms];
#pragma unroll
    for (int u = 0; u < kLbTerms; u++)
    {
        const int m = threadIdx.x + u * kLbThreads;
        if (m < nt * nt)
        {
            const int k = m / nt, j = m - k * nt;
            ts[u]       = 0.5 * gs[m] + 0.5 * gs[j * nt + k];
            te[u]       = (ge[m] + ge[j * nt + k]) * (eps[j] / (2.0 * sqrt(eps[k] * eps[j])));
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kLbTerms; u++)
    {
        const int m = threadIdx.x + u * kLbThreads;
        if (m < nt * nt)
        {
            gs[m] = ts[u];
            ge[m] = te[u];
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nt; k += blockDim.x)
    {
        double as = 0.0, ae = 0.0;
        for (int j = 0; j < nt; j++)
        {
            as += gs[k * nt + j];
            ae += ge[k * nt + j];
        }
        gsig[k] = as;
        geps[k] = ae;
    }
}

} // namespace

int adjoint_max_types1()
{
    return kAdjMaxTypes1;
}

cudaError_t launch_lb_table(const double* sig, const double* eps, int nt, double* table, cudaStream_t s)
{
    launch_pdl(k_lb_table, 1, 256, 0, s, sig, eps, nt, table);
    return cudaGetLastError();
}

cudaError_t launch_lb_table_backward(const double* sig, const double* eps, int nt, const double* gtable,
                                     double* gsig, double* geps, cudaStream_t s)
{
    launch_pdl(k_lb_table_backward, 1, kLbThreads, 2 * sizeof(double) * nt * nt, s, sig, eps, nt, gtable, gsig, geps);
    return cudaGetLastError();
}

namespace
{

template<bool kEwald, bool kGE, bool kBig>
cudaError_t backward_t(const DeviceView& v, const float4* gnb, float4* dnb, double* gnbfp, int* counter,
                       const double* gE, int num_sms, cudaStream_t s)
{
    constexpr size_t smem = adj_smem<kBig>();
    cudaError_t      e    = smem_optin<k_backward<kEwald, kGE, kBig>>(smem, smem);
    if (e == cudaSuccess)
    {
        e = launch_pdl(k_backward<kEwald, kGE, kBig>, num_sms * kAdjBlocksPerSm, kAdjThreads, smem, s, v, gnb, dnb,
                       gnbfp, counter, gE);
    }
    return e;
}

template<bool kEwald, bool kGE, bool kBig>
cudaError_t batch_backward_t(const DeviceView& cv, const BatchSys* sys, const int* prefix, int nsys, double* gnbfp,
                             int* counter, const double* gE, int num_sms, cudaStream_t s)
{
    constexpr size_t smem = adj_smem<kBig>();
    cudaError_t      e    = smem_optin<k_batch_backward<kEwald, kGE, kBig>>(smem, smem);
    if (e == cudaSuccess)
    {
        e = launch_pdl(k_batch_backward<kEwald, kGE, kBig>, num_sms * kAdjBlocksPerSm, kAdjThreads, smem, s, cv, sys,
                       prefix, nsys, gnbfp, counter, gE);
    }
    return e;
}

// More types than the 8 rows (and columns) of one tensor-core tile, which the filler type does not count
// toward: its pairs are never in range.
bool adj_big(const DeviceView& v)
{
    return v.ntypes1 - 1 > 8;
}

} // namespace

cudaError_t launch_backward(const DeviceView& v, const float* d_x, const float* d_gF, const double* d_gE,
                            float4* gnb, float4* dnb, double* d_gnbfp, int* counter, float* d_gx, float* d_gq,
                            double* d_gnbfp_out, int num_sms, cudaStream_t s)
{
    const int tb    = 256;
    const int slots = v.g.cells_capacity * kSc;
    launch_pdl(k_adj_prepare, (slots + tb - 1) / tb, tb, 0, s, v, d_x, d_gF, gnb, dnb, counter, d_gnbfp,
               2 * v.ntypes1 * v.ntypes1);
    using Launch = cudaError_t (*)(const DeviceView&, const float4*, float4*, double*, int*, const double*, int,
                                   cudaStream_t);
    // [Ewald][energy gradients][more than 8 types]
    static const Launch table[2][2][2] = {
        { { backward_t<false, false, false>, backward_t<false, false, true> },
          { backward_t<false, true, false>, backward_t<false, true, true> } },
        { { backward_t<true, false, false>, backward_t<true, false, true> },
          { backward_t<true, true, false>, backward_t<true, true, true> } },
    };
    const cudaError_t e = table[v.coulomb == 0][d_gE != nullptr][adj_big(v)](v, gnb, dnb, d_gnbfp, counter, d_gE,
                                                                              num_sms, s);
    if (e != cudaSuccess)
    {
        return e;
    }
    launch_pdl(k_adj_finish, std::max(1, (v.n + tb - 1) / tb), tb, 0, s, v, dnb, d_gE, d_gx, d_gq, d_gnbfp,
               d_gnbfp_out);
    return cudaGetLastError();
}

cudaError_t launch_batch_backward(const DeviceView& cv, const BatchSys* sys, const int* prefix, int nsys,
                                  const BatchMap& map, const float* d_gF, const double* d_gE,
                                  double* d_gnbfp, int* counter, float* d_gx, float* d_gq, int num_sms, cudaStream_t s)
{
    launch_pdl(k_batch_adj_prepare, map.nslots, kBatchPart, 0, s, sys, map, d_gF, counter, d_gnbfp,
               2 * cv.ntypes1 * cv.ntypes1);
    using Launch = cudaError_t (*)(const DeviceView&, const BatchSys*, const int*, int, double*, int*, const double*,
                                   int, cudaStream_t);
    // [Ewald][energy gradients][more than 8 types]
    static const Launch table[2][2][2] = {
        { { batch_backward_t<false, false, false>, batch_backward_t<false, false, true> },
          { batch_backward_t<false, true, false>, batch_backward_t<false, true, true> } },
        { { batch_backward_t<true, false, false>, batch_backward_t<true, false, true> },
          { batch_backward_t<true, true, false>, batch_backward_t<true, true, true> } },
    };
    const cudaError_t e = table[cv.coulomb == 0][d_gE != nullptr][adj_big(cv)](cv, sys, prefix, nsys, d_gnbfp, counter,
                                                                                d_gE, num_sms, s);
    if (e != cudaSuccess)
    {
        return e;
    }
    launch_pdl(k_batch_adj_finish, map.natoms, kBatchPart, 0, s, cv, sys, map, d_gE, d_gx, d_gq);
    return cudaGetLastError();
}

cudaError_t launch_batch_set_q(const BatchSys* sys, const BatchMap& map, const float* d_q, cudaStream_t s)
{
    launch_pdl(k_batch_set_q, map.nslots, kBatchPart, 0, s, sys, map, d_q);
    return cudaGetLastError();
}

cudaError_t launch_match_loss(const float* d_f, const float* d_ft, size_t n3, float* d_gF, double* d_loss,
                              int num_sms, cudaStream_t s)
{
    cudaMemsetAsync(d_loss, 0, sizeof(double), s);
    const size_t need = (n3 + kLossThreads - 1) / kLossThreads;
    launch_pdl(k_match_loss, (int)std::max<size_t>(1, std::min<size_t>(need, num_sms * 4)), kLossThreads, 0, s, d_f, d_ft,
               n3, d_gF, d_loss);
    return cudaGetLastError();
}

cudaError_t launch_set_nbfp(const DeviceView& v, const float* d_nbfp, cudaStream_t s)
{
    return launch_set_parameters(v, nullptr, d_nbfp, s);
}

// Charges and LJ parameters for force matching: q (atom order) into xq.w and the
// nbfp table (with the all-zero filler type); the self energy follows the charges.
__global__ void k_set_q(DeviceView v, const float* q)
{
    pdl_begin();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= v.hdr->num_cells * kSc)
    {
        return;
    }
    const int a = v.atom_indices[k];
    if (a >= 0)
    {
        v.xq[k].w = q[a];
    }
}

__global__ void k_set_nbfp(float2* nbfp, const float* src, int nt)
{
    pdl_begin();
    const int m   = blockIdx.x * blockDim.x + threadIdx.x;
    const int nt1 = nt + 1;
    if (m >= nt1 * nt1)
    {
        return;
    }
    const int i = m / nt1, j = m % nt1;
    nbfp[m]     = (i < nt && j < nt) ? make_float2(src[2 * (i * nt + j)], src[2 * (i * nt + j) + 1])
                                     : make_float2(0.0f, 0.0f);
}

__global__ void k_compact_gnbfp(const double* padded, double* out, int nt)
{
    pdl_begin();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nt * nt)
    {
        return;
    }
    const int i = m / nt, j = m % nt;
    out[2 * m]     = padded[2 * (i * (nt + 1) + j)];
    out[2 * m + 1] = padded[2 * (i * (nt + 1) + j) + 1];
}

cudaError_t launch_compact_gnbfp(const double* padded, double* out, int nt, cudaStream_t s)
{
    launch_pdl(k_compact_gnbfp, (nt * nt + 255) / 256, 256, 0, s, padded, out, nt);
    return cudaGetLastError();
}

cudaError_t launch_set_parameters(const DeviceView& v, const float* d_q, const float* d_nbfp, cudaStream_t s)
{
    const int tb = 256;
    if (d_q)
    {
        cudaMemcpyAsync(const_cast<float*>(v.q), d_q, sizeof(float) * v.n, cudaMemcpyDeviceToDevice, s);
        launch_pdl(k_set_q, (v.g.cells_capacity * kSc + tb - 1) / tb, tb, 0, s, v, d_q);
    }
    if (d_nbfp)
    {
        const int nt = v.ntypes1 - 1;
        launch_pdl(k_set_nbfp, (v.ntypes1 * v.ntypes1 + tb - 1) / tb, tb, 0, s, const_cast<float2*>(v.nbfp), d_nbfp,
                   nt);
    }
    return cudaGetLastError();
}

} // namespace nbx
