// Cluster-pair search on the GPU into the nbnxm GPU list layout.
//
// Follows nbnxn_make_pairlist_part (src/gromacs/nbnxm/pairlist.cpp:3076-3582)
// for one grid with full periodicity and a rectangular box, with
// make_cluster_list_supersub (:1090-1244), get_cell_range (:286-309),
// boundingbox_only_distance2 (:2841-2878), setSelfAndNewtonExclusionsGpu
// (:880-904) and setExclusionsForIEntry for GPU lists (:1874-1972).
//
// Count pass: one block per i-cell (super-cluster), with the reference's single-precision
// arithmetic (this file is compiled with --fmad=false).  Its shifts, a lane each, give the
// candidate columns; a thread per column finds its z-range of j-cells; the flat sequence of
// j-cells, in the reference's order, goes through shared memory a window at a time: a warp
// tests four of them at once, lane (cell, j-cluster) its j-cluster's bounding box against the
// 8 i-clusters.  The j-clusters found are stored as per-cell records (index, 8-bit i-cluster
// mask) in order, with one code per entry, and the cell's entry / cj4 counts are written.  After
// a prefix sum of the counts, the emit pass (one block per list entry) turns the records into
// sci / cj4 entries at fixed offsets, with the outer masks and per-group pair counts, and sets
// the diagonal and topology exclusion masks.
#include "nbx_internal.cuh"

#include <cstddef>

namespace nbx
{
namespace
{

constexpr int kMaxCj4PerEntry = 1024;  // per (i-cell, shift) entry; beyond it the list overflows

__device__ __forceinline__ void set_status(ListHeader* hdr, unsigned bits)
{
    atomicOr(&hdr->status, bits);
}

__device__ __forceinline__ float sq(float x)
{
    return x * x;
}

// get_cell_range (pairlist.cpp:286-309), lower corner 0.
__device__ void get_cell_range(float b0, float b1, int numCells, float cellSize, float invCellSize, float d2,
                               float rlist, int* cf, int* cl)
{
    const float listRangeBBToCell2 = rlist * rlist;
    const float distanceInCells    = (b0 - 0.0f) * invCellSize;
    int         f                  = max((int)distanceInCells, 0);
    while (f > 0 && d2 + sq((b0 - 0.0f) - (float)(f - 1 + 1) * cellSize) < listRangeBBToCell2)
    {
        f--;
    }
    int l = min((int)((b1 - 0.0f) * invCellSize), numCells - 1);
    while (l < numCells - 1 && d2 + sq((float)(l + 1) * cellSize - (b1 - 0.0f)) < listRangeBBToCell2)
    {
        l++;
    }
    *cf = f;
    *cl = l;
}

__device__ __forceinline__ float max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Every operation rounded: packed products and sums would be contracted into fused multiply-adds
// whatever the compiler is told, so these are scalar.
__device__ __forceinline__ float norm2(float dx, float dy, float dz)
{
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// clusterBoundingBoxDistance2 (pairlist.cpp:351-372) of i-clusters i and i + 1 to one j-cluster, both
// differences of a dimension in packed arithmetic (the same roundings).
// x, y: {lower x, -upper x, lower y, -upper y}, z: {lower z, -upper z} of both; jx, jy, jz: {-upper, lower}.
__device__ __forceinline__ float2 bb_dist2(const float4 xy0, const float4 xy1, const float4 z, const float2 jx,
                                           const float2 jy, const float2 jz)
{
    const float2 x0 = __fadd2_rn(make_float2(xy0.x, xy0.y), jx), x1 = __fadd2_rn(make_float2(xy1.x, xy1.y), jx);
    const float2 y0 = __fadd2_rn(make_float2(xy0.z, xy0.w), jy), y1 = __fadd2_rn(make_float2(xy1.z, xy1.w), jy);
    const float2 z0 = __fadd2_rn(make_float2(z.x, z.y), jz), z1 = __fadd2_rn(make_float2(z.z, z.w), jz);
    return make_float2(norm2(max3(x0.x, x0.y, 0.0f), max3(y0.x, y0.y, 0.0f), max3(z0.x, z0.y, 0.0f)),
                       norm2(max3(x1.x, x1.y, 0.0f), max3(y1.x, y1.y, 0.0f), max3(z1.x, z1.y, 0.0f)));
}

constexpr int kEmitStage = 512;  // j-lists up to this length are staged in shared memory for the
                                 // exclusion lookups

constexpr int kShiftSlots   = kCentral + 1;  // shifts 0 .. central, the visiting order
constexpr int kManyCells    = 1200;          // grid capacity from which a cell takes two warps
constexpr int kCellWindow   = 128;           // candidate j-cells in shared memory at a time
static_assert(kShiftSlots <= kMaxEntriesPerCell && kShiftSlots <= 32, "one lane and one entry code per shift");

// The i-cell under one shift: its bounds, the candidate columns (cx major) and their first number
// among the columns of all shifts.
struct ShiftRange
{
    float bx0, bx1, by0, by1, bz0, bz1;
    float d2z, bz1_frac;
    float shx, shy, shz;
    int   cxf, cyf, ny;
};

struct CountSmem
{
    float4        bbi_xy[kShiftSlots][kNcl];  // shifted cluster bounding boxes: {lower, -upper} of x and y
    float2        bbi_z[kShiftSlots][kNcl];   // and of z
    uint2         masks[kCellWindow];                                    // i-cluster masks of the 8 j-clusters
    int           cell[kCellWindow];                                     // candidate j-cells
    unsigned char cell_shift[kCellWindow];
    ShiftRange    sr[kShiftSlots];
    int           col0[32];  // first column of each shift
    int           nj[32];    // j-clusters found per shift
    int           warp_sum[2][4];
    int           ncols, ci_x, ci_y, pairs;
    unsigned      active;  // shifts with candidate columns
    int2          flag[4][32];  // per warp: {j-cluster, shift * 8 + i-cluster} to check by atoms
};

// Inclusive prefix sum over the block; *total receives the sum of all threads.
template<int kWarps>
__device__ __forceinline__ int block_scan(int x, int* warp_sum, int* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int       incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
        {
            incl += t;
        }
    }
    if (lane == 31)
    {
        warp_sum[warp] = incl;
    }
    __syncthreads();
    int sum = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++)
    {
        incl += w < warp ? warp_sum[w] : 0;
        sum += warp_sum[w];
    }
    *total = sum;
    return incl;
}

// The shifts of i-cell ci, lane = shift (one warp): their ranges of candidate columns.
__device__ __forceinline__ void shift_ranges(const DeviceView& v, int ci, CountSmem& sm)
{
    const unsigned full = 0xffffffffu;
    const int      lane = threadIdx.x & 31;
    const float*   box  = v.g.box;
    const float    rlist = v.rlist, rlist2 = v.rlist2;
    const float2   bbcz_i = v.bbcz[ci];
    // column of this cell (next_ci, pairlist.cpp:2808-2836): the last that starts at or before it; the
    // window shrinks 32-fold per step
    int ci_xy = 0;
    for (int len = v.g.ncol; len > 1;)
    {
        const int  step = (len + 31) / 32;
        const int  c    = ci_xy + lane * step;
        const bool le   = c < ci_xy + len && v.cxy_ind[c] <= ci;
        const int  lo   = ci_xy + (__popc(__ballot_sync(full, le)) - 1) * step;
        len             = min(step, ci_xy + len - lo);
        ci_xy           = lo;
    }
    const int ci_x = ci_xy / v.g.ncy;
    const int ci_y = ci_xy - ci_x * v.g.ncy;
    const int shp_x = (box[0] < rlist) ? 2 : 1;
    const int tz = lane / 15 - 1, ty = lane / 5 % 3 - 1, tx = lane % 5 - 2;
    int       ncol = 0;
    if (lane < kShiftSlots && abs(tx) <= shp_x)
    {
        const float d2cx = 0.0f;
        const float shz  = (float)tz * box[2];
        const float bz0  = bbcz_i.x + shz;
        const float bz1  = bbcz_i.y + shz;
        float       d2z;
        if (tz == 0)
        {
            d2z = 0.0f;
        }
        else if (tz < 0)
        {
            d2z = sq(bz1);
        }
        else
        {
            d2z = sq(bz0 - box[2]);
        }
        const float d2z_cx = d2z + d2cx;
        if (!(d2z_cx >= rlist2))
        {
            float bz1_frac = bz1 / (float)(v.cxy_ind[ci_xy + 1] - v.cxy_ind[ci_xy]);
            if (bz1_frac < 0.0f)
            {
                bz1_frac = 0.0f;
            }
            const float shy = (float)ty * box[1] + (float)tz * 0.0f;
            const float by0 = 0.0f + (float)ci_y * v.g.cs[1] + shy;
            const float by1 = 0.0f + ((float)ci_y + 1.0f) * v.g.cs[1] + shy;
            int         cyf, cyl;
            get_cell_range(by0, by1, v.g.ncy, v.g.cs[1], v.g.ics[1], d2z_cx, rlist, &cyf, &cyl);
            float d2z_cy = d2z;
            if (by1 < 0.0f)
            {
                d2z_cy = d2z_cy + sq(0.0f - by1);
            }
            else if (by0 > box[1])
            {
                d2z_cy = d2z_cy + sq(by0 - box[1]);
            }
            const float shx = (float)tx * box[0] + (float)ty * 0.0f + (float)tz * 0.0f;
            const float bx0 = 0.0f + (float)ci_x * v.g.cs[0] + shx;
            const float bx1 = 0.0f + ((float)ci_x + 1.0f) * v.g.cs[0] + shx;
            int         cxf = 0, cxl = -1;
            if (cyf <= cyl)
            {
                get_cell_range(bx0, bx1, v.g.ncx, v.g.cs[0], v.g.ics[0], d2z_cy, rlist, &cxf, &cxl);
            }
            if (cxf <= cxl)
            {
                if (lane == kCentral && cxf < ci_x)
                {
                    cxf = ci_x;
                }
                const int ny = cyl - cyf + 1;
                ncol         = max(cxl - cxf + 1, 0) * ny;
                sm.sr[lane]  = { bx0, bx1, by0, by1, bz0, bz1, d2z, bz1_frac, shx, shy, shz, cxf, cyf, ny };
            }
        }
    }
    int incl = ncol;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int t = __shfl_up_sync(full, incl, o);
        if (lane >= o)
        {
            incl += t;
        }
    }
    sm.col0[lane]         = incl - ncol;
    sm.nj[lane]           = 0;
    const unsigned active = __ballot_sync(full, ncol > 0);
    if (lane == 31)
    {
        sm.active = active;
        sm.ncols = incl;
        sm.ci_x  = ci_x;
        sm.ci_y  = ci_y;
        sm.pairs = 0;
    }
}

// The z-range of j-cells of candidate column c (numbered over all shifts); *count 0 when none.
__device__ __forceinline__ void column_cells(const DeviceView& v, int ci, const CountSmem& sm, int c, int* shift,
                                             int* first, int* count)
{
    int s = 0;
    for (unsigned m = sm.active; m; m &= m - 1u)
    {
        const int q = __ffs(m) - 1;
        s           = sm.col0[q] <= c ? q : s;
    }
    const ShiftRange& r = sm.sr[s];
    *shift              = s;
    const float rlist2  = v.rlist2;
    const float listRangeBBToJCell2 = v.rlist * v.rlist;
    const float d2z = r.d2z, bz0 = r.bz0, bz1 = r.bz1;
    const int   k  = c - sm.col0[s];
    const int   cx = r.cxf + k / r.ny;
    const int   cy = r.cyf + k % r.ny;
    const int   columnStart = v.cxy_ind[cx * v.g.ncy + cy];
    const int   columnEnd   = v.cxy_ind[cx * v.g.ncy + cy + 1];
    const float cx_real = (float)cx;
    float       d2zx    = d2z;
    if (0.0f + cx_real * v.g.cs[0] > r.bx1)
    {
        d2zx = d2zx + sq(0.0f + cx_real * v.g.cs[0] - r.bx1);
    }
    else if (0.0f + (cx_real + 1.0f) * v.g.cs[0] < r.bx0)
    {
        d2zx = d2zx + sq(0.0f + (cx_real + 1.0f) * v.g.cs[0] - r.bx0);
    }
    const int   cyf_x   = (cx == 0 && s == kCentral && r.cyf < sm.ci_y) ? sm.ci_y : r.cyf;
    const float cy_real = (float)cy;
    float       d2zxy   = d2zx;
    if (0.0f + cy_real * v.g.cs[1] > r.by1)
    {
        d2zxy = d2zxy + sq(0.0f + cy_real * v.g.cs[1] - r.by1);
    }
    else if (0.0f + (cy_real + 1.0f) * v.g.cs[1] < r.by0)
    {
        d2zxy = d2zxy + sq(0.0f + (cy_real + 1.0f) * v.g.cs[1] - r.by0);
    }
    if (!(cy >= cyf_x && columnStart < columnEnd && d2zxy < listRangeBBToJCell2))
    {
        return;
    }
    int midCell = columnStart + (int)(r.bz1_frac * (float)(columnEnd - columnStart));
    if (midCell >= columnEnd)
    {
        midCell = columnEnd - 1;
    }
    const float d2xy = d2zxy - d2z;
    // the walks up and down from the middle cell read four cells' bounds at a time
    int  down = midCell;
    bool more = true;
    while (more && down >= columnStart)
    {
        float u[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            u[q] = v.bbcz[max(down - q, columnStart)].y;
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            more = more && down >= columnStart && (u[q] >= bz0 || d2xy + sq(u[q] - bz0) < rlist2);
            down -= more ? 1 : 0;
        }
    }
    int firstCell = down + 1;
    int up        = midCell + 1;
    more          = true;
    while (more && up < columnEnd)
    {
        float l[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            l[q] = v.bbcz[min(up + q, columnEnd - 1)].x;
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            more = more && up < columnEnd && (l[q] <= bz1 || d2xy + sq(l[q] - bz1) < rlist2);
            up += more ? 1 : 0;
        }
    }
    const int lastCell = up - 1;
    if (s == kCentral && firstCell < ci)
    {
        firstCell = ci;
    }
    if (lastCell >= firstCell)
    {
        *first = firstCell;
        *count = lastCell - firstCell + 1;
    }
}

// Bound by latency: a cell at a corner of the box has eight shifts with columns of their own.  With one warp a
// cell, which took shift after shift, 45k atoms needed 47.4 us, now 19.6 us; 960k atoms fill the GPU and
// stay at 126 us (windows of 512 j-cells, 14 KB a block, leave less L1: 149 us).
template<int kWarps>
__global__ void __launch_bounds__(32 * kWarps, 32 / kWarps) k_search_count(DeviceView v)
{
    constexpr int kThreads = 32 * kWarps;
    pdl_begin();
    __shared__ CountSmem sm;
    const int            ci = blockIdx.x;
    if (ci >= v.hdr->num_cells)
    {
        return;
    }
    const unsigned full  = 0xffffffffu;
    const int      tid   = threadIdx.x;
    const int      lane  = tid & 31;
    const int      warp  = tid >> 5;
    const float    rlist2 = v.rlist2, rbb2 = v.rbb2;
    if (warp == 0)
    {
        shift_ranges(v, ci, sm);
    }
    __syncthreads();
    // shifted i-cluster bounding boxes (set_icell_bb, pairlist.cpp:2260-2303)
    if (lane < kNcl)
    {
        const float4 l = v.bb[2 * (ci * kNcl + lane)];
        const float4 h = v.bb[2 * (ci * kNcl + lane) + 1];
        int          w = 0;
        for (unsigned m = sm.active; m; m &= m - 1u)
        {
            if (w == warp)
            {
                const int         s = __ffs(m) - 1;
                const ShiftRange& r = sm.sr[s];
                sm.bbi_xy[s][lane]  = make_float4(l.x + r.shx, -(h.x + r.shx), l.y + r.shy, -(h.y + r.shy));
                sm.bbi_z[s][lane]   = make_float2(l.z + r.shz, -(h.z + r.shz));
            }
            w = w + 1 == kWarps ? 0 : w + 1;
        }
    }
    int* const           rec_cj = v.rec_cj + (size_t)ci * v.rec_cap;
    unsigned char* const rec_m  = v.rec_m + (size_t)ci * v.rec_cap;
    int                  rec_n  = 0;  // records of this cell so far
    unsigned             pairs  = 0u;  // cluster pairs found by this lane
    const int            ncols  = sm.ncols;
    // The candidate columns of all shifts (the reference's visiting order), a thread each; a block scan turns
    // their cell counts into offsets of one flat sequence of j-cells, increasing within a shift.
    for (int c0 = 0; c0 < ncols; c0 += kThreads)
    {
        int shift = 0, first = 0, count = 0, total = 0;
        if (c0 + tid < ncols)
        {
            column_cells(v, ci, sm, c0 + tid, &shift, &first, &count);
        }
        const int start = block_scan<kWarps>(count, sm.warp_sum[0], &total) - count;
        for (int w0 = 0; w0 < total; w0 += kCellWindow)
        {
            const int wn = min(total - w0, kCellWindow);
            for (int q = max(w0 - start, 0); q < min(count, w0 + wn - start); q++)
            {
                sm.cell[start + q - w0]       = first + q;
                sm.cell_shift[start + q - w0] = (unsigned char)shift;
            }
            __syncthreads();
            // four j-cells per step: lane (kk, jc) tests j-cluster jc of its j-cell against the 8 i-clusters
            // (make_cluster_list_supersub for (ci, scj)); the j-cluster's bounding box is read with the cell's
            // cluster count (empty cluster slots hold far-away boxes, their results are discarded), the next
            // step's while the current one is tested
            const int kk = lane >> 3;
            const int jc = lane & 7;
            int       k0    = 4 * warp;
            int       scj_n = 0, ncl_n = 0;
            float4    jlo{}, jhi{};
            auto      load = [&](int k) {
                ncl_n = 0;
                if (k < wn)
                {
                    scj_n = sm.cell[k];
                    ncl_n = v.nclusters[scj_n];
                    jlo   = v.bb[2 * (scj_n * kNcl + jc)];
                    jhi   = v.bb[2 * (scj_n * kNcl + jc) + 1];
                }
            };
            load(k0 + kk);
            for (; k0 < wn; k0 += 4 * kWarps)
            {
                const int    k     = k0 + kk;
                const int    scj   = scj_n;
                const int    ncl_j = ncl_n;
                const float2 jx = make_float2(-jhi.x, jlo.x), jy = make_float2(-jhi.y, jlo.y),
                             jz = make_float2(-jhi.z, jlo.z);
                load(k + 4 * kWarps);
                const int s     = k < wn ? sm.cell_shift[k] : 0;
                unsigned  im8   = 0u;
                float     d2one = 0.0f;
                if (jc < ncl_j)
                {
#pragma unroll
                    for (int i = 0; i < kNcl; i += 2)
                    {
                        const float2 d2 = bb_dist2(sm.bbi_xy[s][i], sm.bbi_xy[s][i + 1],
                                                   *reinterpret_cast<const float4*>(&sm.bbi_z[s][i]), jx, jy, jz);
                        if (d2.x < rlist2)
                        {
                            im8 |= 1u << i;
                            d2one = d2.x;
                        }
                        if (d2.y < rlist2)
                        {
                            im8 |= 2u << i;
                            d2one = d2.y;
                        }
                    }
                    // empty i-clusters are far away; of the cell's own clusters only i <= j (a single one is
                    // i = j, at distance 0)
                    if (s == kCentral && scj == ci)
                    {
                        im8 &= (2u << jc) - 1u;
                        d2one = 0.0f;
                    }
                }
                // a single cluster pair in range beyond the bounding-box-only distance: check its atom pairs
                // (PRUNE_LIST_CPU_ONE), four flagged j-clusters at a time, eight lanes each (lane jc an i-atom)
                const bool     mine    = __popc(im8) == 1 && d2one >= rbb2;
                const unsigned flagged = __ballot_sync(full, mine);
                if (flagged)
                {
                    const int rank = __popc(flagged & ((1u << lane) - 1u));
                    if (mine)
                    {
                        sm.flag[warp][rank] = make_int2(scj * kNcl + jc, s * kNcl + __ffs(im8) - 1);
                    }
                    __syncwarp();
                    const int nf = __popc(flagged);
                    for (int f0 = 0; f0 < nf; f0 += 4)
                    {
                        bool in = false;
                        if (f0 + kk < nf)
                        {
                            const int2   fl = sm.flag[warp][f0 + kk];
                            const auto&  r  = sm.sr[fl.y >> 3];
                            const float4 xi = v.xq[ci * kSc + (fl.y & 7) * kCl + jc];
                            const float  ix = xi.x + r.shx, iy = xi.y + r.shy, iz = xi.z + r.shz;
                            float        least = 3.0e38f;
#pragma unroll 4
                            for (int h = 0; h < kCl; h++)
                            {
                                const float4 xj = v.xq[fl.x * kCl + h];
                                least           = fminf(least, norm2(ix - xj.x, iy - xj.y, iz - xj.z));
                            }
                            in = least < rlist2;
                        }
                        const unsigned found = __ballot_sync(full, in);
                        if (mine && (rank >> 2) == (f0 >> 2) && ((found >> (8 * (rank & 3))) & 0xffu) == 0u)
                        {
                            im8 = 0u;
                        }
                    }
                    __syncwarp();
                }
                if (k < wn)
                {
                    reinterpret_cast<unsigned char*>(sm.masks)[8 * k + jc] = (unsigned char)im8;
                }
                pairs += __popc(im8);
            }
            __syncthreads();
            // the records of the window in order, a j-cell per thread
            for (int b = 0; b < wn; b += kThreads)
            {
                const int   k = b + tid;
                const uint2 m = k < wn ? sm.masks[k] : make_uint2(0u, 0u);
                int         found = 0, sum = 0;
#pragma unroll
                for (int q = 0; q < 8; q++)
                {
                    found += (((q < 4 ? m.x : m.y) >> (8 * (q & 3))) & 0xffu) != 0u ? 1 : 0;
                }
                int r = rec_n + block_scan<kWarps>(found, sm.warp_sum[1], &sum) - found;
                if (found > 0)
                {
                    atomicAdd(&sm.nj[sm.cell_shift[k]], found);
                    const int cj = sm.cell[k] * kNcl;
#pragma unroll
                    for (int q = 0; q < 8; q++)
                    {
                        const unsigned im = ((q < 4 ? m.x : m.y) >> (8 * (q & 3))) & 0xffu;
                        if (im != 0u)
                        {
                            if (r < v.rec_cap)
                            {
                                rec_cj[r] = cj + q;
                                rec_m[r]  = (unsigned char)im;
                            }
                            r++;
                        }
                    }
                }
                rec_n += sum;
                __syncthreads();  // the window and the scan's sums are free again
            }
        }
        __syncthreads();
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        pairs += __shfl_xor_sync(full, pairs, o);
    }
    if (lane == 0 && pairs > 0u)
    {
        atomicAdd(&sm.pairs, (int)pairs);
    }
    __syncthreads();
    if (warp > 0)
    {
        return;
    }
    // the entries, lane = shift: closeIEntry drops empty ones
    const int      nj   = lane < kShiftSlots ? sm.nj[lane] : 0;
    const unsigned has  = __ballot_sync(full, nj > 0);
    const int      ncj4 = (nj + kJg - 1) / kJg;
    if (nj > 0)
    {
        v.rec_ent[ci * kMaxEntriesPerCell + __popc(has & ((1u << lane) - 1u))] = lane | (nj << 8);
        if (ncj4 > kMaxCj4PerEntry)
        {
            set_status(v.hdr, kStatusEntryOverflow);
        }
    }
    int num_cj4 = ncj4;
    for (int o = 16; o > 0; o >>= 1)
    {
        num_cj4 += __shfl_xor_sync(full, num_cj4, o);
    }
    if (lane == 0)
    {
        v.sci_count[ci] = __popc(has);
        v.cj4_count[ci] = num_cj4;
        // cluster pairs of the list, the count that list balancing splits by
        if (sm.pairs > 0)
        {
            atomicAdd(&v.hdr->num_subpairs, sm.pairs);
        }
        if (rec_n > v.rec_cap)
        {
            atomicMax(&v.hdr->rec_need, rec_n);
            set_status(v.hdr, kStatusRecordOverflow);
        }
    }
}

constexpr int kEmitWarps = 2;    // at least 2: a warp per half of the i-atoms' exclusions
constexpr int kExclStage = 256;  // topology exclusions of a cell's i-atoms staged in shared memory

struct EmitSmem
{
    unsigned      need[2 * kMaxCj4PerEntry / 32];  // per (cj4, half): exclusion mask needed
    int           first[2 * kMaxCj4PerEntry / 32];  // masks needed before the word
    int           diag_pos[kNcl];                   // list positions of the diagonal j-clusters
    int           jl[kEmitStage];                   // the entry's j-clusters (short entries)
    unsigned char jm[kEmitStage];                   // and their i-cluster masks
    int           ex_j[kExclStage];                 // excluded partner's grid slot (-1: itself)
    unsigned char ex_i[kExclStage];                 // the i-atom's slot within the cell
    int           ex_count[2];                      // exclusions of the two halves of the i-atoms
    int           base, masks;                      // first exclusion mask of the entry and their number
};

// Emit pass: one block per list entry (the entries numbered by the prefix sum of the per-cell
// counts) turns its search records into the entry's sci record and cj4 groups.  Each warp finds the
// cell by a 32-way search of the entry offsets and the entry's first record and group from the
// codes of the cell's earlier entries; then the block writes the cj4 groups (one per thread: four
// j-clusters, the i-cluster masks of both warp halves, exclusion index 0 = all interacting), the
// outer masks (the fresh list's masks until a prune refines them) and the group's cluster-pair count
// for balancing; then the exclusions: flag the (cj4, half) pairs that need a mask (self/Newton pairs
// of the diagonal j-clusters and topology exclusions), allocate the flagged masks all interacting,
// clear j <= i on the diagonal (setSelfAndNewtonExclusionsGpu) and the excluded atom pairs
// (setExclusionsForIEntry).  A chain of dependent loads and short loops: with one warp an entry 27.8 us at 45k
// and 90 us at 960k atoms, with two 12.6 and 69 us (with four 12.6 and 82 us).
__global__ void __launch_bounds__(32 * kEmitWarps) k_search_emit(DeviceView v)
{
    pdl_begin();
    constexpr int       kThreads = 32 * kEmitWarps;
    constexpr int       kWords   = 2 * kMaxCj4PerEntry / 32;
    __shared__ EmitSmem sm;
    const int           tid  = threadIdx.x;
    const int           lane = tid & 31;
    const int           warp = tid >> 5;
    const int           e    = blockIdx.x;
    const unsigned      full = 0xffffffffu;
    if (e >= v.hdr->num_sci
        || (v.hdr->status & (kStatusListOverflow | kStatusRecordOverflow | kStatusEntryOverflow)))
    {
        return;
    }
    // the cell of entry e: the last cell whose first entry is at most e (cells without entries
    // share their successor's offset); the search window shrinks 32-fold per step
    int ci = 0;
    {
        int len = v.hdr->num_cells;
        while (len > 1)
        {
            const int  step = (len + 31) / 32;
            const int  c    = ci + lane * step;
            const bool le   = c < ci + len && v.sci_offset[c] <= e;
            const int  cnt  = __popc(__ballot_sync(full, le));
            const int  lo   = ci + (cnt - 1) * step;
            len             = min(step, ci + len - lo);
            ci              = lo;
        }
    }
    // the topology exclusions of the cell's i-atoms, half of them per warp: how many
    int iAtom = -1, x0 = 0, x1 = 0;
    if (warp < 2)
    {
        iAtom = v.atom_indices[ci * kSc + warp * 32 + lane];
        if (iAtom >= 0)
        {
            x0 = v.excl_index[iAtom];
            x1 = v.excl_index[iAtom + 1];
        }
    }
    const int kent = e - v.sci_offset[ci];
    // this entry's code; the records and groups of the cell's earlier entries
    const int cl   = lane <= kent ? v.rec_ent[ci * kMaxEntriesPerCell + lane] : 0;
    int       rec0 = lane < kent ? cl >> 8 : 0;
    int       grp0 = (rec0 + kJg - 1) / kJg;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        rec0 += __shfl_xor_sync(full, rec0, o);
        grp0 += __shfl_xor_sync(full, grp0, o);
    }
    const int            code    = __shfl_sync(full, cl, kent);
    const int            cj4_out = v.cj4_offset[ci] + grp0;
    const int*           rec_cj  = v.rec_cj + (size_t)ci * v.rec_cap + rec0;
    const unsigned char* rec_m   = v.rec_m + (size_t)ci * v.rec_cap + rec0;
    const int            shift   = code & 0xff;
    const int            nj      = code >> 8;
    const int            ncj4    = (nj + kJg - 1) / kJg;
    const bool           excludeSubDiagonal = (shift == kCentral);
    if (tid < kNcl)
    {
        sm.diag_pos[tid] = -1;
    }
    for (int w = tid; w < kWords; w += kThreads)
    {
        sm.need[w] = 0u;
    }
    // the j-list is sorted on cluster index; short lists go to shared memory for the group writes and the
    // exclusion lookups
    const bool staged = nj <= kEmitStage;
    if (staged)
    {
#pragma unroll 4
        for (int p = tid; p < nj; p += kThreads)
        {
            sm.jl[p] = rec_cj[p];
            sm.jm[p] = rec_m[p];
        }
    }
    int ex_off = 0;
    if (warp < 2)
    {
        const int cnt  = x1 - x0;
        int       incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int t = __shfl_up_sync(full, incl, o);
            if (lane >= o)
            {
                incl += t;
            }
        }
        ex_off = incl - cnt;
        if (lane == 31)
        {
            sm.ex_count[warp] = incl;
        }
    }
    __syncthreads();
    // the exclusions as (i-slot, partner grid slot) pairs when they fit; else the entry walks the exclusion lists
    const int  nex       = sm.ex_count[0] + sm.ex_count[1];
    const bool ex_staged = nex <= kExclStage;
    if (ex_staged && warp < 2)
    {
        const int off = ex_off + (warp == 1 ? sm.ex_count[0] : 0);
        // the partners four at a time: their list entries, then their grid slots
        for (int x = x0; x < x1; x += 4)
        {
            int jAtom[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
            {
                jAtom[u] = x + u < x1 ? v.excl_list[x + u] : -1;
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
            {
                if (x + u < x1)
                {
                    sm.ex_j[off + (x + u - x0)] = (jAtom[u] == iAtom) ? -1 : v.cells[jAtom[u]];
                    sm.ex_i[off + (x + u - x0)] = (unsigned char)(warp * 32 + lane);
                }
            }
        }
    }
    const int*           jlist = staged ? sm.jl : rec_cj;
    const unsigned char* mlist = staged ? sm.jm : rec_m;
    for (int g = tid; g < ncj4; g += kThreads)
    {
        Cj4      c;
        unsigned im = 0u;
#pragma unroll
        for (int off = 0; off < kJg; off++)
        {
            const int p = g * kJg + off;
            c.cj[off]   = p < nj ? jlist[p] : 0;
            im |= p < nj ? (unsigned)mlist[p] << (off * kNcl) : 0u;
        }
        c.imei[0].imask    = im;
        c.imei[0].excl_ind = 0;
        c.imei[1]          = c.imei[0];
        v.cj4[cj4_out + g] = c;
        reinterpret_cast<uint2*>(v.imask_outer)[cj4_out + g] = make_uint2(im, im);
        v.grp_pairs[cj4_out + g] = (unsigned char)__popc(im);
    }
    // the diagonal j-clusters (the i-cell's own clusters, central shift)
    if (excludeSubDiagonal)
    {
        for (int p = tid; p < nj; p += kThreads)
        {
            const int cj = jlist[p];
            if ((cj >> 3) == ci)
            {
                sm.diag_pos[cj & (kNcl - 1)] = p;
                atomicOr(&sm.need[(2 * (p / kJg)) / 32], 3u << ((2 * (p / kJg)) % 32));
            }
        }
    }
    if (tid == 0)
    {
        Sci r;
        r.sci       = ci;
        r.shift     = shift;
        r.cj4_start = cj4_out;
        r.cj4_end   = cj4_out + ncj4;
        v.sci[e]    = r;
    }
    __syncthreads();
    // --- topology exclusions (setExclusionsForIEntry, GPU list) ---
    const int cjFirst = jlist[0];
    const int cjLast  = jlist[nj - 1];
    // list position of one excluded atom pair (i-slot i of the cell, partner at grid slot jIndex), -1: not in the entry
    auto position = [&](int i, int jIndex) {
        if (excludeSubDiagonal && jIndex <= ci * kSc + i)
        {
            return -1;
        }
        const int jCluster = jIndex / kCl;
        if (jCluster < cjFirst || jCluster > cjLast)
        {
            return -1;
        }
        int a = 0, b = nj - 1;
        while (a <= b)
        {
            const int m  = (a + b) >> 1;
            const int cm = jlist[m];
            if (cm == jCluster)
            {
                return ((mlist[m] >> (i / kCl)) & 1u) ? m : -1;
            }
            if (cm < jCluster)
            {
                a = m + 1;
            }
            else
            {
                b = m - 1;
            }
        }
        return -1;
    };
    // the (cj4, half) slot of list position index and grid slot jIndex
    auto slot_of = [&](int index, int jIndex) {
        return 2 * (index / kJg) + (jIndex & (kCl - 1)) / (kCl / kSplit);
    };
    auto flag = [&](int slot) { atomicOr(&sm.need[slot / 32], 1u << (slot % 32)); };
    // the mask of a flagged slot: masks are allocated to the flagged slots in order
    auto excl_of_slot = [&](int slot) {
        return sm.base + sm.first[slot / 32] + __popc(sm.need[slot / 32] & ((1u << (slot % 32)) - 1u));
    };
    auto exclude = [&](int i, int jIndex, int index) {
        const unsigned pairMask = 1u << ((index % kJg) * kNcl + i / kCl);
        const int      innerJ   = jIndex & (kCl - 1);
        atomicAnd(&v.excl[excl_of_slot(slot_of(index, jIndex))].pair[(innerJ & (kCl / kSplit - 1)) * kCl + (i & (kCl - 1))],
                  ~pairMask);
    };
    // without staging: f(i-slot, grid slot of the partner) for every exclusion
    auto walk = [&](auto f) {
        for (int i = tid; i < kSc; i += kThreads)
        {
            const int a = v.atom_indices[ci * kSc + i];
            if (a < 0)
            {
                continue;
            }
            for (int x = v.excl_index[a]; x < v.excl_index[a + 1]; x++)
            {
                const int jAtom = v.excl_list[x];
                if (jAtom != a)
                {
                    f(i, v.cells[jAtom]);
                }
            }
        }
    };
    // flag the (cj4, half) pairs that need an exclusion mask; staged positions are kept in the thread's own slots
    int kept[(kExclStage + kThreads - 1) / kThreads];
    if (ex_staged)
    {
#pragma unroll
        for (int u = 0; u < (kExclStage + kThreads - 1) / kThreads; u++)
        {
            const int t = tid + u * kThreads;
            kept[u]     = t < nex && sm.ex_j[t] >= 0 ? position(sm.ex_i[t], sm.ex_j[t]) : -1;
            if (kept[u] >= 0)
            {
                flag(slot_of(kept[u], sm.ex_j[t]));
            }
        }
    }
    else
    {
        walk([&](int i, int jIndex) {
            const int index = position(i, jIndex);
            if (index >= 0)
            {
                flag(slot_of(index, jIndex));
            }
        });
    }
    __syncthreads();
    // allocate the flagged masks
    if (warp == 0)
    {
        constexpr int kPer = kWords / 32;
        int           own  = 0;
#pragma unroll
        for (int u = 0; u < kPer; u++)
        {
            own += __popc(sm.need[lane * kPer + u]);
        }
        int incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int t = __shfl_up_sync(full, incl, o);
            if (lane >= o)
            {
                incl += t;
            }
        }
        int run = incl - own;
#pragma unroll
        for (int u = 0; u < kPer; u++)
        {
            sm.first[lane * kPer + u] = run;
            run += __popc(sm.need[lane * kPer + u]);
        }
        if (lane == 31)
        {
            sm.masks = incl;
            sm.base  = incl > 0 ? atomicAdd(&v.hdr->num_excl, incl) : 0;
        }
    }
    __syncthreads();
    if (sm.masks == 0)
    {
        return;
    }
    if (sm.base + sm.masks > v.hdr->excl_capacity)
    {
        if (tid == 0)
        {
            set_status(v.hdr, kStatusExclOverflow);
        }
        return;
    }
    // all interacting
    for (int w = warp; w < (2 * ncj4 + 31) / 32; w += kEmitWarps)
    {
        unsigned bits = sm.need[w];
        int      run  = sm.base + sm.first[w];
        while (bits)
        {
            const int slot = w * 32 + __ffs(bits) - 1;
            bits &= bits - 1;
            v.excl[run].pair[lane] = 0xffffffffu;
            if (lane == 0)
            {
                v.cj4[cj4_out + slot / 2].imei[slot % 2].excl_ind = run;
            }
            run++;
        }
    }
    __syncthreads();
    // self and Newton exclusions of the diagonal cluster pairs (setSelfAndNewtonExclusionsGpu): clear j <= i;
    // lane = (jIndexInPart, i): word jIndexInPart * 8 + i
    for (int k = warp; k < kNcl * kSplit; k += kEmitWarps)
    {
        const int dj = k / kSplit, part = k % kSplit;
        const int pos = sm.diag_pos[dj];
        const int jip = lane >> 3, ii = lane & 7;
        if (pos >= 0 && ii >= part * (kCl / kSplit) + jip)
        {
            atomicAnd(&v.excl[excl_of_slot(2 * (pos / kJg) + part)].pair[jip * kCl + ii],
                      ~(1u << (pos % kJg * kNcl + dj)));
        }
    }
    if (ex_staged)
    {
#pragma unroll
        for (int u = 0; u < (kExclStage + kThreads - 1) / kThreads; u++)
        {
            const int t = tid + u * kThreads;
            if (kept[u] >= 0)
            {
                exclude(sm.ex_i[t], sm.ex_j[t], kept[u]);
            }
        }
    }
    else
    {
        walk([&](int i, int jIndex) {
            const int index = position(i, jIndex);
            if (index >= 0)
            {
                exclude(i, jIndex, index);
            }
        });
    }
}

// four values from index i, those at n and beyond as 0
__device__ __forceinline__ int4 load4(const int* p, int i, int n)
{
    if (i + 4 <= n)
    {
        return *reinterpret_cast<const int4*>(p + i);
    }
    return make_int4(i < n ? p[i] : 0, i + 1 < n ? p[i + 1] : 0, i + 2 < n ? p[i + 2] : 0, 0);
}

__device__ __forceinline__ void store4(int* p, int i, int n, int4 x)
{
    if (i + 4 <= n)
    {
        *reinterpret_cast<int4*>(p + i) = x;
        return;
    }
    if (i < n) p[i] = x.x;
    if (i + 1 < n) p[i + 1] = x.y;
    if (i + 2 < n) p[i + 2] = x.z;
}

// Exclusive prefix sums of the per-cell entry and cj4 counts, one block, four cells a thread: rows of 4096 cells
// with the next one loaded ahead.  15.6k cells took 21 us with a contiguous run of cells per thread.
__global__ void __launch_bounds__(1024) k_scan_counts(DeviceView v)
{
    pdl_begin();
    __shared__ int ws[2][32];
    const int      n    = v.hdr->num_cells;
    const int      lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int            base_s = 0, base_c = 0;
    int            i  = 4 * threadIdx.x;
    int4           sn = load4(v.sci_count, i, n), cn = load4(v.cj4_count, i, n);
    for (int row = 0; row < n; row += 4096, i += 4096)
    {
        const int4 s = sn, c = cn;
        sn           = load4(v.sci_count, i + 4096, n);
        cn           = load4(v.cj4_count, i + 4096, n);
        const int ls = s.x + s.y + s.z + s.w, lc = c.x + c.y + c.z + c.w;
        int       is = ls, ic = lc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int ts = __shfl_up_sync(0xffffffffu, is, o);
            const int tc = __shfl_up_sync(0xffffffffu, ic, o);
            if (lane >= o)
            {
                is += ts;
                ic += tc;
            }
        }
        __syncthreads();  // the row before has been read
        if (lane == 31)
        {
            ws[0][warp] = is;
            ws[1][warp] = ic;
        }
        __syncthreads();
        // every warp scans the 32 warps' sums
        int a = ws[0][lane], b = ws[1][lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int ta = __shfl_up_sync(0xffffffffu, a, o);
            const int tb = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o)
            {
                a += ta;
                b += tb;
            }
        }
        const int wa = __shfl_sync(0xffffffffu, a, max(warp - 1, 0)), wb = __shfl_sync(0xffffffffu, b, max(warp - 1, 0));
        const int rs = base_s + is - ls + (warp > 0 ? wa : 0);
        const int rc = base_c + ic - lc + (warp > 0 ? wb : 0);
        store4(v.sci_offset, i, n, make_int4(rs, rs + s.x, rs + s.x + s.y, rs + s.x + s.y + s.z));
        store4(v.cj4_offset, i, n, make_int4(rc, rc + c.x, rc + c.x + c.y, rc + c.x + c.y + c.z));
        base_s += __shfl_sync(0xffffffffu, a, 31);
        base_c += __shfl_sync(0xffffffffu, b, 31);
    }
    if (threadIdx.x == 0)
    {
        v.sci_offset[n] = base_s;
        v.cj4_offset[n] = base_c;
        v.hdr->num_sci  = base_s;
        v.hdr->num_cj4  = base_c;
        v.hdr->num_excl = 1;
        if (base_s > v.hdr->sci_capacity || base_c > v.hdr->cj4_capacity)
        {
            set_status(v.hdr, kStatusListOverflow);
        }
    }
}

} // namespace

// count (+ records) -> prefix sum | emit.  All sizes stay on the device; the host reads them
// between the two halves to check the list and record capacities.
cudaError_t launch_search_count(const DeviceView& v, cudaStream_t s)
{
    const int cap    = v.g.cells_capacity;
    // num_subpairs .. rec_need: accumulated by the count pass or set by balancing
    cudaMemsetAsync(&v.hdr->num_subpairs, 0,
                    offsetof(ListHeader, rec_need) + sizeof(int) - offsetof(ListHeader, num_subpairs), s);
    // two warps a cell once the cells alone fill the GPU, four while a cell's latency counts.  The host knows the
    // grid's capacity, not its cells; at 100 / 50 / 25 atoms per nm^3 and a capacity of 1018 the pass takes
    // 23.0 / 20.0 / 18.0 us with four and 28.1 / 22.1 / 20.0 us with two, at 1365 27.2 / 24.4 / 24.1 and 24.2 / 21.0 /
    // 20.0 us, at 4474 53.6 / 42.9 / 44.5 and 48.6 / 36.5 / 37.3 us (at 2653 and 3008, 100 per nm^3, equal)
    if (cap > kManyCells)
    {
        launch_pdl(k_search_count<2>, cap, 64, 0, s, v);
    }
    else
    {
        launch_pdl(k_search_count<4>, cap, 128, 0, s, v);
    }
    launch_pdl(k_scan_counts, 1, 1024, 0, s, v);
    return cudaGetLastError();
}

cudaError_t launch_search_write(const DeviceView& v, int num_entries, cudaStream_t s)
{
    if (num_entries > 0)
    {
        launch_pdl(k_search_emit, num_entries, 32 * kEmitWarps, 0, s, v);
    }
    return cudaGetLastError();
}

} // namespace nbx
