// GPU list balancing after a search: split long entries, then sort entries by size.
//
// Restates, on the device, what the reference does on the host for GPU lists:
//  - split_sci_entry (src/gromacs/nbnxm/pairlist.cpp:2077-2165), without the
//    progressive variant: an entry with more cluster pairs than the target is cut
//    into pieces of close to nsp_max pairs (pairs counted as the bits of
//    imei[0].imask), the last two pieces evened out;
//  - the target of get_nsubpair_target (pairlist.cpp:2485-2585): no splitting
//    when the grid has at least min_ci_balanced cells, else
//    max(36, round(pairs / min_ci_balanced)), here with the exact pair count of
//    the list instead of the geometric estimate;
//  - sort_sci (pairlist.cpp:3827-3873): a stable counting sort on the number of
//    cj4 groups, large entries first, sizes above twice the average sharing one
//    class (the class count is capped at 255 here).
// The cj4 array is untouched: only entry boundaries and order change, so the set
// of cluster pairs is the same.  The persistent force kernel takes entries from an
// atomic queue in list order, so large-first order and even piece sizes shorten
// the tail of the launch.
//
// Sequence (no host synchronisation): count pieces per entry -> exclusive scan ->
// write pieces -> sort into the final list, all sizes from the list header.
#include "nbx_internal.cuh"

#include <algorithm>

namespace nbx
{
namespace
{

constexpr int kMinTarget    = 36;   // nsubpair_target_min, pairlist.cpp:2495
constexpr int kMaxSizeClass = kSizeClasses - 1;
constexpr int kSortThreads  = kSizeClasses;  // a thread per class in the offsets
constexpr int kSortWarps    = kSortThreads / 32;
constexpr int kSortBatch    = 2;  // entries per lane loaded at a time by the sort
constexpr int kScanBatch    = 8;  // piece counts per thread loaded at a time by the scan

__device__ __forceinline__ int balance_target(const ListHeader* hdr, int min_ci_balanced)
{
    const int ncells = hdr->num_cells;
    if (min_ci_balanced <= 0 || ncells >= min_ci_balanced || ncells == 0)
    {
        return 0;
    }
    const long long nsp = hdr->num_subpairs;
    const long long t   = (2 * nsp + min_ci_balanced) / (2 * (long long)min_ci_balanced);
    return t > kMinTarget ? (int)t : kMinTarget;
}

// Cuts entry e into pieces, one warp, a cj4 group per lane, and returns their number; piece(start, end) is called
// with each, in order, by all lanes.  With P the prefix sum of the groups' cluster pairs (grp_pairs, the bits of
// imei[0].imask, written by the search) the open piece that starts at s is cut before the first group j with
// nsp_max - nsp < nsp + pairs(j) - nsp_max, nsp = P[j] - P[s]: P[j] + P[j + 1] > 2 (nsp_max + P[s]), found by a ballot.
// The last two pieces are evened out by moving one group.
template<class Piece>
__device__ __forceinline__ int split_entry(const unsigned char* grp_pairs, Sci e, int nsp_max,
                                           const Piece& piece)
{
    const unsigned full  = 0xffffffffu;
    const int      lane  = threadIdx.x & 31;
    const int      j4len = e.cj4_end - e.cj4_start;
    if (!(nsp_max > 0 && j4len > 1 && j4len * kNcl * kJg > nsp_max))
    {
        piece(e.cj4_start, e.cj4_end);
        return 1;
    }
    int n     = 1;
    int start = e.cj4_start, p_start = 0;          // the open piece and P at its start
    int prev_start = e.cj4_start, prev_pairs = 0;  // the last closed piece (it ends at start) and its pairs
    int last_pairs = 0, last_in_prev = 0;          // pairs of the group before the chunk, of the closed piece's last group
    int carry = 0;
    for (int c0 = e.cj4_start; c0 < e.cj4_end; c0 += 32)
    {
        const int j     = c0 + lane;
        const int pairs = j < e.cj4_end ? grp_pairs[j] : 0;
        int       incl  = pairs;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int t = __shfl_up_sync(full, incl, o);
            if (lane >= o)
            {
                incl += t;
            }
        }
        incl += carry;
        const int below  = incl - pairs;
        int       before = __shfl_up_sync(full, pairs, 1);  // pairs of group j - 1
        before           = lane == 0 ? last_pairs : before;
        for (;;)
        {
            const unsigned cut =
                    __ballot_sync(full, j < e.cj4_end && below > p_start && below + incl > 2 * (nsp_max + p_start));
            if (cut == 0u)
            {
                break;
            }
            const int src = __ffs(cut) - 1;
            if (n > 1)
            {
                piece(prev_start, start);
            }
            prev_start   = start;
            start        = c0 + src;
            const int ps = __shfl_sync(full, below, src);
            prev_pairs   = ps - p_start;
            last_in_prev = __shfl_sync(full, before, src);
            p_start      = ps;
            n++;
        }
        last_pairs = __shfl_sync(full, pairs, 31);
        carry      = __shfl_sync(full, incl, 31);
    }
    if (n > 1)
    {
        const int cut = prev_pairs - last_in_prev >= carry - p_start + last_in_prev ? start - 1 : start;
        piece(prev_start, cut);
        start = cut;
    }
    piece(start, e.cj4_end);
    return n;
}

// Entries per chunk and class (see sci_pieces).
__device__ __forceinline__ int* sort_hist(const DeviceView& v)
{
    return v.sci_pieces + v.sci_cap + 1;
}

// The largest size class of a list of n entries: sizes above twice the average share it; 0: one class, order kept.
__device__ __forceinline__ int largest_class(const ListHeader* hdr, int n)
{
    const int m = hdr->num_cj4 > n ? (int)((2LL * hdr->num_cj4) / n) : 0;
    return m > kMaxSizeClass ? kMaxSizeClass : m;
}

__device__ __forceinline__ int sort_chunk(int n)
{
    return (n + kSortChunks - 1) / kSortChunks;
}

__global__ void k_balance_count(DeviceView v, int min_ci_balanced)
{
    pdl_begin();
    const ListHeader* hdr = v.hdr;
    if (hdr->status & (kStatusListOverflow | kStatusExclOverflow | kStatusGridOverflow))
    {
        return;
    }
    const int nsp_max = balance_target(hdr, min_ci_balanced);
    const int nsci    = hdr->num_sci;
    const int t       = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0)
    {
        v.hdr->nsp_max         = nsp_max;
        v.hdr->num_sci_unsplit = nsci;
    }
    for (int k = t; k < kSortChunks * kSizeClasses; k += gridDim.x * blockDim.x)
    {
        sort_hist(v)[k] = 0;
    }
    // nothing is split: every entry is one piece, at its own place
    const int e = t >> 5;
    if (nsp_max > 0 && e < nsci)
    {
        const int n = split_entry(v.grp_pairs, v.sci[e], nsp_max, [](int, int) {});
        if ((t & 31) == 0)
        {
            v.sci_pieces[e] = n;
        }
    }
}

// Exclusive scan of the piece counts in place (one block, each thread a contiguous run); the
// total goes to num_sci_split.
__global__ void __launch_bounds__(1024) k_balance_scan(DeviceView v)
{
    pdl_begin();
    __shared__ int    warp_sums[32];
    const ListHeader* hdr = v.hdr;
    if (hdr->status & (kStatusListOverflow | kStatusExclOverflow | kStatusGridOverflow))
    {
        return;
    }
    const int n    = hdr->num_sci_unsplit;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (hdr->nsp_max == 0)
    {
        if (threadIdx.x == 0)
        {
            v.hdr->num_sci_split = n;
        }
        return;
    }
    const int per  = (n + blockDim.x - 1) / blockDim.x;
    const int i0   = min(n, (int)threadIdx.x * per);
    const int i1   = min(n, i0 + per);
    int       own  = 0;
    for (int b = i0; b < i1; b += kScanBatch)
    {
        int val[kScanBatch];
#pragma unroll
        for (int u = 0; u < kScanBatch; u++)
        {
            val[u] = b + u < i1 ? v.sci_pieces[b + u] : 0;
        }
#pragma unroll
        for (int u = 0; u < kScanBatch; u++)
        {
            own += val[u];
        }
    }
    int inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o)
        {
            inc += t;
        }
    }
    if (lane == 31)
    {
        warp_sums[warp] = inc;
    }
    __syncthreads();
    if (warp == 0)
    {
        int w = (lane < (int)(blockDim.x >> 5)) ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o)
            {
                w += t;
            }
        }
        warp_sums[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    int run = (warp > 0 ? warp_sums[warp - 1] : 0) + inc - own;
    for (int b = i0; b < i1; b += kScanBatch)
    {
        int val[kScanBatch];
#pragma unroll
        for (int u = 0; u < kScanBatch; u++)
        {
            val[u] = b + u < i1 ? v.sci_pieces[b + u] : 0;
        }
#pragma unroll
        for (int u = 0; u < kScanBatch; u++)
        {
            if (b + u < i1)
            {
                v.sci_pieces[b + u] = run;
                run += val[u];
            }
        }
    }
    if (threadIdx.x == blockDim.x - 1)
    {
        v.hdr->num_sci_split = run;
    }
}

__global__ void k_balance_write(DeviceView v)
{
    pdl_begin();
    const ListHeader* hdr = v.hdr;
    if (hdr->status & (kStatusListOverflow | kStatusExclOverflow | kStatusGridOverflow))
    {
        return;
    }
    // entries per chunk and class for the sort
    const int m     = largest_class(hdr, hdr->num_sci_split);
    const int chunk = sort_chunk(hdr->num_sci_split);
    auto      put   = [&](int p, const Sci& e, int start, int end) {
        const int len = end - start;
        v.sci_tmp[p]  = Sci{ e.sci, e.shift, start, end };
        atomicAdd(&sort_hist(v)[p / chunk * kSizeClasses + (len < m ? len : m)], 1);
    };
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (hdr->nsp_max == 0)
    {
        if (t < hdr->num_sci_unsplit)
        {
            const Sci e = v.sci[t];
            put(t, e, e.cj4_start, e.cj4_end);
        }
        return;
    }
    const int i = t >> 5;
    if (i < hdr->num_sci_unsplit)
    {
        const Sci e = v.sci[i];
        int       p = v.sci_pieces[i];
        split_entry(v.grp_pairs, e, hdr->nsp_max, [&](int start, int end) {
            if ((t & 31) == 0)
            {
                put(p, e, start, end);
            }
            p++;
        });
    }
}

// Stable counting sort of sci_tmp into sci, size classes descending; a block per chunk of the entries.  From the
// chunks' class counts (k_balance_write) thread c gets the class's place in the list and the chunk's place in the
// class; warp w owns the w-th run of the chunk: per-warp class counts, then each warp places its run in order, the
// rank among equal classes of 32 entries from __match_any_sync.  One block of 1024 threads for the whole list took
// 13.6 us for 7k entries and 36 us for 18k.
__global__ void __launch_bounds__(kSortThreads) k_sort_entries(DeviceView v)
{
    pdl_begin();
    __shared__ int hist[kSortWarps][kSizeClasses];  // counts, then each warp's next position
    __shared__ int warp_sums[kSortWarps];
    ListHeader*    hdr = v.hdr;
    if (hdr->status & (kStatusListOverflow | kStatusExclOverflow | kStatusGridOverflow))
    {
        return;
    }
    const int n    = hdr->num_sci_split;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        hdr->num_sci = n;
    }
    if (n == 0)
    {
        return;
    }
    const int m     = largest_class(hdr, n);
    const int chunk = sort_chunk(n);
    const int c0    = blockIdx.x * chunk;
    const int run   = (chunk + kSortWarps - 1) / kSortWarps;
    const int e0    = min(n, c0 + min(chunk, warp * run));
    const int e1    = min(n, c0 + min(chunk, (warp + 1) * run));
    // the class of this thread: its entries in the chunks before this one and in all
    const int cls0   = m - (int)threadIdx.x;
    int       before = 0, total = 0;
    if (cls0 >= 0)
    {
#pragma unroll 16
        for (int b = 0; b < kSortChunks; b++)
        {
            const int h = sort_hist(v)[b * kSizeClasses + cls0];
            before += b < (int)blockIdx.x ? h : 0;
            total += h;
        }
    }
    for (int k = threadIdx.x; k < kSortWarps * kSizeClasses; k += kSortThreads)
    {
        (&hist[0][0])[k] = 0;
    }
    int incl = total;
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
        warp_sums[warp] = incl;
    }
    __syncthreads();
    for (int e = e0 + lane; e < e1; e += 32)
    {
        const int len = v.sci_tmp[e].cj4_end - v.sci_tmp[e].cj4_start;
        atomicAdd(&hist[warp][len < m ? len : m], 1);
    }
    __syncthreads();
    if (cls0 >= 0)
    {
        int pos = incl - total + before;
        for (int w = 0; w < warp; w++)
        {
            pos += warp_sums[w];
        }
#pragma unroll
        for (int w = 0; w < kSortWarps; w++)
        {
            const int h   = hist[w][cls0];
            hist[w][cls0] = pos;
            pos += h;
        }
    }
    __syncthreads();
    for (int b = e0; b < e1; b += 32 * kSortBatch)
    {
        Sci sv[kSortBatch];
#pragma unroll
        for (int u = 0; u < kSortBatch; u++)
        {
            const int e = b + u * 32 + lane;
            sv[u]       = e < e1 ? v.sci_tmp[e] : Sci{ 0, 0, 0, -1 };
        }
#pragma unroll
        for (int u = 0; u < kSortBatch; u++)
        {
            const int      len   = sv[u].cj4_end - sv[u].cj4_start;
            const int      cls   = len < 0 ? -1 : (len < m ? len : m);
            const unsigned peers = __match_any_sync(0xffffffffu, cls);
            const unsigned lower = peers & ((1u << lane) - 1u);
            if (cls >= 0)
            {
                v.sci[hist[warp][cls] + __popc(lower)] = sv[u];
            }
            __syncwarp();
            if (cls >= 0 && lower == 0u)
            {
                hist[warp][cls] += __popc(peers);
            }
            __syncwarp();
        }
    }
}

} // namespace

cudaError_t launch_balance(const DeviceView& v, int num_entries, int min_ci_balanced, cudaStream_t s)
{
    // a warp per entry: a thread per entry walked its groups one after the other (45k atoms, 1165 entries of 40
    // groups: writing 11.3 us, now 6.4 us; counting 4.7 us as before)
    const int tb     = 256;
    const int blocks = std::max((num_entries + tb / 32 - 1) / (tb / 32), 1);
    launch_pdl(k_balance_count, blocks, tb, 0, s, v, min_ci_balanced);
    launch_pdl(k_balance_scan, 1, 1024, 0, s, v);
    launch_pdl(k_balance_write, blocks, tb, 0, s, v);
    launch_pdl(k_sort_entries, kSortChunks, kSortThreads, 0, s, v);
    return cudaGetLastError();
}

} // namespace nbx
