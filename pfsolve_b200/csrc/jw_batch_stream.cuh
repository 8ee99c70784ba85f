// jw_batch_stream.cuh -- uneven batches of real systems on the streaming solve.
//
// One launch over (entry, system range) items, each entry a matrix and its
// systems (PfSolveBatch*).  A CTA takes an item, builds the entry's coefficient
// table with all its threads, and solves the item's systems on groups whose
// shape fits the entry's rows: 4, 8 or 16 rows per thread of one warp, 16 of
// two or four.  Rows move by element copies (StElem): any row count and stride.
//
// Against the group kernel's batches (jw_batch_kernel): there every group of
// warps rebuilds the coefficients of each item in its registers, at the width of
// the longest entry, and 255 registers a thread leave 8 warps an SM; here a
// table serves 16 warps.  32 mixed-precision requests of 42 to 970 rows (22 466
// systems, 109 MB): 545 -> 88 us (388 with the faster table builds alone).
// The bound is shared memory, as in the streaming kernel, plus one table build
// an item, so the host cuts the entries into few items
// (batch_configure_stream in api.cpp).
#pragma once
#include "jw_stream.cuh"

namespace pfb {

constexpr int kBsThreads = 512, kBsWarps = kBsThreads / 32, kBsBufs = 2;

template <int KL, int KU, int SV, int PREC>
struct BsCfg {
    template <int R, int W>
    using St = StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC>;
};

// Shape index of M rows (kBsShapes: longer systems do not run here).
constexpr int kBsShapes = 5;
__host__ __device__ constexpr int bs_shape(int64_t M)
{
    return M <= 128 ? 0 : (M <= 256 ? 1 : (M <= 512 ? 2 : (M <= 1024 ? 3 : (M <= 2048 ? 4 : kBsShapes))));
}
__host__ __device__ inline int bs_warps(int shape) { return shape <= 2 ? 1 : (shape == 3 ? 2 : 4); }

// Barriers: one per staging buffer and group of each group width (their
// arrival counts differ): 16 groups of one warp, 8 of two, 4 of four.
constexpr int kBsBars = kBsBufs * (kBsWarps + kBsWarps / 2 + kBsWarps / 4);

// Shared memory: descriptor | item slots | barriers | scratch | table |
// (align 1024) | staging buffers (every shape's groups fill the same bytes per
// warp at 16 rows per thread).  The table holds the shapes up to the longest
// entry's (Mmax rows): beside the staging buffers the four-warp table of six
// planes does not fit, so the mixed mode's 3-band kind runs here up to 1 024
// rows.  It is at least the exchange area the table build borrows from it.
template <class CF>
__host__ __device__ constexpr size_t bs_table_bytes(int64_t Mmax)
{
    size_t t = (size_t)kBsWarps * kScratchPerWarp * sizeof(double);
    const size_t by_shape[kBsShapes] = {CF::template St<4, 1>::TBL, CF::template St<8, 1>::TBL,
                                        CF::template St<16, 1>::TBL, CF::template St<16, 2>::TBL,
                                        CF::template St<16, 4>::TBL};
    for (int k = 0; k < kBsShapes && k <= bs_shape(Mmax); ++k)
        if (by_shape[k] > t) t = by_shape[k];
    return (t + 15) / 16 * 16;
}
constexpr size_t kBsHead = (sizeof(BatchEntryDev) + 15) / 16 * 16 + 16 + (size_t)kBsBars * 8 +
                           (size_t)kBsWarps * kScratchPerWarp * sizeof(double);
template <class CF>
__host__ __device__ constexpr size_t bs_smem_bytes(int64_t Mmax)
{
    return kBsHead + bs_table_bytes<CF>(Mmax) + 1024 + (size_t)kBsWarps * kBsBufs * 32 * 16 * sizeof(double);
}

// One item on groups of shape C; bi and par are this group's buffer and phase
// among the barriers of its width.
template <class C>
__device__ __forceinline__ bool bs_item(const BatchEntryDev& e, int64_t y0, int64_t y1, void* table_mem,
                                        double* scratch_all, unsigned char* bufs, uint64_t* bars, int& bi,
                                        uint32_t& par)
{
    using CT = typename C::CT;
    constexpr int W = C::W, G = kBsWarps / W;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = warp / W, wg = warp - grp * W;
    CT* table = reinterpret_cast<CT*>(table_mem);
    StElem<C> ld;
    ld.io = &e.io;
    ld.base = bufs + (size_t)(kBsBufs * grp) * C::BUF;
    ld.bars = bars + kBsBufs * grp;
    ld.wg = wg;
    ld.lane = lane;
    const int64_t sys = y0 + grp;
    if (sys < y1) ld.load(bi, sys);  // in flight while the table is built
    st_prologue<C>(e.op, table, scratch_all);
    __syncthreads();
    GroupCtx g;
    g.lane = lane;
    g.wg = wg;
    g.W = W;
    g.nthr = C::T;
    g.bar_id = 1 + grp;
    g.seq = 0;
    g.scratch = scratch_all + (size_t)grp * W * kScratchPerWarp;
    return st_run<C>(e.op, e.io, table, g, ld, kBsBufs, sys, G, y1, bi, par);
}

template <class CF>
__global__ void __launch_bounds__(kBsThreads, 1) jw_batch_stream_kernel(const BatchEntryDev* __restrict__ entries,
                                                                       const WorkItem* __restrict__ items,
                                                                       const int nitems,
                                                                       unsigned int* __restrict__ counter,
                                                                       const int table_bytes)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BatchEntryDev& e = *reinterpret_cast<BatchEntryDev*>(smem_raw);
    int* slot = reinterpret_cast<int*>(smem_raw + (sizeof(BatchEntryDev) + 15) / 16 * 16);
    uint64_t* bars = reinterpret_cast<uint64_t*>(slot + 4);
    double* scratch_all = reinterpret_cast<double*>(bars + kBsBars);
    unsigned char* table = smem_raw + kBsHead;
    unsigned char* after = table + table_bytes;
    unsigned char* bufs = after + ((1024u - (smem_u32(after) & 1023u)) & 1023u);
    uint64_t* bars2 = bars + kBsBufs * kBsWarps;
    uint64_t* bars4 = bars2 + kBsBufs * (kBsWarps / 2);
    for (int k = threadIdx.x; k < kBsBars; k += blockDim.x)
        mbar_init(smem_u32(&bars[k]), &bars[k] < bars2 ? 32 : (&bars[k] < bars4 ? 64 : 128));
    mbar_init_fence();
    int bi1 = 0, bi2 = 0, bi4 = 0;
    uint32_t par1 = 0, par2 = 0, par4 = 0;
    // The first items go to the CTAs in order; the counter (only touched, and
    // only cleared by the host, when there are more items) hands out the rest.
    int it = blockIdx.x;
    while (it < nitems) {
        const WorkItem wi = items[it];
        const int* src = reinterpret_cast<const int*>(entries + wi.entry);
        for (int k = threadIdx.x; k < (int)(sizeof(BatchEntryDev) / 4); k += blockDim.x)
            reinterpret_cast<int*>(&e)[k] = src[k];
        __syncthreads();
        bool ok = true;
        switch (bs_shape(e.op.M)) {
        case 0:
            ok = bs_item<typename CF::template St<4, 1>>(e, wi.y0, wi.y1, table, scratch_all, bufs, bars, bi1, par1);
            break;
        case 1:
            ok = bs_item<typename CF::template St<8, 1>>(e, wi.y0, wi.y1, table, scratch_all, bufs, bars, bi1, par1);
            break;
        case 2:
            ok = bs_item<typename CF::template St<16, 1>>(e, wi.y0, wi.y1, table, scratch_all, bufs, bars, bi1, par1);
            break;
        case 3:
            ok = bs_item<typename CF::template St<16, 2>>(e, wi.y0, wi.y1, table, scratch_all, bufs, bars2, bi2, par2);
            break;
        default:
            ok = bs_item<typename CF::template St<16, 4>>(e, wi.y0, wi.y1, table, scratch_all, bufs, bars4, bi4, par4);
            break;
        }
        if (nitems <= (int)gridDim.x) break;
        // the item is taken when this CTA is free for it; the barriers also
        // end the reads of the last item's table and descriptor
        if (threadIdx.x == 0) *slot = (int)(gridDim.x + atomicAdd(counter, 1u));
        if (__syncthreads_and(ok) == 0) break;  // a completion wait ran out: the status word says so
        it = *slot;
        __syncthreads();
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

}  // namespace pfb
