// batch_stream_variants.cu -- instantiations of the uneven-batch kernel on the
// streaming solve (the real-system kinds of the group kernel's batches).
#include "jw_batch_stream.cuh"
#include "jw_variants.h"
#include "stream_variant_defs.h"

namespace pfb {

template <class CF>
static void bs_launch_fn(dim3 grid, cudaStream_t st, const BatchEntryDev* entries, const WorkItem* items, int nitems,
                         unsigned int* counter, int64_t Mmax)
{
    jw_batch_stream_kernel<CF><<<grid, kBsThreads, bs_smem_bytes<CF>(Mmax), st>>>(entries, items, nitems, counter,
                                                                                 (int)bs_table_bytes<CF>(Mmax));
}

template <class CF>
static size_t bs_smem_fn(int64_t Mmax)
{
    static_assert(bs_smem_bytes<CF>(1024) <= 227 * 1024, "every compiled kind runs batches of up to 1 024 rows");
    return bs_smem_bytes<CF>(Mmax);
}

#define PFB_BST(KL, KU, SV, P)                                                                                    \
    BatchStreamVariant{KL, KU, SV, P, (const void*)&jw_batch_stream_kernel<BsCfg<KL, KU, SV, P>>,                \
                       &bs_smem_fn<BsCfg<KL, KU, SV, P>>, &bs_launch_fn<BsCfg<KL, KU, SV, P>>}

static const BatchStreamVariant kBatchStreamVariants[] = {
    PFB_BST(1, 1, SV_UPPER, PREC_F64),
    PFB_BST(1, 1, SV_UPPER, PREC_MIXED),
    PFB_BST(0, 0, SV_TRI, PREC_F64),
    PFB_BST(0, 0, SV_TRI, PREC_MIXED),
    PFB_BST(0, 0, SV_UPPER, PREC_F64),
    PFB_BST(0, 0, SV_UPPER, PREC_MIXED),
    PFB_BST(0, 0, SV_LOWER, PREC_MIXED),
    PFB_BST(0, 1, SV_LOWER, PREC_MIXED),
    PFB_BST(1, 0, SV_UPPER, PREC_MIXED),
};

const BatchStreamVariant* find_batch_stream_variant(int KL, int KU, int SV, int PREC)
{
    for (const BatchStreamVariant& v : kBatchStreamVariants)
        if (v.KL == KL && v.KU == KU && v.SV == SV && v.PREC == PREC) return &v;
    return nullptr;
}

int batch_stream_shape(int64_t M) { return bs_shape(M); }
int batch_stream_groups(int64_t M) { return kBsWarps / bs_warps(bs_shape(M)); }
int64_t batch_stream_max_rows() { return 2048; }

PFB_STREAM_STATUS_ACCESSOR(batch_stream_status_fetch_clear)

}  // namespace pfb
