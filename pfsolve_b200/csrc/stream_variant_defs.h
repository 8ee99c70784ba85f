// stream_variant_defs.h -- helpers and macros that instantiate streaming
// JW-step kernel variants into the per-file variant tables.  Every file that
// includes it gets its own copy of the device status word (g_stream_status)
// and defines an accessor for it.
#pragma once
#include <cuda.h>

#include "jw_stream.cuh"
#include "jw_variants.h"

namespace pfb {

template <class C>
inline size_t st_smem_fn(int G, int NB)
{
    return st_smem_bytes<C>(G, NB);
}

template <class C>
inline int st_threads_fn(int G)
{
    static_assert(st_scan_fits<C>(), "the scan's exchange stays clear of the barriers");
    return st_threads<C>(G);
}

template <class C>
inline void st_launch_fn(dim3 grid, dim3 block, size_t smem, cudaStream_t st, const CUtensorMap* in,
                         const CUtensorMap* out, const JwOperator& op, const StreamIO& io)
{
    jw_stream_kernel<C><<<grid, block, smem, st>>>(*in, *out, op, io);
}

// Element copies in place of tensor copies (jw_stream_elem_kernel).
template <class C>
inline void st_elem_launch_fn(dim3 grid, dim3 block, size_t smem, cudaStream_t st, const CUtensorMap*,
                              const CUtensorMap*, const JwOperator& op, const StreamIO& io)
{
    jw_stream_elem_kernel<C><<<grid, block, smem, st>>>(op, io);
}
#define PFB_SVE(R, W, KL, KU, SV, LIN, LOUT, SC, P)                                                     \
    StreamVariant{R, W, KL, KU, SV, LIN, LOUT, SC, P, StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>::kMaxThreads, \
                  (const void*)&jw_stream_elem_kernel<StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>>,            \
                  &st_smem_fn<StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>>, 0, 0,                              \
                  &st_elem_launch_fn<StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>>, 0,                          \
                  &st_threads_fn<StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>>, 1}
// real systems: M <= 128, 256, 512, 1024, 2048 and 4096
#define PFB_SEREAL(KL, KU, SV, P)                                                                            \
    PFB_SVE(4, 1, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), PFB_SVE(8, 1, KL, KU, SV, LAY_REAL, LAY_REAL, false, P),       \
        PFB_SVE(16, 1, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), PFB_SVE(16, 2, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), \
        PFB_SVE(16, 4, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), PFB_SVE(32, 4, KL, KU, SV, LAY_REAL, LAY_REAL, false, P)
// complex XXII right-hand sides written packed: M <= 512 and 1024 (32 rows per
// thread of two warps measured slower than the group kernel: 1 184 systems of
// 2 000 rows, 60 against 45 us)
#define PFB_SECPLX(KL, KU, SV, SC, P)                                                                        \
    PFB_SVE(16, 1, KL, KU, SV, LAY_XXII, LAY_PACKED, SC, P), PFB_SVE(16, 2, KL, KU, SV, LAY_XXII, LAY_PACKED, SC, P)
#define PFB_SVP(R, W, KL, KU, SV, LIN, LOUT, SC, P)                                                     \
    StreamVariant{R, W, KL, KU, SV, LIN, LOUT, SC, P, StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>::kMaxThreads, \
                  (const void*)&jw_stream_kernel<StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>>,                 \
                  &st_smem_fn<StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>>,                                    \
                  StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>::IB, StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>::IBO, \
                  &st_launch_fn<StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>>, 0,                               \
                  &st_threads_fn<StCfg<R, W, KL, KU, SV, LIN, LOUT, SC, P>>}
#define PFB_SV(R, W, KL, KU, SV, LIN, LOUT, SC) PFB_SVP(R, W, KL, KU, SV, LIN, LOUT, SC, PREC_F64)
// ALT stride-2 mode: real FP64 row sets, each holding two systems
#define PFB_SVA(R, W, KL, KU, SV)                                                                              \
    StreamVariant{R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64,                                      \
                  StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>::kMaxThreads,                \
                  (const void*)&jw_stream_kernel<StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>>, \
                  &st_smem_fn<StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>>,                 \
                  StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>::IB,                          \
                  StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>::IBO,                         \
                  &st_launch_fn<StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>>, 1,               \
                  &st_threads_fn<StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>>}
// ALT by element copies: row sets of M <= 256, 512, 1024, 2048 and 4096 rows
#define PFB_SVAE(R, W, KL, KU, SV)                                                                             \
    StreamVariant{R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64,                                      \
                  StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>::kMaxThreads,                \
                  (const void*)&jw_stream_elem_kernel<StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>>, \
                  &st_smem_fn<StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>>, 0, 0,           \
                  &st_elem_launch_fn<StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>>, 1,      \
                  &st_threads_fn<StCfg<R, W, KL, KU, SV, LAY_REAL, LAY_REAL, false, PREC_F64, 1>>, 1}
#define PFB_SALTE(KL, KU, SV)                                                                                 \
    PFB_SVAE(8, 1, KL, KU, SV), PFB_SVAE(16, 1, KL, KU, SV), PFB_SVAE(16, 2, KL, KU, SV), PFB_SVAE(16, 4, KL, KU, SV), \
        PFB_SVAE(32, 4, KL, KU, SV)
// 8, 16 and 32 rows per thread, 1, 2 and 4 warps per row set (M <= 4096)
#define PFB_SALT(KL, KU, SV)                                                                                  \
    PFB_SVA(8, 1, KL, KU, SV), PFB_SVA(8, 2, KL, KU, SV), PFB_SVA(8, 4, KL, KU, SV), PFB_SVA(16, 1, KL, KU, SV), \
        PFB_SVA(16, 2, KL, KU, SV), PFB_SVA(16, 4, KL, KU, SV), PFB_SVA(32, 1, KL, KU, SV),                    \
        PFB_SVA(32, 2, KL, KU, SV), PFB_SVA(32, 4, KL, KU, SV)
// real systems: 8 rows per thread (M <= 256, 512, 1024), 16 (M <= 512, 1024,
// 2048) and 32 (M <= 1024, 2048, 4096)
#define PFB_SREALP(KL, KU, SV, P)                                                                        \
    PFB_SVP(8, 1, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), PFB_SVP(8, 2, KL, KU, SV, LAY_REAL, LAY_REAL, false, P),   \
        PFB_SVP(8, 4, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), PFB_SVP(16, 1, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), \
        PFB_SVP(16, 2, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), PFB_SVP(16, 4, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), \
        PFB_SVP(32, 1, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), PFB_SVP(32, 2, KL, KU, SV, LAY_REAL, LAY_REAL, false, P), \
        PFB_SVP(32, 4, KL, KU, SV, LAY_REAL, LAY_REAL, false, P)
#define PFB_SREAL(KL, KU, SV) PFB_SREALP(KL, KU, SV, PREC_F64)
// complex XXII right-hand sides written packed
#define PFB_SCPLXP(KL, KU, SV, SC, P)                                                                             \
    PFB_SVP(16, 1, KL, KU, SV, LAY_XXII, LAY_PACKED, SC, P), PFB_SVP(16, 2, KL, KU, SV, LAY_XXII, LAY_PACKED, SC, P), \
        PFB_SVP(32, 1, KL, KU, SV, LAY_XXII, LAY_PACKED, SC, P), PFB_SVP(32, 2, KL, KU, SV, LAY_XXII, LAY_PACKED, SC, P)
#define PFB_SCPLX(KL, KU, SV, SC) PFB_SCPLXP(KL, KU, SV, SC, PREC_F64)
// real systems two at a time, as XXII complex ones (a pair shares every table
// read): by tensor copies and by element copies
#define PFB_SPAIR(R, W, KL, KU, SV, P)                                                                          \
    PFB_SVP(R, W, KL, KU, SV, LAY_XXII, LAY_XXII, false, P), PFB_SVE(R, W, KL, KU, SV, LAY_XXII, LAY_XXII, false, P)

// Status word of this translation unit's kernels: read and clear.
#define PFB_STREAM_STATUS_ACCESSOR(name)                                          \
    unsigned name()                                                               \
    {                                                                             \
        unsigned v = 0, zero = 0;                                                 \
        if (cudaMemcpyFromSymbol(&v, g_stream_status, sizeof(v)) != cudaSuccess) \
            return ~0u;                                                           \
        if (v) cudaMemcpyToSymbol(g_stream_status, &zero, sizeof(zero));          \
        return v;                                                                 \
    }

}  // namespace pfb
