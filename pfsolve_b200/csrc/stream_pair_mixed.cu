// stream_pair_mixed.cu -- streaming kernel variants that solve real systems in pairs, FP32 solve with FP64 refinement.
#include "stream_variant_defs.h"

namespace pfb {

// Measured, 2^25 rows, tridiagonal, singly and in pairs: N = 512 160 -> 130 us, 701 348 -> 320,
// 1 001 264 -> 240; at 8 rows per thread pairs were slower (N = 96 370 -> 412) and are not compiled.
#define PFB_PAIRS(KL, KU, SV) \
    PFB_SPAIR(16, 1, KL, KU, SV, PREC_MIXED), \
    PFB_SPAIR(16, 2, KL, KU, SV, PREC_MIXED), \
    PFB_SPAIR(16, 4, KL, KU, SV, PREC_MIXED)
static const StreamVariant kPart[] = {
    PFB_PAIRS(0, 0, SV_TRI),
    PFB_PAIRS(0, 0, SV_LOWER),
    PFB_PAIRS(0, 0, SV_UPPER),
    PFB_PAIRS(0, 1, SV_LOWER),
    PFB_PAIRS(1, 0, SV_UPPER),
};

const StreamVariant* stream_pair_mixed(int* count)
{
    *count = (int)(sizeof(kPart) / sizeof(kPart[0]));
    return kPart;
}

PFB_STREAM_STATUS_ACCESSOR(stream_pair_status_mixed)

}  // namespace pfb
