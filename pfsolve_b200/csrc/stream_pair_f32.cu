// stream_pair_f32.cu -- streaming kernel variants that solve real systems in pairs, FP32 storage and arithmetic.
#include "stream_variant_defs.h"

namespace pfb {

// Measured, 2^25 rows, tridiagonal, singly and in pairs: N = 96 116 -> 93 us, 701 126 -> 98, 1 001
// 102 -> 83; at 16 rows per thread of one warp pairs were slower (131 072 x 512 100 -> 105) and are not compiled.
#define PFB_PAIRS(KL, KU, SV) \
    PFB_SPAIR(8, 1, KL, KU, SV, PREC_F32), \
    PFB_SPAIR(16, 2, KL, KU, SV, PREC_F32), \
    PFB_SPAIR(16, 4, KL, KU, SV, PREC_F32)
static const StreamVariant kPart[] = {
    PFB_PAIRS(0, 0, SV_TRI),
    PFB_PAIRS(0, 0, SV_LOWER),
    PFB_PAIRS(0, 0, SV_UPPER),
    PFB_PAIRS(0, 1, SV_LOWER),
    PFB_PAIRS(1, 0, SV_UPPER),
};

const StreamVariant* stream_pair_f32(int* count)
{
    *count = (int)(sizeof(kPart) / sizeof(kPart[0]));
    return kPart;
}

PFB_STREAM_STATUS_ACCESSOR(stream_pair_status_f32)

}  // namespace pfb
