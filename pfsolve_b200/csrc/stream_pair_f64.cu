// stream_pair_f64.cu -- streaming kernel variants that solve real systems in pairs, FP64.
#include "stream_variant_defs.h"

namespace pfb {

// Measured, 2^25 rows, tridiagonal, singly and in pairs: N = 256 126 -> 98 us, 401 130 -> 108,
// 512 95.9 -> 94.2, 701 171 -> 166; 60 000 x 1 001 242 -> 234.
#define PFB_PAIRS(KL, KU, SV) \
    PFB_SPAIR(8, 1, KL, KU, SV, PREC_F64), \
    PFB_SPAIR(16, 1, KL, KU, SV, PREC_F64), \
    PFB_SPAIR(16, 2, KL, KU, SV, PREC_F64), \
    PFB_SPAIR(16, 4, KL, KU, SV, PREC_F64)
static const StreamVariant kPart[] = {
    PFB_PAIRS(0, 0, SV_TRI),
    PFB_PAIRS(0, 0, SV_LOWER),
    PFB_PAIRS(0, 0, SV_UPPER),
    PFB_PAIRS(0, 1, SV_LOWER),
    PFB_PAIRS(1, 0, SV_UPPER),
};

const StreamVariant* stream_pair_f64(int* count)
{
    *count = (int)(sizeof(kPart) / sizeof(kPart[0]));
    return kPart;
}

PFB_STREAM_STATUS_ACCESSOR(stream_pair_status_f64)

}  // namespace pfb
