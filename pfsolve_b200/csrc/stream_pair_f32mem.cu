// stream_pair_f32mem.cu -- streaming kernel variants that solve real systems in pairs, FP64 arithmetic on FP32 storage.
#include "stream_variant_defs.h"

namespace pfb {

// Measured, 2^25 rows, tridiagonal, singly and in pairs: N = 201 121 -> 92 us, 512 65.8 -> 56.7; of
// two warps pairs were slower (N = 1 001 114.5 -> 122) and are not compiled.
#define PFB_PAIRS(KL, KU, SV) \
    PFB_SPAIR(8, 1, KL, KU, SV, PREC_F64_F32MEM), \
    PFB_SPAIR(16, 1, KL, KU, SV, PREC_F64_F32MEM)
static const StreamVariant kPart[] = {
    PFB_PAIRS(0, 0, SV_TRI),
    PFB_PAIRS(0, 0, SV_LOWER),
    PFB_PAIRS(0, 0, SV_UPPER),
    PFB_PAIRS(0, 1, SV_LOWER),
    PFB_PAIRS(1, 0, SV_UPPER),
};

const StreamVariant* stream_pair_f32mem(int* count)
{
    *count = (int)(sizeof(kPart) / sizeof(kPart[0]));
    return kPart;
}

PFB_STREAM_STATUS_ACCESSOR(stream_pair_status_f32mem)

}  // namespace pfb
