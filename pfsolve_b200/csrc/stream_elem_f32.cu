// stream_elem_f32.cu -- streaming kernel variants with element copies, FP32 storage and arithmetic.
#include "stream_variant_defs.h"

namespace pfb {

static const StreamVariant kPart[] = {
    PFB_SEREAL(0, 0, SV_TRI, PREC_F32),
    PFB_SEREAL(0, 1, SV_LOWER, PREC_F32),
    PFB_SEREAL(0, 1, SV_NONE, PREC_F32),
    PFB_SEREAL(0, 0, SV_LOWER, PREC_F32),
    PFB_SEREAL(1, 0, SV_UPPER, PREC_F32),
    PFB_SEREAL(1, 0, SV_NONE, PREC_F32),
    PFB_SEREAL(0, 0, SV_UPPER, PREC_F32),
    PFB_SEREAL(1, 1, SV_UPPER, PREC_F32),
    PFB_SEREAL(2, 2, SV_TRI, PREC_F32),
    PFB_SECPLX(2, 2, SV_TRI, false, PREC_F32),
    PFB_SECPLX(2, 2, SV_TRI, true, PREC_F32),
    PFB_SECPLX(1, 1, SV_UPPER, true, PREC_F32),
};

const StreamVariant* stream_elem_f32(int* count)
{
    *count = (int)(sizeof(kPart) / sizeof(kPart[0]));
    return kPart;
}

PFB_STREAM_STATUS_ACCESSOR(stream_elem_status_f32)

}  // namespace pfb
