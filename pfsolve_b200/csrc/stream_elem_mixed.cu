// stream_elem_mixed.cu -- streaming kernel variants with element copies, FP32 solve with FP64 refinement.
#include "stream_variant_defs.h"

namespace pfb {

static const StreamVariant kPart[] = {
    PFB_SEREAL(0, 0, SV_TRI, PREC_MIXED),
    PFB_SEREAL(0, 1, SV_LOWER, PREC_MIXED),
    PFB_SEREAL(0, 0, SV_LOWER, PREC_MIXED),
    PFB_SEREAL(1, 0, SV_UPPER, PREC_MIXED),
    PFB_SEREAL(0, 0, SV_UPPER, PREC_MIXED),
    PFB_SEREAL(1, 1, SV_UPPER, PREC_MIXED),
    PFB_SECPLX(2, 2, SV_TRI, false, PREC_MIXED),
};

const StreamVariant* stream_elem_mixed(int* count)
{
    *count = (int)(sizeof(kPart) / sizeof(kPart[0]));
    return kPart;
}

PFB_STREAM_STATUS_ACCESSOR(stream_elem_status_mixed)

}  // namespace pfb
