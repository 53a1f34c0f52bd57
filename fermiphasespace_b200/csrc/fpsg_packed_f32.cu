// fpsg_packed_f32.cu — FP32 configurations of k_pair_packed.
#include "fpsg_resident.h"

namespace fpsg {

template <>
const std::vector<QuadCfg<float>>& packed_cfgs<float>()
{
    static const std::vector<QuadCfg<float>> v = {
        FPSG_PACKED(float, 512, 6, false), FPSG_PACKED(float, 512, 8, false), FPSG_PACKED(float, 512, 11, true),
    };
    return v;
}

}  // namespace fpsg
