// fpsg_pair_f32.cu — FP32 configurations of k_pair.
#include "fpsg_resident.h"

namespace fpsg {

template <>
const std::vector<ResCfg<float>>& pair_cfgs<float>()
{
    static const std::vector<ResCfg<float>> v = {
        FPSG_PAIR(float, 128, 1, false), FPSG_PAIR(float, 128, 2, false), FPSG_PAIR(float, 256, 2, false),
        FPSG_PAIR(float, 256, 4, false), FPSG_PAIR(float, 512, 4, false), FPSG_PAIR(float, 512, 5, false),
        FPSG_PAIR(float, 256, 5, true), FPSG_PAIR(float, 512, 4, true), FPSG_PAIR(float, 512, 5, true),
    };
    return v;
}

}  // namespace fpsg
