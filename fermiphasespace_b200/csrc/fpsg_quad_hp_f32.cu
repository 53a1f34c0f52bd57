// fpsg_quad_hp_f32.cu — FP32 configurations of k_resident_quad_hp.
#include "fpsg_resident.h"

namespace fpsg {

template <>
const std::vector<QuadCfg<float>>& quad_hp_cfgs<float>()
{
    static const std::vector<QuadCfg<float>> v = {
        FPSG_QUAD_HP32(256, 4, 1), FPSG_QUAD_HP32(512, 5, 1), FPSG_QUAD_HP32(512, 12, 1), FPSG_QUAD_HP32(512, 6, 2), FPSG_QUAD_HP32(512, 11, 2),
    };
    return v;
}

}  // namespace fpsg
