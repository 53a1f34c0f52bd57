// fpsg_vjp_f32.cu — FP32 configurations of k_vjp_segment.
#include "fpsg_resident.h"

namespace fpsg {

template <>
const std::vector<VjpCfg<float>>& vjp_cfgs<float>()
{
    static const std::vector<VjpCfg<float>> v = {
        FPSG_VJP(float, 128, 3), FPSG_VJP(float, 256, 4), FPSG_VJP(float, 512, 5),
    };
    return v;
}

}  // namespace fpsg
