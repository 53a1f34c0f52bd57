// fpsg_quad_hp_f64.cu — FP64 configurations of k_resident_quad_hp.
#include "fpsg_resident.h"

namespace fpsg {

template <>
const std::vector<QuadCfg<double>>& quad_hp_cfgs<double>()
{
    static const std::vector<QuadCfg<double>> v = {
        FPSG_QUAD_HP64(512, 5), FPSG_QUAD_HP64(640, 4), FPSG_QUAD_HP64(384, 7),
    };
    return v;
}

}  // namespace fpsg
