// fpsg_quad_hp1_f64.cu — FP64 configurations of k_resident_quad_hp with one CTA per spin.
#include "fpsg_resident.h"

namespace fpsg {

const std::vector<QuadCfg<double>>& quad_hp1_cfgs_f64()
{
    static const std::vector<QuadCfg<double>> v = {
        FPSG_QUAD_HP64(256, 4, 1), FPSG_QUAD_HP64(512, 4, 1), FPSG_QUAD_HP64(512, 6, 1),
    };
    return v;
}

}  // namespace fpsg
