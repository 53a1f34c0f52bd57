// fpsg_quad_hp_f64.cu — FP64 configurations of k_resident_quad_hp.
#include "fpsg_resident.h"

namespace fpsg {

const std::vector<QuadCfg<double>>& quad_hp1_cfgs_f64();     // one CTA per spin

template <>
const std::vector<QuadCfg<double>>& quad_hp_cfgs<double>()
{
    static const std::vector<QuadCfg<double>> v = [] {
        std::vector<QuadCfg<double>> c = quad_hp1_cfgs_f64();
        c.push_back(QuadCfg<double>FPSG_QUAD_HP64(512, 3, 2));
        c.push_back(QuadCfg<double>FPSG_QUAD_HP64(512, 4, 2));
        c.push_back(QuadCfg<double>FPSG_QUAD_HP64(512, 5, 2));
        c.push_back(QuadCfg<double>FPSG_QUAD_HP64(640, 4, 2));
        c.push_back(QuadCfg<double>FPSG_QUAD_HP64(384, 7, 2));
        return c;
    }();
    return v;
}

}  // namespace fpsg
