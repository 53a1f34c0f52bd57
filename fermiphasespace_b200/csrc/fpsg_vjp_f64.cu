// fpsg_vjp_f64.cu — FP64 configurations of k_vjp_segment.
#include "fpsg_resident.h"

namespace fpsg {

template <>
const std::vector<VjpCfg<double>>& vjp_cfgs<double>()
{
    static const std::vector<VjpCfg<double>> v = {
        FPSG_VJP(double, 128, 3), FPSG_VJP(double, 256, 4), FPSG_VJP(double, 512, 5),
    };
    return v;
}

}  // namespace fpsg
