// fpsg_packed_f64.cu — FP64 configurations of k_pair_packed.
#include "fpsg_resident.h"

namespace fpsg {

template <>
const std::vector<QuadCfg<double>>& packed_cfgs<double>()
{
    static const std::vector<QuadCfg<double>> v = {
        FPSG_PACKED(double, 512, 3, false), FPSG_PACKED(double, 512, 4, false), FPSG_PACKED(double, 512, 5, false),
    };
    return v;
}

}  // namespace fpsg
