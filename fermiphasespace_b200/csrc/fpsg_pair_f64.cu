// fpsg_pair_f64.cu — FP64 configurations of k_pair.
#include "fpsg_resident.h"

namespace fpsg {

template <>
const std::vector<ResCfg<double>>& pair_cfgs<double>()
{
    static const std::vector<ResCfg<double>> v = {
        FPSG_PAIR(double, 128, 1, false), FPSG_PAIR(double, 128, 2, false), FPSG_PAIR(double, 256, 2, false),
        FPSG_PAIR(double, 256, 4, false), FPSG_PAIR(double, 256, 4, true), FPSG_PAIR(double, 256, 5, true),
        FPSG_PAIR(double, 512, 4, true),
    };
    return v;
}

}  // namespace fpsg
