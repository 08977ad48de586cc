// 1-D steps of lengths 1200 to 2400.
#include "pkde_steps1d_len.cuh"

namespace pkde {

extern const OnePass kOnePasses3[kOneTable];
const OnePass kOnePasses3[kOneTable] = {
    one_pass<1200>(), one_pass<1215>(), one_pass<1250>(), one_pass<1280>(), one_pass<1296>(), one_pass<1350>(),
    one_pass<1440>(), one_pass<1458>(), one_pass<1500>(), one_pass<1536>(), one_pass<1600>(), one_pass<1620>(),
    one_pass<1728>(), one_pass<1800>(), one_pass<1875>(), one_pass<1920>(), one_pass<1944>(), one_pass<2000>(),
    one_pass<2025>(), one_pass<2160>(), one_pass<2187>(), one_pass<2250>(), one_pass<2304>(), one_pass<2400>(),
};

}  // namespace pkde
