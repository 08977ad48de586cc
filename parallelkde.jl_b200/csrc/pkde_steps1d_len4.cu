// 1-D steps of lengths 2430 to 4050.
#include "pkde_steps1d_len.cuh"

namespace pkde {

extern const OnePass kOnePasses4[kOneTable];
const OnePass kOnePasses4[kOneTable] = {
    one_pass<2430>(), one_pass<2500>(), one_pass<2560>(), one_pass<2592>(), one_pass<2700>(), one_pass<2880>(),
    one_pass<2916>(), one_pass<3000>(), one_pass<3072>(), one_pass<3125>(), one_pass<3200>(), one_pass<3240>(),
    one_pass<3375>(), one_pass<3456>(), one_pass<3600>(), one_pass<3645>(), one_pass<3750>(), one_pass<3840>(),
    one_pass<3888>(), one_pass<4000>(), one_pass<4050>(),
};

}  // namespace pkde
