// 1-D steps of lengths 480 to 1152.
#include "pkde_steps1d_len.cuh"

namespace pkde {

extern const OnePass kOnePasses2[kOneTable];
const OnePass kOnePasses2[kOneTable] = {
    one_pass<480>(), one_pass<486>(), one_pass<500>(), one_pass<540>(), one_pass<576>(), one_pass<600>(),
    one_pass<625>(), one_pass<640>(), one_pass<648>(), one_pass<675>(), one_pass<720>(), one_pass<729>(),
    one_pass<750>(), one_pass<768>(), one_pass<800>(), one_pass<810>(), one_pass<864>(), one_pass<900>(),
    one_pass<960>(), one_pass<972>(), one_pass<1000>(), one_pass<1080>(), one_pass<1125>(), one_pass<1152>(),
};

}  // namespace pkde
