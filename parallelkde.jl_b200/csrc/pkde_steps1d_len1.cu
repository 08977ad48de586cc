// 1-D steps of lengths 144 to 450.
#include "pkde_steps1d_len.cuh"

namespace pkde {

extern const OnePass kOnePasses1[kOneTable];
const OnePass kOnePasses1[kOneTable] = {
    one_pass<144>(), one_pass<150>(), one_pass<160>(), one_pass<162>(), one_pass<180>(), one_pass<192>(),
    one_pass<200>(), one_pass<216>(), one_pass<225>(), one_pass<240>(), one_pass<243>(), one_pass<250>(),
    one_pass<270>(), one_pass<288>(), one_pass<300>(), one_pass<320>(), one_pass<324>(), one_pass<360>(),
    one_pass<375>(), one_pass<384>(), one_pass<400>(), one_pass<405>(), one_pass<432>(), one_pass<450>(),
};

}  // namespace pkde
