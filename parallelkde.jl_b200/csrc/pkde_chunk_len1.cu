// Passes of lengths 96 to 250.
#include "pkde_chunk_len.cuh"

namespace pkde {

extern const LenPasses kLenPasses1[kLenTable];
const LenPasses kLenPasses1[kLenTable] = {
    len_passes<96>(), len_passes<100>(), len_passes<108>(), len_passes<120>(), len_passes<125>(), len_passes<135>(),
    len_passes<144>(), len_passes<150>(), len_passes<160>(), len_passes<162>(), len_passes<180>(), len_passes<192>(),
    len_passes<200>(), len_passes<216>(), len_passes<225>(), len_passes<240>(), len_passes<243>(), len_passes<250>(),
};

}  // namespace pkde
