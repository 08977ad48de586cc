// Passes of lengths 270 to 600.
#include "pkde_chunk_len.cuh"

namespace pkde {

extern const LenPasses kLenPasses2[kLenTable];
const LenPasses kLenPasses2[kLenTable] = {
    len_passes<270>(), len_passes<288>(), len_passes<300>(), len_passes<320>(), len_passes<324>(), len_passes<360>(),
    len_passes<375>(), len_passes<384>(), len_passes<400>(), len_passes<405>(), len_passes<432>(), len_passes<450>(),
    len_passes<480>(), len_passes<486>(), len_passes<500>(), len_passes<540>(), len_passes<576>(), len_passes<600>(),
};

}  // namespace pkde
