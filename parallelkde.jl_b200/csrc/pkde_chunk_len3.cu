// Passes of lengths 625 to 1000.
#include "pkde_chunk_len.cuh"

namespace pkde {

extern const LenPasses kLenPasses3[kLenTable];
const LenPasses kLenPasses3[kLenTable] = {
    len_passes<625>(), len_passes<640>(), len_passes<648>(), len_passes<675>(), len_passes<720>(), len_passes<729>(),
    len_passes<750>(), len_passes<768>(), len_passes<800>(), len_passes<810>(), len_passes<864>(), len_passes<900>(),
    len_passes<960>(), len_passes<972>(), len_passes<1000>(),
};

}  // namespace pkde
