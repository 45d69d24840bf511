// Register-band cDTW of listed windows, several per thread
// (see cdtw_reg.cuh); one translation unit per band range for a parallel
// build.
#include "cdtw_reg.cuh"

namespace cdtw {

void regn_fill_part0(void** eu, void** mh) {
    RegNRange<0, kMaxReg2W>::fill((RegKernel*)eu, (RegKernel*)mh);
}

}  // namespace cdtw
