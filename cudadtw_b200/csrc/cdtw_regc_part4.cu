// All-windows register-band cDTW over consecutive windows
// (see cdtw_reg.cuh); one translation unit per band range for a parallel
// build.
#include "cdtw_reg.cuh"

namespace cdtw {

void regc_fill_part4(void** eu, void** mh) {
    RegCRange<83, 96>::fill((RegCKernel*)eu, (RegCKernel*)mh);
}

}  // namespace cdtw
