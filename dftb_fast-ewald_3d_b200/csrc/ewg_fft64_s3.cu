// FP64 transform passes (ewg_fft64.cuh) of a batch, length class 3.
#include "ewg_fft64.cuh"

namespace ewg {

void launch64_seg3(const Launch64& l) { Class64<3>::launch(l); }

}  // namespace ewg
