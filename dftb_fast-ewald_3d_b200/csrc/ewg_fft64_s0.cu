// FP64 transform passes (ewg_fft64.cuh) of a batch, length class 0.
#include "ewg_fft64.cuh"

namespace ewg {

void launch64_seg0(const Launch64& l) { Class64<0>::launch(l); }

}  // namespace ewg
