// FP64 transform passes (ewg_fft64.cuh) of a batch, length class 1.
#include "ewg_fft64.cuh"

namespace ewg {

void launch64_seg1(const Launch64& l) { Class64<1>::launch(l); }

}  // namespace ewg
