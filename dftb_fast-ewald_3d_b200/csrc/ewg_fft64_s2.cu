// FP64 transform passes (ewg_fft64.cuh) of a batch, length class 2.
#include "ewg_fft64.cuh"

namespace ewg {

void launch64_seg2(const Launch64& l) { Class64<2>::launch(l); }

}  // namespace ewg
