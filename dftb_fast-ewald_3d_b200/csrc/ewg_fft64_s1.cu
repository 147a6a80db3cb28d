// FP64 transform passes (ewg_fft64.cuh) of a batch, length class 1.
#include "ewg_fft64.cuh"

namespace ewg {

void launch64_seg1(const Launch64& l) {
  Seg64<TwoPass<72, 9, 8>,
        TwoPass<80, 10, 8>,
        TwoPass<96, 12, 8>>::launch(l);
}

}  // namespace ewg
