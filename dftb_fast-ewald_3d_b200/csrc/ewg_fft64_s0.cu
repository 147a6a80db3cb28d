// FP64 transform passes (ewg_fft64.cuh) of a batch, length class 0.
#include "ewg_fft64.cuh"

namespace ewg {

void launch64_seg0(const Launch64& l) {
  Seg64<TwoPass<16, 4, 4>,
        TwoPass<24, 6, 4>,
        TwoPass<32, 8, 4>,
        TwoPass<40, 8, 5>,
        TwoPass<48, 8, 6>,
        TwoPass<56, 8, 7>,
        TwoPass<64, 8, 8>>::launch(l);
}

}  // namespace ewg
