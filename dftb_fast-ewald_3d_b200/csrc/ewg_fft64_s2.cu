// FP64 transform passes (ewg_fft64.cuh) of a batch, length class 2.
#include "ewg_fft64.cuh"

namespace ewg {

void launch64_seg2(const Launch64& l) {
  Seg64<TwoPass<112, 14, 8>,
        TwoPass<120, 12, 10>,
        TwoPass<128, 16, 8>,
        TwoPass<144, 12, 12>,
        TwoPass<160, 16, 10>,
        TwoPass<168, 14, 12>,
        TwoPass<192, 16, 12>,
        TwoPass<224, 16, 14>,
        TwoPass<240, 16, 15>,
        TwoPass<256, 16, 16>>::launch(l);
}

}  // namespace ewg
