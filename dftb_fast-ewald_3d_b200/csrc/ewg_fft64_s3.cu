// FP64 transform passes (ewg_fft64.cuh) of a batch, length class 3.
#include "ewg_fft64.cuh"

namespace ewg {

void launch64_seg3(const Launch64& l) {
  Seg64<TwoPass<200, 20, 10>,
        TwoPass<216, 18, 12>,
        TwoPass<280, 20, 14>,
        TwoPass<288, 18, 16>,
        TwoPass<320, 20, 16>,
        TwoPass<336, 21, 16>,
        TwoPass<360, 20, 18>,
        TwoPass<384, 24, 16>,
        TwoPass<400, 20, 20>,
        TwoPass<432, 24, 18>,
        TwoPass<480, 24, 20>,
        TwoPass<576, 24, 24>>::launch(l);
}

}  // namespace ewg
