// FP64 transform passes (ewg_fft64.cuh), instantiated for part of the lengths.
#include "ewg_fft64.cuh"

namespace ewg {

bool launch64_b(int n, const Launch64& l) {
  switch (n) {
    case 24: launch64<TwoPass<24, 6, 4>>(l); break;
    case 80: launch64<TwoPass<80, 10, 8>>(l); break;
    case 144: launch64<TwoPass<144, 12, 12>>(l); break;
    case 200: launch64<TwoPass<200, 20, 10>>(l); break;
    case 480: launch64<TwoPass<480, 24, 20>>(l); break;
    default: return false;
  }
  return true;
}

}  // namespace ewg
