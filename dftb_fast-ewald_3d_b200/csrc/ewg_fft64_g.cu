// FP64 transform passes (ewg_fft64.cuh), instantiated for part of the lengths.
#include "ewg_fft64.cuh"

namespace ewg {

bool launch64_g(int n, const Launch64& l) {
  switch (n) {
    case 96: launch64<TwoPass<96, 12, 8>>(l); break;
    case 160: launch64<TwoPass<160, 16, 10>>(l); break;
    case 320: launch64<TwoPass<320, 20, 16>>(l); break;
    case 336: launch64<TwoPass<336, 21, 16>>(l); break;
    default: return false;
  }
  return true;
}

}  // namespace ewg
