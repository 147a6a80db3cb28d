// FP64 transform passes (ewg_fft64.cuh), instantiated for part of the lengths.
#include "ewg_fft64.cuh"

namespace ewg {

bool launch64_d(int n, const Launch64& l) {
  switch (n) {
    case 120: launch64<TwoPass<120, 12, 10>>(l); break;
    case 128: launch64<TwoPass<128, 16, 8>>(l); break;
    case 288: launch64<TwoPass<288, 18, 16>>(l); break;
    case 384: launch64<TwoPass<384, 24, 16>>(l); break;
    default: return false;
  }
  return true;
}

}  // namespace ewg
