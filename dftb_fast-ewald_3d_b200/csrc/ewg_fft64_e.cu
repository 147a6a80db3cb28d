// FP64 transform passes (ewg_fft64.cuh), instantiated for part of the lengths.
#include "ewg_fft64.cuh"

namespace ewg {

bool launch64_e(int n, const Launch64& l) {
  switch (n) {
    case 40: launch64<TwoPass<40, 8, 5>>(l); break;
    case 64: launch64<TwoPass<64, 8, 8>>(l); break;
    case 192: launch64<TwoPass<192, 16, 12>>(l); break;
    case 256: launch64<TwoPass<256, 16, 16>>(l); break;
    case 400: launch64<TwoPass<400, 20, 20>>(l); break;
    default: return false;
  }
  return true;
}

}  // namespace ewg
