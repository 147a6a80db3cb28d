// FP64 transform passes (ewg_fft64.cuh), instantiated for part of the lengths.
#include "ewg_fft64.cuh"

namespace ewg {

bool launch64_c(int n, const Launch64& l) {
  switch (n) {
    case 32: launch64<TwoPass<32, 8, 4>>(l); break;
    case 72: launch64<TwoPass<72, 9, 8>>(l); break;
    case 168: launch64<TwoPass<168, 14, 12>>(l); break;
    case 240: launch64<TwoPass<240, 16, 15>>(l); break;
    case 432: launch64<TwoPass<432, 24, 18>>(l); break;
    default: return false;
  }
  return true;
}

}  // namespace ewg
