// FP64 transform passes (ewg_fft64.cuh), instantiated for part of the lengths.
#include "ewg_fft64.cuh"

namespace ewg {

bool launch64_a(int n, const Launch64& l) {
  switch (n) {
    case 16: launch64<TwoPass<16, 4, 4>>(l); break;
    case 48: launch64<TwoPass<48, 8, 6>>(l); break;
    case 112: launch64<TwoPass<112, 14, 8>>(l); break;
    case 216: launch64<TwoPass<216, 18, 12>>(l); break;
    case 576: launch64<TwoPass<576, 24, 24>>(l); break;
    default: return false;
  }
  return true;
}

}  // namespace ewg
