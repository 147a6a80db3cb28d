// FP64 transform passes (ewg_fft64.cuh), instantiated for part of the lengths.
#include "ewg_fft64.cuh"

namespace ewg {

bool launch64_f(int n, const Launch64& l) {
  switch (n) {
    case 56: launch64<TwoPass<56, 8, 7>>(l); break;
    case 224: launch64<TwoPass<224, 16, 14>>(l); break;
    case 280: launch64<TwoPass<280, 20, 14>>(l); break;
    case 360: launch64<TwoPass<360, 20, 18>>(l); break;
    default: return false;
  }
  return true;
}

}  // namespace ewg
