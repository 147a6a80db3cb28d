// FP64 transform passes (ewg_fft64.cuh) of a single cell, the lengths of this file.
#include "ewg_fft64.cuh"

namespace ewg {

bool launch64_g(int n, const Launch64& l) { return launch64_unit<6>(n, l); }

}  // namespace ewg
