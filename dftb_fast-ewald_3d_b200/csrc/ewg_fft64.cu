// ewg_fft64.cu -- lengths and dispatch of the FP64 transform passes.
#include "ewg_kernels.h"

namespace ewg {

bool launch64_a(int n, const Launch64& l);
bool launch64_b(int n, const Launch64& l);
bool launch64_c(int n, const Launch64& l);
bool launch64_d(int n, const Launch64& l);
bool launch64_e(int n, const Launch64& l);
bool launch64_f(int n, const Launch64& l);
bool launch64_g(int n, const Launch64& l);
void launch64_seg0(const Launch64& l);
void launch64_seg1(const Launch64& l);
void launch64_seg2(const Launch64& l);
void launch64_seg3(const Launch64& l);

// Whole tiles of 8 points that factor into two radices of at most 24.  The class
// of a length bounds the registers, threads (64, 96, 128, 192) and shared memory
// that a batch's launch gives every block.
int fft64_class(int n) {
  switch (n) {
    case 16: case 24: case 32: case 40: case 48: case 56: case 64:
      return 0;
    case 72: case 80: case 96:
      return 1;
    case 112: case 120: case 128: case 144: case 160: case 168: case 192: case 224: case 240: case 256:
      return 2;
    case 200: case 216: case 280: case 288: case 320: case 336: case 360: case 384: case 400: case 432: case 480: case 576:
      return 3;
    default: return -1;
  }
}

void fft64_launch(int n, const Launch64& l) {
  launch64_a(n, l) || launch64_b(n, l) || launch64_c(n, l) || launch64_d(n, l) || launch64_e(n, l) || launch64_f(n, l) || launch64_g(n, l);
}

void fft64_launch_seg(int klass, const Launch64& l) {
  switch (klass) {
    case 0: return launch64_seg0(l);
    case 1: return launch64_seg1(l);
    case 2: return launch64_seg2(l);
    default: return launch64_seg3(l);
  }
}

}  // namespace ewg
