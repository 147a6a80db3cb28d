// ewg_fft64.cu -- lengths and dispatch of the FP64 transform passes.
#include "ewg_fft64.cuh"

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

namespace {
// Every length once, in ascending order, with a file and a class that launch it.
constexpr bool lengths_ok() {
  for (int i = 0; i < kCount64; ++i) {
    const Length64& e = kLengths64[i];
    if (e.r0 * e.r1 != e.n || e.n % 8 != 0 || e.unit < 0 || e.unit >= kUnits64 || e.klass < 0 ||
        e.klass >= kClass64 || (i > 0 && e.n <= kLengths64[i - 1].n))
      return false;
  }
  return true;
}
static_assert(lengths_ok() && kUnits64 == 7 && kClass64 == 4, "fft64_launch and fft64_launch_seg");

// Classes by n / 8 (a batch asks some thousand times).
struct ClassTable {
  signed char k[kLengths64[kCount64 - 1].n / 8 + 1];
};
constexpr ClassTable class_table() {
  ClassTable t{};
  for (signed char& k : t.k) k = -1;
  for (const Length64& e : kLengths64) t.k[e.n / 8] = static_cast<signed char>(e.klass);
  return t;
}
constexpr ClassTable kClasses = class_table();
}  // namespace

int fft64_class(int n) {
  return n > 0 && n % 8 == 0 && n <= kLengths64[kCount64 - 1].n ? kClasses.k[n / 8] : -1;
}

bool fft64_launch(int n, const Launch64& l) {
  return launch64_a(n, l) || launch64_b(n, l) || launch64_c(n, l) || launch64_d(n, l) ||
         launch64_e(n, l) || launch64_f(n, l) || launch64_g(n, l);
}

void fft64_launch_seg(int klass, const Launch64& l) {
  switch (klass) {
    case 0: return launch64_seg0(l);
    case 1: return launch64_seg1(l);
    case 2: return launch64_seg2(l);
    case 3: return launch64_seg3(l);
  }
}

}  // namespace ewg
