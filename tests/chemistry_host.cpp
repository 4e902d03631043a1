// The chemistry of the kernels compiled for the host: what it computes does not depend on where.
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __forceinline__ inline
static inline int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
static inline double __longlong_as_double(long long v) {
  double d;
  std::memcpy(&d, &v, 8);
  return d;
}
static inline float rsqrtf(float v) { return 1.0f / std::sqrt(v); }
using std::fmin;

#include "chemistry_device.cuh"

using Solver = swk::ChemSolver<false>;

extern "C" {

// FP64: recombination rate alpha and its derivative, cooling per n_e^2 of a fully ionized gas
// (recombination and free-free) at the temperatures t
void fits(int n, const double* t, double* alpha, double* dalpha, double* cooling) {
  for (int i = 0; i < n; ++i) {
    const swk::Fits64 f = swk::fits64(t[i]);
    Solver::recombination(f, alpha[i], dalpha[i]);
    Solver s{};
    s.x = 1.0;
    s.temperature = t[i];
    s.density = swk::Units::kProtonMass;
    s.volume = s.length = s.scale_factor = 1.0;
    s.rate = 0.0;
    s.prepare(1.0);
    s.compton_cell = 0.0;
    double slope;
    s.cooling(f, cooling[i], slope);
  }
}

void small_enough(int n, const double* value, const double* change, const double* safety, uint8_t* out) {
  for (int i = 0; i < n; ++i) out[i] = Solver::small(value[i], change[i], safety[i]) ? 1 : 0;
}
}
