// Hydrogen-only chemistry on the device: the semi-implicit x_HII / temperature
// update of Rosdahl et al. (2015) with recursive timestep halving, as in
// src/chemistry/hydrogen_only/mod.rs:125-461 of the reference.
//
// The reference recurses (perform_timestep_internal, 394-424): a failed attempt
// over dt is replaced by two attempts over dt/2, depth <= 100.  Here the recursion
// is an explicit loop.  At any time at most one second half is pending per depth,
// and pending halves are taken deepest first, so the pending set is a bitmask
// over depths and the next interval is its highest set bit.  The result (state and
// the timescale of the last accepted substep) is the same as the recursion's.
//
// kCarryNeutral = false restates the reference exactly: the neutral fraction is
// recomputed as (1 - x) wherever it is used.  kCarryNeutral = true (mixed path)
// additionally carries y = 1 - x as its own FP64 state, updated by -dx, so the
// neutral density keeps full relative precision near complete ionisation; the
// smaller of x and y is the accurate one and the other is re-derived from it.
//
// What bounds it: the FP64 unit, 64 cycles for a warp's instruction in a quarter of an SM, and
// in small runs the chain of the attempts of one cell (hundreds beside a source).  Hence
//   what depends on the state alone is formed once per state (begin()) and not for every
//   attempt from it: a rejected attempt is repeated with half the step for a few operations;
//   FP64: the fits at the temperature that an attempt accepts are the next state's;
//   the recommended steps are formed for the last accepted attempt only.
// None of it changes a rounding: near equilibrium a state's timescale is its value over a small
// difference of large terms, which shows the last bits of every one of them.  Against factors formed
// per attempt, ms a sweep: 128^3 mixed, 14 attempts a cell 10.9 -> 9.4, one 0.97 -> 0.91; 64^3 FP64,
// 27 attempts 15.9 -> 14.0, 1.6 attempts 0.88 -> 0.74, one 0.33 -> 0.32; 256^3 FP64 219 -> 181.
// The mixed path evaluates the rate fits in FP32 (Fits32); the densities, the sums, the
// implicit updates and their accept / reject tests are FP64 in both.
#pragma once

#include <cfloat>
#include <cstdint>

namespace swk {

// src/units/mod.rs:14-108, every quantity a plain SI double.
struct Units {
  static constexpr double kCentimeters = 0.01;
  static constexpr double kCentimetersSquared = kCentimeters * kCentimeters;
  static constexpr double kCubicCentimeters = 1e-6;
  static constexpr double kSeconds = 1.0;
  static constexpr double kCentimetersCubedPerS = kCubicCentimeters / kSeconds;
  static constexpr double kErgs = 1e-7;
  static constexpr double kErgsCentimetersCubedPerS = kErgs * kCentimetersCubedPerS;
  static constexpr double kErgsPerS = kErgs / kSeconds;
  static constexpr double kElectronVolts = 1.602176634e-19;
  static constexpr double kBoltzmann = 1.380649e-23;
  static constexpr double kProtonMass = 1.67262192369e-27;
  static constexpr double kGamma = 5.0 / 3.0;
  static constexpr double kSigma = 2.9580524545305314e-18 * kCentimetersSquared;
  static constexpr double kPhotonAverageEnergy = 18.028356312818811 * kElectronVolts;
  static constexpr double kRydberg = 13.65693 * kElectronVolts;
};

constexpr int kChemMaxDepth = 100;               // hydrogen_only/mod.rs:34
constexpr double kIonizedFractionEpsilon = 1e-10;  // hydrogen_only/mod.rs:38

enum ChemProcess : int { kProcTemperature = 0, kProcIonization = 1, kProcPhotonRate = 2 };

struct Timescale {
  double time;
  int process;
};

// chemistry/timescale.rs:114-120: strict <, so NaN selects `b`.
__device__ __forceinline__ Timescale ts_min(Timescale a, Timescale b) {
  return a.time < b.time ? a : b;
}

// Mixed path: the Rosdahl et al. (2015) rate fits and their temperature derivatives
// (hydrogen_only/mod.rs:161-273) evaluated in FP32 in the fits' own units (erg cm^3/s,
// cm^3/s), at one temperature: the shared factors as in the FP64 forms below (one
// reciprocal of T, rsqrt for both square roots, exp / log1p for the powers).  The
// values carry ~1e-6 relative error; they enter the FP64 update as coefficients.
struct Fits32 {
  float fit, fitd;          // collision_fit and its derivative (161-173)
  float exc, dexc;          // collisional excitation cooling / 7.5e-19-scaled form, and d/dT (237-253)
  float recc, drecc;        // case B recombination cooling and d/dT (196-216)
  float brems, dbrems;      // bremsstrahlung cooling and d/dT (255-263)
  float alpha, dalpha;      // case B recombination rate and d/dT (175-194)
};

__device__ __forceinline__ Fits32 fits32(float t) {
  Fits32 f;
  const float inv_t = 1.0f / t;
  const float rsq = rsqrtf(t);
  const float sq = t * rsq;                      // sqrt(t)
  const float s5 = sq * 0.0031622777f;           // sqrt(t / 1e5)
  const float inv_s5 = rsq * 316.22776f;         // 1 / sqrt(t / 1e5)
  const float inv_1s5 = 1.0f / (1.0f + s5);
  // collision fit
  const float c1 = 1e-5f, c2 = 157809.1f;
  const float e = expf(-c2 * inv_t);
  f.fit = sq * inv_1s5 * e;
  f.fitd = (e * (c1 * c2 * t + 0.5f * s5 * (2.0f * c2 + t))) * (inv_t * rsq) * inv_s5 * (inv_1s5 * inv_1s5);
  // collisional excitation cooling
  const float c2e = 118348.0f;
  const float e_exc = expf(-c2e * inv_t);
  f.exc = 7.5e-19f * inv_1s5 * e_exc;
  f.dexc = (7.5e-19f * e_exc * (c2e * c1 * t - 0.5f * c1 * (t * t) + c2e * s5)) * (inv_t * inv_t) * inv_s5 *
           (inv_1s5 * inv_1s5);
  // case B recombination cooling: lambda^1.97 and (lambda / 2.25)^0.376 from one logarithm
  const float lambda = 315614.0f * inv_t;
  const float ln_lambda = logf(lambda);
  const float l197 = expf(1.97f * ln_lambda);
  const float q = expf(0.376f * (ln_lambda - 0.81093021f));  // ln 2.25
  const float inv_a = expf(-3.72f * log1pf(q));               // (1 + q)^-3.72
  f.recc = 3.435e-30f * t * l197 * inv_a;
  f.drecc = 3.435e-30f * ((inv_a / (1.0f + q)) * (1.0f - 1.97f + (1.0f - 1.97f + 0.376f * 3.72f) * q) * l197);
  // bremsstrahlung
  f.brems = 1.42e-27f * sq;
  f.dbrems = 1.42e-27f * 0.5f * rsq;
  // case B recombination rate: (lambda / 2.74)^0.407, (1 + p)^-2.242
  const float sl = 561.79534f * rsq;                          // sqrt(lambda)
  const float p = expf(0.407f * (ln_lambda - 1.0079579f));    // ln 2.74
  const float inv_b = expf(-2.242f * log1pf(p));
  f.alpha = 2.753e-14f * (lambda * sl) * inv_b;
  const float da = -sl * (inv_b / (p + 1.0f)) * (0.407f * 2.242f * p - 1.5f * p - 1.5f);
  f.dalpha = (2.753e-14f * da) * (-lambda * inv_t);  // d lambda / dT = -lambda / T
  return f;
}

// FP64: what the rate fits and their temperature derivatives (hydrogen_only/mod.rs:161-302) share
// at one temperature.
struct Fits64 {
  double t, sq, s5, lambda;  // temperature, sqrt(t), sqrt(t / 1e5), 315614 / t
  double fit, fitd;          // collision_fit 161-166 and its derivative 167-173
};

__device__ __forceinline__ Fits64 fits64(double t) {
  Fits64 f;
  f.t = t;
  f.sq = sqrt(t);
  f.s5 = sqrt(t / 1e5);
  f.lambda = 315614.0 / t;
  const double c1 = 1.0 / 1e5, c2 = 157809.1;
  const double e = exp(-c2 / t);
  f.fit = f.sq / (1.0 + f.s5) * e;
  f.fitd = (e * (c1 * c2 * t + 0.5 * f.s5 * (2.0 * c2 + t))) / ((t * f.sq) * f.s5 * ((f.s5 + 1.0) * (f.s5 + 1.0)));
  return f;
}

__device__ __forceinline__ void set_fits(Fits64& f, double t) { f = fits64(t); }
__device__ __forceinline__ void set_fits(Fits32& f, double t) { f = fits32((float)t); }

template <bool kCarryNeutral>
struct ChemFits {
  using Type = Fits64;
};
template <>
struct ChemFits<true> {
  using Type = Fits32;
};

template <bool kCarryNeutral>
struct ChemSolver {
  using Fits = typename ChemFits<kCarryNeutral>::Type;
  double x;   // ionized hydrogen fraction
  double y;   // neutral fraction (only meaningful when kCarryNeutral)
  double temperature;
  double density, volume, length, rate, scale_factor;
  bool has_floor;
  double floor_t, floor_x;
  bool clamp_invalid;
  // per-cell factors of the update (prepare())
  double nh, k_cell, compton_cell, xx_cell;
  double step_rate;  // photons of the whole timestep (FP64), rate per volume (mixed)
  // factors of the state that every attempt from it shares (begin()), and the fits at its
  // temperature
  double m, photo, heat_step, cool_step;
  Fits fits;
  double fits_t;  // temperature of `fits`

  __device__ void prepare(double timestep) {
    nh = density / Units::kProtonMass;
    k_cell = (Units::kGamma - 1.0) * Units::kProtonMass / (density * Units::kBoltzmann);
    step_rate = kCarryNeutral ? rate / volume : timestep * rate;
    xx_cell = 2.727 / scale_factor;
    const double x2 = xx_cell * xx_cell;
    compton_cell = 1.017e-37 * (x2 * x2);
    if (kCarryNeutral) compton_cell *= Units::kErgsPerS;
    fits_t = -1.0;  // of no cell
  }

  __device__ __forceinline__ double neutral() const { return kCarryNeutral ? y : (1.0 - x); }
  __device__ __forceinline__ double n_ionized() const { return nh * x; }
  __device__ __forceinline__ double n_neutral() const { return nh * neutral(); }

  // cooling_rate 275-287 and cooling_rate_derivative 289-302 at the current state:
  // collisional ionization / excitation cooling (237-253), case B recombination cooling
  // (196-216), bremsstrahlung and Compton cooling (265-273).  Mixed path: from the FP32 fits;
  // the densities, the sums and the unit factors in FP64.
  // (every term in the order in which it has always been rounded)
  __device__ void cooling(const Fits32& f, double& lambda_c, double& dlambda_c) const {
    const double t = temperature;
    const double ne = n_ionized();
    const double nhn = n_neutral();
    const double nhi = n_ionized();
    const double u = Units::kErgsCentimetersCubedPerS;
    const double compton = compton_cell * (t - xx_cell);
    const double dcompton = compton_cell;
    const double coll = ((double)f.exc + 1.27e-21 * (double)f.fit) * u * ne * nhn;
    const double dcoll = ((double)f.dexc + 1.27e-21 * (double)f.fitd) * u * ne * nhn;
    lambda_c = coll + ((double)f.recc + (double)f.brems) * u * ne * nhi + compton * ne;
    dlambda_c = dcoll + ((double)f.drecc + (double)f.dbrems) * u * ne * nhi + dcompton * ne;
  }
  // FP64: each derivative is the reference's formula with the powers taken from the fit; the
  // values agree with separate evaluation to rounding.
  __device__ void cooling(const Fits64& f, double& lambda_c, double& dlambda_c) const {
    const double t = f.t;
    const double ne = n_ionized();
    const double nhn = n_neutral();
    const double nhi = n_ionized();
    constexpr double u = Units::kErgsCentimetersCubedPerS;
    // excitation cooling and its derivative
    const double c3 = 1.0 / 1e5, c2e = 118348.0;
    const double e_exc = exp(-c2e / t);
    const double exc = (7.5e-19 / (1.0 + f.s5) * e_exc) * u;
    const double dexc = ((7.5e-19 * e_exc * (c2e * c3 * t - 0.5 * c3 * (t * t) + c2e * f.s5)) /
                         ((t * t) * f.s5 * ((1.0 + f.s5) * (1.0 + f.s5)))) * u;
    // case B recombination cooling and its derivative: lambda^1.97 and (lambda / 2.25)^0.376 from
    // one logarithm
    const double c2r = 1.97, c3r = 0.376, c4r = 3.72;
    const double ln_lambda = log(f.lambda);
    const double l197 = exp(c2r * ln_lambda);
    const double q = exp(c3r * (ln_lambda - 0.81093021621632877));  // ln 2.25
    const double a = pow(1.0 + q, c4r);
    const double recomb_rate = (3.435e-30 * t * l197 / a) * u;
    const double drecomb_rate =
        (3.435e-30 * ((1.0 / (a * (1.0 + q))) * (1.0 - c2r + (1.0 - c2r + c3r * c4r) * q) * l197)) * u;
    const double compton = (compton_cell * (temperature - xx_cell)) * Units::kErgsPerS;
    const double dcompton = compton_cell * Units::kErgsPerS;
    const double coll = (exc + (1.27e-21 * f.fit) * u) * ne * nhn;
    const double recomb = recomb_rate * ne * nhi;
    const double brems = ((1.42e-27 * f.sq) * u) * ne * nhi;
    lambda_c = coll + recomb + brems + compton * ne;
    const double dcoll = (dexc + (1.27e-21 * f.fitd) * u) * ne * nhn;
    const double drecomb = drecomb_rate * ne * nhi;
    const double dbrems = ((1.42e-27 / (2.0 * f.sq)) * u) * ne * nhi;
    dlambda_c = dcoll + drecomb + dbrems + dcompton * ne;
  }

  // case B recombination rate and its derivative, 175-194
  __device__ static void recombination(const Fits32& f, double& alpha, double& dalpha) {
    alpha = (double)f.alpha * Units::kCentimetersCubedPerS;
    dalpha = (double)f.dalpha * Units::kCentimetersCubedPerS;
  }
  __device__ static void recombination(const Fits64& f, double& alpha, double& dalpha) {
    const double c2a = 0.407, c3a = 2.242;
    const double dlambda_dt = -315614.0 / (f.t * f.t);
    const double sl = sqrt(f.lambda);
    const double p = pow(f.lambda / 2.74, c2a);
    const double b = pow(1.0 + p, c3a);
    alpha = (2.753e-14 * (f.lambda * sl) / b) * Units::kCentimetersCubedPerS;
    const double da = -sl * (1.0 / (b * (p + 1.0))) * (c2a * c3a * p - 1.5 * p - 1.5);
    dalpha = ((2.753e-14 * da) * Units::kCentimetersCubedPerS) * dlambda_dt;
  }

  // 312-319: photons absorbed per photon arriving, 1 - exp(-n_HI sigma size); both
  // updates of an attempt use it with the x of the attempt's start.  Mixed path:
  // -expm1 in FP32, accurate to ~1e-7 relative also for optically thin cells.
  __device__ double absorbed_fraction() const {
    if (kCarryNeutral) return -(double)expm1f((float)(-n_neutral() * Units::kSigma * length));
    return 1.0 - exp(-n_neutral() * Units::kSigma * length);
  }

  // What the attempts from the current state share.  The reference forms the photon terms with
  // the attempt's step and divides by it: a power of two times the whole timestep, so the whole
  // one gives the same numbers.
  __device__ void begin(double timestep) {
    const double absorbed = absorbed_fraction();
    m = 1.0 / (x + 1.0);  // mu
    double lc, dlc, heating;
    if (kCarryNeutral) {  // (FP32: evaluated apart for either use, so that both keep their roundings)
      Fits f;
      set_fits(f, temperature);
      cooling(f, lc, dlc);
    } else {
      if (!(fits_t == temperature)) {
        set_fits(fits, temperature);
        fits_t = temperature;
      }
      cooling(fits, lc, dlc);
    }
    constexpr double kEnergy = Units::kPhotonAverageEnergy - Units::kRydberg;
    if (kCarryNeutral) {  // photoheating_rate 321-325, photoionization_rate 327-332
      heating = (step_rate * absorbed) * kEnergy;
      photo = (step_rate * absorbed) / n_neutral();
    } else {
      heating = ((step_rate * absorbed) / volume) * kEnergy / timestep;
      photo = ((step_rate * absorbed) / (n_neutral() * volume)) / timestep;
    }
    const double lambda = heating - lc;
    const double dlambdadt = -dlc;
    heat_step = k_cell * m * lambda;
    cool_step = k_cell * m * dlambdadt;
  }

  // 334-354, case B rate at the temperature t of `f` that the attempt has reached
  __device__ double ionized_fraction_change(double timestep, const Fits& f, double t) const {
    const double ne = n_ionized();
    double alpha, dalpha;
    recombination(f, alpha, dalpha);
    const double n_h = nh;
    double beta = (5.85e-11 * (double)f.fit) * Units::kCentimetersCubedPerS;
    double dbeta = (5.85e-11 * (double)f.fitd) * Units::kCentimetersCubedPerS;
    double c = beta * ne + photo;
    double d = alpha * ne;
    double xhii = x;
    double rhsc = ne * t * m * 1.0 * dbeta;
    double dcdx = n_h * beta - rhsc;
    double rhsd = ne * t * m * 1.0 * dalpha;
    double dddx = n_h * alpha - rhsd;
    double j = dcdx - (c + d) - xhii * (dcdx + dddx);
    return timestep * (c - xhii * (c + d)) / (1.0 - j * timestep);
  }

  // 356-369 with Rust f64::clamp semantics (asserts min <= max: flagged here).
  __device__ void clamp() {
    double xf = has_floor ? floor_x : kIonizedFractionEpsilon;
    const double xmax = 1.0 - kIonizedFractionEpsilon;
    if (!(xf <= xmax)) clamp_invalid = true;
    if (kCarryNeutral) {
      if (x < xf) { x = xf; y = 1.0 - x; }
      if (x > xmax) { x = xmax; y = kIonizedFractionEpsilon; }
    } else {
      if (x < xf) x = xf;
      if (x > xmax) x = xmax;
    }
    if (has_floor && temperature < floor_t) temperature = floor_t;
  }

  // relative change of update() 444-461, and whether it is small enough.  Away from equality the
  // product decides as the quotient does (2^-50 covers the roundings of both); at it, and where
  // the product leaves the normal range or the cap of the relative change plays a part, the
  // quotient itself.
  __device__ __forceinline__ static double relative(double value, double change) {
    return fmin(fabs(change / value), 1.0 / DBL_EPSILON);
  }
  __device__ __forceinline__ static bool small(double value, double change, double safety) {
    constexpr double kNear = 8.8817841970012523e-16;  // 2^-50
    const double c = fabs(change), most = safety * fabs(value);
    if (most > 1e-290 && safety < 1.0 / DBL_EPSILON) {
      if (c < most * (1.0 - kNear)) return true;
      if (c > most * (1.0 + kNear)) return false;
    }
    return !(relative(value, change) > safety);
  }

  // perform_timestep 426-441 with perform_timestep_internal 394-424 unrolled, and the attempts
  // (try_timestep_update 371-392, temperature_change 304-310): the state changes when both changes
  // of an attempt are small enough.  The temperature's test takes a few operations, so a lane
  // repeats it until it holds before the warp goes on to the fits at the new temperature.
  __device__ Timescale perform_timestep(double timestep, double safety, bool& failed,
                                        uint32_t& attempts) {
    uint64_t pend_lo = 0, pend_hi = 0;  // pending second halves at depths 1..127
    int depth = 0;
    clamp();
    bool moved = true;  // (one place for begin(): the same roundings for every state)
    while (true) {
      if (moved) begin(timestep);
      moved = false;
      double sub, tc;
      while (true) {
        if (depth > kChemMaxDepth) {
          failed = true;
          return Timescale{timestep / 10.0, kProcTemperature};
        }
        // timestep / 2^depth, exact
        sub = timestep * __longlong_as_double((long long)(1023 - depth) << 52);
        ++attempts;
        tc = heat_step * sub / (1.0 - cool_step * sub);
        if (small(temperature, tc, safety)) break;
        reject(depth, pend_lo, pend_hi);
      }
      const double t = temperature + tc;
      Fits f;
      set_fits(f, t);
      const double xc = ionized_fraction_change(sub, f, t);
      if (!small(x, xc, safety)) {
        reject(depth, pend_lo, pend_hi);
        continue;
      }
      const double t0 = temperature, x0 = x;
      temperature = t;
      if (!kCarryNeutral) {
        fits = f;
        fits_t = t;
      }
      x += xc;
      if (kCarryNeutral) {
        y -= xc;
        // keep the smaller fraction exact and derive the other from it
        if (x < 0.5) y = 1.0 - x; else x = 1.0 - y;
      }
      clamp();
      if (pend_hi) {
        depth = 127 - __clzll((long long)pend_hi);
        pend_hi &= ~(1ull << (depth - 64));
      } else if (pend_lo) {
        depth = 63 - __clzll((long long)pend_lo);
        pend_lo &= ~(1ull << depth);
      } else {
        failed = false;
        return ts_min(Timescale{sub * (safety / relative(t0, tc)), kProcTemperature},
                      Timescale{sub * (safety / relative(x0, xc)), kProcIonization});
      }
      moved = true;
    }
  }

  // halves the step: its second half is pending
  __device__ __forceinline__ static void reject(int& depth, uint64_t& pend_lo, uint64_t& pend_hi) {
    ++depth;
    if (depth < 64) pend_lo |= (1ull << depth); else pend_hi |= (1ull << (depth - 64));
  }
};

}  // namespace swk
