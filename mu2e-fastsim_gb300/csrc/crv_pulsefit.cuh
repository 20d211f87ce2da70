// Pulse reconstruction: reco waveforms -> pulses (crv/crvfastsim/reco/pulsefit.py:49-316).
//
// Per waveform: pedestal (DB value, or the first sample when it undershoots the DB value by more than the
// threshold); then rounds: FindNextPeak from `start` (rising edge, optional plateau, falling edge with the plateau
// value above min_adc_difference), a fit window of up to samples_before / samples_after monotonic samples (one dropped
// on each side when more than one was added), a bounded Gumbel least-squares fit in sine-mapped internal coordinates
// (40 Levenberg-Marquardt steps, then 8 Gauss-Newton steps with halving, EDM and Hessian checks), the failed-fit
// fallback, then the rounded fit is subtracted from every sample and the search resumes at the window end.
//
// GPU mapping: one lane per fit, its samples in a global scratch mirror; a lane keeps its waveform until its last pulse
// (k_pf_persist) or for one pulse per launch (k_pf_round).  What is the lane's own: the fit's state, the sums (sequential
// over the window, as the reference's contractions), the 3x3 solve, the Hessian check, the pulse records (per-waveform
// slots; a waveform has at most half as many pulses as samples).  What the warp does together in k_pf_persist: copies and
// long searches of samples, and the FP64 evaluations (pf_eval_warp).  R = double: every step in FP64, the solve by LU with
// partial pivoting.  R = float (mixed): parameter mapping, residuals, Jacobians, sums and the fit state in FP32 relative to
// the window's first sample; the normal-equation solve in float-float arithmetic on the FP32 pipe (FP64 for values outside
// FP32's comfortable range); absolute pulse times in FP64.
#pragma once
#include "crv_device.cuh"

namespace crv {

struct PulseRec {            // one reconstructed pulse (shared-memory staging)
  double pe, peph, time, height, beta, chi2, letime, ped, A, mu, b;
  int32_t seq;
  uint8_t failed, zerondf, pedfromdb, pad;
};

struct WaveIn {
  long long nw;              // waveforms (an upper bound when nw_dev is set)
  const long long* nw_dev;   // device count of waveforms, or null
  const long long* off;      // first sample of waveform w in the sample array
  const int32_t* n;          // valid samples
  const long long* start_tdc;
  const double* ped_db;
  const double* area;
  const double* height;
  const int16_t* adc16;      // samples (one of adc16 / adc64)
  const long long* adc64;
  long long nsamples;        // rows of the sample array: every waveform must lie inside it
};

__device__ __forceinline__ double round_half_away(double x) {
  double a = floor(fabs(x) + 0.5);
  return x < 0.0 ? -a : (x > 0.0 ? a : 0.0 * x);
}

// |x| as an integer in the order of |x|
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}
// a / b from y = 1 / b rounded (quotient); operands outside 2^-500 .. 2^500 (quotient and remainder could leave the normal
// range; zero) take the division
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const int ea = int((abs_bits(a) >> 52)), eb = int((abs_bits(b) >> 52));
  if (unsigned(eb - 523) > 1000u || unsigned(ea - 523) > 1000u) return a / b;
  return quotient(a, b, y);
}

// whether |x| > |y| (false with a NaN, as the floating-point compare)
__device__ __forceinline__ bool abs_greater(double x, double y) {
  return abs_bits(x) > abs_bits(y) && abs_bits(x) <= 0x7FF0000000000000ull;
}

// LU with partial pivoting (largest |a| in the column, first on ties), then substitution.  Returns false on a zero
// pivot (singular).  The pivots' reciprocals serve the substitution's divisions too, and the comparisons are integer
// ones: of the solve's FP64 instructions a third.
static __device__ __noinline__ bool solve3(const double M[3][3], const double r[3], double x[3]) {
  double a[3][3], b[3], inv[3];
  for (int i = 0; i < 3; ++i) {
    b[i] = r[i];
    for (int j = 0; j < 3; ++j) a[i][j] = M[i][j];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    int piv = k;
    double mx = a[k][k];
#pragma unroll
    for (int i = k + 1; i < 3; ++i)
      if (abs_greater(a[i][k], mx)) { mx = a[i][k]; piv = i; }
    if (abs_bits(mx) == 0ull) return false;
#pragma unroll
    for (int i = k + 1; i < 3; ++i)
      if (piv == i) {
        for (int j = 0; j < 3; ++j) { double tmp = a[k][j]; a[k][j] = a[i][j]; a[i][j] = tmp; }
        double tb = b[k]; b[k] = b[i]; b[i] = tb;
      }
    inv[k] = 1.0 / a[k][k];
#pragma unroll
    for (int i = k + 1; i < 3; ++i) {
      double l = a[i][k] * inv[k];
      a[i][k] = l;
      for (int j = k + 1; j < 3; ++j) a[i][j] -= l * a[k][j];
      b[i] -= l * b[k];
    }
  }
#pragma unroll
  for (int i = 2; i >= 0; --i) {
    double s = b[i];
#pragma unroll
    for (int j = i + 1; j < 3; ++j) s -= a[i][j] * x[j];
    x[i] = div_by(s, a[i][i], inv[i]);
  }
  return true;
}

// eigenvalues of a symmetric 3x3 matrix (cyclic Jacobi), ascending
static __device__ __noinline__ void eig3(const double M[3][3], double e[3]) {
  double a[3][3];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) a[i][j] = M[i][j];
  for (int sweep = 0; sweep < 50; ++sweep) {
    double off = fabs(a[0][1]) + fabs(a[0][2]) + fabs(a[1][2]);
    double dg = fabs(a[0][0]) + fabs(a[1][1]) + fabs(a[2][2]);
    if (off == 0.0 || off <= 1e-300 || off < 1e-18 * dg) break;
    for (int p = 0; p < 2; ++p)
      for (int q = p + 1; q < 3; ++q) {
        double apq = a[p][q];
        if (apq == 0.0) continue;
        double th = (a[q][q] - a[p][p]) / (2.0 * apq);
        double t = (th >= 0.0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
        double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < 3; ++k) {        // A <- J^T A J
          double akp = a[k][p], akq = a[k][q];
          a[k][p] = c * akp - s * akq;
          a[k][q] = s * akp + c * akq;
        }
        for (int k = 0; k < 3; ++k) {
          double apk = a[p][k], aqk = a[q][k];
          a[p][k] = c * apk - s * aqk;
          a[q][k] = s * apk + c * aqk;
        }
      }
  }
  e[0] = a[0][0]; e[1] = a[1][1]; e[2] = a[2][2];
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2 - i; ++j)
      if (e[j] > e[j + 1]) { double tmp = e[j]; e[j] = e[j + 1]; e[j + 1] = tmp; }
}

constexpr int FIT_KEEP = 16;   // window points whose time the fit, and whose exponentials an evaluation, keeps

// FP64 evaluation of one lane at internal parameters u over the window points yw[0..P), times (tdc_fs + i) * period (the first FIT_KEEP of them in tw):
// chi2, and when it is below `bound` (or always: `first`) the normal equations too (a rejected step does not need them).
// Returns whether it is below.  Sums are sequential over the points (the reference's contractions are sequential); every operation rounds as
// written (no contraction).
static __device__ __noinline__ bool eval_f64(const double lo[3], const double w[3], const double u[3], const double* yw,
                                             const double* tw, long long tdc_fs, double period, int P, bool first, double bound, double* chi2, double H[6],
                                             double g[3]) {
  double s0, c0, s1, c1, s2, c2;
  sincos(u[0], &s0, &c0);
  sincos(u[1], &s1, &c1);
  sincos(u[2], &s2, &c2);
  const double A = lo[0] + w[0] * (s0 + 1.0) * 0.5;
  const double mu = lo[1] + w[1] * (s1 + 1.0) * 0.5;
  const double b = lo[2] + w[2] * (s2 + 1.0) * 0.5;
  const double y = 1.0 / b;
  double ez_[FIT_KEEP], gg_[FIT_KEEP], z_[FIT_KEEP];
  double c = 0.0;
#pragma unroll 1
  for (int i = 0; i < P; ++i) {
    const double t = i < FIT_KEEP ? tw[i] : double(tdc_fs + i) * period;
    const double z = div_by(t - mu, b, y);
    const double ez = exp(-z);
    const double gg = exp(-z - ez);
    if (i < FIT_KEEP) { z_[i] = z; ez_[i] = ez; gg_[i] = gg; }
    const double r = yw[i] - A * gg;
    c += r * r;
  }
  *chi2 = c;
  const bool below = c < bound;
  if (!below && !first) return false;
  const double d0 = w[0] * 0.5 * c0, d1 = w[1] * 0.5 * c1, d2 = w[2] * 0.5 * c2;
  const double nb = -1.0 / b;
  double h00 = 0, h01 = 0, h02 = 0, h11 = 0, h12 = 0, h22 = 0, g0 = 0, g1 = 0, g2 = 0;
#pragma unroll 1
  for (int i = 0; i < P; ++i) {
    double z, ez, gg;
    if (i < FIT_KEEP) {
      z = z_[i]; ez = ez_[i]; gg = gg_[i];
    } else {
      const double t = double(tdc_fs + i) * period;
      z = div_by(t - mu, b, y);
      ez = exp(-z);
      gg = exp(-z - ez);
    }
    const double f = A * gg;
    const double r = yw[i] - f;
    const double fz = f * (ez - 1.0);
    const double j0 = gg * d0;
    const double j1 = fz * nb * d1;
    const double j2 = fz * div_by(-z, b, y) * d2;
    h00 += j0 * j0; h01 += j0 * j1; h02 += j0 * j2;
    h11 += j1 * j1; h12 += j1 * j2; h22 += j2 * j2;
    g0 += j0 * r; g1 += j1 * r; g2 += j2 * r;
  }
  H[0] = h00; H[1] = h01; H[2] = h02; H[3] = h11; H[4] = h12; H[5] = h22;
  g[0] = g0; g[1] = g1; g[2] = g2;
  return below;
}

__device__ __forceinline__ void sym3(const double H[6], double M[3][3]) {
  M[0][0] = H[0]; M[0][1] = M[1][0] = H[1]; M[0][2] = M[2][0] = H[2];
  M[1][1] = H[3]; M[1][2] = M[2][1] = H[4]; M[2][2] = H[5];
}

// Whether the smallest eigenvalue of H exceeds 1e-12 of the largest.  A matrix far inside (positive leading minors and
// 4 det / trace^2, a lower bound of the smallest eigenvalue, above 1e-9 of the trace, where the minors' rounding of a
// few 1e-16 of trace^3 does not matter) is told without the eigenvalues.
static __device__ __noinline__ bool hessian_ok64(const double H[6]) {
  const double tr = H[0] + H[3] + H[5];
  const double m2 = H[0] * H[3] - H[1] * H[1];
  const double det = H[0] * (H[3] * H[5] - H[4] * H[4]) - H[1] * (H[1] * H[5] - H[4] * H[2]) +
                     H[2] * (H[1] * H[4] - H[3] * H[2]);
  if (tr > 1e-90 && tr < 1e90 && H[0] > 0.0 && m2 > 1e-9 * tr * tr && 4.0 * det > 1e-9 * tr * tr * tr) return true;
  double M[3][3], e[3];
  sym3(H, M);
  eig3(M, e);
  return e[0] > 1e-12 * fmax(e[2], 1e-300);
}

// the same bits (integer compares; equal values of other bits, a signed zero, only cost an evaluation)
__device__ __forceinline__ bool same3(const double a[3], const double b[3]) {
  return __double_as_longlong(a[0]) == __double_as_longlong(b[0]) &&
         __double_as_longlong(a[1]) == __double_as_longlong(b[1]) &&
         __double_as_longlong(a[2]) == __double_as_longlong(b[2]);
}

// near-threshold local maximum among positions [a, b]
template <typename Y>
__device__ __forceinline__ bool near_lane(const Y* y, int n, int a, int b, Y thr, Y edge) {
  if (a < 0) a = 0;
  if (b > n - 1) b = n - 1;
  for (int i = a; i <= b; ++i) {
    Y left = i > 0 ? y[i - 1] : Y(-1e9);
    Y right = i + 1 < n ? y[i + 1] : Y(-1e9);
    Y d = y[i] - thr;
    if (y[i] >= left && y[i] > right && (d < Y(0) ? -d : d) <= edge) return true;
  }
  return false;
}

// FindNextPeak of one lane over positions [b, end): whether a peak was found (first and last position of its plateau), or
// the state at `end` (rising, and since where)
struct PeakScan {
  int b, ps;
  bool rising, found;
};
template <typename Y>
__device__ __forceinline__ void peak_scan(const Y* y, int end, Y thr, PeakScan& s) {
  for (; s.b < end; ++s.b) {
    const Y prev = y[s.b - 1], cur = y[s.b];
    if (prev < cur) { s.rising = true; s.ps = s.b; }
    else if (prev == cur) {}
    else if (s.rising) {                          // (the plateau's last position is the one before)
      if (prev > thr) { s.found = true; break; }
      s.rising = false;
    }
  }
}

// the same by the warp, 32 positions at a time, from the state b, ps, rising (uniform)
template <typename Y>
__device__ __forceinline__ PeakScan peak_scan_warp(const Y* y, int n, Y thr, int b, int ps, bool rising) {
  const int lane = lane_id();
  const unsigned lt = (1u << lane) - 1u;
  for (; b < n; b += 32) {
    const int i = b + lane;
    const Y prev = i < n ? y[i - 1] : Y(0), cur = i < n ? y[i] : Y(0);
    const bool up = prev < cur, down = !up && prev != cur;
    const unsigned U = __ballot_sync(0xffffffffu, up), D = __ballot_sync(0xffffffffu, down);
    const unsigned before = (U | D) & lt;         // steps that are not level before this one: the last says whether it rises
    const int last = 31 - __clz(before);
    const bool r = before ? (U >> last) & 1u : rising;
    const int from = before ? b + last : ps;
    const unsigned C = __ballot_sync(0xffffffffu, down && r && prev > thr);
    if (C) {
      const int l = __ffs(C) - 1;
      return PeakScan{b + l, __shfl_sync(0xffffffffu, from, l), true, true};
    }
    if (U | D) {
      const int l = 31 - __clz(U | D);
      rising = (U >> l) & 1u;
      ps = b + l;
    }
  }
  return PeakScan{n, ps, rising, false};
}

// fit window around the plateau [ps, pe]
template <typename Y>
__device__ __forceinline__ void peak_window(const CrvParams& p, const Y* y, int n, int ps, int pe, int* fs_o, int* fe_o) {
  int fs = ps - 1, fe = pe + 1;
  for (int k = 1; k <= p.samples_before; ++k) {
    int i = ps - k;
    if (i < 0 || !(y[i] <= y[i + 1])) break;
    fs = i;
    if (i == 0) break;
  }
  for (int k = 1; k <= p.samples_after; ++k) {
    int i = pe + k;
    if (i >= n || !(y[i - 1] >= y[i])) break;
    fe = i;
  }
  if (ps - fs > 1) fs += 1;
  if (fe - pe > 1) fe -= 1;
  *fs_o = fs; *fe_o = fe;
}

struct PulseSlots {
  const long long* off;      // per waveform: first record slot
  const int32_t* cap;        // per waveform: slots (rounds bound)
  int32_t* count;            // per waveform: pulses
  uint8_t* near;             // per waveform: wf_near_threshold
  PulseRec* rec;
  long long rc;              // record slots of the workspace: every waveform's slots must lie inside it
};

// A waveform's samples [off, off + n) lie in the sample array and its record slots in the workspace.  Waveforms that
// break this (inconsistent offsets or lengths from the caller) are not read; the status reports CRV_ST_BOUNDS.
__device__ __forceinline__ bool wave_in_bounds(long long off, int n, long long nsamples) {
  return off >= 0 && n >= 0 && off <= nsamples && (long long)n <= nsamples - off;
}

__device__ __forceinline__ float round_half_away_f(float x) {
  float a = floorf(fabsf(x) + 0.5f);
  return x < 0.0f ? -a : (x > 0.0f ? a : 0.0f * x);
}

// subtract round(fit) from the samples it reaches: walk out from the mode while the rounded value can be non-zero
__device__ __forceinline__ void subtract_lane(const CrvParams& p, double* y, int n, long long st_tdc, double A,
                                              double mu, double b, int* lo_o, int* hi_o) {
  long long im = (long long)floor(mu / p.period) - st_tdc;
  if (im < 0) im = 0;
  if (im > n - 1) im = n - 1;
  int lo = int(im), hi = int(im);
  for (int dir = -1; dir <= 1; dir += 2) {
    for (int i = int(im) + (dir > 0 ? 1 : 0); i >= 0 && i < n; i += dir) {
      double t = double(st_tdc + i) * p.period;
      double z = (t - mu) / b;
      double gv = A * exp(-z - exp(-z));
      y[i] -= round_half_away(gv);
      if (dir < 0) lo = i; else hi = i;
      // unimodal: past the mode the value only shrinks; stop well below the rounding threshold
      if (fabs(gv) < 0.25 && ((dir < 0 && t < mu) || (dir > 0 && t > mu))) break;
    }
  }
  *lo_o = lo;
  *hi_o = hi;
}

// ---- FP32-mixed fit: evaluation, mapping and state in FP32, the normal-equation solve in float-float ----------------
//
// residuals / normal equations at internal parameters u; window sample i at time i * period
__device__ __forceinline__ void eval_f32(const float lo[3], const float w[3], const float u[3], const float* yw,
                                         float period, int P, float* chi2, float H[6], float g[3]) {
  float s0, c0, s1, c1, s2, c2;
  sincosf(u[0], &s0, &c0);
  sincosf(u[1], &s1, &c1);
  sincosf(u[2], &s2, &c2);
  const float A = lo[0] + w[0] * (s0 + 1.0f) * 0.5f;
  const float mu = lo[1] + w[1] * (s1 + 1.0f) * 0.5f;
  const float b = lo[2] + w[2] * (s2 + 1.0f) * 0.5f;
  const float d0 = w[0] * 0.5f * c0, d1 = w[1] * 0.5f * c1, d2 = w[2] * 0.5f * c2;
  const float ib = 1.0f / b;
  float c = 0, h00 = 0, h01 = 0, h02 = 0, h11 = 0, h12 = 0, h22 = 0, g0 = 0, g1 = 0, g2 = 0;
  for (int i = 0; i < P; ++i) {
    const float z = (float(i) * period - mu) * ib;
    // e^-z overflows FP32 beyond 88; at 80 the Gumbel factor e^(-z - e^-z) is already exactly 0
    const float mz = fminf(-z, 80.0f);
    const float ez = __expf(mz);
    const float gg = __expf(mz - ez);
    const float f = A * gg;
    const float r = yw[i] - f;
    const float fz = f * (ez - 1.0f);
    const float j0 = gg * d0;
    const float j1 = -fz * ib * d1;
    const float j2 = -fz * z * ib * d2;
    c += r * r;
    h00 += j0 * j0; h01 += j0 * j1; h02 += j0 * j2;
    h11 += j1 * j1; h12 += j1 * j2; h22 += j2 * j2;
    g0 += j0 * r; g1 += j1 * r; g2 += j2 * r;
  }
  *chi2 = c;
  H[0] = h00; H[1] = h01; H[2] = h02; H[3] = h11; H[4] = h12; H[5] = h22;
  g[0] = g0; g[1] = g1; g[2] = g2;
}

// symmetric 3x3 solve M x = b (M packed 00 01 02 11 12 22): cofactors, determinant and adjugate product in FP64
// (products of FP32 inputs are exact there), the final division by the determinant in FP32.  The fit calls it only
// for values outside FP32's comfortable range (solve_sym_ff below does the rest).
static __device__ __noinline__ bool solve_sym64(const float M[6], const float b[3], float x[3]) {
  const double m00 = f2d(M[0]), m01 = f2d(M[1]), m02 = f2d(M[2]), m11 = f2d(M[3]), m12 = f2d(M[4]), m22 = f2d(M[5]);
  const double c00 = m11 * m22 - m12 * m12;
  const double c01 = m12 * m02 - m01 * m22;
  const double c02 = m01 * m12 - m11 * m02;
  const double det = m00 * c00 + m01 * c01 + m02 * c02;
  if (!finite_nonzero(det)) return false;
  const double c11 = m00 * m22 - m02 * m02;
  const double c12 = m01 * m02 - m00 * m12;
  const double c22 = m00 * m11 - m01 * m01;
  const double b0 = f2d(b[0]), b1 = f2d(b[1]), b2 = f2d(b[2]);
  const double y0 = c00 * b0 + c01 * b1 + c02 * b2;
  const double y1 = c01 * b0 + c11 * b1 + c12 * b2;
  const double y2 = c02 * b0 + c12 * b1 + c22 * b2;
  const float df = d2f_trunc(det);
  const float r = 1.0f / df;
  if (!(fabsf(r) < 1e30f) || !(fabsf(r) > 1e-30f)) {       // determinant outside the comfortable FP32 range
    const double rd = 1.0 / det;
    x[0] = float(y0 * rd); x[1] = float(y1 * rd); x[2] = float(y2 * rd);
    return true;
  }
  x[0] = d2f_trunc(y0) * r; x[1] = d2f_trunc(y1) * r; x[2] = d2f_trunc(y2) * r;
  return true;
}

// The same solve in float-float arithmetic on the FP32 pipe: every product of two FP32 values split exactly into a
// rounded product and its error (fmaf), sums of such pairs with their rounding errors carried (Dekker's and Knuth's
// error-free transformations), so the cofactors, the determinant and the adjugate product keep ~46 significant bits,
// reduced to the FP32 result's 24 by the final truncation, as the FP64 solve's 53 are.  Values outside FP32's
// comfortable range (or a non-finite or zero determinant) go to the FP64 solve.  Measured on the 9,358,230 pulses of
// 65,536 workload events against the FP64 solve: the same pulses, flags and clusters; the sum of pulse PE moves by
// 3e-14 relative; the fit takes 48 % less time (it was bound by the FP64 pipe: ~24 FP64 operations per solve, at
// 1/64 of the FP32 rate, against ~350 FP32 operations for a whole window evaluation).
struct FF {
  float hi, lo;
};
__device__ __forceinline__ FF ff_two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return FF{p, fmaf(a, b, -p)};
}
__device__ __forceinline__ FF ff_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return FF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ FF ff_norm(float a, float b) {       // |a| >= |b| or a == 0
  const float s = __fadd_rn(a, b);
  return FF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF ff_mul2m(float a, float b, float c, float d) {   // a*b - c*d
  const FF p = ff_two_prod(a, b), q = ff_two_prod(c, d);
  const FF s = ff_two_sum(p.hi, -q.hi);
  return ff_norm(s.hi, __fadd_rn(s.lo, __fsub_rn(p.lo, q.lo)));
}
__device__ __forceinline__ FF ff_mul(float x, FF y) {
  const FF p = ff_two_prod(x, y.hi);
  return ff_norm(p.hi, fmaf(x, y.lo, p.lo));
}
__device__ __forceinline__ FF ff_add(FF a, FF b) {
  const FF s = ff_two_sum(a.hi, b.hi);
  return ff_norm(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ bool ff_safe(float x) { return fabsf(x) < 1e36f; }   // finite, headroom for the sums

static __device__ __noinline__ bool solve_sym_ff(const float M[6], const float b[3], float x[3]) {
  const float m00 = M[0], m01 = M[1], m02 = M[2], m11 = M[3], m12 = M[4], m22 = M[5];
  const FF c00 = ff_mul2m(m11, m22, m12, m12);
  const FF c01 = ff_mul2m(m12, m02, m01, m22);
  const FF c02 = ff_mul2m(m01, m12, m11, m02);
  const FF det = ff_add(ff_add(ff_mul(m00, c00), ff_mul(m01, c01)), ff_mul(m02, c02));
  const FF c11 = ff_mul2m(m00, m22, m02, m02);
  const FF c12 = ff_mul2m(m01, m02, m00, m12);
  const FF c22 = ff_mul2m(m00, m11, m01, m01);
  const FF y0 = ff_add(ff_add(ff_mul(b[0], c00), ff_mul(b[1], c01)), ff_mul(b[2], c02));
  const FF y1 = ff_add(ff_add(ff_mul(b[0], c01), ff_mul(b[1], c11)), ff_mul(b[2], c12));
  const FF y2 = ff_add(ff_add(ff_mul(b[0], c02), ff_mul(b[1], c12)), ff_mul(b[2], c22));
  const float df = __fadd_rz(det.hi, det.lo);
  const float r = 1.0f / df;
  if (!(ff_safe(c00.hi) && ff_safe(c01.hi) && ff_safe(c02.hi) && ff_safe(c11.hi) && ff_safe(c12.hi) &&
        ff_safe(c22.hi) && ff_safe(det.hi) && ff_safe(y0.hi) && ff_safe(y1.hi) && ff_safe(y2.hi)) ||
      !(fabsf(df) > 1e-30f) || !(fabsf(r) < 1e30f) || !(fabsf(r) > 1e-30f))
    return solve_sym64(M, b, x);
  x[0] = __fadd_rz(y0.hi, y0.lo) * r;
  x[1] = __fadd_rz(y1.hi, y1.lo) * r;
  x[2] = __fadd_rz(y2.hi, y2.lo) * r;
  return true;
}

// Hessian check of the FP32-mixed fit: the smallest eigenvalue above 1e-12 of the matrix's scale, as H - tau I
// positive definite (Sylvester: every leading principal minor positive), tau = 1e-12 max(trace, 1e-300); the trace
// stands in for the largest eigenvalue (within a factor 3 of it for a positive semi-definite H).
__device__ __forceinline__ bool hessian_ok(const float H[6]) {
  const double h00 = f2d(H[0]), h01 = f2d(H[1]), h02 = f2d(H[2]), h11 = f2d(H[3]), h12 = f2d(H[4]), h22 = f2d(H[5]);
  const double tr = h00 + h11 + h22;
  const double tau = 1e-12 * (tr > 1e-300 ? tr : 1e-300);
  const double a = h00 - tau, d = h11 - tau, f = h22 - tau;
  const double m2 = a * d - h01 * h01;
  const double m3 = a * (d * f - h12 * h12) - h01 * (h01 * f - h12 * h02) + h02 * (h01 * h12 - d * h02);
  return a > 0.0 && m2 > 0.0 && m3 > 0.0;
}

__device__ __forceinline__ bool same3(const float a[3], const float b[3]) {
  return a[0] == b[0] && a[1] == b[1] && a[2] == b[2];
}

// ---- the fit as a machine of single evaluations ---------------------------------------------------------------------
//
// The reference's schedule (40 LM steps, 8 Gauss-Newton steps with halving, EDM and Hessian checks), step for step, one
// evaluation at a time, so that the lanes of a warp evaluate together wherever each stands in its own schedule.  next()
// goes on to the next point to evaluate, or to the end of the fit, with at most one solve; take() takes the point's chi2
// and, when it is lower, its normal equations.  One place evaluates and one solves, so the FP32 evaluation is inlined and
// the state stays in registers (addresses of it are never taken).
//
// What bounds it.  FP32: issue slots, half of them in lanes that differ (fits take 5 to 40 evaluations, 19 on average;
// 21 of 32 lanes active per instruction on the workload's fits, 11 on uneven waveforms).  Lanes that are done were served
// and refilled while others still fitted, from a third or a half of the lanes on: 9.1 -> 13 and 12 ms at 65,536 events (a
// service costs as much as 4 to 9 evaluations whoever takes part), so a warp serves when all its fits are done.  FP64: the
// FP64 pipe, which takes 64 cycles
// of a scheduler (19 of an SM with four warps busy) per warp instruction whatever the number of its active lanes; most of
// an evaluation is exponentials.  Hence divisions from a reciprocal, derivatives only for accepted steps, comparisons on
// integers, the points dealt out (pf_eval_warp), small batches spread over every scheduler.
// Measured, ms at the start -> with the skipped work -> now: 262,144 uneven waveforms FP32 3.78 -> 3.78 -> 3.20; 10,007 in
// FP64 17.9 -> 11.4 -> 6.6; the fits of 1,500 events in FP64 17.4 -> 11.1 -> 8.0; of 65,536 events FP32 9.1 -> 9.1 -> 8.5.
//
// Work whose outcome is known is left out, which changes no result: a step that leaves the parameters as they are has the
// same chi2 and is rejected, and so (FP64) is the point rejected last (while the damping is small it changes the step by
// less than the parameters' last bit; chi2 only falls); a rejected step at the clamped damping, and a Gauss-Newton step
// that no scale improves, leave the state as it was, so the rest of their loops would repeat them, and the final solve is
// that Gauss-Newton step's.  One departure, for the FP32-mixed fits only: the LM phase ends at the first solved step that
// leaves the FP32 parameters unchanged (the schedule would go on raising the damping, which makes the step smaller still).
// Measured on the 9,358,230 pulses of 65,536 workload events: the same pulses, sequence numbers and flags; 10 PE values
// differ from the full schedule's, by at most 2.5e-7 relative (one FP32 rounding), one time by 1e-6 ns; the fit takes 28 %
// less time.

enum : int { FIT_NONE = 0, FIT_DONE = 1, FIT_FIRST = 2, FIT_LM = 3, FIT_GN = 4, FIT_TRY = 5, FIT_LAST = 6 };

__device__ __forceinline__ bool fit_solve(const double H[6], double d0, double d3, double d5, const double g[3],
                                          double x[3]) {
  const double M[3][3] = {{d0, H[1], H[2]}, {H[1], d3, H[4]}, {H[2], H[4], d5}};
  return solve3(M, g, x);
}
__device__ __forceinline__ bool fit_solve(const float H[6], float d0, float d3, float d5, const float g[3], float x[3]) {
  const float M[6] = {d0, H[1], H[2], d3, H[4], d5};
  return solve_sym_ff(M, g, x);
}
__device__ __forceinline__ bool fit_hessian_ok(const double H[6]) {
  const double h[6] = {H[0], H[1], H[2], H[3], H[4], H[5]};
  return hessian_ok64(h);
}
__device__ __forceinline__ bool fit_hessian_ok(const float H[6]) { return hessian_ok(H); }
// x + lam (x + 1e-12) and u + s du, in FP32 with the product fused into the sum
__device__ __forceinline__ double fit_damped(double x, double lam) { return x + lam * (x + 1e-12); }
__device__ __forceinline__ float fit_damped(float x, float lam) { return fmaf(lam, x + 1e-12f, x); }
__device__ __forceinline__ double fit_move(double u, double s, double du) { return u + s * du; }
__device__ __forceinline__ float fit_move(float u, float s, float du) { return fmaf(s, du, u); }

__device__ __forceinline__ bool fit_finite(double x) { return abs_bits(x) < 0x7FF0000000000000ull; }
__device__ __forceinline__ bool fit_finite(float x) { return isfinite(x); }

template <typename R>
struct Fit {
  R lo[3], w[3];                 // lower bounds and spans (FP32: time relative to the window's first sample)
  R u[3], un[3], du[3], g[3], H[6], chi2, lam;
  R rej[sizeof(R) == 8 ? 3 : 1]; // FP64: the last point whose chi2 was not below chi2
  int it;
  int8_t phase, sc;
  bool solved;

  __device__ __forceinline__ bool running() const { return phase > FIT_DONE; }

  // start values: the external parameters p0
  __device__ __forceinline__ void start(const R p0[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const R c = R(2) * (p0[k] - lo[k]) / w[k] - R(1);
      if constexpr (sizeof(R) == 8) un[k] = asin(fmin(fmax(c, -1.0), 1.0));
      else un[k] = asinf(fminf(fmaxf(c, -1.0f), 1.0f));
      if constexpr (sizeof(R) == 8) rej[k] = NAN;
    }
    phase = FIT_FIRST;
  }

  __device__ __forceinline__ bool known() const {      // un's chi2 is known not to be below chi2
    if constexpr (sizeof(R) == 8) return same3(un, u) || same3(un, rej);
    else return same3(un, u);
  }

  __device__ __forceinline__ void damp(bool better, int iters) {
    R ln;
    if constexpr (sizeof(R) == 8) ln = fmin(fmax(better ? lam * 0.3 : lam * 10.0, 1e-9), 1e9);
    else ln = fminf(fmaxf(better ? lam * 0.3f : lam * 10.0f, 1e-9f), 1e9f);
    if (!better && ln == lam) it = iters;
    else ++it;
    lam = ln;
    if (it >= iters) { phase = FIT_GN; it = 0; }
  }

  // to the next point (un) that is to be evaluated, or as far as one solve goes; false: not there yet, or done
  __device__ __forceinline__ bool next(int iters) {
    if (phase == FIT_FIRST) return true;
    if (phase != FIT_TRY) {                            // LM step, Gauss-Newton step, final solve
      const bool lm = phase == FIT_LM;
      const R e = R(1e-12);
      // (copies: the called solve takes addresses, and an address of the state would put all of it into memory)
      const R r[3] = {g[0], g[1], g[2]};
      R x[3] = {du[0], du[1], du[2]};
      solved = fit_solve(H, lm ? fit_damped(H[0], lam) : H[0] + e, lm ? fit_damped(H[3], lam) : H[3] + e,
                         lm ? fit_damped(H[5], lam) : H[5] + e, r, x);
#pragma unroll
      for (int k = 0; k < 3; ++k) du[k] = x[k];
      if (phase == FIT_LAST || (!lm && !solved)) { phase = FIT_DONE; return false; }
      if (lm) {
#pragma unroll
        for (int k = 0; k < 3; ++k) un[k] = u[k] + (solved ? du[k] : R(0));
        if (!known()) return true;
        if (sizeof(R) == 4 && solved) { phase = FIT_GN; it = 0; }
        else damp(false, iters);
        return false;
      }
      phase = FIT_TRY;
      sc = 0;
    }
    for (; sc < 4; ++sc) {
      const R s = sc == 0 ? R(1) : (sc == 1 ? R(0.5) : (sc == 2 ? R(0.25) : R(0.125)));
#pragma unroll
      for (int k = 0; k < 3; ++k) un[k] = fit_move(u[k], s, fit_finite(du[k]) ? du[k] : R(0));
      if (!known()) return true;
    }
    phase = FIT_DONE;                                  // no scale improves: du is the final solve's
    return false;
  }

  // un's chi2 and, when it is below chi2 (or un is the first point), its normal equations
  __device__ __forceinline__ void take(bool better, R c2, const R Hn[6], const R gn[3], int iters) {
    if (better) {
#pragma unroll
      for (int k = 0; k < 3; ++k) { u[k] = un[k]; g[k] = gn[k]; }
#pragma unroll
      for (int k = 0; k < 6; ++k) H[k] = Hn[k];
      chi2 = c2;
    } else if constexpr (sizeof(R) == 8) {
#pragma unroll
      for (int k = 0; k < 3; ++k) rej[k] = un[k];
    }
    if (phase == FIT_FIRST) {
      lam = R(1e-3);
      it = 0;
      phase = iters > 0 ? FIT_LM : FIT_GN;
    } else if (phase == FIT_LM) {
      damp(better, iters);
    } else if (better) {
      phase = ++it >= 8 ? FIT_LAST : FIT_GN;
    } else {
      ++sc;
    }
  }

  // convergence by the estimated distance to the minimum, and the Hessian check
  __device__ __forceinline__ void verdict(bool* conv, bool* hok) const {
    R edm;
    if (solved) {
      edm = R(0.5) * (g[0] * du[0] + g[1] * du[1] + g[2] * du[2]);
      *hok = fit_hessian_ok(H);
    } else {
      edm = R(INFINITY);
      *hok = false;
    }
    if constexpr (sizeof(R) == 8) *conv = isfinite(edm) && (edm <= 1e-3 * fmax(chi2, 1.0));
    else *conv = isfinite(edm) && (edm <= 1e-3f * fmaxf(chi2, 1.0f));
  }
};

// ---- rounds over a device task list (an alternative launch shape: k_pf_persist is the default) ------------------------
//
// A waveform's pulses are found one per round.  Round 0 (k_pf_begin) prepares every waveform and finds its first
// peak; each later launch (k_pf_round) fits one pulse of every waveform still pending, records it, subtracts it and
// searches the next peak, appending the waveform to the next round's list.  Lanes of a warp therefore run the same
// fit schedule on different waveforms instead of one lane per waveform for all its rounds.  After a fixed number of
// rounds a tail launch finishes the few waveforms left, one lane each.  Results depend only on the waveform, so the
// (atomic) order of the lists does not matter.

struct PfState {             // per waveform, carried between rounds
  double ped;
  int32_t start, cnt, ps, pe, fs, fe;
  uint8_t under, fb, near, pad[5];
};

// a lane's waveform of more samples is copied by the warp
constexpr int PF_WARP_COPY = 48, PF_LANE_SCAN = 32;

struct PfQueue {
  PfState* st;               // [nw]
  long long* list[2];        // [nw] each: waveforms pending in even / odd rounds
  long long* counts;         // [rounds + 2]: tasks per round (zeroed before round 0)
  int rounds;                // round launches before the tail launch
  int threads;               // launch shape of the round kernels: threads per block
  int blocks_per_sm;         //   and blocks per SM (grid = min(needed, SMs x blocks_per_sm))
};

__device__ __forceinline__ void push_task(long long* list, long long* count, long long w, bool pend) {
  const unsigned m = __ballot_sync(0xffffffffu, pend);
  if (!m) return;
  const int lane = lane_id();
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(reinterpret_cast<unsigned long long*>(count), (unsigned long long)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (pend) list[base + __popc(m & ((1u << lane) - 1u))] = w;
}

// a waveform's pedestal and start state
__device__ __forceinline__ void pf_open(const CrvParams& p, const WaveIn& W, long long w, PfState& st) {
  const long long off = W.off[w];
  const double pdb = W.ped_db[w];
  const double x0 = W.n[w] > 0 ? (W.adc16 ? double(W.adc16[off]) : double(W.adc64[off])) : 0.0;
  const bool under = (W.n[w] > 0) && (pdb - x0 > p.pedestal_undershoot);
  st.ped = under ? x0 : pdb;
  st.under = under;
  st.start = 0;
  st.cnt = 0;
  st.fb = 0;
  st.near = 0;
}

// sample i of a waveform at `off`, less its pedestal
template <typename R>
__device__ __forceinline__ R pf_sample(const WaveIn& W, long long off, int i, double ped) {
  if (sizeof(R) == 8) return R((W.adc16 ? double(W.adc16[off + i]) : double(W.adc64[off + i])) - ped);
  return R((W.adc16 ? float(W.adc16[off + i]) : float(W.adc64[off + i])) - float(ped));
}

// sample copy and near-threshold scan by one lane
template <typename R>
__device__ __forceinline__ void pf_copy_lane(const CrvParams& p, const WaveIn& W, double* yscr, long long w, PfState& st) {
  const int n = W.n[w];
  const long long off = W.off[w];
  R* y = reinterpret_cast<R*>(yscr) + off;
  for (int i = 0; i < n; ++i) y[i] = pf_sample<R>(W, off, i, st.ped);
  st.near = near_lane<R>(y, n, 0, n - 1, R(p.min_adc_difference), R(p.knife_edge_adc));
}

// the same by the warp, 32 samples at a time (coalesced; the next 32 are loaded for the last lane's right neighbour):
// whether a near-threshold maximum is there
template <typename R>
__device__ __forceinline__ bool pf_copy_warp(const CrvParams& p, const WaveIn& W, double* yscr, long long off, int n,
                                             double ped) {
  R* y = reinterpret_cast<R*>(yscr) + off;
  const R thr = R(p.min_adc_difference), edge = R(p.knife_edge_adc);
  const int lane = lane_id();
  bool near = false;
  R carry = R(-1e9);
  R v = lane < n ? pf_sample<R>(W, off, lane, ped) : R(-1e9);
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const R nx = i + 32 < n ? pf_sample<R>(W, off, i + 32, ped) : R(-1e9);
    const R up = __shfl_up_sync(0xffffffffu, v, 1), down = __shfl_down_sync(0xffffffffu, v, 1);
    const R first = __shfl_sync(0xffffffffu, nx, 0);
    const R left = lane == 0 ? carry : up, right = lane == 31 ? first : down;
    if (i < n) {
      y[i] = v;
      const R d = v - thr;
      near = near || (v >= left && v > right && (d < R(0) ? -d : d) <= edge);
    }
    carry = __shfl_sync(0xffffffffu, v, 31);
    v = nx;
  }
  return __any_sync(0xffffffffu, near);
}

// FP64: times of the window's first points; FP32: none kept
template <typename R>
struct FitTimes {
  double t[sizeof(R) == 8 ? FIT_KEEP : 1];
};

// bounds and start values of the pending pulse's fit.  FP32-mixed: the window relative to its first sample
template <typename R>
__device__ __forceinline__ void pf_setup(const CrvParams& p, const WaveIn& W, const double* yscr, long long w,
                                         const PfState& st, Fit<R>& F, FitTimes<R>& tw) {
  const R* y = reinterpret_cast<const R*>(yscr) + W.off[w];
  const int ps = st.ps, pe = st.pe, fs = st.fs;
  if constexpr (sizeof(R) == 4) {
    const float E = 2.718281828459045f;
    const float Pf = float(p.period);
    const float yps = y[ps];
    const float mtd = float(p.max_time_difference);
    F.lo[0] = yps * E * float(p.min_height_ratio);
    F.w[0] = yps * E * float(p.max_height_ratio) - F.lo[0];
    F.lo[1] = float(ps - fs) * Pf - mtd;
    F.w[1] = float(pe - ps) * Pf + 2.0f * mtd;
    F.lo[2] = float(p.min_beta);
    F.w[2] = float(p.max_beta) - F.lo[2];
    const float tpk_rel = 0.5f * float(ps + pe - 2 * fs) * Pf;    // peak time relative to the window start
    const float p0[3] = {yps * E, tpk_rel, float(p.default_beta)};
    F.start(p0);
  } else {
    const double E = 2.718281828459045;
    const long long st_tdc = W.start_tdc[w];
    const double yps = double(y[ps]);
    const double t_ps = double(st_tdc + ps) * p.period;
    const double t_pe = double(st_tdc + pe) * p.period;
    const double t_peak = 0.5 * (t_ps + t_pe);
    F.lo[0] = yps * E * p.min_height_ratio; F.w[0] = yps * E * p.max_height_ratio - F.lo[0];
    F.lo[1] = t_ps - p.max_time_difference; F.w[1] = t_pe + p.max_time_difference - F.lo[1];
    F.lo[2] = p.min_beta; F.w[2] = p.max_beta - F.lo[2];
    const double p0[3] = {yps * E, t_peak, p.default_beta};
    F.start(p0);
    for (int i = 0; i < FIT_KEEP && i <= st.fe - fs; ++i) tw.t[i] = double(st_tdc + fs + i) * p.period;
  }
}

// evaluate the fit's point and take the outcome
template <typename R>
__device__ __forceinline__ void pf_eval(const CrvParams& p, const WaveIn& W, const double* yscr, long long w,
                                        const PfState& st, Fit<R>& F, const FitTimes<R>& tw) {
  const R* yw = reinterpret_cast<const R*>(yscr) + W.off[w] + st.fs;
  const int P = st.fe - st.fs + 1;
  R c2, Hn[6], gn[3];
  bool better;
  if constexpr (sizeof(R) == 4) {
    eval_f32(F.lo, F.w, F.un, yw, float(p.period), P, &c2, Hn, gn);
    better = F.phase == FIT_FIRST || c2 < F.chi2;
  } else {
    const bool first = F.phase == FIT_FIRST;
    const double lo[3] = {F.lo[0], F.lo[1], F.lo[2]}, wd[3] = {F.w[0], F.w[1], F.w[2]};
    const double un[3] = {F.un[0], F.un[1], F.un[2]};
    better = eval_f64(lo, wd, un, yw, tw.t, W.start_tdc[w] + st.fs, p.period, P, first, first ? INFINITY : F.chi2,
                      &c2, Hn, gn) || first;
  }
  F.take(better, c2, Hn, gn, p.lm_iterations);
}

// FP64 evaluation by the warp: the window points of all lanes, and their sines, spread over the lanes.  A warp instruction
// takes the FP64 pipe 64 cycles whatever the number of its active lanes, so 19 lanes with windows of 4 to 7 points spend
// 7 rounds of exponentials when each lane goes through its own window, 3 when the points are dealt out.  Every value
// comes from the same operations, and each lane adds its own sums in the order of its points, as eval_f64.
constexpr int PF_POINTS = 192;               // points dealt out at a time (whole windows)
struct PfWarp {
  double v[9][PF_POINTS];                    // per point: z, e^-z, Gumbel factor, residual, its square; then the nine products
  double arg[96], sn[96], cs[96];            // per parameter
  double A[32], mu[32], b[32], y[32], d0[32], d1[32], d2[32];
  const double* yw[32];
  long long tdc[32];
  int base[32], at[32];                      // first point of each lane (in v; among the accepted lanes')
  uint8_t own[PF_POINTS];
};

// where each lane's n points lie among those of the lanes before it; end: behind its last
__device__ __forceinline__ int points_before(int n, int* end) {
  int x = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, x, o);
    if (lane_id() >= o) x += v;
  }
  *end = x;
  return x - n;
}

__device__ __forceinline__ void pf_eval_warp(PfWarp& S, const CrvParams& p, const WaveIn& W, const double* yscr, bool point,
                                             long long w, const PfState& st, Fit<double>& F, const FitTimes<double>& tw) {
  const int lane = lane_id();
  const int P = st.fe - st.fs + 1;
  if (point && P > FIT_KEEP) pf_eval<double>(p, W, yscr, w, st, F, tw);     // a long plateau: by its own lane
  bool left = point && P <= FIT_KEEP;
  const unsigned act = __ballot_sync(0xffffffffu, left);
  if (!act) return;
  const int k0 = 3 * __popc(act & ((1u << lane) - 1u)), nk = 3 * __popc(act);
  if (left)
    for (int k = 0; k < 3; ++k) S.arg[k0 + k] = F.un[k];
  __syncwarp();
  for (int q = lane; q < nk; q += 32) sincos(S.arg[q], &S.sn[q], &S.cs[q]);
  __syncwarp();
  if (left) {
    const double A = F.lo[0] + F.w[0] * (S.sn[k0] + 1.0) * 0.5;
    const double mu = F.lo[1] + F.w[1] * (S.sn[k0 + 1] + 1.0) * 0.5;
    const double b = F.lo[2] + F.w[2] * (S.sn[k0 + 2] + 1.0) * 0.5;
    S.A[lane] = A;
    S.mu[lane] = mu;
    S.b[lane] = b;
    S.y[lane] = 1.0 / b;
    S.yw[lane] = yscr + W.off[w] + st.fs;
    S.tdc[lane] = W.start_tdc[w] + st.fs;
  }
  const bool first = F.phase == FIT_FIRST;
#pragma unroll 1
  while (__any_sync(0xffffffffu, left)) {
    int end;
    const int base = points_before(left ? P : 0, &end);
    const bool in = left && end <= PF_POINTS;
    const int np = __reduce_max_sync(0xffffffffu, in ? end : 0);
    if (in) {
      S.base[lane] = base;
      for (int i = 0; i < P; ++i) S.own[base + i] = uint8_t(lane);
    }
    __syncwarp();
#pragma unroll 1
    for (int q = lane; q < np; q += 32) {
      const int l = S.own[q], i = q - S.base[l];
      const double t = double(S.tdc[l] + i) * p.period;
      const double z = div_by(t - S.mu[l], S.b[l], S.y[l]);
      const double ez = exp(-z);
      const double gg = exp(-z - ez);
      const double r = S.yw[l][i] - S.A[l] * gg;
      S.v[0][q] = z;
      S.v[1][q] = ez;
      S.v[2][q] = gg;
      S.v[3][q] = r;
      S.v[4][q] = r * r;
    }
    __syncwarp();
    double c = 0.0, H[6] = {}, g[3] = {};
    if (in)
      for (int i = 0; i < P; ++i) c += S.v[4][base + i];
    const bool better = in && (first || c < F.chi2);
    int end2;
    const int at = points_before(better ? P : 0, &end2);
    const int na = __shfl_sync(0xffffffffu, end2, 31);
    if (better) {
      S.at[lane] = at;
      for (int i = 0; i < P; ++i) S.own[at + i] = uint8_t(lane);
      S.d0[lane] = F.w[0] * 0.5 * S.cs[k0];
      S.d1[lane] = F.w[1] * 0.5 * S.cs[k0 + 1];
      S.d2[lane] = F.w[2] * 0.5 * S.cs[k0 + 2];
    }
    __syncwarp();
#pragma unroll 1
    for (int q = lane; q < na; q += 32) {
      const int l = S.own[q], s = S.base[l] + q - S.at[l];
      const double z = S.v[0][s], ez = S.v[1][s], gg = S.v[2][s], r = S.v[3][s];
      const double f = S.A[l] * gg;
      const double fz = f * (ez - 1.0);
      const double j0 = gg * S.d0[l];
      const double j1 = fz * -S.y[l] * S.d1[l];          // (-1 / b is -(1 / b))
      const double j2 = fz * div_by(-z, S.b[l], S.y[l]) * S.d2[l];
      S.v[0][s] = j0 * j0; S.v[1][s] = j0 * j1; S.v[2][s] = j0 * j2;
      S.v[3][s] = j1 * j1; S.v[4][s] = j1 * j2; S.v[5][s] = j2 * j2;
      S.v[6][s] = j0 * r; S.v[7][s] = j1 * r; S.v[8][s] = j2 * r;
    }
    __syncwarp();
    if (better)
      for (int i = 0; i < P; ++i) {
#pragma unroll
        for (int k = 0; k < 6; ++k) H[k] += S.v[k][base + i];
#pragma unroll
        for (int k = 0; k < 3; ++k) g[k] += S.v[6 + k][base + i];
      }
    if (in) F.take(better, c, H, g, p.lm_iterations);
    left = left && !in;
    __syncwarp();
  }
}

// FP32-mixed: record the fitted pulse and subtract it; fitted values relative to the window's first sample in FP32, FP64
// for the window's absolute time and the absolute pulse times derived from it.  Returns whether the search goes on.
__device__ __forceinline__ bool pf_close(const CrvParams& p, const WaveIn& W, double* yscr, int max_pulses,
                                         const PulseSlots& S, long long w, PfState& st, const Fit<float>& F) {
  const float E = 2.718281828459045f;
  const int n = W.n[w];
  float* y = reinterpret_cast<float*>(yscr) + W.off[w];
  const long long st_tdc = W.start_tdc[w];
  const int ps = st.ps, pe = st.pe, fs = st.fs, fe = st.fe;
  const int P = fe - fs + 1;
  const float Pf = float(p.period);
  const float yps = y[ps];
  const float tpk_rel = 0.5f * float(ps + pe - 2 * fs) * Pf;      // peak time relative to the window start
  bool conv, hok;
  F.verdict(&conv, &hok);
  const int ndf = P - 3;
  bool nearlim = false;
  float par[3];
  const float tol = float(p.limit_tolerance);
  for (int k = 0; k < 3; ++k) {
    const float fr = (sinf(F.u[k]) + 1.0f) * 0.5f;                   // (par - lo) / span
    par[k] = F.lo[k] + F.w[k] * fr;
    if (fr < tol || 1.0f - fr < tol) nearlim = true;
  }
  const bool failed = !conv || !hok || nearlim;
  const double t0 = double(st_tdc + fs) * p.period;               // absolute time of the window's first sample
  const float A = par[0], b = par[2];
  const double mu = t0 + f2d(par[1]);
  const float height = failed ? yps : A / E;
  const float beta = failed ? float(p.default_beta) : b;
  const double tp = failed ? t0 + f2d(tpk_rel) : mu;
  const bool fseq = failed || st.fb;
  const int seq = st.cnt;
  if (seq < S.cap[w]) {
    PulseRec& r = S.rec[S.off[w] + seq];
    r.pe = f2d((failed ? yps * E * float(p.default_beta) : A * b) / d2f_trunc(W.area[w]));
    r.peph = f2d(height / d2f_trunc(W.height[w]));
    r.time = tp;
    r.height = f2d(height);
    r.beta = f2d(beta);
    r.chi2 = (failed || ndf <= 0) ? -1.0 : f2d(F.chi2 / float(ndf > 1 ? ndf : 1));
    r.letime = tp - p.le_time_factor * f2d(beta);
    r.ped = st.ped;
    r.A = f2d(A); r.mu = mu; r.b = f2d(b);
    r.seq = seq;
    r.failed = fseq; r.zerondf = ndf <= 0; r.pedfromdb = !st.under; r.pad = 0;
  }
  st.cnt = seq + 1;
  st.fb = fseq;
  // subtract round(fit) walking out from the mode's sample
  int im = fs + int(floorf(par[1] / Pf));
  if (im < 0) im = 0;
  if (im > n - 1) im = n - 1;
  int lo = im, hi = im;
  {
    const float mu_rel = par[1] - float(im - fs) * Pf;             // mode relative to sample im
    const float inv_b = 1.0f / b;
    for (int dir = -1; dir <= 1; dir += 2) {
      for (int i = im + (dir > 0 ? 1 : 0); i >= 0 && i < n; i += dir) {
        const float tr = float(i - im) * Pf;
        const float z = (tr - mu_rel) * inv_b;
        const float gv = A * __expf(-z - __expf(-z));
        y[i] -= round_half_away_f(gv);
        if (dir < 0) lo = i; else hi = i;
        if (fabsf(gv) < 0.25f && ((dir < 0 && tr < mu_rel) || (dir > 0 && tr > mu_rel))) break;
      }
    }
  }
  st.near = st.near || near_lane<float>(y, n, lo - 1, hi + 1, float(p.min_adc_difference), float(p.knife_edge_adc));
  st.start = fe;
  return st.cnt < max_pulses;
}

// FP64
__device__ __forceinline__ bool pf_close(const CrvParams& p, const WaveIn& W, double* yscr, int max_pulses,
                                         const PulseSlots& S, long long w, PfState& st, const Fit<double>& F) {
  const double E = 2.718281828459045;
  const int n = W.n[w];
  double* y = yscr + W.off[w];
  const long long st_tdc = W.start_tdc[w];
  const int ps = st.ps, pe = st.pe, fs = st.fs, fe = st.fe;
  const int P = fe - fs + 1;
  const double yps = y[ps];
  const double t_ps = double(st_tdc + ps) * p.period;
  const double t_pe = double(st_tdc + pe) * p.period;
  const double t_peak = 0.5 * (t_ps + t_pe);
  const double top[3] = {yps * E * p.max_height_ratio, t_pe + p.max_time_difference, p.max_beta};
  bool conv, hok;
  F.verdict(&conv, &hok);
  double par[3];
  for (int k = 0; k < 3; ++k) par[k] = F.lo[k] + F.w[k] * (sin(F.u[k]) + 1.0) * 0.5;
  const int ndf = P - 3;
  bool nearlim = false;
  for (int k = 0; k < 3; ++k) {
    const double span = F.w[k];
    if ((par[k] - F.lo[k]) / span < p.limit_tolerance || (top[k] - par[k]) / span < p.limit_tolerance)
      nearlim = true;
  }
  const bool failed = !conv || !hok || nearlim;
  const double A = par[0], mu = par[1], b = par[2];
  const double height = failed ? yps : A / E;
  const double beta = failed ? p.default_beta : b;
  const double tp = failed ? t_peak : mu;
  const bool fseq = failed || st.fb;
  const int seq = st.cnt;
  if (seq < S.cap[w]) {
    PulseRec& r = S.rec[S.off[w] + seq];
    r.pe = (failed ? yps * E * p.default_beta : A * b) / W.area[w];
    r.peph = height / W.height[w];
    r.time = tp;
    r.height = height;
    r.beta = beta;
    r.chi2 = (failed || ndf <= 0) ? -1.0 : F.chi2 / double(ndf > 1 ? ndf : 1);
    r.letime = tp - p.le_time_factor * beta;
    r.ped = st.ped;
    r.A = A; r.mu = mu; r.b = b;
    r.seq = seq;
    r.failed = fseq; r.zerondf = ndf <= 0; r.pedfromdb = !st.under; r.pad = 0;
  }
  st.cnt = seq + 1;
  st.fb = fseq;
  int lo, hi;
  subtract_lane(p, y, n, st_tdc, A, mu, b, &lo, &hi);
  st.near = st.near || near_lane<double>(y, n, lo - 1, hi + 1, p.min_adc_difference, p.knife_edge_adc);
  st.start = fe;
  return st.cnt < max_pulses;
}

// the next peak; false: none is left
template <typename R>
__device__ __forceinline__ bool pf_search(const CrvParams& p, const WaveIn& W, const double* yscr, long long w,
                                          PfState& st) {
  const R* y = reinterpret_cast<const R*>(yscr) + W.off[w];
  const int n = W.n[w];
  PeakScan s{st.start > 0 ? st.start + 1 : 1, 0, false, false};
  peak_scan<R>(y, n, R(p.min_adc_difference), s);
  if (!s.found) return false;
  st.ps = s.ps;
  st.pe = s.b - 1;
  peak_window<R>(p, y, n, st.ps, st.pe, &st.fs, &st.fe);
  return true;
}

// the same for the lanes that want it (every lane of the warp calls it): PF_LANE_SCAN positions by each lane, then the
// warp goes on for one lane after the other
template <typename R>
__device__ __forceinline__ bool pf_search_warp(const CrvParams& p, const WaveIn& W, const double* yscr, bool want,
                                               long long w, PfState& st) {
  const R thr = R(p.min_adc_difference);
  __syncwarp();                        // a lane's samples (copied, or less its pulse) are read by the others below
  const long long off = want ? W.off[w] : 0;
  const int n = want ? W.n[w] : 0;
  const R* y = reinterpret_cast<const R*>(yscr) + off;
  PeakScan s{want && st.start > 0 ? st.start + 1 : 1, 0, false, false};
  if (want) peak_scan<R>(y, n - s.b > PF_LANE_SCAN ? s.b + PF_LANE_SCAN : n, thr, s);
  for (unsigned m = __ballot_sync(0xffffffffu, want && !s.found && s.b < n); m; m &= m - 1) {
    const int l = __ffs(m) - 1;
    const PeakScan f = peak_scan_warp<R>(reinterpret_cast<const R*>(yscr) + __shfl_sync(0xffffffffu, off, l),
                                         __shfl_sync(0xffffffffu, n, l), thr, __shfl_sync(0xffffffffu, s.b, l),
                                         __shfl_sync(0xffffffffu, s.ps, l), __shfl_sync(0xffffffffu, int(s.rising), l));
    if (lane_id() == l) s = f;
  }
  if (!want || !s.found) return false;
  st.ps = s.ps;
  st.pe = s.b - 1;
  peak_window<R>(p, y, n, st.ps, st.pe, &st.fs, &st.fe);
  return true;
}

// pedestal, sample copy, near-threshold scan and the first peak; true when a pulse is pending
template <typename R>
__device__ __forceinline__ bool pf_begin(const CrvParams& p, const WaveIn& W, double* yscr, int max_pulses,
                                         long long w, PfState& st) {
  pf_open(p, W, w, st);
  pf_copy_lane<R>(p, W, yscr, w, st);
  return max_pulses > 0 && pf_search<R>(p, W, yscr, w, st);
}

// fit, record and subtract the pending pulse, then search the next one; true when another pulse is pending
template <typename R>
__device__ __forceinline__ bool pf_step(const CrvParams& p, const WaveIn& W, double* yscr, int max_pulses,
                                        const PulseSlots& S, long long w, PfState& st) {
  Fit<R> F;
  FitTimes<R> tw;
  pf_setup<R>(p, W, yscr, w, st, F, tw);
#pragma unroll 1
  while (F.running())
    if (F.next(p.lm_iterations)) pf_eval<R>(p, W, yscr, w, st, F, tw);
  return pf_close(p, W, yscr, max_pulses, S, w, st, F) && pf_search<R>(p, W, yscr, w, st);
}

__device__ __forceinline__ void pf_finish(const PulseSlots& S, Status* status, long long w, const PfState& st) {
  S.count[w] = st.cnt;
  S.near[w] = st.near;
  if (st.cnt > S.cap[w]) set_flag(status, CRV_ST_LIMIT);
}

template <typename R>
__global__ void __launch_bounds__(128) k_pf_begin(CrvParams p, WaveIn W, double* __restrict__ yscr, int max_pulses,
                                                 PulseSlots S, PfQueue Q, Status* status) {
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  const long long nw = bounded_count(W.nw, W.nw_dev);
  for (long long base = (blockIdx.x * (long long)(blockDim.x >> 5) + warp_in_block()) * 32; base < nw;
       base += nwarps * 32) {
    const long long w = base + lane_id();
    bool pend = false;
    if (w < nw && !(wave_in_bounds(W.off[w], W.n[w], W.nsamples) && S.off[w] >= 0 && S.cap[w] >= 0 &&
                    S.off[w] + S.cap[w] <= S.rc)) {
      set_flag(status, CRV_ST_BOUNDS);
      S.count[w] = 0;
      S.near[w] = 0;
    } else if (w < nw) {
      PfState st;
      pend = pf_begin<R>(p, W, yscr, max_pulses, w, st);
      if (pend) Q.st[w] = st;
      else pf_finish(S, status, w, st);
    }
    push_task(Q.list[0], &Q.counts[0], w, pend);
  }
}

// round r: the tasks of list r & 1 (count counts[r]); tail != 0: finish every task in the lane
template <typename R>
__global__ void __launch_bounds__(128) k_pf_round(CrvParams p, WaveIn W, double* __restrict__ yscr, int max_pulses,
                                                 PulseSlots S, PfQueue Q, int r, int tail, Status* status) {
  const long long* in = Q.list[r & 1];
  const long long n_in = Q.counts[r];
  long long* out = Q.list[(r + 1) & 1];
  long long* n_out = &Q.counts[r + 1];
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long base = (blockIdx.x * (long long)(blockDim.x >> 5) + warp_in_block()) * 32; base < n_in;
       base += nwarps * 32) {
    const long long i = base + lane_id();
    long long w = -1;
    bool pend = false;
    if (i < n_in) {
      w = in[i];
      PfState st = Q.st[w];
      pend = pf_step<R>(p, W, yscr, max_pulses, S, w, st);
      if (tail)
        while (pend) pend = pf_step<R>(p, W, yscr, max_pulses, S, w, st);
      if (pend) Q.st[w] = st;
      else pf_finish(S, status, w, st);
    }
    if (!tail) push_task(out, n_out, w, pend);
  }
}

// Lanes of a warp that hold a waveform: all of them, or fewer when the warps of nw waveforms would not be `few` (four an
// SM, one for each scheduler).  A small batch takes as long as its slowest warp, which takes as long as the lanes of it
// that differ most; 100 waveforms of 200 samples took 870 us (FP64: 7.2 ms) in full warps, 568 us (3.3 ms) in warps of one,
// 10,007 of them 972 us (7.6 ms) in full warps, 874 us (6.7 ms) in half warps.
__host__ __device__ inline int pf_lanes(long long nw, long long few) {
  int lanes = 32;
  while (lanes > 1 && (nw + lanes - 1) / lanes < few) lanes >>= 1;
  return lanes;
}

// One launch for every pulse of a batch.  Each lane holds one waveform.  The warp's fits run together, one evaluation of
// each at a time; when all are done the lanes record and subtract their pulses, search their next peaks, and those whose
// waveform is finished take the next unclaimed waveforms of the batch (one warp-aggregated atomicAdd on a device head per
// refill).  Nothing waits on another warp: a warp exits once the waveforms are all claimed and its own lanes are done.  A
// waveform's results depend only on the waveform, so the order of claims does not matter (same outputs as the round
// kernels).  The head is Q.counts[0], zeroed before the launch.
//
// On waveforms of 200 samples half of the time went into copies and searches that a lane did alone while the others
// waited; the warp now does what is longer than PF_WARP_COPY and PF_LANE_SCAN (3.48 -> 3.20 ms for the search, 3.78 -> 3.48
// for the copies and the machine of evaluations; thresholds of 32 and 16 measured the same).
template <typename R>
__global__ void __launch_bounds__(128) k_pf_persist(CrvParams p, WaveIn W, double* __restrict__ yscr, int max_pulses,
                                                    PulseSlots S, PfQueue Q, long long few, Status* status) {
  const long long nw = bounded_count(W.nw, W.nw_dev);
  const int lanes = pf_lanes(nw, few);
  unsigned long long* head = reinterpret_cast<unsigned long long*>(&Q.counts[0]);
  const int lane = lane_id();
  long long w = -1;
  PfState st;
  Fit<R> F;
  FitTimes<R> tw;
  F.phase = FIT_NONE;
  extern __shared__ __align__(16) char pf_smem[];
  bool exhausted = nw <= 0;
#pragma unroll 1
  while (true) {
    // record and subtract the fitted pulses, search the next ones, refill the lanes whose waveform is finished (a
    // waveform without any pulse frees its lane again at once)
    bool search = false, pend = false;
    if (F.phase == FIT_DONE) {
      search = pf_close(p, W, yscr, max_pulses, S, w, st, F);
      if (!search) pf_finish(S, status, w, st);
      F.phase = FIT_NONE;
    }
#pragma unroll 1
    while (true) {
      const bool peak = pf_search_warp<R>(p, W, yscr, search, w, st);
      if (search) {
        pend = peak;
        if (!pend) pf_finish(S, status, w, st);
        search = false;
      }
      if (exhausted) break;
      const unsigned need = __ballot_sync(0xffffffffu, !pend && lane < lanes);
      if (!need) break;
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(head, (unsigned long long)__popc(need));
      base = __shfl_sync(0xffffffffu, base, 0);
      exhausted = (long long)(base + __popc(need)) >= nw;
      bool open = false;
      if (!pend && lane < lanes) {
        const long long c = (long long)base + __popc(need & ((1u << lane) - 1u));
        if (c < nw) {
          w = c;
          if (!(wave_in_bounds(W.off[w], W.n[w], W.nsamples) && S.off[w] >= 0 && S.cap[w] >= 0 &&
                S.off[w] + S.cap[w] <= S.rc)) {
            set_flag(status, CRV_ST_BOUNDS);
            S.count[w] = 0;
            S.near[w] = 0;
          } else {
            pf_open(p, W, w, st);
            open = true;
          }
        }
      }
      // long waveforms by the warp, one after the other; short ones by their lanes
      const int n = open ? W.n[w] : 0;
      const long long off = open ? W.off[w] : 0;
      for (unsigned m = __ballot_sync(0xffffffffu, n > PF_WARP_COPY); m; m &= m - 1) {
        const int l = __ffs(m) - 1;
        const bool near = pf_copy_warp<R>(p, W, yscr, __shfl_sync(0xffffffffu, off, l), __shfl_sync(0xffffffffu, n, l),
                                          __shfl_sync(0xffffffffu, st.ped, l));
        if (lane == l) st.near = near;
      }
      __syncwarp();
      if (open) {
        if (n <= PF_WARP_COPY) pf_copy_lane<R>(p, W, yscr, w, st);
        search = max_pulses > 0;
        if (!search) pf_finish(S, status, w, st);
      }
    }
    if (pend) pf_setup<R>(p, W, yscr, w, st, F, tw);
    __syncwarp();
    if (!__any_sync(0xffffffffu, pend)) break;
    // the fits, an evaluation of each at a time
#pragma unroll 1
    while (__any_sync(0xffffffffu, F.running())) {
      const bool point = F.running() && F.next(p.lm_iterations);
      __syncwarp();
      if constexpr (sizeof(R) == 8)
        pf_eval_warp(reinterpret_cast<PfWarp*>(pf_smem)[warp_in_block()], p, W, yscr, point, w, st, F, tw);
      else if (point) pf_eval<R>(p, W, yscr, w, st, F, tw);
      __syncwarp();
    }
  }
}

}  // namespace crv
