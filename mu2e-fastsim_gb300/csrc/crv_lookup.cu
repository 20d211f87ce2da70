// Lookup-table photon model: the substep kernel of crvfastsim.response.photons._substep_photons
// (crv/crvfastsim/response/photons.py:139-224) over (step, SiPM) rows, with keyed draws.
//
// Built with -fmad=false (FP64 throughout): every operation rounds as written, so the CPU oracle
// (oracle/crv_oracle.c, orc_substep_photons) reproduces the photons bit for bit.
//
// What bounds it: FP64, the FP64 pipe (19 cycles of an SM per warp instruction, conversions and comparisons included), so
// everything that need not be FP64 arithmetic is integer or certain FP32 work: bins and box tests compare ordered bits,
// the binomial draws are decided in FP32 where that is certain, uniforms become integer thresholds (20,011 rows of 137
// photons: count 2.9 -> 0.33 ms, emit 8.1 -> 1.9 ms, of which the fibre-decay logarithms are most).  FP32-mixed:
// instruction issue (200,000 rows: count 1.33 -> 1.23 ms, emit 6.8 -> 2.25 ms).
//
// Layout: a warp per row, lanes over its substeps (a 20 mm crossing has 200).  Pass 1 counts the arrivals of every
// row, an exclusive scan turns the counts into output offsets, pass 2 repeats the draws (keyed: the same numbers) and
// writes the photons in (row, substep, table, arrival) order, each lane at its offset from a warp scan.
#include <cstdint>
#include <cuda_runtime.h>

#include "crv_launch.h"
#include "crv_scan.cuh"

namespace crv {

constexpr uint32_t ST_SUBSTEP = 7;
constexpr int SUB_CALL_BINOMIAL = 0, SUB_CALL_PHOTON = 1, SUB_CALL_GAMMA = 2;
constexpr long long SUB_MAX_SUBSTEPS = 1ll << 20;
constexpr int SUB_MAX_ARRIVALS = 4096, SUB_MAX_EMISSIONS = 128;
constexpr int SUB_ROWS_PER_BLOCK = 8;                         // warps per block

// draw block of row (step, chan), table tb, call, substep k, arrival j
__device__ __forceinline__ U4 sub_block(uint32_t seed, long long step, long long chan, int tb, int call, int idx,
                                        long long k, int j) {
  uint32_t w2 = w2_of(ST_SUBSTEP, uint32_t(tb), uint32_t(idx), uint32_t(call), uint32_t(chan));
  uint32_t w3 = (uint32_t(k) << 12) | uint32_t(j);
  return philox(uint32_t(step), uint32_t((unsigned long long)step >> 32), w2, w3, seed, 0u);
}

// FP64 values without FP64 instructions.  This GPU's FP64 pipe takes a warp instruction of any number of active lanes for
// 19 cycles of the whole SM, conversions and comparisons included; integer and FP32 instructions cost a hundredth.
__device__ __forceinline__ double i2d(unsigned long long v) {       // exact below 2^53
  if (v == 0ull) return 0.0;
  const int lz = __clzll((long long)v);
  const unsigned long long m = v << lz;                              // leading bit at 63
  return __longlong_as_double((long long)(((unsigned long long)(1086 - lz) << 52) + ((m << 1) >> 12)));
}
// integers in the order of the doubles (-0 as +0); NaNs order beyond the infinities of their sign
__device__ __forceinline__ long long ord64(double x) {
  const long long b = __double_as_longlong(x);
  return b >= 0 ? b : (long long)(0x8000000000000000ull - (unsigned long long)b);
}
__device__ __forceinline__ bool is_nan(double x) {
  return ((unsigned long long)__double_as_longlong(x) << 1) > 0xFFE0000000000000ull;
}

// Binomial(n, p): inversion (Kachitvichyanukul & Schmeiser's BINV) on min(p, 1 - p) while the mean is at most 256,
// else the normal approximation rint(mean + sqrt(mean (1 - q)) z) clipped to [0, n]
__device__ __noinline__ long long binomial_64(long long n, double p, const U4 w) {
  if (n <= 0 || !(p > 0.0)) return 0;
  if (p >= 1.0) return n;
  const bool flip = p > 0.5;
  const double q = flip ? 1.0 - p : p;
  const double mean = double(n) * q;
  long long k;
  if (mean > 256.0) {
    double z0, z1;
    Math<double>::normal_pair(w, &z0, &z1);
    double x = rint(mean + sqrt(mean * (1.0 - q)) * z0);
    k = x < 0.0 ? 0 : (x > double(n) ? n : (long long)x);
  } else {
    double u = u01(w.x, w.y);
    const double s = q / (1.0 - q);
    const double a = double(n + 1) * s;
    double r = dexp(double(n) * dlog(1.0 - q));
    k = 0;
    while (u > r && k < n) {
      u = u - r;
      k += 1;
      r = r * (a / double(k) - s);
    }
  }
  return flip ? n - k : k;
}

// The same draw, decided in FP32 where that is certain.  The inversion only compares u with the running terms r, so an
// FP32 run of it gives the FP64 count whenever every comparison's two sides lie further apart than the sum of the
// errors: of r, relative er: its argument n log(1 - q) (q truncated to 2^-23, log1pf and expf within 2 ulp, a product)
// is within 6e-7 relative, so r within 6e-7 |arg| + 4e-7, taken as 1e-6 (|arg| + 1); each step multiplies by a / k - s,
// whose terms are within 6e-7 and at least a factor 2 apart while k <= n / 2, taken as 4e-6 a step; of u, absolute eu:
// 2^-24 of its truncation and a rounding and r's error per subtraction.  FP64's own errors (1e-14) vanish in these.  A
// comparison that is not certain (about one draw in 2,000), a mean above 128 or k above n / 2 takes the FP64 form.  A
// draw costs ~80 FP64 instructions there and none here.
__device__ __forceinline__ long long binomial(long long n, double p, const U4& w) {
  const float pf = d2f_trunc(p);
  if (n > 0 && n < 1000000 && pf > 1e-30f && pf < 0.49f) {
    const int ni = int(n);
    const float arg = float(ni) * log1pf(-pf);
    if (arg > -80.0f && float(ni) * pf < 128.0f) {
      float u = f01(w.x), eu = 6e-8f;
      const float s = __fdividef(pf, 1.0f - pf), a = float(ni + 1) * s;
      float r = expf(arg), er = 1e-6f * (1.0f - arg);
      int k = 0;
      while (2 * k <= ni) {
        const float tol = eu + (er + 2e-7f) * r;
        if (u < r - tol) return k;
        if (!(u > r + tol)) break;                 // not certain
        u = u - r;
        eu = tol + 1.2e-7f;
        ++k;
        r = r * (__fdividef(a, float(k)) - s);
        er = er + 4e-6f;
      }
    }
  }
  return binomial_64(n, p, w);
}

// numpy-style findBin: bin i with e[i] <= v <= e[i+1] (the lower bin on an inner edge), -1 outside
__device__ __forceinline__ int find_bin(const double* __restrict__ e, int ne, double v) {
  const long long x = ord64(v);
  if (is_nan(v) || x < ord64(e[0]) || x > ord64(e[ne - 1])) return -1;
  if (x == ord64(e[0])) return 0;
  int lo = 0, hi = ne;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (ord64(e[mid]) < x) lo = mid + 1; else hi = mid;
  }
  return lo - 1;
}

// the same bins for phi given c = cos phi and ce[j] = cos(phi edge j) (descending): phi > edge j <=> c < ce[j]
__device__ __forceinline__ int find_bin_cos(const double* __restrict__ ce, int ne, double c) {
  const long long x = ord64(c);
  if (is_nan(c) || x > ord64(ce[0]) || x < ord64(ce[ne - 1])) return -1;
  if (x == ord64(ce[0])) return 0;
  int lo = 0, hi = ne;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (ord64(ce[mid]) > x) lo = mid + 1; else hi = mid;
  }
  return lo - 1;
}

// First index j whose running sum of the row's n uint8 weights reaches thr (the number of running sums below thr), n when
// none does.  tab: the table's [nrow][n] weights.  The sums are integers, so sum < thr is sum < ceil(thr), and the row
// is read in aligned 16-byte loads that do not depend on each other, four weights per dp4a, instead of byte by byte with
// a floating-point compare each (two FP64 instructions a weight in the FP64 kernel): emit of 200,000 FP32 rows of 137
// photons and 150 weights 6.8 -> 3.5 ms, of 20,011 FP64 rows 8.1 -> 5.3 ms.  Weights outside the row are masked; a
// load that would leave the table (its ends are rarely aligned) is put together from bytes.
__device__ __forceinline__ uint32_t keep_bytes(uint32_t w, int lo, int hi) {   // bytes [lo, hi) of a word
  lo = min(max(lo, 0), 4);
  hi = min(max(hi, 0), 4);
  if (hi <= lo) return 0u;
  return w & (0xFFFFFFFFu >> (8 * (4 - hi))) & (0xFFFFFFFFu << (8 * lo));
}
__device__ __noinline__ uint4 edge_words(const uint8_t* q, const uint8_t* row, int n) {
  uint32_t v[4] = {0u, 0u, 0u, 0u};
  for (int b = 0; b < 16; ++b)
    if (q + b >= row && q + b < row + n) v[b >> 2] |= uint32_t(q[b]) << (8 * (b & 3));
  return make_uint4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ int first_reaching(const uint8_t* __restrict__ tab, int nrow, int bin, int n, int thr) {
  if (thr <= 0) return 0;
  const uint8_t* row = tab + (long long)bin * n;
  const uint8_t* end = tab + (long long)nrow * n;
  const int head = int(reinterpret_cast<uintptr_t>(row) & 15u);
  uint32_t cum = 0;
#pragma unroll 1
  for (int p0 = -head; p0 < n; p0 += 64) {
    uint4 v[4];                                    // four loads in flight
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int pos = p0 + 16 * b;
      const uint8_t* q = row + pos;
      v[b] = make_uint4(0u, 0u, 0u, 0u);
      if (pos < n) {
        if (q >= tab && q + 16 <= end) v[b] = __ldg(reinterpret_cast<const uint4*>(q));
        else v[b] = edge_words(q, row, n);
      }
    }
    if (p0 < 0) {                                  // the weights before the row
      v[0].x = keep_bytes(v[0].x, -p0, 4);
      v[0].y = keep_bytes(v[0].y, -p0 - 4, 4);
      v[0].z = keep_bytes(v[0].z, -p0 - 8, 4);
      v[0].w = keep_bytes(v[0].w, -p0 - 12, 4);
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int pos = p0 + 16 * b;
      const uint32_t s0 = __dp4a(v[b].x, 0x01010101u, cum), s1 = __dp4a(v[b].y, 0x01010101u, s0);
      const uint32_t s2 = __dp4a(v[b].z, 0x01010101u, s1), s3 = __dp4a(v[b].w, 0x01010101u, s2);
      if (s3 >= uint32_t(thr)) {                   // the word, then the byte; the weights after the row count as n
        const bool x = s0 >= uint32_t(thr), y = s1 >= uint32_t(thr), z = s2 >= uint32_t(thr);
        const uint32_t w = x ? v[b].x : y ? v[b].y : z ? v[b].z : v[b].w;
        uint32_t t = (x ? cum : y ? s0 : z ? s1 : s2) + (w & 0xFFu);
        int j = pos + (x ? 0 : y ? 4 : z ? 8 : 12);
        if (t < uint32_t(thr)) {
          ++j;
          t += (w >> 8) & 0xFFu;
          if (t < uint32_t(thr)) {
            ++j;
            t += (w >> 16) & 0xFFu;
            j += t < uint32_t(thr);
          }
        }
        return min(j, n);
      }
      cum = s3;
    }
  }
  return n;
}
// smallest integer not below thr (at most 2^31 - 1): the threshold on integer sums
__device__ __forceinline__ int sum_threshold(float thr) { return thr < 2147483520.0f ? int(ceilf(thr)) : 2147483647; }

struct SubBins {
  int bin[3];
  double frac, z;
};

// per-row constants of the substep geometry
struct SubRow {
  double s[3], d[3];
  double nsub, inv_nsub;       // inv_nsub: 1 / nsub rounded
  int bb, bth;
};

// Geometry and bins of substep k of a row (photons.py:139-196).  The scintillator's hole and the fibres are tested only
// inside their bounding boxes: outside, ex or ey is at least 1 and so is ex^2 + ey^2, and a radius is at least the
// larger of its two distances, in rounded arithmetic too (rounding is monotone).
__device__ __forceinline__ SubBins substep_bins(const CrvLookup& L, const SubRow& w, long long k) {
  const double k_half = __longlong_as_double(__double_as_longlong(i2d((unsigned long long)(2 * k + 1))) - (1ll << 52));
  const double frac = quotient(k_half, w.nsub, w.inv_nsub);      // (k + 1/2) / nsub
  const double x = w.s[0] + w.d[0] * frac;
  const double y = w.s[1] + w.d[1] * frac;
  const double z = w.s[2] + w.d[2] * frac;
  const double half_sep = L.fiber_separation / 2.0;
  const double ax = fabs(x), ay = fabs(y), az = fabs(z);
  const long long oax = ord64(ax), oay = ord64(ay);
  const bool inz = ord64(az) < ord64(L.half_length) && !is_nan(az);
  // inside the scintillator: box, outside the elliptic fibre hole, not in a rounded corner
  bool insc = oax < ord64(L.half_thickness) && oay < ord64(L.half_width) && inz && !is_nan(ax) && !is_nan(ay);
  const double hy = ay - half_sep;
  const bool hole = L.hole_radius_x > 0.0 && L.hole_radius_y > 0.0;
  if (insc && !(hole && (oax >= ord64(L.hole_radius_x) || ord64(fabs(hy)) >= ord64(L.hole_radius_y)))) {
    const double ex = ax / L.hole_radius_x, ey = hy / L.hole_radius_y;
    insc = ex * ex + ey * ey >= 1.0;
  }
  const double cx = L.half_thickness - L.corner_radius, cy = L.half_width - L.corner_radius;
  if (insc && oax > ord64(cx) && oay > ord64(cy)) {
    const double qx = ax - cx, qy = ay - cy;
    if (sqrt(qx * qx + qy * qy) > L.corner_radius) insc = false;
  }
  const int ny = L.nedges[1] - 1, nz = L.nedges[2] - 1, nb = L.nedges[3] - 1;
  const int nth = L.nedges[4] - 1, nph = L.nedges[5] - 1, nr = L.nedges[6] - 1;
  SubBins S;
  S.frac = frac;
  S.z = z;
  S.bin[0] = S.bin[1] = S.bin[2] = -1;
  const int bz = find_bin(L.edges[2], L.nedges[2], z);
  if (insc && bz >= 0) {
    const int bx = find_bin(L.edges[0], L.nedges[0], ax), by = find_bin(L.edges[1], L.nedges[1], y);
    if (bx >= 0 && by >= 0) {
      S.bin[0] = bz + by * nz + bx * ny * nz;
      if (w.bb >= 0) S.bin[1] = w.bb + bz * nb + by * nz * nb + bx * ny * nz * nb;
    }
  }
  // inside a fibre: radius from the nearer fibre axis and the angle of the step direction to it
  const double y0 = y + half_sep, y1 = y - half_sep;
  const long long ofr = ord64(L.fiber_radius);
  if (inz && !insc && oax <= ofr && (ord64(fabs(y0)) <= ofr || ord64(fabs(y1)) <= ofr)) {
    const double r0 = sqrt(x * x + y0 * y0), r1 = sqrt(x * x + y1 * y1);
    const bool in0 = r0 <= L.fiber_radius, in1 = r1 <= L.fiber_radius;
    if ((in0 || in1) && w.bb >= 0 && w.bth >= 0 && bz >= 0) {
      const double ry = in1 ? y1 : y0, rr = in1 ? r1 : r0;
      const double norm = sqrt(w.d[0] * w.d[0] + w.d[1] * w.d[1]) * rr;
      double c = 1.0;
      if (norm > 0.0) {
        c = (w.d[0] * x + w.d[1] * ry) / norm;
        c = c < -1.0 ? -1.0 : (c > 1.0 ? 1.0 : c);
      }
      const int bph = find_bin_cos(L.cos_phi_edges, L.nedges[5], c), br = find_bin(L.edges[6], L.nedges[6], rr);
      if (bph >= 0 && br >= 0)
        S.bin[2] = bz + br * nz + bph * nr * nz + w.bth * nph * nr * nz + w.bb * nth * nph * nr * nz;
    }
  }
  return S;
}

__device__ __forceinline__ long long photons_per_substep(const CrvSubstepRows& R, int tb, long long r) {
  return tb == 0 ? R.n_scint[r] : (tb == 1 ? R.n_ck_s[r] : R.n_ck_f[r]);
}

// arrivals of table tb at a substep (bin >= 0)
__device__ __forceinline__ long long arrivals(const CrvLookup& L, const CrvSubstepRows& R, uint32_t seed, long long r,
                                              long long step, long long chan, long long k, int tb, int bin, double z) {
  double pr = f2d(L.table[tb].prob[bin]) * R.dev[r];
  if (R.mu) {
    const double mu = R.mu[r];
    if (ord64(mu) != 0) pr = pr * dexp(-mu * z);   // dexp(0) is 1
  }
  if (is_nan(pr) || ord64(pr) >= ord64(1.0)) pr = 1.0;         // (not below 1)
  return binomial(photons_per_substep(R, tb, r), pr, sub_block(seed, step, chan, tb, SUB_CALL_BINOMIAL, 0, k, 0));
}

// ceil(u * sum) of a 53-bit uniform u = k 2^-53 and an integer sum, u * sum rounded to FP64 first: the threshold
// first_reaching compares integer running sums with.  The product k * sum is exact in 84 bits; rounding to 53 of them
// (to nearest, ties to even) and the ceiling are integer work.
__device__ __forceinline__ int ceil_uniform(unsigned long long k, int sum) {
  if (sum <= 0 || k == 0ull) return 0;
  const unsigned long long m = (unsigned long long)(uint32_t)sum;
  unsigned long long hi = __umul64hi(k, m), lo = k * m;
  const int bits = hi ? 128 - __clzll((long long)hi) : 64 - __clzll((long long)lo);
  if (bits > 53) {                                 // round off the lowest `s` bits
    const int s = bits - 53;                       // at most 31
    const unsigned long long rest = lo & ((1ull << s) - 1ull), half = 1ull << (s - 1);
    lo -= rest;
    if (rest > half || (rest == half && ((lo >> s) & 1ull))) {
      const unsigned long long t = lo + (1ull << s);
      hi += t < lo;
      lo = t;
    }
  }
  const unsigned long long q = (hi << 11) | (lo >> 53);
  return int(q) + ((lo & ((1ull << 53) - 1ull)) != 0ull);
}

// delay of arrival j at a substep (photons.py:128-137, :214-218), and its number of emissions in a decaying fibre
__device__ __forceinline__ double arrival_delay(const CrvLookup& L, uint32_t seed, long long step, long long chan,
                                                long long k, int tb, int bin, int j, int* ne) {
  const CrvLookupTable& T = L.table[tb];
  const U4 w = sub_block(seed, step, chan, tb, SUB_CALL_PHOTON, 0, k, j);
  const int thr = ceil_uniform(bits53(w.x, w.y), T.delay_sum[bin]);
  const double d = i2d((unsigned long long)first_reaching(T.delays, T.nbins, bin, T.ndelay, thr));
  if (L.fiber_decay_time > 0.0)
    *ne = first_reaching(T.emis, T.nbins, bin, T.nemis, ceil_uniform(bits53(w.z, w.w), T.emis_sum[bin]));
  return d;
}

// theta bin of a row: from theta, or from cos theta against the cos of the edges
__device__ __forceinline__ int theta_bin(const CrvLookup& L, const CrvSubstepRows& R, long long r) {
  return R.theta ? find_bin(L.edges[4], L.nedges[4], R.theta[r])
                 : find_bin_cos(L.cos_theta_edges, L.nedges[4], R.cos_theta[r]);
}

__device__ __forceinline__ SubRow sub_row(const CrvLookup& L, const CrvSubstepRows& R, long long r, long long nsub) {
  SubRow w;
  for (int x = 0; x < 3; ++x) { w.s[x] = R.s[3 * r + x]; w.d[x] = R.d[3 * r + x]; }
  w.nsub = i2d((unsigned long long)nsub);
  w.inv_nsub = 1.0 / w.nsub;
  w.bb = find_bin(L.edges[3], L.nedges[3], R.beta[r]);
  w.bth = theta_bin(L, R, r);
  return w;
}

__device__ __forceinline__ bool row_ok(const CrvSubstepRows& R, long long r, long long* nsub, Status* status) {
  *nsub = R.nsub[r];
  if (*nsub > SUB_MAX_SUBSTEPS) {
    set_flag(status, CRV_ST_LIMIT);
    return false;
  }
  return *nsub > 0;
}

// Rows a launch takes.  The stage entry point takes every row; the resident chain's dense rows (row 4 step + SiPM,
// every group's rows in one table) take [0, min(nrows, *nrows_dev)) of group gsel, and the seed from *seed_dev (a
// device copy of the chain's parameter-block seed, so that a captured graph of the chain follows a new seed).
struct RowSel {
  const long long* nrows_dev;
  const int8_t* group;
  const uint32_t* seed_dev;
  int gsel;
  uint16_t* kept;                // arrivals of each row's first nkept substeps, from the count to the emission
  int nkept;
};

// The counts drawn for a substep, kept for the emission, which repeats the draws only where they do not fit (counts of 255
// or more) and beyond a row's first nkept substeps.  A substep lies in the scintillator (tables 0 and 1) or in a fibre
// (table 2).  200,000 FP32 rows of 200 substeps: emission 2.70 -> 2.25 ms, count 1.16 -> 1.21; 328,000 rows of a lookup
// chain's 2,048 events 3.70 -> 3.04 and 1.61 -> 1.74.
constexpr int SUB_KEPT = 256;
constexpr uint16_t SUB_REDRAW = 0xFFFF;
__device__ __forceinline__ uint16_t* kept_row(const RowSel& q, long long r) { return q.kept + r * q.nkept; }
__device__ __forceinline__ void keep_counts(uint16_t* kept, int nkept, int k, int scint_or_fibre, int ck) {
  if (k < nkept) kept[k] = (scint_or_fibre | ck) < 255 ? uint16_t(scint_or_fibre | ck << 8) : SUB_REDRAW;
}
__device__ __forceinline__ bool kept_counts(const uint16_t* kept, int nkept, int k, const int bin[3], int a[3]) {
  if (k >= nkept) return false;
  const uint16_t v = kept[k];
  if (v == SUB_REDRAW) return false;
  if (bin[2] >= 0) a[2] = v & 255;
  else { a[0] = v & 255; a[1] = v >> 8; }
  return true;
}
__device__ __forceinline__ long long sel_nrows(const RowSel& q, long long n) {
  if (!q.nrows_dev) return n;
  const long long m = *q.nrows_dev;
  return m < n ? m : n;
}
__device__ __forceinline__ bool sel_row(const RowSel& q, long long r) { return !q.group || q.group[r] == q.gsel; }
__device__ __forceinline__ uint32_t sel_seed(const RowSel& q, uint32_t seed) { return q.seed_dev ? *q.seed_dev : seed; }

__global__ void __launch_bounds__(SUB_ROWS_PER_BLOCK * 32) k_substep_count(CrvLookup L, CrvSubstepRows R,
                                                                           uint32_t seed, long long nrows, RowSel sel,
                                                                           long long* __restrict__ count,
                                                                           Status* status) {
  seed = sel_seed(sel, seed);
  nrows = sel_nrows(sel, nrows);
  const long long warps = (long long)gridDim.x * SUB_ROWS_PER_BLOCK;
  for (long long r = (long long)blockIdx.x * SUB_ROWS_PER_BLOCK + warp_in_block(); r < nrows; r += warps) {
    if (!sel_row(sel, r)) continue;                          // warp-uniform
    long long nsub;
    long long tot = 0;
    if (row_ok(R, r, &nsub, status)) {
      const long long step = R.step[r], chan = R.chan[r];
      const SubRow w = sub_row(L, R, r, nsub);
      uint16_t* const kept = kept_row(sel, r);
      for (long long k = lane_id(); k < nsub; k += 32) {
        const SubBins S = substep_bins(L, w, k);
        int in_or_fibre = 0, ck = 0;
#pragma unroll 1
        for (int tb = 0; tb < 3; ++tb)
          if (S.bin[tb] >= 0) {
            long long a = arrivals(L, R, seed, r, step, chan, k, tb, S.bin[tb], S.z);
            if (a >= SUB_MAX_ARRIVALS) { set_flag(status, CRV_ST_LIMIT); a = 0; }
            tot += a;
            if (tb == 1) ck = int(a); else in_or_fibre = int(a);
          }
        keep_counts(kept, sel.nkept, int(k), in_or_fibre, ck);
      }
    }
    tot = warp_sum(tot);
    if (lane_id() == 0) count[r] = tot;
  }
}

// The arrivals of a warp's row wait in a shared queue, in (substep, table, arrival) order, until 32 of them can be emitted
// together: a 32-substep chunk has 12 to 22 arrivals, so emitting chunk by chunk left half of the lanes idle (emit
// of 200,000 FP32 rows of 137 photons 3.5 -> 3.3 ms, of 326,000 rows of 78 photons 5.1 -> 4.2 ms).
constexpr int SUB_QUEUE = 96;
template <typename T>
struct SubQueue {
  uint32_t key[SUB_QUEUE];       // substep << 12 | arrival
  int bin[SUB_QUEUE];
  T at[SUB_QUEUE];               // substep time (FP64) or its fraction of the row (FP32)
  uint8_t table[SUB_QUEUE];
};

// Queue one chunk's arrivals (a[tb] of the lane's substep k) and call emit(queued, slot, lane's output row) by every lane for every 32 queued,
// after the row's last chunk for what is left too.  c: queued, o: output row of the queue's front.
template <typename T, typename Emit>
__device__ __forceinline__ void queue_chunk(SubQueue<T>& Q, int& c, long long& o, const int a[3], const int bin[3],
                                            uint32_t k, T at, bool last, Emit emit) {
  const int lane = lane_id();
  const int n = a[0] + a[1] + a[2];
  int sum;
  const int pre = warp_excl(n, &sum);
  int off = 0;
  do {
    const int m = min(SUB_QUEUE - c, sum - off);
#pragma unroll 1
    for (int e = max(off - pre, 0); e < n && pre + e < off + m; ++e) {
      const int q = c + pre + e - off;
      const int tb = e < a[0] ? 0 : e < a[0] + a[1] ? 1 : 2;
      const int j = e - (tb > 0 ? a[0] : 0) - (tb > 1 ? a[1] : 0);
      Q.key[q] = (k << 12) | uint32_t(j);
      Q.bin[q] = tb == 0 ? bin[0] : tb == 1 ? bin[1] : bin[2];
      Q.at[q] = at;
      Q.table[q] = uint8_t(tb);
    }
    __syncwarp();
    c += m;
    off += m;
    const bool flush = last && off == sum;
    int b = 0;
#pragma unroll 1
    for (; b + 32 <= c || (flush && b < c); b += 32) {
      emit(b + lane < c, b + lane, o + lane);
      o += 32;
    }
    __syncwarp();
    if (b) {                                       // the rest moves to the front
      const int rest = max(c - b, 0);
      uint32_t key = 0;
      int bn = 0;
      T t = T(0);
      uint8_t tb = 0;
      if (lane < rest) { key = Q.key[b + lane]; bn = Q.bin[b + lane]; t = Q.at[b + lane]; tb = Q.table[b + lane]; }
      __syncwarp();
      if (lane < rest) { Q.key[lane] = key; Q.bin[lane] = bn; Q.at[lane] = t; Q.table[lane] = tb; }
      c = rest;
      __syncwarp();
    }
  } while (off < sum);
}

// The emissions of the warp's arrivals (ne of them each, 0 for none): the sums of their -log u, in order.  The Philox blocks
// of all arrivals, two emissions each, are dealt out over the lanes, 64 at a time, and each lane adds its own terms: with
// its own emissions in each lane the warp went on, a logarithm on the FP64 pipe at a time, until the arrival with the most
// of them was done (20,011 rows of 137 photons: emission 1.81 -> 1.41 ms; in FP32, where a logarithm is cheap, this lost:
// 3.04 -> 3.40 ms in the lookup chain of 2,048 events).
struct SubGamma {
  double x[2][64];
  int before[33], ne[32];        // blocks before each lane's, emissions
};
__device__ __forceinline__ double emission_sum(SubGamma& G, const SubQueue<double>& Q, int b, uint32_t seed, long long step,
                                          long long chan, int ne) {
  const int lane = lane_id();
  int total;
  const int before = warp_excl((ne + 1) >> 1, &total);
  G.before[lane] = before;
  G.ne[lane] = ne;
  if (lane == 31) G.before[32] = total;
  __syncwarp();
  double g = 0.0;
#pragma unroll 1
  for (int base = 0; base < total; base += 64) {
#pragma unroll 1
    for (int q = base + lane; q < min(base + 64, total); q += 32) {
      int l = 0;                                   // the last lane whose blocks start at or before q
#pragma unroll
      for (int step2 = 16; step2 > 0; step2 >>= 1)
        if (G.before[l + step2] <= q) l += step2;
      const int i = q - G.before[l];
      const uint32_t key = Q.key[b + l];
      const U4 v = sub_block(seed, step, chan, Q.table[b + l], SUB_CALL_GAMMA, i, (long long)(key >> 12), int(key & 0xFFFu));
      G.x[0][q - base] = dlog(u01_open(v.x, v.y));
      if (2 * i + 1 < G.ne[l]) G.x[1][q - base] = dlog(u01_open(v.z, v.w));
    }
    __syncwarp();
    for (int q = max(before, base); q < min(before + ((ne + 1) >> 1), base + 64); ++q) {
      g = g - G.x[0][q - base];
      if (2 * (q - before) + 1 < ne) g = g - G.x[1][q - base];
    }
    __syncwarp();
  }
  return g;
}

// o_chan may be null (not written); a row whose offset is negative has no place in the output and is skipped
__global__ void __launch_bounds__(SUB_ROWS_PER_BLOCK * 32) k_substep_emit(CrvLookup L, CrvSubstepRows R, uint32_t seed,
                                                                          long long nrows, RowSel sel,
                                                                          const long long* __restrict__ offset,
                                                                          const long long* __restrict__ total,
                                                                          long long cap, int64_t* __restrict__ o_step,
                                                                          int64_t* __restrict__ o_chan,
                                                                          double* __restrict__ o_time,
                                                                          Status* status) {
  __shared__ SubQueue<double> queue[SUB_ROWS_PER_BLOCK];
  __shared__ SubGamma gamma[SUB_ROWS_PER_BLOCK];
  SubQueue<double>& Q = queue[warp_in_block()];
  if (*total > cap) return;                                    // reported by the capacity check
  seed = sel_seed(sel, seed);
  nrows = sel_nrows(sel, nrows);
  const long long warps = (long long)gridDim.x * SUB_ROWS_PER_BLOCK;
  for (long long r = (long long)blockIdx.x * SUB_ROWS_PER_BLOCK + warp_in_block(); r < nrows; r += warps) {
    if (!sel_row(sel, r) || offset[r] < 0) continue;          // warp-uniform
    long long nsub;
    if (!row_ok(R, r, &nsub, status)) continue;               // warp-uniform
    const long long step = R.step[r], chan = R.chan[r];
    const SubRow w = sub_row(L, R, r, nsub);
    const double t0 = R.t0[r], dt = R.t1[r] - t0;
    auto emit = [&](bool on, int q, long long o) {
      double tt = 0.0;
      int ne = 0;
      if (on) {
        o_step[o] = step;
        if (o_chan) o_chan[o] = chan;
        const uint32_t key = Q.key[q];
        tt = Q.at[q] + arrival_delay(L, seed, step, chan, (long long)(key >> 12), Q.table[q], Q.bin[q], int(key & 0xFFFu), &ne);
        if (ne > SUB_MAX_EMISSIONS) {
          set_flag(status, CRV_ST_LIMIT);
          ne = 0;
        }
      }
      if (L.fiber_decay_time > 0.0) {
        const double g = emission_sum(gamma[warp_in_block()], Q, q - lane_id(), seed, step, chan, ne);
        if (ne > 0) tt = tt + g * L.fiber_decay_time;
      }
      if (on) o_time[o] = tt;
    };
    const uint16_t* const kept = kept_row(sel, r);
    long long o = offset[r];
    int c = 0;
    for (long long k0 = 0; k0 < nsub; k0 += 32) {
      const long long k = k0 + lane_id();
      SubBins S;
      S.bin[0] = S.bin[1] = S.bin[2] = -1;
      S.frac = 0.0;
      int a[3] = {0, 0, 0};
      if (k < nsub) {
        S = substep_bins(L, w, k);
        const bool drawn = kept_counts(kept, sel.nkept, int(k), S.bin, a);
#pragma unroll
        for (int tb = 0; tb < 3; ++tb)
          if (!drawn && S.bin[tb] >= 0) {
            long long x = arrivals(L, R, seed, r, step, chan, k, tb, S.bin[tb], S.z);
            a[tb] = x >= SUB_MAX_ARRIVALS ? 0 : int(x);
          }
      }
      queue_chunk(Q, c, o, a, S.bin, uint32_t(k), t0 + dt * S.frac, k0 + 32 >= nsub, emit);
    }
  }
}

// ---- FP32-mixed variant: geometry, arrival draws and delays in FP32 (24-bit uniforms), edges staged as FP32 in
// shared memory, absolute photon times FP64 (row start time + FP32 offset).  Same keyed counters as the FP64 path,
// different numbers from them; the results agree with the FP64 path statistically.

struct EdgesF {
  const float* e[7];
  const float* cphi;
  const float* cth;
  int n[7];
};

// stage the edges (and cos of the phi / theta edges) of L as FP32 in shared memory; returns the views
__device__ __forceinline__ EdgesF stage_edges_f(const CrvLookup& L, float* sm) {
  EdgesF E;
  int o = 0;
  for (int i = 0; i < 7; ++i) {
    E.n[i] = L.nedges[i];
    for (int j = threadIdx.x; j < L.nedges[i]; j += blockDim.x) sm[o + j] = float(L.edges[i][j]);
    E.e[i] = sm + o;
    o += L.nedges[i];
  }
  for (int j = threadIdx.x; j < L.nedges[5]; j += blockDim.x) sm[o + j] = float(L.cos_phi_edges[j]);
  E.cphi = sm + o;
  o += L.nedges[5];
  for (int j = threadIdx.x; j < L.nedges[4]; j += blockDim.x) sm[o + j] = L.cos_theta_edges ? float(L.cos_theta_edges[j]) : 0.f;
  E.cth = sm + o;
  __syncthreads();
  return E;
}

__device__ __forceinline__ int find_bin_f(const float* e, int ne, float v) {
  if (!(v >= e[0]) || !(v <= e[ne - 1])) return -1;
  if (v == e[0]) return 0;
  int lo = 0, hi = ne;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (e[mid] < v) lo = mid + 1; else hi = mid;
  }
  return lo - 1;
}

__device__ __forceinline__ int find_bin_cos_f(const float* ce, int ne, float c) {
  if (!(c <= ce[0]) || !(c >= ce[ne - 1])) return -1;
  if (c == ce[0]) return 0;
  int lo = 0, hi = ne;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (ce[mid] > c) lo = mid + 1; else hi = mid;
  }
  return lo - 1;
}

// 32-bit counts throughout: conversions between 64-bit integers and floats run on the FP64 pipe.  Where the inversion's first
// term is below FP32's normal range (means from 88 on, from 63 at q = 1/2, up to 256; as 0 it would never let a draw end
// before n) FP64 draws from the same words: with WIDE; else -1 is returned.
template <bool WIDE>
__device__ __forceinline__ int binomial_f(int n, float p, const U4& w) {
  if (n <= 0 || !(p > 0.f)) return 0;
  if (p >= 1.f) return n;
  const bool flip = p > 0.5f;
  const float q = flip ? 1.f - p : p;
  const float mean = float(n) * q;
  int k;
  if (mean > 256.f) {
    float z0, z1;
    Math<float>::normal_pair(w, &z0, &z1);
    const float x = rintf(mean + sqrtf(mean * (1.f - q)) * z0);
    k = x < 0.f ? 0 : (x > float(n) ? n : int(x));
  } else {
    float u = f01(w.x);
    const float s = q / (1.f - q);
    const float a = float(n + 1) * s;
    float r = __expf(float(n) * log1pf(-q));
    if (r < 1.17549435e-38f) {
      if constexpr (WIDE) return int(binomial_64(n, f2d(p), w));
      else return -1;
    }
    k = 0;
    while (u > r && k < n) {
      u = u - r;
      k += 1;
      r = r * (a / float(k) - s);
    }
  }
  return flip ? n - k : k;
}

// a row in FP32: local start, step vector, and per-row constants
struct RowF {
  float s[3], d[3], dev, mu, dt, inv_nsub;
  double t0;
  long long step, chan;
  int nsub, bb, bth, n[3];
  int cy, cz;                  // y and z bin of every substep when the row's ends share one, else -2
};

// double -> float on the integer pipe (truncating; zeros by their bits): every lane of the warp converts the same
// row values, and an FP64-pipe conversion costs a whole warp slot of GB300's FP64 pipe
__device__ __forceinline__ float to_f(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  if ((b << 1) == 0ull) return __uint_as_float(uint32_t(b >> 32));
  return d2f_trunc(x);
}

__device__ __forceinline__ RowF load_row_f(const CrvSubstepRows& R, const EdgesF& E, long long r) {
  RowF w;
  for (int x = 0; x < 3; ++x) {
    w.s[x] = to_f(R.s[3 * r + x]);
    w.d[x] = to_f(R.d[3 * r + x]);
  }
  w.dev = to_f(R.dev[r]);
  w.mu = R.mu ? to_f(R.mu[r]) : 0.f;
  w.t0 = R.t0[r];
  w.dt = to_f(R.t1[r] - R.t0[r]);
  w.nsub = int(R.nsub[r]);                                     // at most 2^20 (checked by row_ok)
  w.inv_nsub = 1.f / float(w.nsub);
  w.step = R.step[r];
  w.chan = R.chan[r];
  const long long n3[3] = {R.n_scint[r], R.n_ck_s[r], R.n_ck_f[r]};
  for (int t = 0; t < 3; ++t) w.n[t] = n3[t] < 0 ? 0 : (n3[t] > 0x7FFFFFFFll ? 0x7FFFFFFF : int(n3[t]));
  // a coordinate runs from one end to the other without leaving their interval (rounding is monotone), and the bins do
  // not decrease along it
  const int y0 = find_bin_f(E.e[1], E.n[1], w.s[1]), y1 = find_bin_f(E.e[1], E.n[1], w.s[1] + w.d[1]);
  const int z0 = find_bin_f(E.e[2], E.n[2], w.s[2]), z1 = find_bin_f(E.e[2], E.n[2], w.s[2] + w.d[2]);
  w.cy = y0 == y1 && y0 >= 0 ? y0 : -2;
  w.cz = z0 == z1 && z0 >= 0 ? z0 : -2;
  w.bb = find_bin_f(E.e[3], E.n[3], to_f(R.beta[r]));
  w.bth = R.theta ? find_bin_f(E.e[4], E.n[4], to_f(R.theta[r])) : find_bin_cos_f(E.cth, E.n[4], to_f(R.cos_theta[r]));
  return w;
}

struct GeoF {
  float ht, hw, hl, half_sep, hrx, hry, fr, cr;
};

__device__ __forceinline__ GeoF geo_f(const CrvLookup& L) {
  return {float(L.half_thickness), float(L.half_width), float(L.half_length), float(L.fiber_separation / 2.0),
          float(L.hole_radius_x), float(L.hole_radius_y), float(L.fiber_radius), float(L.corner_radius)};
}

__device__ __forceinline__ void substep_bins_f(const GeoF& g, const EdgesF& E, const RowF& w, int k, int bin[3],
                                               float* z_out, float* frac_out) {
  const float frac = (float(k) + 0.5f) * w.inv_nsub;
  const float x = fmaf(w.d[0], frac, w.s[0]), y = fmaf(w.d[1], frac, w.s[1]), z = fmaf(w.d[2], frac, w.s[2]);
  const float ax = fabsf(x), ay = fabsf(y);
  const bool inz = fabsf(z) < g.hl;
  bool insc = ax < g.ht && ay < g.hw && inz;
  // hole and fibres only inside their bounding boxes, as in substep_bins
  const float hy = ay - g.half_sep;
  if (insc && !(g.hrx > 0.f && g.hry > 0.f && (ax >= g.hrx || fabsf(hy) >= g.hry))) {
    const float ex = ax / g.hrx, ey = hy / g.hry;
    insc = ex * ex + ey * ey >= 1.f;
  }
  const float cx = g.ht - g.cr, cy = g.hw - g.cr;
  if (insc && ax > cx && ay > cy) {
    const float qx = ax - cx, qy = ay - cy;
    if (sqrtf(qx * qx + qy * qy) > g.cr) insc = false;
  }
  const int ny = E.n[1] - 1, nz = E.n[2] - 1, nb = E.n[3] - 1, nth = E.n[4] - 1, nph = E.n[5] - 1, nr = E.n[6] - 1;
  bin[0] = bin[1] = bin[2] = -1;
  const int bz = w.cz > -2 ? w.cz : find_bin_f(E.e[2], E.n[2], z);
  if (insc && bz >= 0) {
    const int bx = find_bin_f(E.e[0], E.n[0], ax), by = w.cy > -2 ? w.cy : find_bin_f(E.e[1], E.n[1], y);
    if (bx >= 0 && by >= 0) {
      bin[0] = bz + by * nz + bx * ny * nz;
      if (w.bb >= 0) bin[1] = w.bb + bz * nb + by * nz * nb + bx * ny * nz * nb;
    }
  }
  const float y0 = y + g.half_sep, y1 = y - g.half_sep;
  if (inz && !insc && ax <= g.fr && (fabsf(y0) <= g.fr || fabsf(y1) <= g.fr)) {
    const float r0 = sqrtf(x * x + y0 * y0), r1 = sqrtf(x * x + y1 * y1);
    const bool in0 = r0 <= g.fr, in1 = r1 <= g.fr;
    if ((in0 || in1) && w.bb >= 0 && w.bth >= 0 && bz >= 0) {
      const float ry = in1 ? y1 : y0, rr = in1 ? r1 : r0;
      const float norm = sqrtf(w.d[0] * w.d[0] + w.d[1] * w.d[1]) * rr;
      float c = 1.f;
      if (norm > 0.f) c = fminf(1.f, fmaxf(-1.f, (w.d[0] * x + w.d[1] * ry) / norm));
      const int bph = find_bin_cos_f(E.cphi, E.n[5], c), br = find_bin_f(E.e[6], E.n[6], rr);
      if (bph >= 0 && br >= 0) bin[2] = bz + br * nz + bph * nr * nz + w.bth * nph * nr * nz + w.bb * nth * nph * nr * nz;
    }
  }
  *z_out = z;
  *frac_out = frac;
}

template <bool WIDE>
__device__ __forceinline__ int arrivals_f(const CrvLookup& L, const CrvSubstepRows& R, const RowF& w, uint32_t seed,
                                          int k, int tb, int bin, float z) {
  float pr = L.table[tb].prob[bin] * w.dev;
  if (R.mu) pr = pr * __expf(-w.mu * z);
  pr = fminf(pr, 1.f);
  return binomial_f<WIDE>(w.n[tb], pr, sub_block(seed, w.step, w.chan, tb, SUB_CALL_BINOMIAL, 0, k, 0));
}

// offset of arrival j from the row start time (FP32: substep time, delay, fibre decay)
__device__ __forceinline__ float arrival_offset_f(const CrvLookup& L, float decay, uint32_t seed, const RowF& w,
                                                  int k, int tb, int bin, int j, float frac, Status* status) {
  const CrvLookupTable& T = L.table[tb];
  const U4 v = sub_block(seed, w.step, w.chan, tb, SUB_CALL_PHOTON, 0, k, j);
  float off = w.dt * frac + float(first_reaching(T.delays, T.nbins, bin, T.ndelay,
                                                 sum_threshold(f01(v.x) * float(T.delay_sum[bin]))));
  if (decay > 0.f) {
    const int ne = first_reaching(T.emis, T.nbins, bin, T.nemis, sum_threshold(f01(v.z) * float(T.emis_sum[bin])));
    if (ne > SUB_MAX_EMISSIONS) {
      set_flag(status, CRV_ST_LIMIT);
    } else if (ne > 0) {
      float g = 0.f;
      for (int i = 0; i < ne; i += 2) {
        const U4 q = sub_block(seed, w.step, w.chan, tb, SUB_CALL_GAMMA, i >> 1, k, j);
        g -= __logf(f01_open(q.x));
        if (i + 1 < ne) g -= __logf(f01_open(q.z));
      }
      off += g * decay;
    }
  }
  return off;
}

// arrivals of row r, by the warp; -1 when one of its draws needs FP64 (not with WIDE)
template <bool WIDE>
__device__ __forceinline__ long long count_row_f(const CrvLookup& L, const CrvSubstepRows& R, const EdgesF& E, const GeoF& g,
                                                 uint32_t seed, const RowSel& sel, long long r, Status* status) {
  long long nsub;
  long long tot = 0;
  int low = 0;
  if (row_ok(R, r, &nsub, status)) {
    const RowF w = load_row_f(R, E, r);
    uint16_t* const kept = kept_row(sel, r);
    int sum = 0;
    for (int k = lane_id(); k < w.nsub; k += 32) {
      int bin[3];
      float z, frac;
      substep_bins_f(g, E, w, k, bin, &z, &frac);
      int in_or_fibre = 0, ck = 0;
      for (int tb = 0; tb < 3; ++tb)
        if (bin[tb] >= 0) {
          int a = arrivals_f<WIDE>(L, R, w, seed, k, tb, bin[tb], z);
          if (!WIDE) low = min(low, a);
          if (a >= SUB_MAX_ARRIVALS) { set_flag(status, CRV_ST_LIMIT); a = 0; }
          sum += a;
          if (tb == 1) ck = a; else in_or_fibre = a;
        }
      keep_counts(kept, sel.nkept, k, in_or_fibre, ck);
    }
    tot = sum;
  }
  tot = warp_sum(tot);
  return !WIDE && __any_sync(0xffffffffu, low < 0) ? -1 : tot;
}

__global__ void __launch_bounds__(SUB_ROWS_PER_BLOCK * 32) k_substep_count_f32(CrvLookup L, CrvSubstepRows R,
                                                                               uint32_t seed, long long nrows,
                                                                               RowSel sel,
                                                                               long long* __restrict__ count,
                                                                               Status* status) {
  extern __shared__ float edges_sm[];
  const EdgesF E = stage_edges_f(L, edges_sm);
  const GeoF g = geo_f(L);
  seed = sel_seed(sel, seed);
  nrows = sel_nrows(sel, nrows);
  const long long warps = (long long)gridDim.x * SUB_ROWS_PER_BLOCK;
  for (long long r = (long long)blockIdx.x * SUB_ROWS_PER_BLOCK + warp_in_block(); r < nrows; r += warps) {
    if (!sel_row(sel, r)) continue;                          // warp-uniform
    const long long tot = count_row_f<false>(L, R, E, g, seed, sel, r, status);
    if (lane_id() == 0) count[r] = tot;
  }
}

// The rows that k_substep_count_f32 left at -1, counted with FP64 draws where they are needed.  Ordinary tables have none
// (means below 5), and the FP64 draw among the others takes registers from every warp: 200,000 rows 1.21 -> 1.34 ms, as a
// call for a whole row 1.29; marked rows and this launch, a lane per row until one is found, 1.21 -> 1.23 + 0.01 ms.
__global__ void __launch_bounds__(SUB_ROWS_PER_BLOCK * 32) k_substep_count_wide(CrvLookup L, CrvSubstepRows R,
                                                                                uint32_t seed, long long nrows,
                                                                                RowSel sel,
                                                                                long long* __restrict__ count,
                                                                                Status* status) {
  extern __shared__ float edges_sm[];
  seed = sel_seed(sel, seed);
  nrows = sel_nrows(sel, nrows);
  const long long tiles = (nrows + blockDim.x - 1) / blockDim.x;
  for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    const long long r0 = t * blockDim.x + threadIdx.x;
    const bool mine = r0 < nrows && sel_row(sel, r0) && count[r0] < 0;
    if (!__syncthreads_or(mine)) continue;
    const EdgesF E = stage_edges_f(L, edges_sm);
    const GeoF g = geo_f(L);
    for (unsigned m = __ballot_sync(0xffffffffu, mine); m; m &= m - 1u) {
      const long long r = r0 - lane_id() + __ffs(m) - 1;
      const long long tot = count_row_f<true>(L, R, E, g, seed, sel, r, status);
      if (lane_id() == 0) count[r] = tot;
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(SUB_ROWS_PER_BLOCK * 32) k_substep_emit_f32(CrvLookup L, CrvSubstepRows R,
                                                                              uint32_t seed, long long nrows,
                                                                              RowSel sel,
                                                                              const long long* __restrict__ offset,
                                                                              const long long* __restrict__ total,
                                                                              long long cap,
                                                                              int64_t* __restrict__ o_step,
                                                                              int64_t* __restrict__ o_chan,
                                                                              double* __restrict__ o_time,
                                                                              Status* status) {
  extern __shared__ float edges_sm[];
  __shared__ SubQueue<float> queue[SUB_ROWS_PER_BLOCK];
  SubQueue<float>& Q = queue[warp_in_block()];
  if (*total > cap) return;                                    // block-uniform, before the staging barrier
  const EdgesF E = stage_edges_f(L, edges_sm);
  const GeoF g = geo_f(L);
  const float decay = float(L.fiber_decay_time);
  seed = sel_seed(sel, seed);
  nrows = sel_nrows(sel, nrows);
  const long long warps = (long long)gridDim.x * SUB_ROWS_PER_BLOCK;
  for (long long r = (long long)blockIdx.x * SUB_ROWS_PER_BLOCK + warp_in_block(); r < nrows; r += warps) {
    if (!sel_row(sel, r) || offset[r] < 0) continue;          // warp-uniform
    long long nsub;
    if (!row_ok(R, r, &nsub, status)) continue;
    const RowF w = load_row_f(R, E, r);
    auto emit = [&](bool on, int q, long long o) {
      if (!on) return;
      o_step[o] = w.step;
      if (o_chan) o_chan[o] = w.chan;
      const uint32_t key = Q.key[q];
      o_time[o] = w.t0 + f2d(arrival_offset_f(L, decay, seed, w, int(key >> 12), Q.table[q], Q.bin[q], int(key & 0xFFFu),
                                              Q.at[q], status));
    };
    const uint16_t* const kept = kept_row(sel, r);
    long long o = offset[r];
    int c = 0;
    for (int k0 = 0; k0 < w.nsub; k0 += 32) {
      const int k = k0 + lane_id();
      int bin[3] = {-1, -1, -1};
      float z = 0.f, frac = 0.f;
      int a[3] = {0, 0, 0};
      if (k < w.nsub) {
        substep_bins_f(g, E, w, k, bin, &z, &frac);
        const bool drawn = kept_counts(kept, sel.nkept, k, bin, a);
#pragma unroll
        for (int tb = 0; tb < 3; ++tb)
          if (!drawn && bin[tb] >= 0) {
            a[tb] = arrivals_f<true>(L, R, w, seed, k, tb, bin[tb], z);
            if (a[tb] >= SUB_MAX_ARRIVALS) a[tb] = 0;
          }
      }
      queue_chunk(Q, c, o, a, bin, uint32_t(k), frac, k0 + 32 >= w.nsub, emit);
    }
  }
}

// FP32 edges of a table in shared memory: up to EDGES_MOST bytes are taken.  The emission holds its queues beside them, and
// what does not fit the ordinary 48 KB together needs the kernel's opt-in.
constexpr size_t EDGES_MOST = 48 * 1024;
static size_t edges_smem(const CrvLookup& L) {
  int nedge = 0;
  for (int i = 0; i < 7; ++i) nedge += L.nedges[i];
  return sizeof(float) * size_t(nedge + L.nedges[5] + L.nedges[4]);
}
static cudaError_t allow_edges(size_t bytes) {
  if (bytes + sizeof(SubQueue<float>) * SUB_ROWS_PER_BLOCK <= 48 * 1024) return cudaSuccess;
  return allow_dynamic_smem(k_substep_emit_f32);
}

static void launch_count_f32(const CrvLookup& L, const CrvSubstepRows& R, uint32_t seed, long long nrows, const RowSel& sel,
                             long long* count, Status* status, unsigned grid, cudaStream_t s) {
  constexpr int TH = SUB_ROWS_PER_BLOCK * 32;
  {
    crv::Mark mark_("k_substep_count", s);
    k_substep_count_f32<<<grid, TH, edges_smem(L), s>>>(L, R, seed, nrows, sel, count, status);
  }
  const long long blocks = (nrows + TH - 1) / TH;
  crv::Mark mark_("k_substep_count_wide", s);
  k_substep_count_wide<<<(unsigned)(blocks < (long long)grid ? blocks : (long long)grid), TH, edges_smem(L), s>>>(
      L, R, seed, nrows, sel, count, status);
}

struct SubWs {
  long long *count, *offset, *parts, *total;
  uint16_t* kept;
};

// least: the bytes without the kept counts, which come last
static SubWs sub_layout(char* base, long long n, size_t* bytes, size_t* least) {
  size_t off = 0;
  auto take = [&](long long cnt) {
    off = (off + 255) & ~size_t(255);
    long long* p = base ? reinterpret_cast<long long*>(base + off) : nullptr;
    off += size_t(cnt > 0 ? cnt : 1) * sizeof(long long);
    return p;
  };
  SubWs w;
  w.count = take(n);
  w.offset = take(n);
  w.parts = take(scan_parts_len(n) + 1);
  w.total = take(1);
  *least = ((off + 255) & ~size_t(255)) + 256;
  w.kept = reinterpret_cast<uint16_t*>(take(n * (SUB_KEPT / 4)));
  *bytes = off + 256;
  return w;
}

}  // namespace crv

using namespace crv;

extern "C" int64_t crv_substeps_workspace(int64_t nrows) {
  if (nrows < 0) return -1;
  size_t b = 0, least = 0;
  sub_layout(nullptr, nrows, &b, &least);
  return (int64_t)b;
}

extern "C" int crv_substep_photons(const CrvLookup* L, uint32_t seed, const CrvSubstepRows* rows, int64_t nrows,
                                   int64_t* o_step, int64_t* o_chan, double* o_time, int64_t cap, int64_t* n_out_dev,
                                   void* workspace, int64_t workspace_bytes, void* stream, CrvStatus* status_dev) {
  if (!L || !rows || !n_out_dev || !status_dev || nrows < 0 || cap < 0) return CRV_ERR_ARG;
  for (int i = 0; i < 7; ++i)
    if (!L->edges[i] || L->nedges[i] < 2) return CRV_ERR_ARG;
  if (!L->cos_phi_edges || L->precision < 0 || L->precision > 1) return CRV_ERR_ARG;
  for (int t = 0; t < 3; ++t) {
    const CrvLookupTable& T = L->table[t];
    if (!T.prob || !T.delays || !T.delay_sum || !T.emis || !T.emis_sum || T.ndelay < 1 || T.nemis < 1) return CRV_ERR_ARG;
  }
  const int nb = L->nedges[3] - 1, nx = L->nedges[0] - 1, ny = L->nedges[1] - 1, nz = L->nedges[2] - 1;
  const int nth = L->nedges[4] - 1, nph = L->nedges[5] - 1, nr = L->nedges[6] - 1;
  if ((long long)L->table[0].nbins < (long long)nx * ny * nz || (long long)L->table[1].nbins < (long long)nx * ny * nz * nb ||
      (long long)L->table[2].nbins < (long long)nb * nth * nph * nr * nz)
    return CRV_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (nrows == 0) {
    if (cudaMemsetAsync(n_out_dev, 0, sizeof(long long), s) != cudaSuccess) return CRV_ERR_CUDA;
    return CRV_OK;
  }
  if (!rows->s || !rows->d || !rows->t0 || !rows->t1 || !rows->beta || !rows->dev || !rows->nsub || !rows->step ||
      !rows->chan || !rows->n_scint || !rows->n_ck_s || !rows->n_ck_f)
    return CRV_ERR_ARG;
  if (!rows->theta && (!rows->cos_theta || !L->cos_theta_edges)) return CRV_ERR_ARG;
  size_t whole = 0, least = 0;
  sub_layout(nullptr, nrows, &whole, &least);
  if (!workspace || (long long)least > workspace_bytes) return CRV_ERR_ARG;
  // counts kept for as many substeps of each row as there is room for (the others are drawn again)
  const long long room = (workspace_bytes - (long long)least) / (2 * nrows);
  const int nkept = int(room < SUB_KEPT ? room : SUB_KEPT) & ~31;
  char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255));
  SubWs w = sub_layout(base, nrows, &whole, &least);
  Status* S = reinterpret_cast<Status*>(status_dev);
  const long long blocks = (nrows + SUB_ROWS_PER_BLOCK - 1) / SUB_ROWS_PER_BLOCK;
  const long long maxb = (long long)device_info().sms * 8;
  const unsigned grid = (unsigned)(blocks < maxb ? blocks : maxb);
  const bool f32 = L->precision == 1;
  const RowSel sel{nullptr, nullptr, nullptr, 0, w.kept, nkept};
  const size_t esm = edges_smem(*L);
  if (f32 && esm > EDGES_MOST) return CRV_ERR_ARG;
  if (f32 && allow_edges(esm) != cudaSuccess) return CRV_ERR_CUDA;
  if (f32) {
    launch_count_f32(*L, *rows, seed, nrows, sel, w.count, S, grid, s);
  } else {
    crv::Mark mark_("k_substep_count", s);
    k_substep_count<<<grid, SUB_ROWS_PER_BLOCK * 32, 0, s>>>(*L, *rows, seed, nrows, sel, w.count, S);
  }
  if (cudaGetLastError() != cudaSuccess) return CRV_ERR_CUDA;
  if (exclusive_scan(column(w.count, w.offset), nrows, nullptr,
                     scan_end(w.total, n_out_dev).check(S, CRV_NEED_PHOTONS_OUT, cap), w.parts, s) != cudaSuccess)
    return CRV_ERR_CUDA;
  if (f32) {
    crv::Mark mark_("k_substep_emit", s);
    k_substep_emit_f32<<<grid, SUB_ROWS_PER_BLOCK * 32, esm, s>>>(*L, *rows, seed, nrows, sel, w.offset,
                                                                 w.total, cap,
                                                                 o_step, o_chan, o_time, S);
  } else {
    crv::Mark mark_("k_substep_emit", s);
    k_substep_emit<<<grid, SUB_ROWS_PER_BLOCK * 32, 0, s>>>(*L, *rows, seed, nrows, sel, w.offset, w.total,
                                                            cap, o_step,
                                                            o_chan, o_time, S);
  }
  if (cudaGetLastError() != cudaSuccess) return CRV_ERR_CUDA;
  return CRV_OK;
}

// ---- row preparation (photons.iter_rows) -----------------------------------------------------------------------------

namespace crv {

constexpr uint32_t ST_LROWS = 8;
constexpr double LROW_PRECISION_MM = 0.1;
constexpr double AMU_MEV = 931.49410242;       // atomic mass unit (CODATA 2018)

// mass [MeV] and charge [e] of a particle code: table lookup, ions 100ZZZAAAI decoded, unknown (0, 0)
__device__ __forceinline__ void particle(const CrvLookupGroup& G, long long pdg, double* m, double* q) {
  int lo = 0, hi = G.npdg;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (G.pdg_code[mid] < pdg) lo = mid + 1; else hi = mid;
  }
  if (lo < G.npdg && G.pdg_code[lo] == pdg) {
    *m = G.pdg_mass[lo];
    *q = G.pdg_charge[lo];
    return;
  }
  const long long a = pdg < 0 ? -pdg : pdg;
  if (a >= 1000000000ll) {
    *m = double((a / 10) % 1000) * AMU_MEV;
    *q = double((a / 10000) % 1000) * (pdg < 0 ? -1.0 : 1.0);
  } else {
    *m = 0.0;
    *q = 0.0;
  }
}

// Cherenkov photons per mm: linear in beta from (0, 0) through the map, flat beyond its end, times |charge|
__device__ __forceinline__ double cerenkov_per_mm(const double* __restrict__ map, int n, double beta, double q) {
  double x0 = 0.0, y0 = 0.0, v;
  int j = 0;
  while (j < n && map[2 * j] <= beta) { x0 = map[2 * j]; y0 = map[2 * j + 1]; ++j; }
  if (beta < 0.0) v = 0.0;
  else if (j == n) v = n > 0 ? map[2 * (n - 1) + 1] : 0.0;
  else v = (map[2 * j + 1] - y0) / (map[2 * j] - x0) * (beta - x0) + y0;
  return v * fabs(q);
}

// photons per substep: rint(draw / nsub) of Gauss(avg, sqrt avg) for avg > 10, else Poisson(avg) by inversion
__device__ __forceinline__ long long per_substep(double avg, long long nsub, const U4& w) {
  double x;
  if (avg > 10.0) {
    double z0, z1;
    Math<double>::normal_pair(w, &z0, &z1);
    x = avg + sqrt(avg) * z0;
  } else {
    const double lam = avg > 0.0 ? avg : 0.0;
    const double u = u01(w.x, w.y);
    double p = dexp(-lam), F = p;
    int k = 0;
    while (u >= F && k < 200) {
      k += 1;
      p = p * lam / double(k);
      F = F + p;
    }
    x = double(k);
  }
  const double n = rint(x / double(nsub));
  return n > 0.0 ? (long long)n : 0;
}

__device__ __forceinline__ bool in_lgroup(const CrvLookupGroup& G, const CrvLookupSteps& S, long long i) {
  const int b = S.bar[i];
  return b >= 0 && b < G.nbars && G.in_group[b] && isfinite(S.t0[i]) && isfinite(S.t1[i]);
}

__global__ void k_lrows_flag(CrvLookupGroup G, CrvLookupSteps S, long long n, int32_t* __restrict__ flag) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    flag[i] = in_lgroup(G, S, i) ? 1 : 0;
}

// The rows of step i (a step of group G) for each simulated SiPM: row index(si, output channel) of O
template <typename Index>
__device__ __forceinline__ void lrows_of_step(const CrvLookupGroup& G, const CrvLookupSteps& S, uint32_t seed, long long i,
                                              const CrvSubstepRowsOut& O, Index index) {
  const int nsim = G.reflector == 0 ? 4 : 2;
  const int b = S.bar[i];
  const double* c = G.center + 3 * b;
  const double ws[3] = {S.x0[i] - c[0], S.y0[i] - c[1], S.z0[i] - c[2]};
  const double we[3] = {S.x1[i] - c[0], S.y1[i] - c[1], S.z1[i] - c[2]};
  double sl[3], el[3];
  for (int k = 0; k < 3; ++k) {
    const int ax = G.l2w[3 * b + k];
    sl[k] = ws[ax];
    el[k] = we[ax];
  }
  if (G.reflector < 0) { sl[2] = -sl[2]; el[2] = -el[2]; }
  double m, q;
  particle(G, S.pdg[i], &m, &q);
  const double p0 = sqrt(S.px0[i] * S.px0[i] + S.py0[i] * S.py0[i] + S.pz0[i] * S.pz0[i]);
  const double e = 0.5 * (sqrt(p0 * p0 + m * m) + sqrt(S.p1[i] * S.p1[i] + m * m));
  double beta = 1.0;
  if (m > 0.0) {
    const double g = e / m;
    double b2 = 1.0 - 1.0 / (g * g);
    b2 = b2 < 0.0 ? 0.0 : (b2 > 1.0 ? 1.0 : b2);
    beta = sqrt(b2);
  }
  const double avg_s = G.yield[b] * S.edep[i];
  const double avg_cs = cerenkov_per_mm(G.ck_scint, G.nck_scint, beta, q) * S.len[i];
  const double avg_cf = cerenkov_per_mm(G.ck_fiber, G.nck_fiber, beta, q) * S.len[i];
  const double k = G.speed_k[b];
  for (int si = 0; si < nsim; ++si) {
    const int s = G.reflector == 0 ? si : 2 * si;
    double a[3] = {sl[0], sl[1], sl[2]}, bb[3] = {el[0], el[1], el[2]};
    if (s == 1 || s == 3) { a[2] = -a[2]; bb[2] = -bb[2]; }
    if (s == 2 || s == 3) { a[1] = -a[1]; bb[1] = -bb[1]; }
    const double d[3] = {bb[0] - a[0], bb[1] - a[1], bb[2] - a[2]};
    const double dl = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
    double ct = 1.0;
    if (dl > 0.0) {
      ct = d[2] / dl;
      ct = ct < -1.0 ? -1.0 : (ct > 1.0 ? 1.0 : ct);
    }
    long long nsub = (long long)(dl / LROW_PRECISION_MM);
    nsub = nsub > 1 ? nsub : 1;
    const long long chan_dev = 4ll * b + s;
    const long long chan_out = 4ll * b + (G.reflector < 0 ? s + 1 : s);
    const long long o = index(si, chan_out);
    for (int x = 0; x < 3; ++x) {
      O.s[3 * o + x] = a[x];
      O.d[3 * o + x] = d[x];
    }
    O.t0[o] = S.t0[i] + k * (a[2] + G.half_length);
    O.t1[o] = S.t1[i] + k * (bb[2] + G.half_length);
    O.nsub[o] = nsub;
    O.beta[o] = beta;
    O.cos_theta[o] = ct;
    O.dev[o] = G.dev[chan_dev];
    O.mu[o] = G.mu[b];
    O.step[o] = i;
    O.chan[o] = chan_out;
    const uint32_t lo = uint32_t(i), hi = uint32_t((unsigned long long)i >> 32);
    O.n_scint[o] = per_substep(avg_s, nsub, philox(lo, hi, w2_of(ST_LROWS, 0, 0, 0, uint32_t(chan_dev)), 0u, seed, 0u));
    O.n_ck_s[o] = per_substep(avg_cs, nsub, philox(lo, hi, w2_of(ST_LROWS, 1, 0, 0, uint32_t(chan_dev)), 0u, seed, 0u));
    O.n_ck_f[o] = per_substep(avg_cf, nsub, philox(lo, hi, w2_of(ST_LROWS, 2, 0, 0, uint32_t(chan_dev)), 0u, seed, 0u));
  }
}

__global__ void k_lrows_fill(CrvLookupGroup G, CrvLookupSteps S, uint32_t seed, long long n,
                             const long long* __restrict__ rank, const long long* __restrict__ total,
                             CrvSubstepRowsOut O) {
  const long long ng = *total;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (!in_lgroup(G, S, i)) continue;
    const long long r0 = rank[i];
    lrows_of_step(G, S, seed, i, O, [&](int si, long long) { return (long long)si * ng + r0; });
  }
}

__global__ void k_lrows_count(const long long* __restrict__ total, int nsim, long long* __restrict__ n_rows) {
  *n_rows = *total * nsim;
}

}  // namespace crv

extern "C" int64_t crv_lookup_rows_workspace(int64_t nsteps) {
  if (nsteps < 0) return -1;
  size_t off = 0;
  auto take = [&](size_t bytes) { off = ((off + 255) & ~size_t(255)) + (bytes ? bytes : 1); };
  take(sizeof(int32_t) * nsteps);
  take(sizeof(long long) * nsteps);
  take(sizeof(long long) * (scan_parts_len(nsteps) + 1));
  take(sizeof(long long));
  return (int64_t)(off + 512);
}

extern "C" int crv_lookup_rows(const CrvLookupGroup* G, uint32_t seed, const CrvLookupSteps* st, int64_t nsteps,
                               CrvSubstepRowsOut* out, int64_t cap, int64_t* n_rows_dev, void* workspace,
                               int64_t workspace_bytes, void* stream, CrvStatus* status_dev) {
  if (!G || !st || !out || !n_rows_dev || !status_dev || nsteps < 0) return CRV_ERR_ARG;
  if (G->reflector < -1 || G->reflector > 1 || G->nbars < 1 || G->npdg < 0 || G->nck_scint < 0 || G->nck_fiber < 0)
    return CRV_ERR_ARG;
  if (!G->center || !G->l2w || !G->in_group || !G->yield || !G->speed_k || !G->mu || !G->dev ||
      (G->nck_scint && !G->ck_scint) || (G->nck_fiber && !G->ck_fiber) ||
      (G->npdg && (!G->pdg_code || !G->pdg_mass || !G->pdg_charge)))
    return CRV_ERR_ARG;
  const int nsim = G->reflector == 0 ? 4 : 2;
  if (cap < nsim * nsteps) return CRV_ERR_ARG;                 // every step of the group gives nsim rows
  cudaStream_t s = (cudaStream_t)stream;
  if (nsteps == 0) return cudaMemsetAsync(n_rows_dev, 0, sizeof(long long), s) == cudaSuccess ? CRV_OK : CRV_ERR_CUDA;
  if (!st->x0 || !st->y0 || !st->z0 || !st->x1 || !st->y1 || !st->z1 || !st->px0 || !st->py0 || !st->pz0 ||
      !st->p1 || !st->t0 || !st->t1 || !st->edep || !st->len || !st->bar || !st->pdg)
    return CRV_ERR_ARG;
  if (!out->s || !out->d || !out->t0 || !out->t1 || !out->beta || !out->cos_theta || !out->dev || !out->mu ||
      !out->nsub || !out->step || !out->chan || !out->n_scint || !out->n_ck_s || !out->n_ck_f)
    return CRV_ERR_ARG;
  if (crv_lookup_rows_workspace(nsteps) > workspace_bytes || !workspace) return CRV_ERR_ARG;
  char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255));
  size_t off = 0;
  auto take = [&](size_t bytes) {
    off = (off + 255) & ~size_t(255);
    char* p = base + off;
    off += bytes ? bytes : 1;
    return p;
  };
  int32_t* flag = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * nsteps));
  long long* rank = reinterpret_cast<long long*>(take(sizeof(long long) * nsteps));
  long long* parts = reinterpret_cast<long long*>(take(sizeof(long long) * (scan_parts_len(nsteps) + 1)));
  long long* total = reinterpret_cast<long long*>(take(sizeof(long long)));
  const long long blocks = (nsteps + 255) / 256, maxb = (long long)device_info().sms * 8;
  const unsigned grid = (unsigned)(blocks < maxb ? blocks : maxb);
  {
    crv::Mark mark_("k_lrows_flag", s);
    k_lrows_flag<<<grid, 256, 0, s>>>(*G, *st, nsteps, flag);
  }
  if (exclusive_scan(column(flag, rank), nsteps, nullptr, scan_end(total), parts, s) != cudaSuccess) return CRV_ERR_CUDA;
  {
    crv::Mark mark_("k_lrows_fill", s);
    k_lrows_fill<<<grid, 256, 0, s>>>(*G, *st, seed, nsteps, rank, total, *out);
  }
  {
    crv::Mark mark_("k_lrows_count", s);
    k_lrows_count<<<1, 1, 0, s>>>(total, nsim, reinterpret_cast<long long*>(n_rows_dev));
  }
  (void)status_dev;
  return cudaGetLastError() == cudaSuccess ? CRV_OK : CRV_ERR_CUDA;
}

// ---- the lookup-table model inside the resident chain ------------------------------------------------------------
//
// Rows are dense: row 4 i + c for step i and output channel c = chan & 3, one table of rows for every group; a row of
// no group (a SiPM the group does not simulate, a step of no group or with a non-finite time) has group -1.  The
// counts and the photons then run once per group over the rows of that group (RowSel), with that group's table.

namespace crv {

struct LGroups {
  CrvLookupGroup g[CRV_LOOKUP_CHAIN_GROUPS];
  int n;
};

// rows of every step of the batch; the first thread also writes the row bound and the parameter block's seed
__global__ void k_lrows_chain(CrvParams p, LGroups K, CrvLookupSteps S, const long long* __restrict__ nsteps_dev,
                              long long step_cap, CrvSubstepRowsOut O, int8_t* __restrict__ row_group,
                              long long* __restrict__ nrows, uint32_t* __restrict__ seed_dev) {
  long long n = *nsteps_dev;
  n = n < step_cap ? (n > 0 ? n : 0) : step_cap;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *nrows = 4 * n;
    *seed_dev = p.seed;
  }
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    for (int c = 0; c < 4; ++c) row_group[4 * i + c] = -1;
    int gi = -1;
    for (int k = 0; k < K.n && gi < 0; ++k)
      if (in_lgroup(K.g[k], S, i)) gi = k;
    if (gi < 0) continue;
    lrows_of_step(K.g[gi], S, p.seed, i, O, [&](int, long long chan) {
      const long long o = 4 * i + (chan & 3);
      row_group[o] = int8_t(gi);
      return o;
    });
  }
}

// per-row counts into the chain's int32 per-(step, SiPM) counts (0 for rows of no group; a row beyond the int32
// range is reported and leaves its group, so that no pass writes its photons)
__global__ void k_lcount_narrow(const long long* __restrict__ nrows_dev, long long cap, int8_t* __restrict__ row_group,
                                const long long* __restrict__ c64, int32_t* __restrict__ c32, Status* status) {
  long long n = *nrows_dev;
  n = n < cap ? n : cap;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n; r += (long long)gridDim.x * blockDim.x) {
    long long v = row_group[r] < 0 ? 0 : c64[r];
    if (v > 0x7FFFFFFFll) {
      set_flag(status, CRV_ST_LIMIT);
      row_group[r] = -1;
      v = 0;
    }
    c32[r] = int32_t(v);
  }
}

static CrvSubstepRows rows_in(const CrvSubstepRowsOut& o) {
  CrvSubstepRows r{};
  r.s = o.s; r.d = o.d; r.t0 = o.t0; r.t1 = o.t1; r.beta = o.beta; r.theta = nullptr; r.dev = o.dev; r.mu = o.mu;
  r.nsub = o.nsub; r.step = o.step; r.chan = o.chan; r.n_scint = o.n_scint; r.n_ck_s = o.n_ck_s; r.n_ck_f = o.n_ck_f;
  r.cos_theta = o.cos_theta;
  return r;
}

static unsigned step_grid(long long n) {
  const long long blocks = (n + 255) / 256;
  const long long maxb = (long long)device_info().sms * 8;
  return (unsigned)(blocks < 1 ? 1 : (blocks < maxb ? blocks : maxb));
}

static unsigned row_grid(long long nrows) {
  const long long blocks = (nrows + SUB_ROWS_PER_BLOCK - 1) / SUB_ROWS_PER_BLOCK;
  const long long maxb = (long long)device_info().sms * 8;
  return (unsigned)(blocks < 1 ? 1 : (blocks < maxb ? blocks : maxb));
}

cudaError_t lookup_chain_rows(const CrvParams& p, const CrvLookupChain& K, const long long* nsteps_dev,
                              long long step_cap, const LookupChainWs& w, cudaStream_t s) {
  LGroups G{};
  G.n = K.ngroups;
  for (int k = 0; k < K.ngroups; ++k) G.g[k] = K.group[k];
  const unsigned grid = step_grid(step_cap);
  crv::Mark mark_("k_lrows_chain", s);
  k_lrows_chain<<<grid, 256, 0, s>>>(p, G, K.steps, nsteps_dev, step_cap, w.rows, w.row_group, w.nrows, w.seed);
  return cudaGetLastError();
}

cudaError_t lookup_chain_count(const CrvLookupChain& K, const LookupChainWs& w, long long row_cap, int32_t* count32,
                               Status* status, cudaStream_t s) {
  const CrvSubstepRows R = rows_in(w.rows);
  const unsigned grid = row_grid(row_cap);
  for (int k = 0; k < K.ngroups; ++k) {
    const CrvLookup& L = K.table[k];
    if (L.precision == 1 && edges_smem(L) > EDGES_MOST) return cudaErrorInvalidValue;
    const RowSel sel{w.nrows, w.row_group, w.seed, k, w.kept, w.nkept};
    if (L.precision == 1) {
      launch_count_f32(L, R, 0u, row_cap, sel, w.count, status, grid, s);
    } else {
      crv::Mark mark_("k_substep_count", s);
      k_substep_count<<<grid, SUB_ROWS_PER_BLOCK * 32, 0, s>>>(L, R, 0u, row_cap, sel, w.count, status);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  crv::Mark mark_("k_lcount_narrow", s);
  k_lcount_narrow<<<step_grid(row_cap), 256, 0, s>>>(w.nrows, row_cap, w.row_group, w.count, count32, status);
  return cudaGetLastError();
}

cudaError_t lookup_chain_emit(const CrvLookupChain& K, const LookupChainWs& w, long long row_cap,
                              const long long* total, long long cap, Status* status, cudaStream_t s) {
  const CrvSubstepRows R = rows_in(w.rows);
  const unsigned grid = row_grid(row_cap);
  for (int k = 0; k < K.ngroups; ++k) {
    const CrvLookup& L = K.table[k];
    const RowSel sel{w.nrows, w.row_group, w.seed, k, w.kept, w.nkept};
    if (L.precision == 1) {
      const cudaError_t e = allow_edges(edges_smem(L));
      if (e != cudaSuccess) return e;
    }
    crv::Mark mark_("k_substep_emit", s);
    if (L.precision == 1)
      k_substep_emit_f32<<<grid, SUB_ROWS_PER_BLOCK * 32, edges_smem(L), s>>>(L, R, 0u, row_cap, sel, w.row_off,
                                                                             total, cap, w.o_step, nullptr,
                                                                             w.o_time, status);
    else
      k_substep_emit<<<grid, SUB_ROWS_PER_BLOCK * 32, 0, s>>>(L, R, 0u, row_cap, sel, w.row_off, total, cap,
                                                              w.o_step, nullptr, w.o_time, status);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace crv
