// Waveform stage: SiPM charges -> zero-suppressed 12-sample digis.
//
// Semantics of the reference synthesis (crv/crvfastsim/reco/waveform.py:65-172, chain.py:219-270):
//   * TDC0 per (event, FEB): one uniform x width (keyed by event and FEB key, so no global order is needed);
//   * charges of a SiPM split into clusters where consecutive times differ by more than max_time + 4 periods; a
//     cluster is kept if n_charges * max(template) >= min_voltage;
//   * the cluster waveform starts at t_start = ceil((t_first - P - TDC0) / P) P + TDC0 and is
//     max(floor((t_last - t_first + max_time) / P), last reached sample + 1) samples long;
//   * every charge adds template[rint((J P + t_start - t) / precision)] * charge / q_ref to samples J >= ceil((t -
//     t_start)/P) within ceil(max_time/P) + 2 samples; electronics noise sigma * z(event, channel, tick) is added to
//     every sample (keyed normals);
//   * zero suppression: a digi starts at sample i if a sample in i-2..i+2 exceeds min_voltage, i >= the end of the
//     previous digi and t_start + i P lies in the window; ADC = clip(int16(V * conv + pedestal + 0.5), min, max);
//     startTDC = rint((start - TDC0) / P).
//
// GPU mapping: one warp per SiPM; the cluster waveform is a shared-memory tile (lanes own samples); each sample sums
// the charges that reach it in charge order (a contiguous range found by binary search), so FP64 sums round exactly
// as the reference's scatter-add; the zero-suppression scan proceeds 32 samples per ballot.
#pragma once
#include "crv_device.cuh"

namespace crv {

struct WfGroups {
  const long long* n;            // device: number of SiPM groups
  const long long* start;        // first charge row of the group
  const int32_t* count;          // charges in the group
  const long long* label;        // SiPM label
  const uint32_t* run;           // run per group (keys), may be null (run 0)
};

// The longest cluster above this many samples is noted (*longest): without one the synthesis passes for longer clusters
// end before they look at a group (passes that found nothing took 25 us of 130 at 2,048 events, 0.33 ms at 65,536)
constexpr int WF_LONG = 64;

struct DigiSlots {
  const long long* off;          // first slot of the group
  const int32_t* cap;            // slots of the group
  int32_t* n;                    // digis written
  long long* chan;
  double* start;
  double* tdc0;
  long long* starttdc;
  double* volt;                  // [slots, 12]; null: volts not kept
  int16_t* adc;                  // [slots, 12]
};

__device__ __forceinline__ int32_t feb_key(const CrvParams& p, const CrvChannels& ch, int c) {
  return p.feb_key_mode == 1 ? ch.feb[c] : ch.roc[c] * 1000 + ch.feb[c];
}

__device__ __forceinline__ double tdc0_of(const CrvParams& p, const CrvChannels& ch, long long label, uint32_t run) {
  long long evk = label / 32768;
  int c = int(label % 32768);
  EvKey ek{uint32_t(evk & 0xFFFFF), uint32_t(evk >> 20), run};
  U4 w = keyed(p.seed, ek, ST_TDC0 << 28, uint32_t(feb_key(p, ch, c)));
  return u01(w.x, w.y) * p.feb_phase_width;
}

__device__ __forceinline__ int reach_samples(const CrvParams& p) { return int(ceil(p.spe_max_time / p.period)) + 2; }

// first sample a charge at time t reaches in a cluster starting at ts
__device__ __forceinline__ long long first_sample(const CrvParams& p, double t, double ts) {
  double v = ceil((t - ts) / p.period);
  return v > 0.0 ? (long long)v : 0;
}

// x / d, exactly: a multiplication by 1/d when d is a power of two (the quotient rounds identically), else a division
__device__ __forceinline__ double exact_div(double x, double d) {
  int e;
  double m = frexp(d, &e);
  return m == 0.5 ? x * ldexp(1.0, 1 - e) : x / d;
}

// template index of sample J for a charge at t (returns -1 when the pair does not contribute)
__device__ __forceinline__ int tmpl_index(const CrvParams& p, long long J, double t, double ts, int tlen) {
  double st = double(J) * p.period + ts - t;
  if (!(st >= 0.0)) return -1;
  double ti = rint(exact_div(st, p.spe_precision));
  return ti < double(tlen) ? int(ti) : -1;
}

// FP32-mixed forms on dt = t - t_start (one FP64 subtraction per charge, then FP32)
__device__ __forceinline__ int first_sample_f(float dt, float P) {
  float v = ceilf(dt / P);
  return v > 0.0f ? int(v) : 0;
}

__device__ __forceinline__ int tmpl_index_f(int J, float dt, float P, float inv_prec, int tlen) {
  float st = float(J) * P - dt;
  if (!(st >= 0.0f)) return -1;
  float ti = rintf(st * inv_prec);
  return ti < float(tlen) ? int(ti) : -1;
}

// A kept cluster, computed once per cluster by the prepass (a lane per cluster): t_start = k0 P + TDC0, charge rows
// [a, b) relative to the group start, length in samples, and the samples whose start lies in the window [ilo, ihi]
// (valid while the length fits a synthesis pass, at most 16,384 samples).
struct WfCluster {
  double ts;
  long long k0;
  int32_t a, b, L;
  int16_t ilo, ihi;
};

// t_start of a cluster, rounded the same way wherever it is formed (no contraction into an FMA)
__device__ __forceinline__ double cluster_ts(long long k0, double period, double tdc0) {
  return __dadd_rn(__dmul_rn(double(k0), period), tdc0);
}

// samples of a cluster whose start lies in the window: [i_lo, i_hi] (monotone predicates)
__device__ __forceinline__ void window_bounds(const CrvParams& p, double ts, int L, int* lo_o, int* hi_o) {
  if (ts >= p.window_lo && __dadd_rn(ts, __dmul_rn(double(L - 1), p.period)) <= p.window_hi) {
    *lo_o = 0;
    *hi_o = L - 1;
    return;
  }
  double a0 = ceil((p.window_lo - ts) / p.period);
  long long c = (long long)fmax(a0 - 1.0, 0.0);
  while (c < L && !(__dadd_rn(ts, __dmul_rn(double(c), p.period)) >= p.window_lo)) ++c;
  while (c > 0 && __dadd_rn(ts, __dmul_rn(double(c - 1), p.period)) >= p.window_lo) --c;
  double b0 = floor((p.window_hi - ts) / p.period);
  long long d = (long long)fmin(b0 + 1.0, double(L - 1));
  while (d >= 0 && !(__dadd_rn(ts, __dmul_rn(double(d), p.period)) <= p.window_hi)) --d;
  while (d + 1 < L && __dadd_rn(ts, __dmul_rn(double(d + 1), p.period)) <= p.window_hi) ++d;
  *lo_o = int(c);
  *hi_o = int(d);
}

constexpr int WF_FX = 32;                      // fractional bits of fixed-point times

// trunc(x * 2^32) for |x| < 2^30; false for non-finite or larger values
__device__ __forceinline__ bool d2fx(double x, long long* out) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = int((b >> 52) & 0x7FF);
  if (e == 0x7FF || e >= 1023 + 30) return false;
  if (e < 1023 - WF_FX - 1) {                  // |x| < 2^-33: below the resolution
    *out = 0;
    return true;
  }
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const int sh = e - 1075 + WF_FX;             // in [-54, 10]
  const unsigned long long v = sh >= 0 ? (m << sh) : (m >> (-sh));
  *out = (b >> 63) ? -(long long)v : (long long)v;
  return true;
}

// order-preserving unsigned key of a double's bits (larger key = larger value), so a maximum over a table is
// integer work: a warp-wide FP64 instruction costs ~60-70 FP32 issue slots on this GPU
__device__ __forceinline__ unsigned long long dkey(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double dkey_value(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}

// the template's maximum (NaN entries ignored, as fmax does) by every thread of the block; call from all threads
__device__ __forceinline__ double block_tmpl_max(const double* tmpl, int tlen, unsigned long long* slot) {
  if (threadIdx.x == 0) *slot = dkey(-1e300);
  __syncthreads();
  unsigned long long m = dkey(-1e300);
  for (int i = threadIdx.x; i < tlen; i += blockDim.x) {
    const double v = tmpl[i];
    const unsigned long long k = dkey(v);
    if (v == v && k > m) m = k;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long x = __shfl_xor_sync(0xffffffffu, m, o);
    if (x > m) m = x;
  }
  if (lane_id() == 0) atomicMax(slot, m);
  __syncthreads();
  return dkey_value(*slot);
}

// Cluster starts waiting for a warp's lanes, and the totals of the tile's groups.
constexpr int PREP_QUEUE = 96;
struct PrepQueue {
  int first[PREP_QUEUE];         // first charge of the cluster in its group
  uint8_t group[PREP_QUEUE];     // its group in the tile
  int nk[32], bound[32], maxlen[32];
};

// The prepass of both precisions (Prep: Prep32, Prep64): the groups' kept clusters, TDC0, digi bounds and longest
// clusters.  Warps take tiles of groups: lanes over the groups (TDC0), over each group's charges (cluster starts), then
// over the clusters of all the tile's groups, which wait in a shared queue.
template <typename Prep>
__global__ void __launch_bounds__(256, 3) k_wf_prep(CrvParams p, CrvChannels ch, WfGroups G,
                                                 const double* __restrict__ time, const double* __restrict__ tmpl,
                                                 int tlen, const double* __restrict__ tdc0_rows,
                                                 double* __restrict__ g_tdc0, int32_t* __restrict__ g_bound,
                                                 int32_t* __restrict__ g_maxlen, int32_t* __restrict__ g_nkept,
                                                 int32_t* __restrict__ g_digis, int* __restrict__ longest, int* __restrict__ taken,
                                                 typename Prep::Record* __restrict__ cl, Status* status) {
  __shared__ PrepQueue queue[8];
  __shared__ typename Prep::Consts K_s;
  __shared__ unsigned long long vmax_s;
  const double vmax = block_tmpl_max(tmpl, tlen, &vmax_s);
  if (threadIdx.x == 0) K_s = Prep::consts(p, vmax);           // FP64 scalars once per block, in one thread
  __syncthreads();
  const typename Prep::Consts& K = K_s;
  if (Prep::LIMIT && (!Prep::ok(K) || tlen > 1024)) {
    if (threadIdx.x == 0 && blockIdx.x == 0) set_flag(status, CRV_ST_LIMIT);
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < *G.n; g += (long long)gridDim.x * blockDim.x) {
      g_bound[g] = 0;              // no group has a cluster or a digi: what follows reads these columns
      g_maxlen[g] = 0;
      g_nkept[g] = 0;
      g_digis[g] = 0;
      g_tdc0[g] = 0.0;
    }
    return;
  }
  const int zs = p.samples_zs;
  const int lane = lane_id();
  const unsigned lt = (1u << lane) - 1u;
  PrepQueue& Q = queue[warp_in_block()];
  const long long ng = *G.n;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  const int tile = tile_taken(ng, warps);
  for (long long ti = blockIdx.x * (long long)(blockDim.x >> 5) + warp_in_block(); ti * tile < ng;
       ti = next_tile(taken, warps)) {
    const long long g0 = ti * tile;
    // lane = group of the tile: its rows and its keyed TDC0 (unless the caller gives one per cluster)
    const int ntile = int(min((long long)tile, ng - g0));
    const long long gl = g0 + lane;
    int n_l = 0;
    long long q0_l = 0;
    typename Prep::Tdc0 tdc0_l = 0;
    if (lane < ntile) {
      n_l = G.count[gl];
      q0_l = G.start[gl];
      if (!tdc0_rows) tdc0_l = Prep::tdc0(p, ch, K, G.label[gl], G.run ? G.run[gl] : 0u);
    }
    Q.nk[lane] = 0;
    Q.bound[lane] = 0;
    Q.maxlen[lane] = 0;
    __syncwarp();
    // The clusters queued in Q (start rows, in order), the first `full` of them with known ends: keep rule, start tick,
    // length, window range, digi bound, one cluster per lane.
    auto clusters = [&](int cnt, int full) {
#pragma unroll 1
      for (int base = 0; base < full; base += 32) {
        const int e = base + lane;
        const bool on = e < full;
        const int gi = on ? Q.group[e] : 0, a = on ? Q.first[e] : 0;
        const int gn = e + 1 < cnt ? int(Q.group[e + 1]) : -1;
        const int n = __shfl_sync(0xffffffffu, n_l, gi);
        const long long q0 = __shfl_sync(0xffffffffu, q0_l, gi);
        const typename Prep::Tdc0 tdc0g = __shfl_sync(0xffffffffu, tdc0_l, gi);
        const int b = on && gn == gi ? Q.first[e + 1] : n;
        const bool keep = on && Prep::keep(p, K, b - a);
        typename Prep::Record rec{};
        int L = 0;
        if (keep) {
          const typename Prep::Tdc0 tdc0 = tdc0_rows ? Prep::caller_tdc0(tdc0_rows[q0 + a], status) : tdc0g;
          rec = Prep::record(p, K, time + q0, a, b, tdc0, tlen);
          L = rec.L;
        }
        const unsigned mine = __match_any_sync(0xffffffffu, on ? gi : 32 + lane);
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        if (keep) cl[q0 + Q.nk[gi] + __popc(km & mine & lt)] = rec;
        __syncwarp();
        if (keep) {
          if ((km & mine & lt) == 0u) Q.nk[gi] += __popc(km & mine);
          atomicAdd(&Q.bound[gi], (L + zs - 1) / zs);
          atomicMax(&Q.maxlen[gi], L);
        }
        __syncwarp();
      }
    };
    // cluster starts of every group: a new cluster where consecutive fixed-point times differ by more than the gap
    int cnt = 0, gi = 0, base = 0, n = __shfl_sync(0xffffffffu, n_l, 0);
    long long q0 = __shfl_sync(0xffffffffu, q0_l, 0), prev = 0;
    unsigned bad = 0;
    bool odd = false, prev_ok = false;
#pragma unroll 1
    while (true) {
      if (gi < ntile && base >= n) {               // next group
        if (Prep::LIMIT && __any_sync(0xffffffffu, odd)) {
          bad |= 1u << gi;
          if (lane == 0) set_flag(status, CRV_ST_LIMIT);
        }
        odd = false;
        ++gi;
        base = 0;
        n = __shfl_sync(0xffffffffu, n_l, gi & 31);
        q0 = __shfl_sync(0xffffffffu, q0_l, gi & 31);
        if (gi < ntile && n <= 0) continue;
      }
      const bool end = gi >= ntile;
      if (end || cnt > PREP_QUEUE - 32) {          // all clusters, or those with known ends to make room for 32 more
        clusters(cnt, end ? cnt : cnt - 1);
        if (end) break;
        const int f = Q.first[cnt - 1];
        const uint8_t q = Q.group[cnt - 1];
        __syncwarp();
        if (lane == 0) { Q.first[0] = f; Q.group[0] = q; }
        cnt = 1;
        __syncwarp();
      }
      const int q = base + lane;
      long long tf = 0;
      const bool known = q < n && d2fx(time[q0 + q], &tf);
      odd |= q < n && !known;
      long long tp = __shfl_up_sync(0xffffffffu, tf, 1);
      const unsigned okm = __ballot_sync(0xffffffffu, known);
      bool pk = (okm >> ((lane + 31) & 31)) & 1u;
      if (lane == 0) { tp = prev; pk = prev_ok; }
      const bool isnew = q < n && (q == 0 || Prep::is_new(K, tf, tp, known && pk, time + q0 + q));
      const unsigned m = __ballot_sync(0xffffffffu, isnew);
      if (isnew) {
        const int at = cnt + __popc(m & lt);
        Q.first[at] = q;
        Q.group[at] = uint8_t(gi);
      }
      cnt += __popc(m);
      prev = __shfl_sync(0xffffffffu, tf, 31);
      prev_ok = okm >> 31;
      base += 32;
      __syncwarp();
    }
    __syncwarp();
    if (lane < ntile) {
      const bool drop = (bad >> lane) & 1u;
      g_bound[gl] = drop ? 0 : Q.bound[lane];
      g_maxlen[gl] = drop ? 0 : Q.maxlen[lane];
      g_nkept[gl] = drop ? 0 : Q.nk[lane];
      g_digis[gl] = 0;         // the synthesis writes the groups with kept clusters only
      if (!drop && Q.maxlen[lane] > WF_LONG) atomicMax(longest, Q.maxlen[lane]);
      g_tdc0[gl] = drop ? 0.0 : Prep::tdc0_value(tdc0_l);
    }
    __syncwarp();
  }
}

// FP64 form of the prepass.  The gap test on consecutive times is decided on fixed-point copies (2^-32 ns, truncated)
// unless they lie within a few units of the gap; everything else runs once per cluster, 32 clusters at a time.
struct Prep64 {
  using Record = WfCluster;
  static constexpr bool LIMIT = false;
  struct Consts {
    double vmax, gap;
    long long gap_fx;
    int nr, gap_ok;
  };
  static __device__ __forceinline__ Consts consts(const CrvParams& p, double vmax) {
    Consts K;
    K.vmax = vmax;
    K.gap = p.spe_max_time + 4.0 * p.period;
    K.nr = reach_samples(p);
    K.gap_ok = d2fx(K.gap, &K.gap_fx);
    return K;
  }
  static __device__ __forceinline__ bool ok(const Consts&) { return true; }
  static __device__ __forceinline__ bool is_new(const Consts& K, long long tf, long long tp, bool known,
                                                const double* t) {
    if (known && K.gap_ok) {
      const long long d = tf - tp - K.gap_fx;      // within 2 units of the difference
      if (d > 4 || d < -4) return d > 0;
    }
    return t[0] - t[-1] > K.gap;
  }
  static __device__ __forceinline__ bool keep(const CrvParams& p, const Consts& K, int n) {
    return double(n) * K.vmax >= p.min_voltage;
  }
  using Tdc0 = double;
  static __device__ __forceinline__ double tdc0(const CrvParams& p, const CrvChannels& ch, const Consts&,
                                                long long label, uint32_t run) {
    return tdc0_of(p, ch, label, run);
  }
  static __device__ __forceinline__ double caller_tdc0(double x, Status*) { return x; }
  static __device__ __forceinline__ double tdc0_value(double v) { return v; }
  static __device__ __forceinline__ WfCluster record(const CrvParams& p, const Consts& K, const double* t, int a, int b,
                                                     double tdc0, int tlen) {
    const long long k0 = (long long)ceil((t[a] - p.period - tdc0) / p.period);
    const double ts = cluster_ts(k0, p.period, tdc0);
    const long long est = (long long)floor((t[b - 1] - t[a] + p.spe_max_time) / p.period);
    // the last charge reaches the last sample: a later charge's sample times are no larger, so its reach is no shorter
    long long used = 0;
    const long long j0 = first_sample(p, t[b - 1], ts);
#pragma unroll 1
    for (int k = K.nr - 1; k >= 0; --k)
      if (tmpl_index(p, j0 + k, t[b - 1], ts, tlen) >= 0) {
        used = j0 + k + 1;
        break;
      }
    const int L = int(est > used ? est : used);
    int ilo = 0, ihi = -1;
    if (L <= 16384) window_bounds(p, ts, L, &ilo, &ihi);
    return WfCluster{ts, k0, a, b, L, int16_t(ilo), int16_t(ihi)};
  }
};

constexpr int WF_QSTAGE = 512;    // charges of a cluster staged in shared memory (larger clusters: on the fly)
constexpr int WF_TMPL = 1024;     // template entries kept in shared memory (longer templates: from global memory)

__host__ __device__ inline size_t wf_smem_per_warp(int cap) {
  return (size_t(cap) * 8 + size_t(WF_QSTAGE) * 16 + 15) & ~size_t(15);
}

__device__ __forceinline__ int16_t adc_of(const CrvParams& p, double v) {
  double x = v * p.adc_conversion + double(p.adc_pedestal) + 0.5;
  long long i;
  if (!(x == x)) i = (long long)-2147483648ll;
  else if (x >= 2147483647.0) i = 2147483647ll;
  else if (x <= -2147483648.0) i = -2147483648ll;
  else i = (long long)trunc(x);
  int16_t s = int16_t(uint16_t(uint32_t(int32_t(i)) & 0xFFFFu));
  int r = s;
  if (r < p.min_adc) r = p.min_adc;
  if (r > p.max_adc) r = p.max_adc;
  return int16_t(r);
}

// ADC of an FP32 sample: v * conversion + pedestal + 0.5 is exact in FP64 for an FP32 v (a 24-bit by 12-bit
// product plus a small offset), so one FP32 FMA (one rounding) truncates to the same integer unless it lands on an
// integer itself; only then, or out of range, is the FP64 form evaluated.
__device__ __forceinline__ int16_t adc_of_f(const CrvParams& p, float v, float conv, float off) {
  const float x = fmaf(v, conv, off);
  if (!(fabsf(x) < 1e9f) || x == truncf(x)) return adc_of(p, f2d(v));
  int r = int16_t(uint16_t(uint32_t(int32_t(truncf(x))) & 0xFFFFu));
  if (r < p.min_adc) r = p.min_adc;
  if (r > p.max_adc) r = p.max_adc;
  return int16_t(r);
}

#if defined(CRV_REAL_IS_FLOAT) && !CRV_REAL_IS_FLOAT    // the FP64 kernels' unit
// Synthesis in FP64 without FP64 decisions.  A warp-wide FP64 instruction takes 19 cycles of the whole SM, so only the
// arithmetic whose rounding is the result (sample sums, noise, volts, start times) is FP64; what a comparison or a
// rounding to an integer decides is decided on fixed-point copies where that is certain, and by the FP64 form elsewhere:
//   first sample  ceil((t - ts) / P) from t - ts in units of 2^-32 ns, unless it lies within j + 8 units of a sample;
//   template index rint((J P + ts - t) / precision) and the sign of the time, from 32-bit differences in 2^-20 ns (a
//                 charge of the sample's range lies within the template's length, so the differences fit; both
//                 terms truncated, J P within J 2^-32: 7 units at most; the FP32 quotient within 2^-22), unless within
//                 four times those errors of a half (4e-4 here) or 16 units of 0;
//   ADC           truncation of v conversion + pedestal + 1/2, from FP32 unless within 0.01 of an integer.
// 1,500 events: synthesis 5.9 -> 2.9 ms, of which the noise normals are a third, prepass (Prep64) 2.9 -> 0.5 ms.
struct WfFixed {
  long long P;                   // period, 2^-32 ns
  float P_ns, inv_P;
  double inv_ref;                // 1 / reference charge, rounded
  float unit, half;              // 2^-20 ns in template steps; 1/2 less the index quotient's error
  float conv, off;
  int plain;                     // settings outside the fixed-point forms' range: FP64 forms only
};

__device__ __forceinline__ WfFixed wf_fixed(const CrvParams& p) {
  WfFixed F;
  const double reach = p.spe_max_time + 3.0 * p.period;
  F.plain = !d2fx(p.period, &F.P) || !(p.period > 0.5) || !(p.spe_max_time >= 0.0 && reach < 1000.0) ||
            !(p.spe_precision > 0.0 && reach / p.spe_precision < 4000.0) || !(fabs(p.adc_conversion) < 1e6) ||
            !(fabs(double(p.adc_pedestal)) < 8000.0);
  F.P_ns = float(p.period);
  F.inv_P = float(1.0 / p.period);
  F.inv_ref = 1.0 / p.spe_ref_charge;
  F.unit = float(0x1p-20 / p.spe_precision);
  F.half = 0.5f - 4.0f * (float(reach / p.spe_precision) * 0x1p-22f + 16.0f * F.unit);
  F.conv = float(p.adc_conversion);
  F.off = float(double(p.adc_pedestal) + 0.5);
  return F;
}

// first sample of a charge whose time from the cluster start is x (2^-32 ns), given where that is certain
__device__ __forceinline__ bool first_sample_fx(const WfFixed& F, long long x, int* j) {
  if (x <= -16) { *j = 0; return true; }
  if (x < 16 || x > (1ll << 50)) return false;
  long long k = (long long)(__int2float_rn(int(x >> 32)) * F.inv_P);    // floor estimate, within a sample or two
  while (k * F.P > x) --k;
  while ((k + 1) * F.P <= x) ++k;
  const long long r = x - k * F.P, tol = k + 8;                          // in [0, P)
  if (r < tol || F.P - r < tol) return false;
  *j = int(k) + 1;
  return true;
}

__device__ __forceinline__ int16_t adc_near(const CrvParams& p, const WfFixed& F, double v) {
  if (!F.plain) {
    const float x = fmaf(d2f_trunc(v), F.conv, F.off), t = truncf(x), d = fabsf(x - t);
    // value, conversion and offset in FP32: within 2^-22 of |v conversion| + |off|, 4e-3 below 16,000
    if (fabsf(x) < 8000.0f && d > 0.01f && d < 0.99f) {
      int r = int(t);
      if (r < p.min_adc) r = p.min_adc;
      if (r > p.max_adc) r = p.max_adc;
      return int16_t(r);
    }
  }
  return adc_of(p, v);
}

// normal of one sample: the pair of the block, only the half that is used
__device__ __noinline__ double noise_normal(U4 w, int odd) {
  const double u1 = u01_open(w.x, w.y), u2 = u01(w.z, w.w);
  const double r = sqrt(-2.0 * dlog(u1));
  double s, c;
  dsincospi(2.0 * u2, &s, &c);
  return r * (odd ? s : c);
}

// Synthesis + zero suppression of the groups whose longest kept cluster is in (lo, cap].
__global__ void __launch_bounds__(256, 3) k_wf_synth(CrvParams p, WfGroups G, const double* __restrict__ time,
                                                  const double* __restrict__ charge, const double* __restrict__ tmpl,
                                                  int tlen, const double* __restrict__ tdc0_rows,
                                                  const double* __restrict__ g_tdc0,
                                                  const int32_t* __restrict__ g_maxlen,
                                                  const int32_t* __restrict__ g_nkept,
                                                  const WfCluster* __restrict__ cl, int lo, int cap, int last_pass,
                                                  const int* __restrict__ longest, int* __restrict__ taken,
                                                  DigiSlots D, Status* status) {
  extern __shared__ __align__(16) char smem[];
  if (lo >= WF_LONG && *longest <= lo) return;
  char* wbase = smem + size_t(warp_in_block()) * wf_smem_per_warp(cap);
  double* wave = reinterpret_cast<double*>(wbase);
  double* qn_s = reinterpret_cast<double*>(wbase + size_t(cap) * 8);
  int32_t* j0_s = reinterpret_cast<int32_t*>(wbase + size_t(cap) * 8 + size_t(WF_QSTAGE) * 8);
  int32_t* dt_s = j0_s + WF_QSTAGE;                // t - ts in 2^-20 ns, modulo 2^32
  __shared__ double tmpl_s[WF_TMPL];
  __shared__ WfFixed F_s;
  for (int i = threadIdx.x; i < tlen && i < WF_TMPL; i += blockDim.x) tmpl_s[i] = tmpl[i];
  if (threadIdx.x == 0) F_s = wf_fixed(p);
  __syncthreads();
  const WfFixed& F = F_s;
  const double* tm = tlen <= WF_TMPL ? tmpl_s : tmpl;
  const int nr = reach_samples(p);
  const int zs = p.samples_zs;
  const double vthr = p.min_voltage;
  const double sigma = p.noise_sigma;
  const int lane = lane_id();
  long long ng = *G.n;
  long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  // groups in tiles per warp: one coalesced load of their longest clusters and a ballot pick this pass's groups
  const int tile = tile_taken(ng, warps);
  for (long long ti = blockIdx.x * (long long)(blockDim.x >> 5) + warp_in_block(); ti * tile < ng;
       ti = next_tile(taken, warps)) {
   const int mll = lane < tile && ti * tile + lane < ng ? g_maxlen[ti * tile + lane] : 0;
   unsigned todo = __ballot_sync(0xffffffffu, mll > lo);
   while (todo) {
    const int bsel = __ffs(todo) - 1;
    todo &= todo - 1;
    const long long g = ti * tile + bsel;
    const int ml = __shfl_sync(0xffffffffu, mll, bsel);
    if (ml > cap) {
      if (last_pass && lane == 0) {
        set_flag(status, CRV_ST_CAPACITY);
        need_at_least(status, CRV_NEED_SAMPLES, ml);
      }
      continue;
    }
    long long q0 = G.start[g];
    const double* t = time + q0;
    const double* qc = charge + q0;
    long long lab = G.label[g];
    uint32_t run = G.run ? G.run[g] : 0u;
    long long evk = lab / 32768;
    EvKey ek{uint32_t(evk & 0xFFFFF), uint32_t(evk >> 20), run};
    uint32_t chan = uint32_t(lab % 32768);
    double tdc0 = g_tdc0[g];
    long long slot = D.off[g];
    int scap = D.cap[g];
    int nd = 0;
    const int nk = g_nkept[g];
    for (int kc = 0; kc < nk; ++kc) {
      const WfCluster C = cl[q0 + kc];
      const int a = C.a, b = C.b, L = C.L;
      const long long k0 = C.k0;
      const double ts = C.ts;
      const double tdc0c = tdc0_rows ? tdc0_rows[q0 + a] : tdc0;
      // stage each charge's first reached sample, time from the cluster start and normalised charge
      const bool staged = (b - a) <= WF_QSTAGE;
      bool fixed = staged && !F.plain;
      if (staged) {
        for (int q = a + lane; q < b; q += 32) {
          const double tq = t[q];
          long long x = 0;
          const bool fx = d2fx(tq - ts, &x);
          int j = 0;
          if (!fx || F.plain || !first_sample_fx(F, x, &j)) j = int32_t(first_sample(p, tq, ts));
          j0_s[q - a] = j;
          dt_s[q - a] = int32_t(x >> 12);
          fixed = fixed && fx;
          const double qq = qc[q];
          const int e = int((__double_as_longlong(qq) >> 52) & 0x7FF);
          qn_s[q - a] = unsigned(e - 723) < 600u && F.inv_ref > 1e-90 && F.inv_ref < 1e90
                            ? quotient(qq, p.spe_ref_charge, F.inv_ref) : qq / p.spe_ref_charge;
        }
        fixed = __all_sync(0xffffffffu, fixed);
        __syncwarp();
      }
      // samples: sum of the charges reaching each sample, in charge order
      for (int j = lane; j < L; j += 32) {
        // charges with first_sample in (j - nr, j]: first_sample is non-decreasing along the cluster.  The staged
        // and the on-the-fly searches are separate loops, so the staged one carries no FP64 work.
        int q1, lo2;
        if (staged) {
          int lo_q = a, hi_q = b;                    // first charge with first_sample > j - nr
          while (lo_q < hi_q) {
            int m = (lo_q + hi_q) >> 1;
            if (j0_s[m - a] > j - nr) hi_q = m; else lo_q = m + 1;
          }
          q1 = lo_q;
          int hi2 = b;                               // first charge with first_sample > j
          lo2 = q1;
          while (lo2 < hi2) {
            int m = (lo2 + hi2) >> 1;
            if (j0_s[m - a] > j) hi2 = m; else lo2 = m + 1;
          }
        } else {
          int lo_q = a, hi_q = b;
          while (lo_q < hi_q) {
            int m = (lo_q + hi_q) >> 1;
            if (first_sample(p, t[m], ts) > (long long)j - nr) hi_q = m; else lo_q = m + 1;
          }
          q1 = lo_q;
          int hi2 = b;
          lo2 = q1;
          while (lo2 < hi2) {
            int m = (lo2 + hi2) >> 1;
            if (first_sample(p, t[m], ts) > (long long)j) hi2 = m; else lo2 = m + 1;
          }
        }
        double acc = 0.0;
        if (fixed) {
          const int32_t JP = int32_t(((long long)j * F.P) >> 12);
#pragma unroll 1
          for (int q = q1; q < lo2; ++q) {
            const int32_t st = int32_t(uint32_t(JP) - uint32_t(dt_s[q - a]));
            const float x = float(st) * F.unit;
            const float r = rintf(x);
            int ti = int(r);
            if (st < 16 || fabsf(x - r) > F.half) ti = st < -16 ? -1 : tmpl_index(p, j, t[q], ts, tlen);
            if (ti >= 0 && ti < tlen) acc += tm[ti] * qn_s[q - a];
          }
        } else {
          for (int q = q1; q < lo2; ++q) {
            int ti = tmpl_index(p, j, t[q], ts, tlen);
            if (ti >= 0) acc += tm[ti] * (staged ? qn_s[q - a] : qc[q] / p.spe_ref_charge);
          }
        }
        if (p.noise_on) {
          long long tk = k0 + j;
          U4 w = keyed(p.seed, ek, (ST_NOISE << 28) | (chan & 0x7FFFu), uint32_t(tk >> 1));
          acc = acc + sigma * noise_normal(w, int(tk & 1));
        }
        wave[j] = acc;
      }
      __syncwarp();
      const int i_lo = C.ilo, i_hi = C.ihi;
      // zero suppression over chunks of 32 samples
      int next_i = 0;
      for (int base = 0; base < L; base += 32) {
        int i = base + lane;
        bool w = false;
        if (i < L) {
          for (int d = -2; d <= 2 && !w; ++d) {
            int k = i + d;
            if (k >= 0 && k < L && above(wave[k], vthr)) w = true;
          }
        }
        bool inwin = i >= i_lo && i <= i_hi;
        unsigned cand = __ballot_sync(0xffffffffu, w && inwin);
        while (true) {
          unsigned m = cand;
          if (next_i > base) m &= (next_i - base >= 32) ? 0u : ~((1u << (next_i - base)) - 1u);
          if (!m) break;
          int i0 = base + __ffs(m) - 1;
          // emit digi at i0; its start TDC (start - TDC0) / P is the integer tick k0 + i0
          if (nd < scap) {
            long long o = slot + nd;
            if (lane < zs) {
              int c = i0 + lane;
              double v = c < L ? wave[c] : 0.0;
              if (D.volt) D.volt[o * zs + lane] = v;
              D.adc[o * zs + lane] = adc_near(p, F, v);
            }
            if (lane == 0) {
              D.chan[o] = lab;
              D.start[o] = __dadd_rn(ts, __dmul_rn(double(i0), p.period));
              D.tdc0[o] = tdc0c;
              D.starttdc[o] = k0 + i0;
            }
          }
          ++nd;
          next_i = i0 + zs;
        }
      }
      __syncwarp();
    }
    if (lane == 0) {
      D.n[g] = nd;
      if (nd > scap) set_flag(status, CRV_ST_CAPACITY);
    }
   }
  }
}

#endif

}  // namespace crv

namespace crv {

struct Digis {
  long long* chan;
  double* start;
  double* tdc0;
  long long* starttdc;
  double* volt;
  int16_t* adc;
};

#ifdef CRV_ENGINE_TU
// a group's digis by the warp
__device__ __forceinline__ void digi_compact_group(const DigiSlots& D, const Digis& O, int nd, long long s0, long long o0,
                                                   int zs) {
  bool sorted = true;
  for (int j = lane_id() + 1; j < nd; j += 32) sorted = sorted && !(D.start[s0 + j] < D.start[s0 + j - 1]);
  if (__all_sync(0xffffffffu, sorted)) {
    for (int i = lane_id(); i < nd; i += 32) {
      O.chan[o0 + i] = D.chan[s0 + i];
      if (O.start) O.start[o0 + i] = D.start[s0 + i];
      if (O.tdc0) O.tdc0[o0 + i] = D.tdc0[s0 + i];
      O.starttdc[o0 + i] = D.starttdc[s0 + i];
    }
    for (long long f = lane_id(); f < (long long)nd * zs; f += 32) {
      if (O.volt) O.volt[o0 * zs + f] = D.volt[s0 * zs + f];
      O.adc[o0 * zs + f] = D.adc[s0 * zs + f];
    }
    return;
  }
  for (int i = 0; i < nd; ++i) {
    // rank of digi i among the group's digis by start, ties by production order
    const double si = D.start[s0 + i];
    int r = 0;
    for (int j = lane_id(); j < nd; j += 32) {
      const double sj = D.start[s0 + j];
      r += (sj < si) || (sj == si && j < i);
    }
    r = warp_sum(r);
    const long long o = o0 + r, s = s0 + i;
    if (lane_id() == 0) {
      O.chan[o] = D.chan[s];
      if (O.start) O.start[o] = D.start[s];
      if (O.tdc0) O.tdc0[o] = D.tdc0[s];
      O.starttdc[o] = D.starttdc[s];
    }
    if (lane_id() < zs) {
      if (O.volt) O.volt[o * zs + lane_id()] = D.volt[s * zs + lane_id()];
      O.adc[o * zs + lane_id()] = D.adc[s * zs + lane_id()];
    }
  }
}

// Move each group's digis from its slots to the output, ordered by start (stable) within the group.
// O.start, O.tdc0 and O.volt may be null (the resident chain reads channel, start TDC and ADC only): not written.
// A tile of groups per warp, a lane per group with at most four digis in order (nearly all: they come out of the synthesis
// in start order, clusters in time order, digis in sample order); the others by the warp.  Bound by the latency of a
// group's few loads when a warp took one group at a time: 65,536 events 1.59 -> 0.22 ms, 2,048 events 44 -> 13 us.
__global__ void k_digi_compact(const long long* __restrict__ ng_dev, DigiSlots D, const long long* __restrict__ out_off,
                               int zs, Digis O, long long out_cap) {
  const long long ng = *ng_dev;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  const int tile = ng < 4 * warps ? 1 : 32;    // few groups: a warp each (1,900 groups: 3 against 10 us)
  // samples of a digi in words of eight bytes: every digi then starts on one
  const bool words = (zs & 3) == 0 && ((reinterpret_cast<uintptr_t>(D.adc) | reinterpret_cast<uintptr_t>(O.adc)) & 7) == 0;
  for (long long ti = blockIdx.x * (long long)(blockDim.x >> 5) + warp_in_block(); ti * tile < ng; ti += warps) {
    const long long gl = ti * tile + lane_id();
    int nd_l = 0;
    long long s0_l = 0, o0_l = 0;
    if (lane_id() < tile && gl < ng) {
      nd_l = D.n[gl];
      s0_l = D.off[gl];
      o0_l = out_off[gl];
      if (nd_l > D.cap[gl] || o0_l + nd_l > out_cap) nd_l = 0;     // (reported by the synthesis or the sum of the counts)
    }
    bool own = tile > 1 && nd_l > 0 && nd_l <= 4;
    for (int i = 1; own && i < nd_l; ++i) own = !(D.start[s0_l + i] < D.start[s0_l + i - 1]);
    if (own)
      for (int i = 0; i < nd_l; ++i) {
        const long long s = s0_l + i, o = o0_l + i;
        O.chan[o] = D.chan[s];
        if (O.start) O.start[o] = D.start[s];
        if (O.tdc0) O.tdc0[o] = D.tdc0[s];
        O.starttdc[o] = D.starttdc[s];
        if (O.volt)
          for (int c = 0; c < zs; ++c) O.volt[o * zs + c] = D.volt[s * zs + c];
        if (words) {
          const long long* a = reinterpret_cast<const long long*>(D.adc + s * zs);
          long long* b = reinterpret_cast<long long*>(O.adc + o * zs);
          for (int c = 0; c < zs >> 2; ++c) b[c] = a[c];
        } else {
          for (int c = 0; c < zs; ++c) O.adc[o * zs + c] = D.adc[s * zs + c];
        }
      }
    for (unsigned m = __ballot_sync(0xffffffffu, nd_l > 0 && !own); m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      digi_compact_group(D, O, __shfl_sync(0xffffffffu, nd_l, l), __shfl_sync(0xffffffffu, s0_l, l),
                         __shfl_sync(0xffffffffu, o0_l, l), zs);
    }
  }
}

// Groups: runs of equal labels in a label-sorted array
struct LabelRuns {
  using V = long long;
  static constexpr bool FLAG = true;
  const long long* label;
  long long *start, *group_label;
  __device__ __forceinline__ long long item(long long i) const { return i == 0 || label[i] != label[i - 1]; }
  __device__ __forceinline__ void put(long long i, long long, long long g) const {
    start[g] = i;
    group_label[g] = label[i];
  }
};

// counts from consecutive starts; run per group from a sorted (event key -> run) table (run 0 if absent)
__global__ void k_group_counts(const long long* __restrict__ ng_dev, long long n, const long long* __restrict__ n_dev,
                               const long long* __restrict__ gstart, const long long* __restrict__ glabel,
                               int32_t* __restrict__ gcount, const long long* __restrict__ ev_keys,
                               const uint32_t* __restrict__ ev_runs, long long n_ev, uint32_t* __restrict__ grun,
                               Status* status) {
  long long ng = *ng_dev;
  n = bounded_count(n, n_dev);
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < ng; g += (long long)gridDim.x * blockDim.x) {
    long long e = (g + 1 < ng ? gstart[g + 1] : n) - gstart[g];
    gcount[g] = int32_t(e);
    uint32_t r = 0;
    if (ev_keys && n_ev > 0) {
      long long k = glabel[g] / 32768;
      long long lo = 0, hi = n_ev;
      while (lo < hi) {
        long long m = (lo + hi) >> 1;
        if (ev_keys[m] < k) lo = m + 1; else hi = m;
      }
      if (lo < n_ev && ev_keys[lo] == k) r = ev_runs[lo];
      else set_flag(status, CRV_ST_ORDER);
    }
    grun[g] = r;
  }
}
#endif

}  // namespace crv
