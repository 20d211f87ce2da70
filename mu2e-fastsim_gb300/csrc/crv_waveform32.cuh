// FP32-mixed waveform stage: SiPM charges -> zero-suppressed digis with no FP64 instruction on the common path.
//
// Same semantics as crv_waveform.cuh (the reference's synthesis, crv/crvfastsim/reco/waveform.py:65-172), different
// arithmetic: GB300 issues FP64 at ~1/70 of the FP32 rate and a warp-wide FP64 instruction costs the same with one
// active lane as with 32, so the per-cluster scalars that the FP64 path computes in double precision (cluster start
// tick, start time, length, window range, TDC0) are computed here in 64-bit fixed point (times x 2^32, integer
// arithmetic), and every sample sums its charges in FP32 on times relative to the cluster start.
//
//   times        t_fx = trunc(t * 2^32) (|t| < 2^30 ns; larger or non-finite times set CRV_ST_LIMIT / NONFINITE);
//                differences are exact integers, converted to FP32 once (dt of a charge from its cluster start);
//   TDC0         keyed draw as in the FP64 path: the same 53 random bits times the phase width, in fixed point;
//   k0           ceil((t_first - P - TDC0) / P) exactly on the fixed-point values (FP32 estimate, integer fix-up);
//   outputs      start and TDC0 of a digi are the fixed-point values converted exactly to double; volts are the
//                FP32 sums widened exactly; ADC as the FP32 stage rule (adc_of_f).
//
// Three kernels:
//   k_wf_prep     (crv_waveform.cuh) a tile of groups per warp: lanes over the groups (TDC0), over each group's charges (cluster split by
//                 the gap test on consecutive fixed-point times, ballots), then over the clusters of all the tile's
//                 groups, which wait in a shared queue: keep rule, start tick, length, window sample range, digi
//                 bound; kept clusters are written to cl[group start + k] (the record layout of WfCluster, with the
//                 fixed-point start in place of the double).  A group has 1.2 clusters, so group by group the
//                 cluster work ran on one or two lanes (65,536 events: 6.1 -> 3.0 ms).
//   k_wf_synth16  the same as k_wf_synth32 for groups whose clusters have at most 16 samples, two groups per warp;
//   k_wf_synth32  per kept cluster: the charges' FP32 offsets from the cluster start and normalised charges are
//                 staged in shared memory (coalesced loads), then lanes own samples (32 per tile) and sum the
//                 template contributions of the staged charges in charge order (deterministic), keyed noise is
//                 added, and the zero-suppression scan emits digis 32 samples per ballot.
#pragma once
#include "crv_waveform.cuh"

namespace crv {

// v * 2^-32 as FP32: integer part and fraction converted separately, one final rounding
__device__ __forceinline__ float fx2f(long long v) {
  const int hi = int(v >> 32);                 // floor(v / 2^32): |v| < 2^62
  const unsigned int lo = (unsigned int)(v & 0xFFFFFFFFll);
  return fmaf(__uint2float_rn(lo), 0x1p-32f, __int2float_rn(hi));
}

// v * 2^-32 as double by integer construction of the bits: exact for |v| < 2^53 (times below 2^21 ns), truncated
// beyond
__device__ __forceinline__ double fx2d(long long v) {
  if (v == 0) return 0.0;
  const unsigned long long a = v < 0 ? (unsigned long long)(-v) : (unsigned long long)v;
  const int lz = __clzll((long long)a);
  const unsigned long long m = lz >= 11 ? a << (lz - 11) : a >> (11 - lz);   // leading bit at 52
  const unsigned long long e = (unsigned long long)(1023 + (63 - lz) - WF_FX);
  return __longlong_as_double((long long)((e << 52) | (m & 0xFFFFFFFFFFFFFull) | (v < 0 ? (1ull << 63) : 0ull)));
}

// ceil(x / d) and floor(x / d) for d > 0 on fixed-point values whose quotient is below 2^30 in magnitude: FP32
// estimate (a 32-bit conversion: the 64-bit one issues at a small fraction of the rate), exact integer correction
__device__ __forceinline__ long long fx_ceil_div(long long x, long long d, float inv_d) {
  long long k = (long long)(int)ceilf(fminf(fmaxf(fx2f(x) * inv_d, -1073741824.0f), 1073741824.0f));
  while (k * d < x) ++k;
  while ((k - 1) * d >= x) --k;
  return k;
}
__device__ __forceinline__ long long fx_floor_div(long long x, long long d, float inv_d) {
  long long k = (long long)(int)floorf(fminf(fmaxf(fx2f(x) * inv_d, -1073741824.0f), 1073741824.0f));
  while (k * d > x) --k;
  while ((k + 1) * d <= x) ++k;
  return k;
}

// keyed TDC0 in fixed point: the FP64 path's 53 random bits times the phase width
__device__ __forceinline__ long long tdc0_fx_of(const CrvParams& p, const CrvChannels& ch, long long label,
                                                uint32_t run, long long width_fx) {
  const long long evk = label / 32768;
  const int c = int(label % 32768);
  EvKey ek{uint32_t(evk & 0xFFFFF), uint32_t(evk >> 20), run};
  U4 w = keyed(p.seed, ek, ST_TDC0 << 28, uint32_t(feb_key(p, ch, c)));
  const unsigned long long u53 = bits53(w.x, w.y);
  return (long long)__umul64hi(u53 << 11, (unsigned long long)width_fx);
}

struct WfFx {                   // per-launch constants of the fixed-point forms
  long long P, gap, maxt, wlo, whi, width;
  float invP;                   // 1 / P in ns (FP32, for the quotient estimates)
  int nmin;                     // smallest charge count of a kept cluster
  bool ok;
};

__device__ __forceinline__ WfFx wf_fx_consts(const CrvParams& p, double vmax) {
  WfFx f;
  f.ok = d2fx(p.period, &f.P) && d2fx(p.spe_max_time + 4.0 * p.period, &f.gap) && d2fx(p.spe_max_time, &f.maxt) &&
         d2fx(fmax(fmin(p.window_lo, 5e8), -5e8), &f.wlo) && d2fx(fmax(fmin(p.window_hi, 5e8), -5e8), &f.whi) &&
         d2fx(p.feb_phase_width, &f.width) && f.P > 0;
  f.invP = float(1.0 / p.period);              // fx_ceil_div / fx_floor_div estimate on times in ns
  // keep rule n * vmax >= min_voltage (n integer, monotone in n): the smallest such n
  int n = vmax > 0.0 ? int(fmin(ceil(p.min_voltage / vmax), 2e9)) : 2000000000;
  if (n < 0) n = 0;
  while (n > 0 && double(n - 1) * vmax >= p.min_voltage) --n;
  while (n < 2000000000 && !(double(n) * vmax >= p.min_voltage)) ++n;
  f.nmin = n;
  return f;
}

// The FP32 path's cluster record: WfCluster's layout with the fixed-point start time in place of the double.
struct WfCluster32 {
  long long ts_fx;
  long long k0;
  int32_t a, b, L;
  int16_t ilo, ihi;
};
static_assert(sizeof(WfCluster32) == sizeof(WfCluster), "FP32 cluster record layout");

// FP32 form of the prepass (k_wf_prep): fixed-point times, cluster records with the fixed-point start
struct Prep32 {
  using Record = WfCluster32;
  static constexpr bool LIMIT = true;          // times beyond the fixed-point range are refused
  struct Consts {
    WfFx F;
    float ip, Pf;
    int nr;
  };
  static __device__ __forceinline__ Consts consts(const CrvParams& p, double vmax) {
    return Consts{wf_fx_consts(p, vmax), float(1.0 / p.spe_precision), float(p.period), reach_samples(p)};
  }
  static __device__ __forceinline__ bool ok(const Consts& K) { return K.F.ok; }
  static __device__ __forceinline__ bool is_new(const Consts& K, long long tf, long long tp, bool, const double*) {
    return tf - tp > K.F.gap;
  }
  static __device__ __forceinline__ bool keep(const CrvParams&, const Consts& K, int n) { return n >= K.F.nmin; }
  using Tdc0 = long long;
  static __device__ __forceinline__ long long tdc0(const CrvParams& p, const CrvChannels& ch, const Consts& K,
                                                   long long label, uint32_t run) {
    return tdc0_fx_of(p, ch, label, run, K.F.width);
  }
  static __device__ __forceinline__ long long caller_tdc0(double x, Status* status) {
    long long v = 0;
    if (!d2fx(x, &v)) {
      set_flag(status, CRV_ST_LIMIT);
      v = 0;
    }
    return v;
  }
  static __device__ __forceinline__ double tdc0_value(long long v) { return fx2d(v); }
  static __device__ __forceinline__ WfCluster32 record(const CrvParams&, const Consts& K, const double* t, int a, int b,
                                                       long long tdc0, int tlen) {
    const WfFx& F = K.F;
    long long tf, tl;
    if (!d2fx(t[a], &tf) || !d2fx(t[b - 1], &tl)) return WfCluster32{};      // the group is dropped
    const long long k0 = fx_ceil_div(tf - F.P - tdc0, F.P, F.invP);
    const long long ts = k0 * F.P + tdc0;
    const long long est = fx_floor_div(tl - tf + F.maxt, F.P, F.invP);
    // the last charge reaches the last sample (the reach only grows with the charge time)
    const float dt = fx2f(tl - ts);
    long long used = 0;
    const int j0 = first_sample_f(dt, K.Pf);
    for (int k = K.nr - 1; k >= 0; --k)
      if (tmpl_index_f(j0 + k, dt, K.Pf, K.ip, tlen) >= 0) {
        used = j0 + k + 1;
        break;
      }
    const int L = int(est > used ? est : used);
    int ilo = 0, ihi = -1;
    if (L <= 16384) {
      const long long last = ts + (long long)(L - 1) * F.P;
      ilo = ts >= F.wlo ? 0 : int(min((long long)L, fx_ceil_div(F.wlo - ts, F.P, F.invP)));
      ihi = last <= F.whi ? L - 1 : int(max(-1ll, fx_floor_div(F.whi - ts, F.P, F.invP)));
    }
    return WfCluster32{ts, k0, a, b, L, int16_t(ilo), int16_t(ihi)};
  }
};

constexpr int WF32_QS = 256;      // charges staged per chunk (per warp)

__host__ __device__ inline size_t wf32_smem_per_warp(int cap) {
  return (size_t(cap) * 4 + size_t(WF32_QS) * 12 + 15) & ~size_t(15);
}

// Per-block scalars of the synthesis (FP64 work once per block, in one thread) and the template in FP32
struct WfBlock32 {
  float tmpl[1024];
  long long P_fx;
  float P, inv_prec, inv_q, vthr, sigma, conv, off;
  int nr;
};
__device__ __forceinline__ void wf_block32(const CrvParams& p, const double* tmpl, int tlen, WfBlock32& B) {
  for (int i = threadIdx.x; i < tlen; i += blockDim.x) B.tmpl[i] = float(tmpl[i]);
  if (threadIdx.x == 0) {
    long long P;
    B.P_fx = d2fx(p.period, &P) ? P : 0;
    B.P = float(p.period);
    B.inv_prec = float(1.0 / p.spe_precision);
    B.inv_q = float(1.0 / p.spe_ref_charge);
    B.vthr = float(p.min_voltage);
    B.sigma = float(p.noise_sigma);
    B.conv = float(p.adc_conversion);
    B.off = float(double(p.adc_pedestal) + 0.5);
    B.nr = reach_samples(p);
  }
  __syncthreads();
}

// Synthesis + zero suppression of the groups whose clusters have at most 16 samples: two groups per warp, a lane per
// sample, the samples in registers, the neighbours' decisions in ballots.  Sums as k_wf_synth32's for such clusters: every
// other charge of a chunk in a sum of its own, the two added.  Bound by instructions: about 1,040 a cluster where each has a
// warp, most of them (noise, decisions, output, the cluster's scalars) on 10 to 14 lanes.  8.9 million clusters of 65,536
// events, all passes: 11.07 -> 7.97 ms; 280,000 of 2,048 events 417 -> 359 us.  Up to `few` groups (a warp for each on the
// chip) are left to k_wf_synth32, where two in turn on one warp would only take longer (1,900 groups: 24 against 47 us).
constexpr int WF16_QS = WF32_QS;  // charges staged per chunk and group: the chunks of k_wf_synth32
__global__ void __launch_bounds__(256, 4) k_wf_synth16(CrvParams p, WfGroups G, const double* __restrict__ time,
                                                    const double* __restrict__ charge, const double* __restrict__ tmpl,
                                                    int tlen, const double* __restrict__ tdc0_rows,
                                                    const double* __restrict__ g_tdc0,
                                                    const int32_t* __restrict__ g_maxlen,
                                                    const int32_t* __restrict__ g_nkept,
                                                    const WfCluster32* __restrict__ cl, long long few,
                                                    int* __restrict__ taken, DigiSlots D, Status* status) {
  extern __shared__ __align__(16) char smem[];
  __shared__ WfBlock32 B;
  const long long ng = *G.n;
  if (ng <= few) return;                       // a warp for each: left to k_wf_synth32
  if (tlen > 1024) return;                     // refused by the host; the table must fit the shared copy
  wf_block32(p, tmpl, tlen, B);
  const int lane = lane_id(), half = lane >> 4, J = lane & 15, sh = half << 4;
  // (time from the cluster start, normalised charge) of the half's charges; two are read at a time
  float2* sq = reinterpret_cast<float2*>(smem) + (size_t(warp_in_block()) * 2 + half) * WF16_QS;
  const long long P_fx = B.P_fx;
  const int zs = p.samples_zs;
  const float ip = B.inv_prec, inv_q = B.inv_q, vthr = B.vthr, sigma = B.sigma;
  const float JP = __fmul_rn(float(J), B.P);   // rounded before the subtraction, never fused with it
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  const int tile = tile_taken(ng, warps);
  for (long long ti = blockIdx.x * (long long)(blockDim.x >> 5) + warp_in_block(); ti * tile < ng;
       ti = next_tile(taken, warps)) {
   const long long g0 = ti * tile;
   const bool in = lane < tile && g0 + lane < ng;
   const int mll = in ? g_maxlen[g0 + lane] : 0;
   unsigned todo = __ballot_sync(0xffffffffu, mll > 0 && mll <= 16);
   while (todo) {
    const int b0 = __ffs(todo) - 1;
    todo &= todo - 1;
    const int b1 = todo ? __ffs(todo) - 1 : -1;
    if (todo) todo &= todo - 1;
    const int bsel = half ? b1 : b0;
    const bool valid = bsel >= 0;
    const long long g = g0 + (valid ? bsel : b0);
    const long long q0 = G.start[g];
    const double* t = time + q0;
    const double* qc = charge + q0;
    const long long lab = G.label[g];
    const uint32_t run = G.run ? G.run[g] : 0u;
    const long long evk = lab / 32768;
    const EvKey ek{uint32_t(evk & 0xFFFFF), uint32_t(evk >> 20), run};
    const uint32_t chan = uint32_t(lab % 32768);
    const double tdc0g = g_tdc0[g];
    const long long slot = D.off[g];
    const int scap = D.cap[g];
    const int nk = valid ? g_nkept[g] : 0;
    int nd = 0;
#pragma unroll 1
    for (int kc = 0; __any_sync(0xffffffffu, kc < nk); ++kc) {
      const bool act = kc < nk;
      WfCluster32 C{};
      if (act) C = cl[q0 + kc];
      const int L = C.L;
      const long long k0 = C.k0, ts = C.ts_fx;
      float wave = 0.0f;
      int left = C.b - C.a, c0 = C.a;
#pragma unroll 1
      while (__any_sync(0xffffffffu, left > 0)) {
        const int nq = min(WF16_QS, max(left, 0));
        const int most = max(nq, __shfl_xor_sync(0xffffffffu, nq, 16));
        __syncwarp();
        for (int i = J; i < most + (most & 1); i += 16) {
          float2 v = make_float2(3e38f, 0.0f);           // (behind the half's charges: later than every sample)
          if (i < nq) {
            long long tf = 0;
            d2fx(t[c0 + i], &tf);
            v = make_float2(fx2f(tf - ts), d2f_trunc(qc[c0 + i]) * inv_q);
          }
          sq[i] = v;
        }
        __syncwarp();
        float even = 0.0f, odd = 0.0f;
#pragma unroll 2
        for (int q = 0; q < most; q += 2) {
          const float4 v = *reinterpret_cast<const float4*>(sq + q);
          // nearest integer of st / precision (ties to even) by the 1.5 x 2^23 shift; |st / precision| < 2^22
          const float se = __fsub_rn(JP, v.x), so = __fsub_rn(JP, v.z);
          const int te = __float_as_int(fmaf(se, ip, 12582912.0f)) - 0x4B400000;
          const int to = __float_as_int(fmaf(so, ip, 12582912.0f)) - 0x4B400000;
          if (se >= 0.0f && te < tlen) even = fmaf(B.tmpl[te], v.y, even);
          if (so >= 0.0f && to < tlen) odd = fmaf(B.tmpl[to], v.w, odd);
        }
        wave = wave + (even + odd);
        left -= WF16_QS;
        c0 += WF16_QS;
      }
      // keyed electronics noise on every sample
      if (p.noise_on && J < L) {
        const long long tk = k0 + J;
        U4 w = keyed(p.seed, ek, (ST_NOISE << 28) | (chan & 0x7FFFu), uint32_t(tk >> 1));
        float z0, z1;
        Math<float>::normal_pair(w, &z0, &z1);
        wave = wave + sigma * ((tk & 1) ? z1 : z0);
      }
      // zero suppression: samples with one above the threshold among their neighbours up to two away, in the window
      const unsigned over = (__ballot_sync(0xffffffffu, J < L && wave > vthr) >> sh) & 0xFFFFu;
      const unsigned near = over | over << 1 | over << 2 | over >> 1 | over >> 2;
      unsigned cand = (__ballot_sync(0xffffffffu, J < L && ((near >> J) & 1u) && J >= C.ilo && J <= C.ihi) >> sh) & 0xFFFFu;
#pragma unroll 1
      while (__any_sync(0xffffffffu, cand != 0u)) {
        const bool on = cand != 0u;
        const int i0 = on ? __ffs(cand) - 1 : 0;
        const bool put = on && nd < scap;
        const long long o = slot + nd;
        for (int k = J; k - J < zs; k += 16) {
          const int c = i0 + k;
          const float x = __shfl_sync(0xffffffffu, wave, sh + (c & 15));
          const float v = c < L ? x : 0.0f;
          if (put && k < zs) {
            if (D.volt) D.volt[o * zs + k] = f2d(v);
            D.adc[o * zs + k] = adc_of_f(p, v, B.conv, B.off);
          }
        }
        if (put && J == 0) {
          D.chan[o] = lab;
          D.start[o] = fx2d(ts + (long long)i0 * P_fx);
          D.tdc0[o] = tdc0_rows ? tdc0_rows[q0 + C.a] : tdc0g;
          D.starttdc[o] = k0 + i0;
        }
        if (on) {
          ++nd;
          cand = i0 + zs < 16 ? cand >> (i0 + zs) << (i0 + zs) : 0u;
        }
      }
    }
    if (valid && J == 0) {
      D.n[g] = nd;
      if (nd > scap) set_flag(status, CRV_ST_CAPACITY);
    }
   }
  }
}

// Synthesis + zero suppression of the groups whose longest kept cluster is in (lo, cap] (FP32-mixed).
__global__ void __launch_bounds__(256, 4) k_wf_synth32(CrvParams p, WfGroups G, const double* __restrict__ time,
                                                    const double* __restrict__ charge, const double* __restrict__ tmpl,
                                                    int tlen, const double* __restrict__ tdc0_rows,
                                                    const double* __restrict__ g_tdc0,
                                                    const int32_t* __restrict__ g_maxlen,
                                                    const int32_t* __restrict__ g_nkept,
                                                    const WfCluster32* __restrict__ cl, int lo, int cap,
                                                    int last_pass, long long few, const int* __restrict__ longest,
                                                    int* __restrict__ taken, DigiSlots D, Status* status) {
  extern __shared__ __align__(16) char smem[];
  if (lo >= WF_LONG && *longest <= lo) return;
  __shared__ WfBlock32 B;
  char* wbase = smem + size_t(warp_in_block()) * wf32_smem_per_warp(cap);
  float* wave = reinterpret_cast<float*>(wbase);
  float2* sq = reinterpret_cast<float2*>(wbase + size_t(cap) * 4);              // (dt, normalised charge)
  int* sj = reinterpret_cast<int*>(wbase + size_t(cap) * 4 + size_t(WF32_QS) * 8);  // first sample reached
  if (tlen > 1024) return;                     // refused by the host; the table must fit the shared copy
  wf_block32(p, tmpl, tlen, B);
  const float* const tmpl_f = B.tmpl;
  const long long P_fx = B.P_fx;
  const int nr = B.nr;
  const int zs = p.samples_zs;
  const int lane = lane_id();
  const float Pf = B.P, ip = B.inv_prec;
  const float inv_q = B.inv_q;
  const float vthr = B.vthr;
  const float sigma = B.sigma;
  const float conv_f = B.conv, off_f = B.off;
  const long long ng = *G.n;
  if (ng <= few && lo == 16) lo = 0;           // (k_wf_synth16 leaves them to this kernel)
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  // groups in tiles per warp: one coalesced load of their longest clusters and a ballot pick this pass's groups
  const int tile = tile_taken(ng, warps);
  for (long long ti = blockIdx.x * (long long)(blockDim.x >> 5) + warp_in_block(); ti * tile < ng;
       ti = next_tile(taken, warps)) {
   const long long g0 = ti * tile;
   const long long gl = g0 + lane;
   const bool in = lane < tile && gl < ng;
   const int mll = in ? g_maxlen[gl] : 0;
   unsigned todo = __ballot_sync(0xffffffffu, in && mll > lo);
   while (todo) {
    const int bsel = __ffs(todo) - 1;
    todo &= todo - 1;
    const long long g = g0 + bsel;
    const int ml = __shfl_sync(0xffffffffu, mll, bsel);
    if (ml > cap) {
      if (last_pass && lane == 0) {
        set_flag(status, CRV_ST_CAPACITY);
        need_at_least(status, CRV_NEED_SAMPLES, ml);
      }
      continue;
    }
    const long long q0 = G.start[g];
    const double* t = time + q0;
    const double* qc = charge + q0;
    const long long lab = G.label[g];
    const uint32_t run = G.run ? G.run[g] : 0u;
    const long long evk = lab / 32768;
    const EvKey ek{uint32_t(evk & 0xFFFFF), uint32_t(evk >> 20), run};
    const uint32_t chan = uint32_t(lab % 32768);
    const double tdc0g = g_tdc0[g];
    const long long slot = D.off[g];
    const int scap = D.cap[g];
    int nd = 0;
    const int nk = g_nkept[g];
    for (int kc = 0; kc < nk; ++kc) {
      const WfCluster32 C = cl[q0 + kc];
      const int a = C.a, b = C.b, L = C.L;
      const long long k0 = C.k0, ts = C.ts_fx;
      const double tdc0c = tdc0_rows ? tdc0_rows[q0 + a] : tdc0g;
      for (int j = lane; j < L; j += 32) wave[j] = 0.0f;
      // charges in chunks: stage (dt, q) and the first sample reached, then every 32-sample tile the chunk reaches
      for (int c0 = a; c0 < b; c0 += WF32_QS) {
        const int nq = min(WF32_QS, b - c0);
        __syncwarp();
        for (int i = lane; i < nq; i += 32) {
          long long tf = 0;
          d2fx(t[c0 + i], &tf);
          const float dt = fx2f(tf - ts);
          sq[i] = make_float2(dt, d2f_trunc(qc[c0 + i]) * inv_q);
          sj[i] = first_sample_f(dt, Pf);
        }
        __syncwarp();
        const int jA = sj[0];
        const int jB = min(sj[nq - 1] + nr - 1, L - 1);
        for (int T = (jA >> 5) << 5; T <= jB; T += 32) {
          // charges of the chunk that can reach the tile: first sample in (T - nr, T + 31]
          int q1 = 0, q2 = nq;
          if (L > 32) {                            // (one tile: all of them)
            int hi = nq;
            while (q1 < hi) {
              const int m = (q1 + hi) >> 1;
              if (sj[m] > T - nr) hi = m; else q1 = m + 1;
            }
            q2 = q1;
            hi = nq;
            while (q2 < hi) {
              const int m = (q2 + hi) >> 1;
              if (sj[m] > T + 31) hi = m; else q2 = m + 1;
            }
          }
          // a cluster of at most 16 samples (most of them) takes two lanes per sample, each summing every other
          // charge; the two partial sums are added in a fixed order, so the result is the same on every run
          const int split = L <= 16 ? 1 : 0;
          const int J = T + (split ? (lane & 15) : lane);
          const int part = split ? (lane >> 4) : 0;
          const float JP = __fmul_rn(float(J), Pf);      // rounded before the subtraction, never fused with it
          float acc = 0.0f;
#pragma unroll 4
          for (int q = q1 + part; q < q2; q += 1 + split) {
            const float2 v = sq[q];
            const float st = __fsub_rn(JP, v.x);
            // nearest integer of st / precision (ties to even) by the 1.5 x 2^23 shift; |st / precision| < 2^22
            const int ti = __float_as_int(fmaf(st, ip, 12582912.0f)) - 0x4B400000;
            if (st >= 0.0f && ti < tlen) acc = fmaf(tmpl_f[ti], v.y, acc);
          }
          const float other = __shfl_down_sync(0xffffffffu, acc, 16);
          if (split) acc = acc + other;
          if (J < L && (split ? lane < 16 : true)) wave[J] = wave[J] + acc;
        }
      }
      __syncwarp();
      // keyed electronics noise on every sample
      if (p.noise_on) {
        for (int j = lane; j < L; j += 32) {
          const long long tk = k0 + j;
          U4 w = keyed(p.seed, ek, (ST_NOISE << 28) | (chan & 0x7FFFu), uint32_t(tk >> 1));
          float z0, z1;
          Math<float>::normal_pair(w, &z0, &z1);
          wave[j] = wave[j] + sigma * ((tk & 1) ? z1 : z0);
        }
        __syncwarp();
      }
      // zero suppression over tiles of 32 samples
      const int i_lo = C.ilo, i_hi = C.ihi;
      int next_i = 0;
      for (int base = 0; base < L; base += 32) {
        const int i = base + lane;
        bool w = false;
        if (i < L) {
          for (int d = -2; d <= 2 && !w; ++d) {
            const int k = i + d;
            if (k >= 0 && k < L && wave[k] > vthr) w = true;
          }
        }
        const bool inwin = i >= i_lo && i <= i_hi;
        const unsigned cand = __ballot_sync(0xffffffffu, w && inwin);
        while (true) {
          unsigned m = cand;
          if (next_i > base) m &= (next_i - base >= 32) ? 0u : ~((1u << (next_i - base)) - 1u);
          if (!m) break;
          const int i0 = base + __ffs(m) - 1;
          if (nd < scap) {
            const long long o = slot + nd;
            if (lane < zs) {
              const int c = i0 + lane;
              const float v = c < L ? wave[c] : 0.0f;
              if (D.volt) D.volt[o * zs + lane] = f2d(v);
              D.adc[o * zs + lane] = adc_of_f(p, v, conv_f, off_f);
            }
            if (lane == 0) {
              D.chan[o] = lab;
              D.start[o] = fx2d(ts + (long long)i0 * P_fx);
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

}  // namespace crv
