// Response stage: CrvSteps -> photons at the SiPMs -> SiPM charges.
//
// Photon counts per (step, SiPM) follow the reference rule Gauss(mean, sqrt mean) if mean > 10 else Poisson(mean),
// rint, floor at 0 (crv/crvfastsim/response/photons.py:102-112) with the analytic yield x two-exponential attenuation
// in place of the lookup tables; SiPMs 0/2 read the -length end and 1/3 the +length end (photons.py:333-356).
//
// The SiPM model is the reference's serial one (crv/crvfastsim/response/sipm.py:141-198): per SiPM, photons in time
// order; a pixel fires with p1 (1 - e^(-v/p2)), v = Vov (1 - e^(-(t - t_last)/tau)); each firing draws cross-talk
// on its 4 neighbours, handled breadth first with multiplicity merging 1 - (1 - p)^m before the next photon; trap
// afterpulses are scheduled per firing and fired after all photons in time order.
//
// GPU mapping: one warp per SiPM.  The warp draws every photon's pixel and fire uniform as it loads it and keeps only
// those that can fire (4 in 10), in time order, in shared memory beside the pixel state (last-discharge time per pixel +
// a fired bitmap); it then steps through them with their first-generation cross-talk, one touch of a pixel per lane
// (simulate_sipm).  Keyed draws make every lane's random numbers independent of the processing order, so the result is
// exactly the serial one.
//
// What bounds the SiPM kernel: instruction issue and instruction fetch.  All warps are at different places of one large
// loop body; DRAM traffic is 2 % of the peak.  Measured on 65,536 workload events (7.8 M SiPMs of 85 photons, FP32):
// evaluating all 85 photons in the serial step 79.3 ms; only those that can fire, with their first generation in the
// step, all inlined (98 KB of code, 59 % of the fetches hit) 79.7 ms; photons and nodes in one lane order (62 KB)
// 42.0 ms; rare paths as calls with one copy of Philox (51 KB) 36.0 ms; all first-pass draws as calls, 20 warps instead
// of 16 per SM 33.0 ms.  FP64, 1,500 events: 14.4 -> 4.3 ms (draws decided on integers, most photons never reach FP64).
#pragma once
#include "crv_device.cuh"
#include "crv_scan.cuh"

namespace crv {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

template <typename S>
__device__ __forceinline__ double ld_real(const void* p, long long i) {
  return double(static_cast<const S*>(p)[i]);
}

__device__ __forceinline__ double step_real(const CrvSteps& st, const void* p, long long i) {
  return st.real_bytes == 4 ? double(static_cast<const float*>(p)[i]) : static_cast<const double*>(p)[i];
}

// ---------------------------------------------------------------------------------------------------------------------
// event preparation: steps of each event grouped by bar (stable), per-step event index, SiPM count per event

constexpr int PREP_THREADS = 256;

#ifdef CRV_ENGINE_TU
// keys: bar << 16 | step-in-event; sorted ascending in shared memory (bitonic, block-wide)
__device__ void block_bitonic_u32(uint32_t* a, int P) {
  for (int size = 2; size <= P; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int q = threadIdx.x; q < (P >> 1); q += blockDim.x) {
        int lo = 2 * stride * (q / stride) + (q % stride);
        int hi = lo + stride;
        bool up = (lo & size) == 0;
        uint32_t x = a[lo], y = a[hi];
        if ((x > y) == up) { a[lo] = y; a[hi] = x; }
      }
      __syncthreads();
    }
  }
}

// mode 0: count SiPMs per event (sipm_count); mode 1: write the SiPM table at sipm_off
__global__ void k_event_prep(CrvEvents ev, long long nevents, CrvSteps st, CrvChannels ch, int masked,
                             int step_cap, int32_t* __restrict__ step_event, int32_t* __restrict__ step_order,
                             int32_t* __restrict__ sipm_count, const long long* __restrict__ sipm_off,
                             int32_t* __restrict__ s_event, int32_t* __restrict__ s_chan,
                             long long* __restrict__ s_seg, int32_t* __restrict__ s_nseg, Status* status, int mode) {
  extern __shared__ uint32_t keys[];
  __shared__ int wcount[PREP_THREADS / 32];
  for (long long e = blockIdx.x; e < nevents; e += gridDim.x) {
    long long f = ev.first_step[e];
    int n = ev.nsteps[e];
    if (mode == 0 && step_event)
      for (int i = threadIdx.x; i < n; i += blockDim.x) step_event[f + i] = int32_t(e);
    if (n > step_cap || n >= 65536) {
      if (threadIdx.x == 0) {
        if (n >= 65536) set_flag(status, CRV_ST_LIMIT);
        else { set_flag(status, CRV_ST_CAPACITY); need_at_least(status, CRV_NEED_STEPS_PER_EVENT, n); }
        if (mode == 0) sipm_count[e] = 0;
      }
      continue;
    }
    int P = 1;
    while (P < n) P <<= 1;
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
      if (i < n) {
        int b = st.bar[f + i];
        keys[i] = (uint32_t(b) << 16) | uint32_t(i);
      } else {
        keys[i] = 0xFFFFFFFFu;
      }
    }
    __syncthreads();
    block_bitonic_u32(keys, P);
    if (mode == 0 && step_order)
      for (int i = threadIdx.x; i < n; i += blockDim.x) step_order[f + i] = int32_t(f + (keys[i] & 0xFFFFu));
    // segments: thread i starts a segment if bar differs from i-1
    int mine = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      uint32_t b = keys[i] >> 16;
      if (i == 0 || (keys[i - 1] >> 16) != b) {
        for (int s = 0; s < 4; ++s) {
          int c = int(b) * 4 + s;
          bool ok = !masked || (ch.status[c] & 0b101) == 0;
          mine += ok;
        }
      }
    }
    if (mode == 0) {
      int tot = warp_sum(mine);
      if (lane_id() == 0) wcount[warp_in_block()] = tot;
      __syncthreads();
      if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += wcount[w];
        sipm_count[e] = t;
      }
      __syncthreads();
    } else {
      // serial write in segment order by thread 0 (events are small; keeps label order)
      if (threadIdx.x == 0) {
        long long o = sipm_off[e];
        for (int i = 0; i < n;) {
          uint32_t b = keys[i] >> 16;
          int j = i;
          while (j < n && (keys[j] >> 16) == b) ++j;
          for (int s = 0; s < 4; ++s) {
            int c = int(b) * 4 + s;
            if (masked && (ch.status[c] & 0b101) != 0) continue;
            s_event[o] = int32_t(e);
            s_chan[o] = c;
            s_seg[o] = f + i;
            s_nseg[o] = j - i;
            ++o;
          }
          i = j;
        }
      }
      __syncthreads();
    }
  }
}

#endif  // CRV_ENGINE_TU

// ---------------------------------------------------------------------------------------------------------------------
// photon counts and arrival times

template <typename R>
__device__ __forceinline__ R readout_distance(R z, R half, int s) {
  R d = (s % 2 == 0) ? (z + half) : (half - z);
  if (d < R(0)) d = R(0);
  if (d > R(2) * half) d = R(2) * half;
  return d;
}

template <typename R>
__device__ __forceinline__ R mean_photons(const CrvParams& p, R edep, R dev, R d) {
  using M = Math<R>;
  R att = R(p.frac_short) * M::exp(-d / R(p.lambda_short)) + R(p.frac_long) * M::exp(-d / R(p.lambda_long));
  return R(p.yield_per_mev) * edep * dev * att;
}

template <typename R>
__device__ __forceinline__ int draw_count(R avg, const U4& w) {
  using M = Math<R>;
  R x;
  if (avg > R(10)) {
    R z0, z1;
    M::normal_pair(w, &z0, &z1);
    x = avg + sqrt(avg) * z0;
  } else {
    R lam = avg > R(0) ? avg : R(0);
    R u = M::uni(w, 0);
    R pk = M::exp(-lam);
    R F = pk;
    int k = 0;
    while (u >= F && k < 200) {
      k += 1;
      pk = pk * lam / R(k);
      F = F + pk;
    }
    x = R(k);
  }
  x = rint(x);
  return x > R(0) ? int(x) : 0;
}


// count[4 * i + s]: photons of step i on SiPM s (masked channels 0 when `masked`)
template <typename R>
__global__ void k_photon_count(CrvParams p, CrvEvents ev, CrvSteps st, CrvBars bars, CrvChannels ch,
                               const int32_t* __restrict__ step_event, long long nsteps,
                               const long long* __restrict__ nsteps_dev, int masked, int32_t* __restrict__ count,
                               Status* status) {
  nsteps = bounded_count(nsteps, nsteps_dev);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nsteps;
       i += (long long)gridDim.x * blockDim.x) {
    int e = step_event[i];
    int sie = int(i - ev.first_step[e]);
    int b = st.bar[i];
    double t = step_real(st, st.t, i);
    if (!isfinite(t)) {
      for (int s = 0; s < 4; ++s) count[4 * i + s] = 0;
      continue;
    }
    int ax = bars.length_axis[b];
    double pos = step_real(st, ax == 0 ? st.x : (ax == 1 ? st.y : st.z), i);
    double z = pos - bars.center_l[b];
    double half = bars.half_l[b];
    R edep = R(step_real(st, st.edep, i));
    EvKey ek{ev.event[e], ev.subrun[e], ev.run[e]};
    for (int s = 0; s < 4; ++s) {
      int c = b * 4 + s;
      int n = 0;
      if (!masked || (ch.status[c] & 0b101) == 0) {
        R d = readout_distance(R(z), R(half), s);
        R avg = mean_photons<R>(p, edep, R(ch.yield_factor[c]), d);
        U4 w = keyed(p.seed, ek, w2_of(ST_COUNT, 0, 0, 0, uint32_t(c)), uint32_t(sie));
        n = draw_count<R>(avg, w);
        if (n > 65536) { set_flag(status, CRV_ST_LIMIT); n = 65536; }
      }
      count[4 * i + s] = n;
    }
  }
}

#ifdef CRV_ENGINE_TU
// per SiPM of the table: photons on it, slot capacity for its charges, photon-id base (event's first step row)
__global__ void k_sipm_sizes(const long long* __restrict__ nsipm_dev, const int32_t* __restrict__ s_event, const int32_t* __restrict__ s_chan,
                             const long long* __restrict__ s_seg, const int32_t* __restrict__ s_nseg,
                             const int32_t* __restrict__ step_order, const int32_t* __restrict__ count,
                             CrvEvents ev, int charge_factor, int32_t* __restrict__ nphot,
                             int32_t* __restrict__ slot_cap, long long* __restrict__ id_base,
                             long long* __restrict__ label, uint32_t* __restrict__ run,
                             int32_t* __restrict__ nmain, int32_t* __restrict__ nap, int32_t* __restrict__ fired) {
  long long nsipm = *nsipm_dev;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < nsipm;
       g += (long long)gridDim.x * blockDim.x) {
    int s = s_chan[g] & 3;
    long long a = s_seg[g];
    int n = 0;
    for (int k = 0; k < s_nseg[g]; ++k) n += count[4 * (long long)step_order[a + k] + s];
    nphot[g] = n;
    slot_cap[g] = n > 0 ? charge_factor * n + 16 : 0;
    int e = s_event[g];
    id_base[g] = ev.first_step[e];
    long long evkey = ((long long)ev.subrun[e] << 20) | (long long)ev.event[e];
    label[g] = evkey * 32768 + s_chan[g];
    run[g] = ev.run[e];
    nmain[g] = 0;                // the SiPM stage writes the SiPMs with photons only, and none at an overflow
    nap[g] = 0;
    fired[g] = 0;
  }
}

#endif  // CRV_ENGINE_TU

// Emission delays, in decay times, of a row of n photons (every lane of the warp calls it): the order statistics of n
// exponential delays by the Renyi representation, S_j = sum_{i <= j} X_i / (n - i) with X_i = -log u_i and u_i photon i's
// keyed uniform.  The delays have the distribution of n independent exponential delays; photon j (key j) takes the j-th
// smallest, so every row's photons come out in time order.  Sums: over 32 photons at a time an inclusive Hillis-Steele
// scan (offsets 1, 2, 4, 8, 16), the earlier ones' total in front; the CPU oracle adds in the same order, so FP64 sums are
// identical.  A Philox block holds two photons' uniforms: a lane draws for two photons where more than 32 are left, and
// the terms move to the lanes of the scans.  emit(j, S_j) is called by the lane of photon j.
template <typename R>
__device__ __forceinline__ R delay_sums(R v, R* carry) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const R y = __shfl_up_sync(0xffffffffu, v, off);
    if (lane_id() >= off) v = v + y;
  }
  const R S = *carry + v;
  *carry = *carry + __shfl_sync(0xffffffffu, v, 31);
  return S;
}
template <typename R, typename Emit>
__device__ __forceinline__ void row_delays(uint32_t seed, const EvKey& ek, uint32_t chan, uint32_t sie, int n, Emit emit) {
  using M = Math<R>;
  const int lane = lane_id();
  const uint32_t w2 = w2_of(ST_PHOTON, 0, 0, 0, chan);
  R carry = R(0);
  for (int c0 = 0; c0 < n; c0 += 64) {
    const bool two = n - c0 > 32;
    const int j0 = c0 + (two ? 2 * lane : lane);
    R x0 = R(0), x1 = R(0);
    if (j0 < n) {
      const U4 w = keyed(seed, ek, w2, (sie << 16) | uint32_t(j0 >> 1));
      x0 = (-M::log(M::uni_open(w, two ? 0 : j0 & 1))) / R(n - j0);
      if (two && j0 + 1 < n) x1 = (-M::log(M::uni_open(w, 1))) / R(n - j0 - 1);
    }
    R a = x0, b = R(0);
    if (two) {
      const R e0 = __shfl_sync(0xffffffffu, x0, lane >> 1), e1 = __shfl_sync(0xffffffffu, x1, lane >> 1);
      const R f0 = __shfl_sync(0xffffffffu, x0, 16 + (lane >> 1)), f1 = __shfl_sync(0xffffffffu, x1, 16 + (lane >> 1));
      a = (lane & 1) ? e1 : e0;
      b = (lane & 1) ? f1 : f0;
    }
    const R S = delay_sums(a, &carry);
    if (c0 + lane < n) emit(c0 + lane, S);
    if (two) {
      const R T = delay_sums(b, &carry);
      if (c0 + 32 + lane < n) emit(c0 + 32 + lane, T);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// SiPM simulation: one warp per SiPM

// scheduled afterpulses per SiPM: a SiPM of at most 256 photons fires at most a few hundred pixels, with trap-0
// probabilities of a few percent; beyond the queue the SiPM reports CRV_ST_LIMIT
__host__ __device__ constexpr int sipm_tcap(int cap) { return cap <= 256 ? 32 : 128; }

struct SipmGroups {
  const long long* n;            // device: number of groups
  const long long* guard[2];     // device totals that must not exceed guard_cap (else the pass is skipped)
  long long guard_cap[2];
  const long long* start;        // first photon row of the group
  const int32_t* count;          // photons in the group
  const long long* label;        // SiPM label
  const uint32_t* run;
  const uint32_t* key32;         // draw key per photon (chain) ...
  const long long* key64;        // ... or per photon as int64 (stage API); neither: the photon's index in its SiPM
  const long long* photon_id;    // photon id per photon (stage API), or null: id = id_base[g] + (key >> 16)
  const long long* id_base;
  const long long* slot_off;     // output slot region of the group
  const int32_t* slot_cap;
  int* taken;                    // counts of tiles taken, one for each pass that hands them out (zeroed before)
};
constexpr int SIPM_PASSES = 2, RESP_COUNTS = SIPM_PASSES + 2;   // counts of tiles taken: passes, photons, compaction

struct SipmOut {
  double* t;
  double* v;
  long long* id;
  int32_t* nmain;                // charges from photons and cascades (time order)
  int32_t* nap;                  // afterpulse charges (time order), stored after the main ones
  int32_t* fired;                // pixels that fired at least once
};

// The staged photons are those that can fire (see k_sipm_sim): time, draw key, and the pixel with a flag.
constexpr uint32_t PH_PIX = 0x7FFu;      // pixel id (below 1,681)
constexpr uint32_t PH_FIRES = 0x8000u;   // its fire uniform is below the firing probability at full overvoltage

// A warp's shared memory: CAP photons; LOC: the photons' positions in the group are kept (ph_loc), for per-photon ids
// (photon_id); without them a warp needs 4 bytes less per photon and more warps fit an SM.  One byte offset and
// compile-time offsets from it, so the layout costs one register, passes to the called functions as it is, and every
// access is a shared-memory one there too.
extern __shared__ __align__(16) char sipm_smem[];
template <typename R, int CAP, bool LOC>
struct SipmShared {
  static constexpr int TCAP = sipm_tcap(CAP);                      // afterpulse queue length
  // Last-discharge times.  First pass: per pixel the number of its last charge record, and the records' times (FT of
  // them; a SiPM of at most 256 photons has at most 272 charge slots, and one with more charges is reported, its
  // results dropped).  Other passes, where a pixel fires over and over: the time per pixel.
  static constexpr bool BY_RECORD = CAP <= 256;
  static constexpr int FT = 288;
  static constexpr int O_FT = NPS_ALLOC * 2;
  static constexpr int O_T = BY_RECORD ? O_FT + FT * int(sizeof(R)) : NPS_ALLOC * int(sizeof(R)), O_TRT = O_T + CAP * int(sizeof(R)),
                       O_TRU = O_TRT + TCAP * int(sizeof(R)), O_TRI = O_TRU + TCAP * int(sizeof(R)),
                       O_KEY = O_TRI + TCAP * 8, O_LOC = O_KEY + CAP * 4, O_BM = O_LOC + (LOC ? CAP * 4 : 0),
                       O_MISC = O_BM + 64 * 4, O_CAND = O_MISC + 16, O_TRP = O_CAND + 256 * 2,
                       O_FRP = O_TRP + TCAP * 2, O_FRM = O_FRP + 64 * 2, O_PIX = O_FRM + 64 * 2,
                       BYTES = (O_PIX + CAP * 2 + 15) / 16 * 16;
  static_assert(O_TRI % 8 == 0, "afterpulse ids on 8 bytes");
  int base;
  template <typename T>
  __device__ __forceinline__ T* at(int off) const { return reinterpret_cast<T*>(sipm_smem + base + off); }
  __device__ __forceinline__ R last(int q) const {
    if constexpr (BY_RECORD) return at<R>(O_FT)[at<uint16_t>(0)[q]];
    else return at<R>(0)[q];
  }
  // pixel q fired at time t, charge record k; `top`: no later touch of q in this step
  __device__ __forceinline__ void set_last(int q, int k, R t, bool top = true) const {
    if constexpr (BY_RECORD) {
      k = min(k, FT - 1);
      at<R>(O_FT)[k] = t;
      if (top) at<uint16_t>(0)[q] = uint16_t(k);
    } else {
      if (top) at<R>(0)[q] = t;
    }
  }
  __device__ __forceinline__ R* ph_t() const { return at<R>(O_T); }
  __device__ __forceinline__ uint32_t* ph_key() const { return at<uint32_t>(O_KEY); }
  __device__ __forceinline__ uint32_t* ph_loc() const { return at<uint32_t>(O_LOC); }
  __device__ __forceinline__ uint16_t* ph_pix() const { return at<uint16_t>(O_PIX); }   // PH_PIX | PH_FIRES
  __device__ __forceinline__ uint32_t* bm() const { return at<uint32_t>(O_BM); }
  __device__ __forceinline__ R* tr_t() const { return at<R>(O_TRT); }
  __device__ __forceinline__ R* tr_uf() const { return at<R>(O_TRU); }
  __device__ __forceinline__ long long* tr_id() const { return at<long long>(O_TRI); }
  __device__ __forceinline__ uint16_t* tr_pix() const { return at<uint16_t>(O_TRP); }
  __device__ __forceinline__ uint16_t* fr_pix() const { return at<uint16_t>(O_FRP); }
  __device__ __forceinline__ uint16_t* fr_m() const { return at<uint16_t>(O_FRM); }
  // 256 cross-talk candidates; also the photon step's 32 node words
  __device__ __forceinline__ uint16_t* cand() const { return at<uint16_t>(O_CAND); }
  __device__ __forceinline__ uint32_t* nodes() const { return at<uint32_t>(O_CAND); }
  __device__ __forceinline__ int* misc() const { return at<int>(O_MISC); }   // [0..3] run_cascade's results
};

__device__ __forceinline__ bool bm_test(const uint32_t* bm, int p) { return (bm[p >> 5] >> (p & 31)) & 1u; }
__device__ __forceinline__ void bm_set(uint32_t* bm, int p) { atomicOr(&bm[p >> 5], 1u << (p & 31)); }

// The integer a uniform is made of (uni = bits * 2^-53 in FP64, * 2^-24 in FP32, both exact) and the threshold T of a
// probability q with bits < T exactly when uni < q: a draw is then decided by one integer compare, without building
// the uniform (in FP64 two conversions, a multiplication and a compare on the FP64 pipe).
template <typename R> struct UniBits;
template <> struct UniBits<double> {
  using T = unsigned long long;
  static __device__ __forceinline__ T of(const U4& w, int h) { return h ? bits53(w.z, w.w) : bits53(w.x, w.y); }
  static __device__ __forceinline__ T below(double q) {
    const double x = q * 0x1p53;
    if (!(x > 0.0)) return 0ull;
    if (x >= 0x1p53) return 1ull << 53;
    const T k = (T)x;
    return k + (double(k) < x ? 1ull : 0ull);
  }
};
template <> struct UniBits<float> {
  using T = uint32_t;
  static __device__ __forceinline__ T of(const U4& w, int h) { return (h ? w.z : w.x) >> 8; }
  static __device__ __forceinline__ T below(float q) {
    const float x = q * 0x1p24f;
    if (!(x > 0.0f)) return 0u;
    if (x >= 0x1p24f) return 1u << 24;
    const T k = (T)x;
    return k + (float(k) < x ? 1u : 0u);
  }
};

// floor(u * 1600) of the pixel draw.  FP64: u = k 2^-53, so the exact product is m 2^-47 with m = 25 k; the FP64
// product rounds it to 53 bits, which reaches the next integer exactly when the fraction lies within half a unit of
// it (at the half the even neighbour is that integer).  Integer instructions, the FP64 product's result.
__device__ __forceinline__ int map_bin(double, unsigned long long k) {
  const unsigned long long m = k * 25ull;
  int b = int(m >> 47);
  const int s = 11 - __clzll((long long)m);      // bits the product is rounded by
  if (s > 0 && (m & ((1ull << 47) - 1ull)) >= (1ull << 47) - (1ull << (s - 1))) ++b;
  return b;
}
__device__ __forceinline__ int map_bin(float, uint32_t k) {
  return int(floorf(float(k) * 0x1p-24f * float(NPX)));
}

// Photon-map bin by the CDF (GetRandom2), then the pixel id of the point: "truncate" keeps the bin, "lrint" rounds
// the point, i.e. moves to the next pixel in x and in y each with probability 1/2 (crv/crvfastsim/response/sipm.py:
// 80-91).  The two halves are bits 0 and 1 of the draw word whose low bits the bin uniform does not use.
static __device__ __noinline__ int map_search(const double* cum, double u) {
  const double v = u * cum[NPX - 1];
  int lo = 0, hi = NPX;
#pragma unroll 1
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (cum[mid] <= v) lo = mid + 1; else hi = mid;
  }
  return lo;
}
template <typename R>
__device__ __forceinline__ int draw_pixel(const CrvParams& p, const CrvPixels& px, const uint32_t* dead, const U4& w) {
  int b;
  if (p.uniform_map) {
    b = map_bin(R(0), UniBits<R>::of(w, 0));
  } else {
    b = map_search(px.cum, double(Math<R>::uni(w, 0)));
  }
  if (b > NPX - 1) b = NPX - 1;
  if (b < 0) b = 0;
  int q = b + b / 40;                            // x * 41 + y of x = b / 40, y = b % 40
  if (p.pixel_lrint) q += PXS * int(w.y & 1u) + int((w.y >> 1) & 1u);
  return ((dead[q >> 5] >> (q & 31)) & 1u) ? -1 : q;
}

// SiPM constants in the compute type, converted once per block (held in shared memory: in the FP32 kernels a
// conversion from the FP64 parameters inside the per-photon code would issue on the narrow FP64 pipe every time)
template <typename R>
struct SipmK {
  R vov, tau, p1, p2, life0, life1, t_end;
  R inv_tau, inv_p2;             // reciprocals, rounded
  int plain;                     // tau or p2 too large or small for div_const
  typename UniBits<R>::T t_ct, t_t0, t_t1;       // cross-talk and trap draws
  typename UniBits<R>::T t_fire;                 // a pixel at full overvoltage fires
  typename UniBits<R>::T t_cand;                 // a photon at or above it fires on no pixel, whatever its state
  float t_end_dn;                // largest float <= t_end: float times compare with it exactly as with t_end
  int ct_on, t0_on, t1_on, npx, npy;
};

// Correctly rounded a / b for a constant b of ordinary size, from y = 1 / b rounded (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990: two corrections by the exact remainder).  Five instructions;
// the division's own sequence and slow path are 1.9 KB of code a copy in FP32, a dozen FP64 instructions in FP64.
// Quotients below the normal range may differ in their last bits and a zero's sign is lost, neither of which an
// exponential of the result sees.  An infinite or NaN first product (a pixel that fired at -infinity) is the quotient: the
// remainder of it would be NaN.
template <typename R>
__device__ __noinline__ R div_plain(R a, R b) { return a / b; }
__device__ __forceinline__ float fma_r(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_r(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_r(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_r(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7F800000u) == 0x7F800000u; }
__device__ __forceinline__ bool not_finite(double x) { return (__double2hiint(x) & 0x7FF00000) == 0x7FF00000; }
template <typename R>
__device__ __forceinline__ R div_const(R a, R b, R y, int plain) {
  if (plain) return div_plain<R>(a, b);
  R q = mul_r(a, y);
  if (not_finite(q)) return q;
  q = fma_r(fma_r(-q, b, a), y, q);
  return fma_r(fma_r(-q, b, a), y, q);
}

template <typename R>
__device__ __forceinline__ R pfire(const SipmK<R>& K, R v) {
  using M = Math<R>;
  return K.p1 * (R(1) - M::exp(div_const<R>(-v, K.p2, K.inv_p2, K.plain)));
}

// probability that a node hit m times fires: 1 - (1 - pfire)^m
template <typename R>
__device__ __forceinline__ R pfire_m(const SipmK<R>& K, R v, int m) {
  R q = R(1) - pfire<R>(K, v);
  R qm = q;
#pragma unroll 1
  for (int i = 1; i < m; ++i) qm = qm * q;
  return R(1) - qm;
}

template <typename R>
__device__ __noinline__ void sipm_consts(const CrvParams& p, SipmK<R>& K) {
  K.vov = R(p.overvoltage); K.tau = R(p.time_constant); K.p1 = R(p.p1); K.p2 = R(p.p2);
  K.life0 = R(p.trap0_lifetime); K.life1 = R(p.trap1_lifetime); K.t_end = R(p.t_end);
  K.t_end_dn = __double2float_rd(p.t_end);
  K.ct_on = p.q_ct > 0.0; K.t0_on = p.q_t0 > 0.0; K.t1_on = p.q_t1 > 0.0;
  K.t_ct = UniBits<R>::below(R(p.q_ct)); K.t_t0 = UniBits<R>::below(R(p.q_t0)); K.t_t1 = UniBits<R>::below(R(p.q_t1));
  K.npx = p.n_pixels_x; K.npy = p.n_pixels_y;
  K.inv_tau = R(1) / K.tau;
  K.inv_p2 = R(1) / K.p2;
  const auto odd = [](R x) { return !((x > R(1e-9) && x < R(1e9)) || (x < R(-1e-9) && x > R(-1e9))); };
  K.plain = odd(K.tau) || odd(K.p2) || !(K.vov > R(-1e9) && K.vov < R(1e9));
  const R pm = pfire_m<R>(K, K.vov, 1);
  K.t_fire = UniBits<R>::below(pm);
  // A recovering pixel has 0 <= v <= overvoltage (photons come in time order), and pfire grows with v, so no state
  // fires a photon that a full pixel would not; 1e-6 covers the rounding of the exponentials many times over.  With
  // constants of other signs every photon on a live pixel is kept.
  const bool grows = K.vov >= R(0) && K.tau > R(0) && K.p1 >= R(0) && K.p2 > R(0);
  K.t_cand = grows ? UniBits<R>::below(pm + R(1e-6)) : UniBits<R>::below(R(2));
}

// recovered overvoltage at time t of a pixel that fired last at t0
template <typename R>
__device__ __forceinline__ R recovered_from(const SipmK<R>& K, R t, R t0) {
  using M = Math<R>;
  return K.vov * (R(1) - M::exp(div_const<R>(-(t - t0), K.tau, K.inv_tau, K.plain)));
}
// recovered overvoltage of pixel q at time t (Vov if it never fired)
template <typename R, int CAP, bool LOC>
__device__ __forceinline__ R recovered(const SipmK<R>& K, const SipmShared<R, CAP, LOC>& S, int q, R t) {
  if (!bm_test(S.bm(), q)) return K.vov;
  return recovered_from<R>(K, t, S.last(q));
}

// Per SiPM context while simulating.
struct SipmCtx {
  EvKey ek;
  uint32_t chan;
  long long slot;          // first output slot
  int cap;                 // output slots
  int nq;                  // main records so far (may exceed cap: counting only)
  int ntr;                 // scheduled afterpulses
  int limit;               // a key/capacity limit was hit
};

// A draw as a call: the kernel's warps are all at different places of a large loop body, so its speed hangs on how much
// of that body the instruction cache holds (with everything inlined 98 KB of code, half of the fetches missed).
static __device__ __noinline__ U4 keyed_call(uint32_t seed, EvKey ek, uint32_t w2, uint32_t w3) {
  return keyed(seed, ek, w2, w3);
}

// The photon step's draws: called in the first pass; inlined in the others, whose few warps per SM wait for their own
// instructions' results more than for the cache.
template <int CAP>
__device__ __forceinline__ U4 draw(uint32_t seed, const EvKey& ek, uint32_t w2, uint32_t w3) {
  if constexpr (CAP <= 256) return keyed_call(seed, ek, w2, w3);
  else return keyed(seed, ek, w2, w3);
}

// Schedule the afterpulses of a fired node (trap0: call 1 (u, u_time), call 4 word 0-1 (u_fire);
// trap1: call 4 word 2-3 (u), call 5 (u_time, u_fire)) from its call-1 draw a.  Returns how many were scheduled into
// (t, uf).
template <typename R>
struct Traps {
  R t[2], uf[2];
  int n;
};
template <typename R>
__device__ __noinline__ Traps<R> schedule_traps(uint32_t seed, const SipmK<R>& K, EvKey ek, uint32_t w2, uint32_t key,
                                                R t, U4 a, bool trap0) {
  using M = Math<R>;
  Traps<R> o;
  o.t[0] = o.t[1] = o.uf[0] = o.uf[1] = R(0);
  o.n = 0;
  const U4 b = keyed_call(seed, ek, w2 | (4u << 15), key);
  if (trap0) {
    o.t[0] = t - K.life0 * M::log(M::uni_open(a, 1));
    o.uf[0] = M::uni(b, 0);
    o.n = 1;
  }
  if (K.t1_on && UniBits<R>::of(b, 1) < K.t_t1) {
    const U4 c = keyed_call(seed, ek, w2 | (5u << 15), key);
    const R t1 = t - K.life1 * M::log(M::uni_open(c, 0)), u1 = M::uni(c, 1);
    if (o.n) { o.t[1] = t1; o.uf[1] = u1; }
    else { o.t[0] = t1; o.uf[0] = u1; }
    ++o.n;
  }
  return o;
}
template <typename R>
__device__ __forceinline__ int node_traps(uint32_t seed, const SipmK<R>& K, const SipmCtx& C, uint32_t gen,
                                          uint32_t idx, uint32_t key, R t, const U4& a, R* tt, R* uf) {
  const bool trap0 = K.t0_on && UniBits<R>::of(a, 0) < K.t_t0;
  if (!trap0 && !K.t1_on) return 0;              // call 4 is only read by a trap-0 afterpulse or the trap-1 draw
  const Traps<R> o = schedule_traps<R>(seed, K, C.ek, w2_of(ST_SIPM, gen, idx, 0, C.chan), key, t, a, trap0);
  tt[0] = o.t[0]; tt[1] = o.t[1];
  uf[0] = o.uf[0]; uf[1] = o.uf[1];
  return o.n;
}

// Neighbours of a pixel in increasing pixel order: bit 0 x - 1, bit 1 y - 1, bit 2 y + 1, bit 3 x + 1.
__device__ __forceinline__ int neighbour(int pix, int q) {
  return pix + (q == 0 ? -PXS : (q == 1 ? -1 : (q == 2 ? 1 : PXS)));
}

// cross-talk candidates of a fired node among the neighbours inside the grid, from its draws: xa / xb bit 0 and bit 1
// set for call 2's (x - 1, x + 1) and call 3's (y - 1, y + 1) uniforms below the cross-talk probability
template <typename R>
__device__ __forceinline__ unsigned crosstalk_mask(const SipmK<R>& K, unsigned xa, unsigned xb, int pix) {
  const int x = pix / PXS, y = pix - PXS * x;
  unsigned m = 0;
  if (x > 0) m |= xa & 1u;
  if (y > 0) m |= (xb & 1u) << 1;
  if (y + 1 < K.npy) m |= (xb & 2u) << 1;
  if (x + 1 < K.npx) m |= (xa & 2u) << 2;
  return m;
}

template <typename R>
__device__ __forceinline__ unsigned node_crosstalk(uint32_t seed, const SipmK<R>& K, const SipmCtx& C,
                                                   uint32_t gen, uint32_t idx, uint32_t key, int pix) {
  using B = UniBits<R>;
  if (!K.ct_on) return 0;
  U4 a = keyed_call(seed, C.ek, w2_of(ST_SIPM, gen, idx, 2, C.chan), key);
  U4 b = keyed_call(seed, C.ek, w2_of(ST_SIPM, gen, idx, 3, C.chan), key);
  const unsigned xa = unsigned(B::of(a, 0) < K.t_ct) | (unsigned(B::of(a, 1) < K.t_ct) << 1);
  const unsigned xb = unsigned(B::of(b, 0) < K.t_ct) | (unsigned(B::of(b, 1) < K.t_ct) << 1);
  if ((xa | xb) == 0u) return 0;
  return crosstalk_mask<R>(K, xa, xb, pix);
}

// Append a charge record (lane-ordered position pos relative to C.nq) if it fits.
// widening to the FP64 output columns (FP32: by integer bit arithmetic, off the FP64 pipe)
__device__ __forceinline__ double widen(double x) { return x; }
__device__ __forceinline__ double widen(float x) { return f2d(x); }

template <typename R>
__device__ __forceinline__ void put_charge(const SipmOut& O, const SipmCtx& C, int pos, R t, R v, long long id) {
  int k = C.nq + pos;
  if (k < C.cap) {
    long long o = C.slot + k;
    O.t[o] = widen(t);
    O.v[o] = widen(v);
    O.id[o] = id;
  }
}

// Queue a lane's n (0..2) scheduled afterpulses at position pos of the queue.
template <typename R, int CAP, bool LOC>
__device__ __forceinline__ void put_traps(const SipmShared<R, CAP, LOC>& S, int pos, int n, const R* tt, const R* uf, int pix,
                                          long long id) {
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    if (a >= n) break;
    const int k = pos + a;
    if (k < S.TCAP) { S.tr_t()[k] = tt[a]; S.tr_uf()[k] = uf[a]; S.tr_pix()[k] = uint16_t(pix); S.tr_id()[k] = id; }
  }
}

// Build the next frontier from the candidate list (lane 0): sort, unique with multiplicity, drop dead.
template <typename R, int CAP, bool LOC>
__device__ __forceinline__ int make_frontier(const SipmShared<R, CAP, LOC>& S, int nc, const uint32_t* dead, int* limit) {
  int nf = 0;
  if (lane_id() == 0) {
#pragma unroll 1
    for (int a = 1; a < nc; ++a) {           // insertion sort (tiny lists)
      uint16_t x = S.cand()[a];
      int b = a - 1;
#pragma unroll 1
      while (b >= 0 && S.cand()[b] > x) { S.cand()[b + 1] = S.cand()[b]; --b; }
      S.cand()[b + 1] = x;
    }
#pragma unroll 1
    for (int a = 0; a < nc;) {
      int b = a;
#pragma unroll 1
      while (b < nc && S.cand()[b] == S.cand()[a]) ++b;
      int q = S.cand()[a];
      if (!((dead[q >> 5] >> (q & 31)) & 1u)) {
        if (nf > MAX_IDX) { *limit = 1; break; }
        S.fr_pix()[nf] = uint16_t(q);
        S.fr_m()[nf] = uint16_t(b - a);
        ++nf;
      }
      a = b;
    }
    S.misc()[3] = nf;
  }
  __syncwarp();
  nf = S.misc()[3];
  __syncwarp();
  return nf;
}

// Append the drawn neighbours ct of every lane's pixel q to the n candidates; returns how many there are then (at most
// 256 are kept).
template <typename R, int CAP, bool LOC>
__device__ __forceinline__ int put_candidates(const SipmShared<R, CAP, LOC>& S, unsigned ct, int q, int n) {
  const int c = __popc(ct);
  const unsigned b0 = __ballot_sync(FULL, c & 1), b1 = __ballot_sync(FULL, c & 2), b2 = __ballot_sync(FULL, c & 4);
  int at = n + __popc(b0 & lanemask_lt()) + 2 * __popc(b1 & lanemask_lt()) + 4 * __popc(b2 & lanemask_lt());
#pragma unroll 1
  for (unsigned m = ct; m; m &= m - 1u, ++at)
    if (at < 256) S.cand()[at] = uint16_t(neighbour(q, __ffs(m) - 1));
  return n + __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
}

// Cross-talk cascade of one photon from generation 2 on; the frontier is spread over the lanes.  ct: the lane's drawn
// neighbours of its pixel pix (0: none, or a node of another photon).  Generation 1 is part of the photon step (simulate_sipm), so this runs for the few photons whose
// cascade goes further; called, not inlined, to keep the photon step's code and registers small.  C.nq, C.ntr and
// C.limit come back in S.misc()[0..2].
template <typename R, int CAP, bool LOC>
__device__ __noinline__ void run_cascade(uint32_t seed, const SipmK<R>& K, SipmShared<R, CAP, LOC> S,
                                         const uint32_t* dead, SipmCtx C, const SipmOut& O, unsigned ct, int pix, int src,
                                         R t, uint32_t key, long long id) {
  t = __shfl_sync(FULL, t, src);
  key = __shfl_sync(FULL, key, src);
  id = __shfl_sync(FULL, id, src);
  int nc = put_candidates(S, ct, pix, 0);
  __syncwarp();
  uint32_t gen = 2;
  int lim = 0;
#pragma unroll 1
  while (true) {
    const int nf = make_frontier(S, nc, dead, &lim);
    lim = __shfl_sync(FULL, lim, 0);
    if (lim || nf == 0) break;
    if (gen > MAX_GEN) { lim = 1; break; }
    int ncand = 0;
#pragma unroll 1
    for (int base = 0; base < nf; base += 32) {
      int i = base + lane_id();
      bool act = i < nf;
      int q = act ? S.fr_pix()[i] : 0;
      R v = R(0);
      bool fire = false;
      if (act) {
        v = recovered(K, S, q, t);
        R pm = pfire_m<R>(K, v, S.fr_m()[i]);
        U4 w = keyed_call(seed, C.ek, w2_of(ST_SIPM, gen, uint32_t(i), 0, C.chan), key);
        fire = Math<R>::uni(w, 1) < pm;
      }
      unsigned fm = __ballot_sync(FULL, fire);
      int pos = __popc(fm & lanemask_lt());
      R tt[2], uf[2];
      int ntr = 0;
      unsigned ct = 0;
      if (fire) {
        put_charge<R>(O, C, pos, t, v, id);
        S.set_last(q, C.nq + pos, t);
        bm_set(S.bm(), q);
        if (K.t0_on || K.t1_on) {
          const U4 a = keyed_call(seed, C.ek, w2_of(ST_SIPM, gen, uint32_t(i), 1, C.chan), key);
          ntr = node_traps<R>(seed, K, C, gen, uint32_t(i), key, t, a, tt, uf);
        }
        ct = node_crosstalk<R>(seed, K, C, gen, uint32_t(i), key, q);
      }
      C.nq += __popc(fm);
      // traps and candidates in node order
      const unsigned a1 = __ballot_sync(FULL, ntr > 0), a2 = __ballot_sync(FULL, ntr > 1);
      put_traps(S, C.ntr + __popc(a1 & lanemask_lt()) + __popc(a2 & lanemask_lt()), ntr, tt, uf, q, id);
      C.ntr += __popc(a1) + __popc(a2);
      ncand = put_candidates(S, ct, q, ncand);
      __syncwarp();
    }
    if (ncand > 256) { lim = 1; break; }
    ++gen;
    nc = ncand;
  }
  lim = __any_sync(FULL, lim) || C.limit;
  if (lane_id() == 0) { S.misc()[0] = C.nq; S.misc()[1] = C.ntr; S.misc()[2] = lim; }
  __syncwarp();
}

// A touch at time t of a pixel that fired last at t0, with fire draw fb: recovered overvoltage and whether it fires.
// Called: few touches meet a pixel that has fired.
template <typename R>
struct Touch {
  R v;
  bool fire;
};
template <typename R>
__device__ __noinline__ Touch<R> touch_again(const SipmK<R>& K, R t, R t0, typename UniBits<R>::T fb) {
  Touch<R> o;
  o.v = recovered_from<R>(K, t, t0);
  o.fire = fb < UniBits<R>::below(pfire_m<R>(K, o.v, 1));
  return o;
}

// Serial-semantics simulation of one SiPM whose n staged photons (those that can fire, in time order) sit in S.ph_*.
//
// The serial order of events is: photon, its first-generation cross-talk nodes in pixel order, the rest of its cascade,
// next photon.  A step takes the next photons and their first-generation nodes (about one photon in eight has any), as
// many as fit a warp, one touch per lane in that order.  All draws are keyed, so the step has them before anything is
// decided.  A touch whose pixel no earlier touch of the step names is decided at once, against the state the step
// starts from; the others (one step in four has one) are decided one at a time in order, each against the last touch
// before it that fired.  A node fires only if its photon did.  The step then commits everything, or, when a fired node
// starts a second generation, everything up to that photon, whose cascade continues in run_cascade.
template <typename R, int CAP, bool LOC>
__device__ __forceinline__ void simulate_sipm(const CrvParams& p, const SipmK<R>& K,
                                              const SipmShared<R, CAP, LOC>& S, const uint32_t* dead, SipmCtx& C,
                                              const SipmOut& O, int n, const long long* photon_id, long long gstart,
                                              long long id_base) {
  using B = UniBits<R>;
  const int lane = lane_id();
  const unsigned lt = lanemask_lt();
  int k = 0;
#pragma unroll 1
  while (k < n) {
    // photons, one per lane: their cross-talk draws (calls 2 and 3) give the first-generation nodes, the drawn
    // neighbours on live pixels in pixel order
    bool has = k + lane < n;
    const uint32_t pkey = has ? S.ph_key()[k + lane] : 0u;
    const uint32_t ppix = has ? uint32_t(S.ph_pix()[k + lane]) : 0u;
    unsigned live = 0;
    if (K.ct_on) {
      unsigned xy = 0;
#pragma unroll 1
      for (uint32_t call = 2; call < 4; ++call) {
        const U4 w = draw<CAP>(p.seed, C.ek, w2_of(ST_SIPM, 0, 0, call, C.chan), pkey);
        xy = (xy >> 2) | (unsigned(B::of(w, 0) < K.t_ct) << 2) | (unsigned(B::of(w, 1) < K.t_ct) << 3);
      }
      if (has && xy) {
        const int pix = int(ppix & PH_PIX);
#pragma unroll 1
        for (unsigned m = crosstalk_mask<R>(K, xy & 3u, xy >> 2, pix); m; m &= m - 1u) {
          const int q = __ffs(m) - 1, np = neighbour(pix, q);
          if (!((dead[np >> 5] >> (np & 31)) & 1u)) live |= 1u << q;
        }
      }
    }
    // the step's touches in serial order: pixel, node flag, index in the generation, photon's lane above, photon's touch
    int take = min(n - k, 32), total = take;
    {
      const int c = has ? 1 + __popc(live) : 0;
      const unsigned b0 = __ballot_sync(FULL, c & 1), b1 = __ballot_sync(FULL, c & 2), b2 = __ballot_sync(FULL, c & 4);
      const int base = __popc(b0 & lt) + 2 * __popc(b1 & lt) + 4 * __popc(b2 & lt);
      has = has && base + c <= 32;
      take = __popc(__ballot_sync(FULL, has));
      total = __shfl_sync(FULL, base + c, take - 1);
      __syncwarp();
      if (has) {
        const uint32_t who = (uint32_t(lane) << 19) | (uint32_t(base) << 24);
        S.nodes()[base] = ppix | who;
        uint32_t at = uint32_t(base), idx = 0;
#pragma unroll 1
        for (unsigned m = live; m; m &= m - 1u, ++idx)
          S.nodes()[++at] = uint32_t(neighbour(int(ppix & PH_PIX), __ffs(m) - 1)) | (1u << 16) | (idx << 17) | who;
      }
      __syncwarp();
    }
    const bool act = lane < total;
    const uint32_t w = act ? S.nodes()[lane] : 0u;
    const int pix = int(w & PH_PIX), pl = int((w >> 19) & 31u), par = int(w >> 24);
    const uint32_t node = (w >> 16) & 1u, idx = (w >> 17) & 3u;
    const uint32_t key = __shfl_sync(FULL, pkey, pl);
    const R t = act ? S.ph_t()[k + pl] : R(0);
    const unsigned same = __match_any_sync(FULL, act ? pix : -1 - lane);
    const bool set = act && bm_test(S.bm(), pix);
    bool dirty = act && (same & lt) != 0u;
    // decisions
    R v = K.vov;
    bool fire = (w & PH_FIRES) != 0u;
    if (__any_sync(FULL, node || set || dirty)) {
      const U4 w0 = draw<CAP>(p.seed, C.ek, w2_of(ST_SIPM, node, idx, 0, C.chan), key);
      const typename B::T fb = B::of(w0, 1);
      if (node) fire = fb < K.t_fire;
      if (set) {
        const Touch<R> o = touch_again<R>(K, t, S.last(pix), fb);
        v = o.v;
        fire = o.fire;
      }
      unsigned dm = __ballot_sync(FULL, dirty);
      dirty = dirty || (node && ((dm >> par) & 1u));
      dm = __ballot_sync(FULL, dirty);
      const bool pfire0 = __shfl_sync(FULL, int(fire && !dirty), par) != 0;
      fire = fire && !dirty && (!node || pfire0);
#pragma unroll 1
      while (dm) {                                 // in serial order
        const int d = __ffs(dm) - 1;
        const int x = __shfl_sync(FULL, pix, d);
        const unsigned m = __ballot_sync(FULL, fire && pix == x) & ((1u << d) - 1u);
        const R tl = __shfl_sync(FULL, t, m ? 31 - __clz(m) : 0);
        const bool pf = __shfl_sync(FULL, int(fire), par) != 0;
        if (lane == d) {
          v = K.vov;
          fire = fb < K.t_fire;
          if (m || set) {
            const Touch<R> o = touch_again<R>(K, t, m ? tl : S.last(pix), fb);
            v = o.v;
            fire = o.fire;
          }
          fire = fire && (!node || pf);
        }
        dm &= dm - 1u;
      }
    }
    // the fired nodes' cross-talk draws, calls 2 and 3 of sixteen nodes per Philox evaluation; the step ends with the
    // first photon that has a node with cross-talk of its own
    unsigned nct = 0;
    int cut = 32;
    const unsigned nfm = __ballot_sync(FULL, fire && node);
    if (nfm && K.ct_on) {
      const bool mine = fire && node;
      const int rank = __popc(nfm & lt), cnt = __popc(nfm);
      if (mine) S.fr_pix()[rank] = uint16_t(lane);
      __syncwarp();
#pragma unroll 1
      for (int g = 0; g < cnt; g += 16) {
        const int j = g + (lane & 15);
        const int src = j < cnt ? S.fr_pix()[j] : 0;
        const uint32_t kk = __shfl_sync(FULL, key, src), ii = __shfl_sync(FULL, idx, src);
        const U4 a = draw<CAP>(p.seed, C.ek, w2_of(ST_SIPM, 1, ii, 2u + uint32_t(lane >> 4), C.chan), kk);
        const unsigned x = unsigned(B::of(a, 0) < K.t_ct) | (unsigned(B::of(a, 1) < K.t_ct) << 1);
        const unsigned xa = __shfl_sync(FULL, x, rank & 15), xb = __shfl_sync(FULL, x, 16 + (rank & 15));
        if (mine && (rank >> 4) == (g >> 4) && (xa | xb)) nct = crosstalk_mask<R>(K, xa, xb, pix);
      }
      const unsigned m2 = __ballot_sync(FULL, nct != 0u);
      if (m2) {
        cut = __shfl_sync(FULL, par, __ffs(m2) - 1);
        fire = fire && par <= cut;
      }
    }
    // commit: charges in serial order, pixel state (the last touch of a pixel stays), afterpulses
    const unsigned fm = __ballot_sync(FULL, fire);
    long long id = 0;
    if (act) id = LOC ? photon_id[gstart + S.ph_loc()[k + pl]] : id_base + (long long)(key >> 16);
    int ntr = 0;
    R tt[2], uf[2];
    if (fire) {
      put_charge<R>(O, C, __popc(fm & lt), t, v, id);
      bm_set(S.bm(), pix);
      S.set_last(pix, C.nq + __popc(fm & lt), t, (same & fm & ~lt) == (1u << lane));
      if (K.t0_on || K.t1_on) {
        const U4 a = draw<CAP>(p.seed, C.ek, w2_of(ST_SIPM, node, idx, 1, C.chan), key);
        ntr = node_traps<R>(p.seed, K, C, node, idx, key, t, a, tt, uf);
      }
    }
    C.nq += __popc(fm);
    const unsigned a1 = __ballot_sync(FULL, ntr > 0);
    if (a1) {
      const unsigned a2 = __ballot_sync(FULL, ntr > 1);
      put_traps(S, C.ntr + __popc(a1 & lt) + __popc(a2 & lt), ntr, tt, uf, pix, id);
      C.ntr += __popc(a1) + __popc(a2);
    }
    __syncwarp();
    if (cut < 32) {
      take = __shfl_sync(FULL, pl, cut) + 1;
      run_cascade(p.seed, K, S, dead, C, O, par == cut ? nct : 0u, pix, cut, t, key, id);
      C.nq = S.misc()[0];
      C.ntr = S.misc()[1];
      C.limit = S.misc()[2];
      __syncwarp();
    }
    k += take;
  }
  if (C.ntr > S.TCAP) C.limit = 1;
}

// Afterpulses after all photons, in (time, schedule order); stored after the main records.  Returns the count.
// Lane 0, one after the other (rare, see run_afterpulses).
template <typename R, int CAP, bool LOC>
__device__ __noinline__ int afterpulses_serial(const SipmK<R>& K, SipmShared<R, CAP, LOC> S, SipmCtx C, const SipmOut& O) {
  const int ntr = min(C.ntr, S.TCAP);
  int nap = 0;
  if (lane_id() == 0) {
    // insertion sort by time (stable: equal times keep schedule order)
#pragma unroll 1
    for (int a = 1; a < ntr; ++a) {
      R x = S.tr_t()[a], xu = S.tr_uf()[a];
      uint16_t xp = S.tr_pix()[a];
      long long xi = S.tr_id()[a];
      int b = a - 1;
#pragma unroll 1
      while (b >= 0 && S.tr_t()[b] > x) {
        S.tr_t()[b + 1] = S.tr_t()[b]; S.tr_uf()[b + 1] = S.tr_uf()[b]; S.tr_pix()[b + 1] = S.tr_pix()[b];
        S.tr_id()[b + 1] = S.tr_id()[b];
        --b;
      }
      S.tr_t()[b + 1] = x; S.tr_uf()[b + 1] = xu; S.tr_pix()[b + 1] = xp; S.tr_id()[b + 1] = xi;
    }
#pragma unroll 1
    for (int a = 0; a < ntr; ++a) {
      R t1 = S.tr_t()[a];
      if (t1 > K.t_end) continue;
      int q = S.tr_pix()[a];
      R v = recovered(K, S, q, t1);
      if (S.tr_uf()[a] < pfire<R>(K, v)) {
        S.set_last(q, C.nq + nap, t1);
        S.bm()[q >> 5] |= 1u << (q & 31);
        put_charge<R>(O, C, nap, t1, v, S.tr_id()[a]);
        ++nap;
      }
    }
  }
  nap = __shfl_sync(FULL, nap, 0);
  __syncwarp();
  return nap;
}

// One per lane when there are at most 32, on pixels that differ: then none decides another.
template <typename R, int CAP, bool LOC>
__device__ __noinline__ int run_afterpulses(const SipmK<R>& K, SipmShared<R, CAP, LOC> S, SipmCtx C,
                                            const SipmOut& O) {
  const int lane = lane_id();
  const bool on = lane < C.ntr;
  const R t = on ? S.tr_t()[lane & (S.TCAP - 1)] : R(0);
  const int q = on ? int(S.tr_pix()[lane & (S.TCAP - 1)]) : 0;
  const unsigned same = __match_any_sync(FULL, on ? q : -1 - lane);
  if (C.ntr > 32 || __any_sync(FULL, on && (same & (same - 1u)) != 0u)) return afterpulses_serial(K, S, C, O);
  R v = R(0);
  bool fire = false;
  if (on && !(t > K.t_end)) {
    v = recovered_from<R>(K, t, S.last(q));        // its pixel has fired
    fire = S.tr_uf()[lane] < pfire<R>(K, v);
  }
  const unsigned fm = __ballot_sync(FULL, fire);
  int pos = 0;                                     // fired before it in (time, schedule) order
#pragma unroll 1
  for (unsigned m = fm; m; m &= m - 1u) {
    const int j = __ffs(m) - 1;
    const R tj = __shfl_sync(FULL, t, j);
    pos += tj < t || (tj == t && j < lane);
  }
  if (fire) put_charge<R>(O, C, pos, t, v, S.tr_id()[lane]);
  return __popc(fm);
}

// Order-preserving integer image of an FP64 time, -0 taken as +0 (as the numeric comparison does): FP64 sort
// comparisons on the integer pipe instead of the FP64 pipe.
__device__ __forceinline__ unsigned long long ord_time(double t) {
  unsigned long long u = (unsigned long long)__double_as_longlong(t);
  if (u == 0x8000000000000000ull) u = 0ull;
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// (ta, ka) > (tb, kb) in (time, key) order
__device__ __forceinline__ bool after(float ta, uint32_t ka, float tb, uint32_t kb) {
  return (ta > tb) || (ta == tb && ka > kb);
}
__device__ __forceinline__ bool after(double ta, uint32_t ka, double tb, uint32_t kb) {
  const unsigned long long a = ord_time(ta), b = ord_time(tb);
  return (a > b) || (a == b && ka > kb);
}

// sort the staged photons by (time, key) (warp bitonic over the next power of two)
template <typename R, int CAP, bool LOC>
__device__ __noinline__ void sort_photons(SipmShared<R, CAP, LOC> S, int n) {
  int P = 1;
  while (P < n) P <<= 1;
#pragma unroll 1
  for (int i = n + lane_id(); i < P; i += 32) {
    S.ph_t()[i] = R(INFINITY);
    S.ph_key()[i] = 0xFFFFFFFFu;
    S.ph_pix()[i] = 0;
    if (LOC) S.ph_loc()[i] = 0xFFFFFFFFu;
  }
  __syncwarp();
#pragma unroll 1
  for (int size = 2; size <= P; size <<= 1) {
#pragma unroll 1
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
#pragma unroll 1
      for (int q = lane_id(); q < (P >> 1); q += 32) {
        const int lo = ((q & ~(stride - 1)) << 1) | (q & (stride - 1));   // stride is a power of two
        const int hi = lo + stride;
        const bool up = (lo & size) == 0;
        const R ta = S.ph_t()[lo], tb = S.ph_t()[hi];
        const uint32_t ka = S.ph_key()[lo], kb = S.ph_key()[hi];
        if (after(ta, ka, tb, kb) == up) {
          S.ph_t()[lo] = tb; S.ph_t()[hi] = ta;
          S.ph_key()[lo] = kb; S.ph_key()[hi] = ka;
          const uint16_t xa = S.ph_pix()[lo];
          S.ph_pix()[lo] = S.ph_pix()[hi]; S.ph_pix()[hi] = xa;
          if (LOC) {
            uint32_t la = S.ph_loc()[lo];
            S.ph_loc()[lo] = S.ph_loc()[hi]; S.ph_loc()[hi] = la;
          }
        }
      }
      __syncwarp();
    }
  }
}

// Errors of a SiPM: more charges than slots, a key limit (limit > 0), more photons than the last pass takes (limit < 0).
static __device__ __noinline__ void sipm_report(Status* status, int charges, int cap, int photons, int limit) {
  if (limit < 0) {
    set_flag(status, CRV_ST_CAPACITY);
    need_at_least(status, CRV_NEED_PHOTONS_PER_SIPM, photons);
    return;
  }
  if (charges > cap) {
    set_flag(status, CRV_ST_CAPACITY);
    const long long per = photons > 0 ? (charges - 16 + photons - 1) / photons : 1;
    need_at_least(status, CRV_NEED_CHARGE_FACTOR, per < 1 ? 1 : per);
  }
  if (limit) set_flag(status, CRV_ST_LIMIT);
}

// Warps per block.  First pass: 24 warps of 8.8 KB of shared memory fit an SM in FP32, as two blocks of 80 registers a
// thread (20 warps of 96 registers: 29.2 instead of 27.3 ms for 65,536 events); 20 of 11.2 KB in FP64 (24 with their
// spills: 2.28 instead of 2.12 ms for 1,500 events).  The later passes have room for 11 warps or fewer, in one block.
template <typename R>
__host__ __device__ constexpr int sipm_block_warps(int cap) { return cap > 256 ? 16 : sizeof(R) == 4 ? 12 : 10; }

// draw key of photon i of a group that starts at row a
template <bool LOC>
__device__ __forceinline__ uint32_t draw_key(const SipmGroups& G, long long a, int i) {
  if constexpr (!LOC) return G.key32[a + i];       // the chain's own photons
  else return G.key64 ? uint32_t(G.key64[a + i]) : uint32_t(i);
}

// SiPM stage over photon groups (PT: storage type of the photon times)
template <typename R, typename PT, int CAP, bool LOC>
__global__ void __launch_bounds__(sipm_block_warps<R>(CAP) * 32, CAP <= 256 ? 2 : 1) k_sipm_sim(const __grid_constant__ CrvParams p, CrvPixels px, SipmGroups G,
                                                 const PT* __restrict__ ph_time, int lo, int last_pass,
                                                 const __grid_constant__ SipmOut O, Status* status) {
  __shared__ uint32_t dead[64];
  __shared__ SipmK<R> K;
  for (int i = threadIdx.x; i < 64; i += blockDim.x) dead[i] = i < DEAD_WORDS ? px.dead_bits[i] : 0u;
  if (threadIdx.x == 0) sipm_consts<R>(p, K);
  __syncthreads();
  const SipmShared<R, CAP, LOC> S{warp_in_block() * SipmShared<R, CAP, LOC>::BYTES};
  for (int q = 0; q < 2; ++q)
    if (G.guard[q] && *G.guard[q] > G.guard_cap[q]) return;
  const long long ngroups = *G.n;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  // groups in tiles per warp: one coalesced load of their counts and a ballot pick the groups of this pass (a
  // later pass, which holds few groups, does not walk every group with a dependent load)
  const int tile = tile_size(ngroups, warps);
  for (long long ti = blockIdx.x * (long long)(blockDim.x >> 5) + warp_in_block(); ti * tile < ngroups;
       ti = CAP > 1024 ? ti + warps : next_tile(G.taken + (CAP > 256), warps)) {
   const long long g0 = ti * tile, gl = g0 + lane_id();
   const bool in = lane_id() < tile && gl < ngroups;
   const int cl = in ? G.count[gl] : 0;
   unsigned todo = __ballot_sync(FULL, in && cl > lo);
   while (todo) {
    const int bsel = __ffs(todo) - 1;
    todo &= todo - 1;
    const long long g = g0 + bsel;
    const int cnt = __shfl_sync(FULL, cl, bsel);
    long long a = G.start[g];
    long long lab = G.label[g];
    SipmCtx C;
    long long evk = lab / 32768;
    C.ek = EvKey{uint32_t(evk & 0xFFFFF), uint32_t(evk >> 20), G.run[g]};
    C.chan = uint32_t(lab % 32768);
    C.slot = G.slot_off[g];
    C.cap = G.slot_cap[g];
    C.nq = 0;
    C.ntr = 0;
    C.limit = 0;
    if (cnt > CAP) {
      if (lane_id() == 0 && last_pass) {
        sipm_report(status, 0, 0, cnt, -1);
        O.nmain[g] = 0; O.nap[g] = 0; O.fired[g] = 0;
      }
      continue;
    }
    // Stage the photons with t <= t_end that can fire: on a live pixel, with a fire uniform below t_cand (4 in 10 of
    // them; the others change nothing).  The next 32 photons are loaded while these are drawn; one copy of the draw
    // in the code (four chunks per step unrolled took 20 KB more of it than the instruction cache has room for).
    int n = 0;
    PT tn = PT(0);
    uint32_t kn = 0;
    if (lane_id() < cnt) {
      tn = ph_time[a + lane_id()];
      kn = draw_key<LOC>(G, a, lane_id());
    }
#pragma unroll 1
    for (int base = 0; base < cnt; base += 32) {
      const int i = base + lane_id();
      const PT tv = tn;
      const uint32_t kv = kn;
      if (i + 32 < cnt) {
        tn = ph_time[a + i + 32];
        kn = draw_key<LOC>(G, a, i + 32);
      }
      bool keep;
      if constexpr (sizeof(PT) == 4) keep = i < cnt && (float(tv) <= K.t_end_dn);
      else keep = i < cnt && (double(tv) <= p.t_end);
      const U4 w = draw<CAP>(p.seed, C.ek, w2_of(ST_SIPM, 0, 0, 0, C.chan), kv);
      const typename UniBits<R>::T fb = UniBits<R>::of(w, 1);
      keep = keep && fb < K.t_cand;
      int pix = -1;
      if (keep) pix = draw_pixel<R>(p, px, dead, w);
      keep = pix >= 0;
      const unsigned km = __ballot_sync(FULL, keep);
      if (keep) {
        const int o = n + __popc(km & lanemask_lt());
        S.ph_t()[o] = R(tv);
        S.ph_key()[o] = kv;
        S.ph_pix()[o] = uint16_t(uint32_t(pix) | (fb < K.t_fire ? PH_FIRES : 0u));
        if (LOC) S.ph_loc()[o] = uint32_t(i);
      }
      n += __popc(km);
    }
    for (int w = lane_id(); w < 64; w += 32) S.bm()[w] = 0u;
    __syncwarp();
    // the photons of one (step, SiPM) row come out of the photon stage in (time, key) order, so a SiPM hit by one
    // step needs no sort: check the order, sort only when it is broken
    bool ordered = true;
#pragma unroll 1
    for (int i = lane_id(); i + 1 < n; i += 32)
      ordered = ordered && !after(S.ph_t()[i], S.ph_key()[i], S.ph_t()[i + 1], S.ph_key()[i + 1]);
    if (!__all_sync(FULL, ordered)) sort_photons(S, n);
    const long long idb = G.id_base ? G.id_base[g] : 0;
    simulate_sipm(p, K, S, dead, C, O, n, G.photon_id, a, idb);
    const int nap = C.ntr ? run_afterpulses(K, S, C, O) : 0;
    int fired = 0;
    for (int w = lane_id(); w < DEAD_WORDS; w += 32) fired += __popc(S.bm()[w]);
    fired = warp_sum(fired);
    if (lane_id() == 0) {
      O.nmain[g] = C.nq;
      O.nap[g] = nap;
      O.fired[g] = fired;
      if (C.nq + nap > C.cap || C.limit) sipm_report(status, C.nq + nap, C.cap, cnt, C.limit);
    }
    __syncwarp();
   }
  }
}

#ifdef CRV_ENGINE_TU
// compaction: merge each group's main and afterpulse runs by time into the output at out_off[g]
__global__ void k_charge_compact(const long long* __restrict__ ngroups_dev, const long long* __restrict__ glabel,
                                 const long long* __restrict__ slot_off, const int32_t* __restrict__ slot_cap,
                                 const int32_t* __restrict__ nmain, const int32_t* __restrict__ nap,
                                 const long long* __restrict__ out_off, const double* __restrict__ st,
                                 const double* __restrict__ sv, const long long* __restrict__ sid, double capacitance,
                                 double overvoltage, int fp32, CrvCharges out, long long out_cap,
                                 int* __restrict__ taken) {
  // out.pe and out.photon may be null (the resident chain reads label, time and charge only): not written
  // FP32-mixed: voltages are FP32 values; charge and PE in FP32 (no FP64 multiply and division per charge)
  const float cap_f = float(capacitance), inv_vov_f = 1.0f / float(overvoltage);
  long long ngroups = *ngroups_dev;
  long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  // groups in tiles per warp: one coalesced load of their sizes and offsets, then the non-empty ones in order
  const int tile = tile_taken(ngroups, warps);
  for (long long ti = blockIdx.x * (long long)(blockDim.x >> 5) + warp_in_block(); ti * tile < ngroups;
       ti = next_tile(taken, warps)) {
   const long long g0 = ti * tile, gl = g0 + lane_id();
   int nm_l = 0, na_l = 0;
   long long s0_l = 0, o0_l = 0, lab_l = 0;
   bool ok = false;
   if (lane_id() < tile && gl < ngroups) {
     nm_l = nmain[gl];
     na_l = nap[gl];
     s0_l = slot_off[gl];
     o0_l = out_off[gl];
     lab_l = glabel[gl];
     // an overflowed group (reported through the status) or one beyond the output is not written
     ok = nm_l + na_l > 0 && nm_l + na_l <= slot_cap[gl] && o0_l + nm_l + na_l <= out_cap;
   }
   unsigned todo = __ballot_sync(0xffffffffu, ok);
   while (todo) {
    const int bsel = __ffs(todo) - 1;
    todo &= todo - 1;
    const int nm = __shfl_sync(0xffffffffu, nm_l, bsel), na = __shfl_sync(0xffffffffu, na_l, bsel);
    const long long s0 = __shfl_sync(0xffffffffu, s0_l, bsel), o0 = __shfl_sync(0xffffffffu, o0_l, bsel);
    const long long lab = __shfl_sync(0xffffffffu, lab_l, bsel);
    // rank of each record in the merged order: main i -> i + #(ap with t < t_main_i);
    // ap j -> j + #(main with t <= t_ap_j)
    for (int i = lane_id(); i < nm + na; i += 32) {
      long long src = s0 + i;
      double t = st[src];
      int r;
      if (i < nm) {
        int c = 0;
        for (int j = 0; j < na; ++j) c += st[s0 + nm + j] < t;
        r = i + c;
      } else {
        int lo = 0, hi = nm;       // main records are time ordered: count main with t_main <= t
        while (lo < hi) {
          int mid = (lo + hi) >> 1;
          if (st[s0 + mid] <= t) lo = mid + 1; else hi = mid;
        }
        r = (i - nm) + lo;
      }
      long long o = o0 + r;
      double v = sv[src];
      out.label[o] = lab;
      out.time[o] = t;
      if (fp32) {
        const float vf = d2f_trunc(v);
        out.charge[o] = f2d(cap_f * vf);
        if (out.pe) out.pe[o] = f2d(vf * inv_vov_f);
      } else {
        out.charge[o] = capacitance * v;
        if (out.pe) out.pe[o] = v / overvoltage;
      }
      if (out.photon) out.photon[o] = sid[src];
    }
   }
  }
}

#endif  // CRV_ENGINE_TU

}  // namespace crv
