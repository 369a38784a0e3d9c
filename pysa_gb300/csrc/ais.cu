// ais.cu -- annealed importance sampling and exact log Z (sm_103a).
//
// k_ais restates ais_sample (pysa/simulation.py:293-317) with the acceptance
// rule of update_spin_ref (pysa/ising.py:66-92, pysa/qubo.py:66-92):
//   full = beta dn + (1 - beta) log(p0(s') / p0(s)),  accept iff full >= 0
//   or log(u) < full.  The uniform reference gives a zero log ratio; the
// Bernoulli reference (pysa/ais.py:198-217) gives +-log((1 - p) / p) when a
// bit goes up / down.  Layout as in the plain sweep (warp = GW samples,
// lanes over columns, local fields in registers) but every sample runs its
// whole anneal inside one launch: samples never interact.  The log weight of
// each anneal step is accumulated in f64 (pysa/simulation.py:312-314), after
// the sweep ("reference" order) or before it ("standard" order).
//
// k_logz_exact enumerates all 2^n states in Gray-code order in f64, with an
// online log-sum-exp per thread.
#include <type_traits>

#include "aux.cuh"
#include "ais_api.h"

namespace pysa_gb {

// accept_full on full = beta dn + (1 - beta) refd.  With the uniform
// reference (refd = 0) full = beta dn is exact in f64 and its f32 rounding
// is the f32 product, so the fast path runs on the FP32 pipe (far faster
// than this GPU's FP64 one) and f64 is left to the band's exact rule; the
// decisions are accept_full's.
__device__ __forceinline__ bool ais_accept(float beta, float dn, bool sbit,
                                           double lr, bool uniform_ref,
                                           uint32_t x) {
  if (!uniform_ref) {
    const double refd = sbit ? -lr : lr;  // bit going down : up
    return accept_full(
        (double)beta * (double)dn + (1.0 - (double)beta) * refd, x);
  }
  if (dn != dn) return false;  // as accept_full on a NaN
  // full >= 0: a zero factor or factors of one sign
  if (dn == 0.0f || beta == 0.0f || ((dn > 0.0f) == (beta > 0.0f)))
    return true;
  const float ff = beta * dn;  // == (float)full
  if (ff < -24.0f) return false;
  const float uf = __uint2float_rn(x) * 0x1p-32f + 0x1p-33f;
  const float lf = __logf(uf);
  const float margin = 3e-5f + 1e-6f * fabsf(ff);
  if (lf < ff - margin) return true;
  if (lf > ff + margin) return false;
  return accept_full_slow((double)beta * (double)dn, x);
}

// Log-weight increment of one temperature step,
// (-beta e - (1 - beta) re) - (-beta_old e - (1 - beta_old) re), re the
// reference's log-probability of the state; with the uniform reference
// re = 0 and only the two f32-rounded products remain (same value)
__device__ __forceinline__ double ais_dlw(float beta, float beta_old, float e,
                                         int n, int ones, double logp,
                                         double log1p_, bool uniform_ref) {
  if (uniform_ref)
    return (double)__fmul_rn(-beta, e) - (double)__fmul_rn(-beta_old, e);
  const double re = -((double)(n - ones) * logp + (double)ones * log1p_);
  return ((double)__fmul_rn(-beta, e) - (1.0 - (double)beta) * re) -
         ((double)__fmul_rn(-beta_old, e) - (1.0 - (double)beta_old) * re);
}

template <int NC, int GW>
__global__ void __launch_bounds__(128) k_ais(const AisArgs a) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int inst = blockIdx.y;
  if (a.replicas[inst] != 1) {
    if (blockIdx.x == 0 && threadIdx.x == 0) set_status(a.status, PYSA_GB_ERR_ARG);
    return;
  }
  const int n = a.n_tab[inst];
  const int ld = a.ld_tab[inst];
  const int64_t samples = a.reads[inst];
  const int64_t cbase = a.chain_off[inst];
  const float* Jp = a.J + a.j_off[inst];
  const int64_t s0 = (int64_t)warp * GW;
  if (s0 >= samples) return;
  const bool ising = a.problem_type == PYSA_GB_ISING;
  const int words = (n + 31) >> 5;

  float H[GW][NC];
  uint32_t spin[GW][NC];  // word m = spins 32m..32m+31 (same in every lane)
#pragma unroll
  for (int g = 0; g < GW; ++g) {
    const int64_t smp = s0 + g;
    const bool valid = smp < samples;
#pragma unroll
    for (int m = 0; m < NC; ++m) {
      const int col = 32 * m + lane;
      H[g][m] = (valid && col < n)
                    ? a.fields[(cbase + smp) * a.field_ld + col] : 0.0f;
      spin[g][m] =
          (valid && m < words) ? a.spins[(cbase + smp) * a.words + m] : 0u;
    }
  }
  const int gl = lane < GW ? lane : 0;
  const bool lane_valid = lane < GW && s0 + lane < samples;
  const int64_t my = s0 + gl;         // sample index within the instance
  const int64_t myc = cbase + my;     // its chain
  double E = lane_valid ? (double)a.energies[myc] : 0.0;
  int ones = 0;  // bits at 1 (spin +1 / x = 1) of lane g's sample
  if (lane_valid)
    for (int w = 0; w < words; ++w) ones += __popc(a.spins[myc * a.words + w]);
  double lw = 0.0;
  float beta_old = 0.0f;
  const double lr = a.ref == 1 ? log((1.0 - a.p) / a.p) : 0.0;
  const double logp = a.ref == 1 ? log(a.p) : 0.0;
  const double log1p_ = a.ref == 1 ? log(1.0 - a.p) : 0.0;

  for (int k = 0; k < a.num_temps; ++k) {
    const float beta = a.temps[k];
    if (a.order == 1) {
      lw += ais_dlw(beta, beta_old, (float)E, n, ones, logp, log1p_,
                    a.ref != 1);
    }
    const int32_t* perm =
        a.perm + ((int64_t)k * a.num_instances + inst) * a.max_n;
    for (int t = 0; t < n; ++t) {
      const int i = a.update == PYSA_GB_RANDOM ? perm[t] : t;
      const int m = i >> 5, l = i & 31;
      float hv = 0.0f;
      uint32_t word = 0;
#pragma unroll
      for (int g = 0; g < GW; ++g) {
        float hm = H[g][0];
        uint32_t wm = spin[g][0];
#pragma unroll
        for (int mm = 1; mm < NC; ++mm) {
          hm = (mm == m) ? H[g][mm] : hm;
          wm = (mm == m) ? spin[g][mm] : wm;
        }
        const float v = __shfl_sync(0xffffffffu, hm, l);
        if (lane == g) {
          hv = v;
          word = wm;
        }
      }
      const bool sbit = (word >> l) & 1u;
      const float dn = ising ? (sbit ? 2.0f * hv : -2.0f * hv)
                             : (sbit ? hv : -hv);
      bool acc = false;
      if (lane_valid) {
        const uint32_t x = draw1(a.seed, TAG_AIS, (uint32_t)inst, (uint32_t)k,
                                 (uint32_t)my, (uint32_t)t);
        acc = ais_accept(beta, dn, sbit, lr, a.ref != 1, x);
      }
      const uint32_t am = __ballot_sync(0xffffffffu, acc);
      const uint32_t sm = __ballot_sync(0xffffffffu, sbit);
      if (acc) {
        E -= (double)dn;
        ones += sbit ? -1 : 1;
      }
      if (am) {
        const float* row = Jp + (int64_t)i * ld;
        float Jr[NC];
#pragma unroll
        for (int mm = 0; mm < NC; ++mm) {
          const int col = 32 * mm + lane;
          Jr[mm] = col < n ? __ldg(row + col) : 0.0f;
        }
#pragma unroll
        for (int g = 0; g < GW; ++g) {
          if ((am >> g) & 1u) {
            const bool sg = (sm >> g) & 1u;
            const float d = ising ? (sg ? -2.0f : 2.0f) : (sg ? -1.0f : 1.0f);
#pragma unroll
            for (int mm = 0; mm < NC; ++mm) {
              H[g][mm] = fmaf(d, Jr[mm], H[g][mm]);
              if (mm == m) spin[g][mm] ^= (1u << l);
            }
          }
        }
      }
    }
    if (a.order == 0) {
      lw += ais_dlw(beta, beta_old, (float)E, n, ones, logp, log1p_,
                    a.ref != 1);
    }
    beta_old = beta;
  }
  if (lane_valid) {
    a.log_w[myc] = lw;
    a.energies[myc] = (float)E;
  }
#pragma unroll
  for (int g = 0; g < GW; ++g) {
    const int64_t smp = s0 + g;
    if (smp < samples) {
#pragma unroll
      for (int m = 0; m < NC; ++m)
        if (m < words && lane == 0)
          a.spins[(cbase + smp) * a.words + m] = spin[g][m];
    }
  }
}

// Thresholds of one beta step in field units (see FieldThreshold): with y =
// +-field signed so that dn = scale y, a move is accepted when y >= th + off
// and rejected when y < tl + off, off shifting both by the reference's log
// ratio for the spin's value; in between, and for a beta that is not a plain
// positive number, ais_accept decides.
struct AisThreshold {
  float tl1, tl0, th1, th0, up, cap;
  __device__ __forceinline__ AisThreshold(float beta, float scale, double lr,
                                          bool uniform_ref) {
    constexpr float kLn2 = 0.69314718056f;
    const bool plain = beta >= 1e-30f && beta < 1e30f;
    const float inv = plain ? 1.0f / (beta * scale) : 0.0f;
    // a set bit going down changes the log ratio by -c
    const float c = uniform_ref ? 0.0f
                                : (float)((1.0 - (double)beta) * lr);
    const float m = fmaf(1e-6f, fabsf(c), 3e-5f) * inv;
    tl1 = kLn2 * 1.000001f * inv;
    th1 = kLn2 * 0.999999f * inv;
    tl0 = plain ? -m : -INFINITY;
    // (NaN: no y is above it, an infinite one included)
    th0 = plain ? m : __int_as_float(0x7fc00000);
    up = plain ? c * inv : 0.0f;
    // the uniform reference accepts every dn >= 0
    cap = !plain ? th0 : uniform_ref ? 0.0f : INFINITY;
  }
  __device__ __forceinline__ void at(uint32_t x, float& tl, float& th) const {
    const float l2 = log2_uniform(x);
    tl = fmaf(tl1, l2, tl0);
    th = fminf(fmaf(th1, l2, th0), cap);
  }
};

// A warp per sample, the visiting positions in turn (n <= 32 NC).  Lane l
// holds the fields of columns l, l + 32, ... in registers and, as bits m of
// one word, the spins 32 m + l; the instance's couplings are in shared
// memory.  Row, thresholds and the fields after a flip do not depend on the
// decision, which only selects: about 60 cycles a position whatever the
// acceptance.  A decision inside the band has its sweep done again with the
// exact rule.  For few samples: the kernels that hold several samples per
// warp or thread need fewer instructions each, but too few warps then leave
// every SM waiting.  A lane keeps the energy change of the position it is
// numbered after; they are added in f64, over the lanes once a sweep.  Measured
// for n = 96, 1000 samples, 200 steps: 12.7 ms with 8 samples per warp, 1.46 ms
// here (random order 1.73).
template <int NC, bool RANDOM>
__global__ void __launch_bounds__(512) k_ais_turn(const AisArgs a) {
  extern __shared__ __align__(16) float Jt[];  // [n][32 NC]
  const int inst = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (a.replicas[inst] != 1) {
    if (blockIdx.x == 0 && tid == 0) set_status(a.status, PYSA_GB_ERR_ARG);
    return;
  }
  const int n = a.n_tab[inst], ld = a.ld_tab[inst];
  const int64_t samples = a.reads[inst];
  const int WPC = blockDim.x >> 5;
  if ((int64_t)blockIdx.x * WPC >= samples) return;  // whole CTA
  const float* Jp = a.J + a.j_off[inst];
  for (int e = tid; e < n * 32 * NC; e += blockDim.x) {
    const int r = e / (32 * NC), c = e % (32 * NC);
    Jt[e] = c < n ? Jp[(int64_t)r * ld + c] : 0.0f;
  }
  __syncthreads();
  const int64_t my = (int64_t)blockIdx.x * WPC + warp;
  if (my >= samples) return;
  const int64_t myc = a.chain_off[inst] + my;
  const bool ising = a.problem_type == PYSA_GB_ISING;
  const float scale = ising ? 2.0f : 1.0f;
  const bool uniform_ref = a.ref != 1;
  const int words = (n + 31) >> 5;
  float h[NC];
  uint32_t sp = 0u;  // bit m: spin 32 m + lane
#pragma unroll
  for (int m = 0; m < NC; ++m) {
    const int col = 32 * m + lane;
    h[m] = col < n ? a.fields[myc * a.field_ld + col] : 0.0f;
    if (m < words)
      sp |= ((a.spins[myc * a.words + m] >> lane) & 1u) << m;
  }
  double E = (double)a.energies[myc];
  double lw = 0.0;
  float beta_old = 0.0f;
  const double lr = uniform_ref ? 0.0 : log((1.0 - a.p) / a.p);
  const double logp = uniform_ref ? 0.0 : log(a.p);
  const double log1p_ = uniform_ref ? 0.0 : log(1.0 - a.p);
  // columns past n hold no spin: their bits stay 0
  auto ones = [&]() {
    return uniform_ref ? 0 : __reduce_add_sync(0xffffffffu, __popc(sp));
  };
  for (int k = 0; k < a.num_temps; ++k) {
    const float beta = a.temps[k];
    if (a.order == 1)
      lw += ais_dlw(beta, beta_old, (float)E, n, ones(), logp, log1p_,
                    uniform_ref);
    const int32_t* perm =
        a.perm + ((int64_t)k * a.num_instances + inst) * a.max_n;
    const AisThreshold at(beta, scale, lr, uniform_ref);
    double dE = 0.0;  // the sweep's energy change, this lane's part
    // one sweep; EXACT asks ais_accept where the thresholds have no answer,
    // otherwise returns whether some decision needed it
    auto sweep = [&](auto exact_t) {
      constexpr bool EXACT = decltype(exact_t)::value;
      uint32_t unsure = 0u;
      for (int b = 0; b < words; ++b) {
        const int t0 = 32 * b;
        int il = t0 + lane;
        if (RANDOM) il = il < n ? perm[il] : 0;
        float tl, th, gain = 0.0f;  // of position t0 + lane
        {
          uint32_t x[4], v[4];
          draw4(a.seed, TAG_AIS, (uint32_t)inst, (uint32_t)k, (uint32_t)my,
                (uint32_t)(8 * b + (lane & 7)), x);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            v[q] = __shfl_sync(0xffffffffu, x[q], lane >> 2);
          const int q = lane & 3;
          at.at(q < 2 ? (q ? v[1] : v[0]) : (q == 2 ? v[2] : v[3]), tl, th);
        }
        auto turn = [&](int t) {
          const int p = t - t0;
          const int i = RANDOM ? __shfl_sync(0xffffffffu, il, p) : t;
          const int mi = i >> 5, l = i & 31;
          const float* row = Jt + i * (32 * NC) + lane;
          const bool sb =
              ((__shfl_sync(0xffffffffu, sp, l) >> mi) & 1u) != 0u;
          const float d = sb ? -scale : scale;
          const float off = sb ? at.up : -at.up;
          const float thp = __shfl_sync(0xffffffffu, th, p) + off;
          const float tlp = __shfl_sync(0xffffffffu, tl, p) + off;
          float hm = h[0];
#pragma unroll
          for (int m = 1; m < NC; ++m) hm = m == mi ? h[m] : hm;
          const float hv = __shfl_sync(0xffffffffu, hm, l);
          float v[NC];
#pragma unroll
          for (int m = 0; m < NC; ++m) v[m] = fmaf(d, row[32 * m], h[m]);
          const float y = sb ? hv : -hv;
          bool acc = y >= thp;
          if constexpr (EXACT) {
            if (!acc && !(y < tlp))
              acc = ais_accept(beta, scale * y, sb, lr, uniform_ref,
                               draw1(a.seed, TAG_AIS, (uint32_t)inst,
                                     (uint32_t)k, (uint32_t)my, (uint32_t)t));
          } else {
            unsure |= (!acc && !(y < tlp)) ? 1u : 0u;
          }
#pragma unroll
          for (int m = 0; m < NC; ++m) h[m] = acc ? v[m] : h[m];
          sp ^= acc && lane == l ? 1u << mi : 0u;
          gain = acc && lane == p ? scale * y : gain;
        };
        const int te = t0 + 32 < n ? t0 + 32 : n;
        if constexpr (EXACT) {
#pragma unroll 1
          for (int t = t0; t < te; ++t) turn(t);
        } else {
#pragma unroll(NC < 8 ? 4 : 2)
          for (int t = t0; t < te; ++t) turn(t);
        }
        dE -= (double)gain;
      }
      return unsure != 0u;
    };
    float h0[NC];
#pragma unroll
    for (int m = 0; m < NC; ++m) h0[m] = h[m];
    const uint32_t sp0 = sp;
    if (sweep(std::false_type{})) {
#pragma unroll
      for (int m = 0; m < NC; ++m) h[m] = h0[m];
      sp = sp0;
      dE = 0.0;
      sweep(std::true_type{});
    }
    E += warp_sum(dE);
    if (a.order == 0)
      lw += ais_dlw(beta, beta_old, (float)E, n, ones(), logp, log1p_,
                    uniform_ref);
    beta_old = beta;
  }
  if (lane == 0) {
    a.log_w[myc] = lw;
    a.energies[myc] = (float)E;
  }
#pragma unroll
  for (int m = 0; m < NC; ++m) {
    const uint32_t w = __ballot_sync(0xffffffffu, (sp >> m) & 1u);
    if (m < words && lane == 0) a.spins[myc * a.words + m] = w;
  }
}

// One sweep's energy change as three f32 (two exact two-sums, Knuth's): to
// 2^-72 of its largest term, more than the f64 sum it stands in for, without
// f64 instructions (1/64 of the rate) for each attempt.  Every sweep's change
// starts at zero and joins the sample's energy, which is f64, at its end.
struct SweepEnergy {
  float a = 0.0f, b = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(float x) {
    const float s = a + x, u = s - a;
    const float e = (a - (s - u)) + (x - u);
    const float t = b + e, v = t - b;
    c += (b - (t - v)) + (e - v);
    a = s;
    b = t;
  }
  // (an infinite or NaN sum has no further parts)
  __device__ __forceinline__ double value() const {
    return fabsf(a) < INFINITY ? (double)a + ((double)b + (double)c)
                               : (double)a;
  }
};

// Two pairs from shared memory.  Volatile: the couplings never change, and
// unrolled code would otherwise try to keep all of them in registers.
__device__ __forceinline__ ulonglong2 load_pairs(uint32_t addr) {
  ulonglong2 v;
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];"
               : "=l"(v.x), "=l"(v.y)
               : "r"(addr));
  return v;
}

// Small instances (n <= NP <= 32), many samples: one thread per sample, its
// spins in one word and its fields in NP registers as pairs, the instance's
// couplings in shared memory (the row of the visited spin is the same for
// every thread: broadcast 16-byte loads).  A position costs NP / 2 paired
// multiply-adds and NP / 4 loads; a rejected attempt adds 0 * J, which changes
// no field but possibly the sign of a zero.  Bound by instruction issue: the
// Philox draw (one per four positions) and the field updates take most of
// it.  Measured for 64 instances of n = 24, 1024 samples, 200 steps: 4.33 ms
// with the fields in shared memory and an f64 addition an attempt, 1.27 ms
// here (random order 4.42 and 1.77).
template <int NP, bool RANDOM>
__global__ void __launch_bounds__(128) k_ais_small(const AisArgs a) {
  __shared__ __align__(16) float Js[NP * NP];
  const uint32_t js_addr = smem_addr(Js);
  const int inst = blockIdx.y;
  const int tid = threadIdx.x;
  if (a.replicas[inst] != 1) {
    if (blockIdx.x == 0 && tid == 0) set_status(a.status, PYSA_GB_ERR_ARG);
    return;
  }
  const int n = a.n_tab[inst];
  const int ld = a.ld_tab[inst];
  const int64_t samples = a.reads[inst];
  if ((int64_t)blockIdx.x * blockDim.x >= samples) return;  // whole CTA
  const float* Jp = a.J + a.j_off[inst];
  for (int e = tid; e < NP * NP; e += blockDim.x) {
    const int r = e / NP, c = e % NP;
    Js[e] = (r < n && c < n) ? Jp[(int64_t)r * ld + c] : 0.0f;
  }
  const int64_t my = (int64_t)blockIdx.x * blockDim.x + tid;
  const bool valid = my < samples;
  const int64_t myc = a.chain_off[inst] + (valid ? my : 0);
  uint64_t H[NP / 2];
#pragma unroll
  for (int c = 0; c < NP / 2; ++c)
    H[c] = pack2(
        valid && 2 * c < n ? a.fields[myc * a.field_ld + 2 * c] : 0.0f,
        valid && 2 * c + 1 < n ? a.fields[myc * a.field_ld + 2 * c + 1]
                               : 0.0f);
  __syncthreads();
  if (!valid) return;
  const bool ising = a.problem_type == PYSA_GB_ISING;
  const float scale = ising ? 2.0f : 1.0f;
  const bool uniform_ref = a.ref != 1;
  uint32_t word = a.spins[myc * a.words];
  double E = (double)a.energies[myc];
  double lw = 0.0;
  float beta_old = 0.0f;
  const double lr = uniform_ref ? 0.0 : log((1.0 - a.p) / a.p);
  const double logp = uniform_ref ? 0.0 : log(a.p);
  const double log1p_ = uniform_ref ? 0.0 : log(1.0 - a.p);
  for (int k = 0; k < a.num_temps; ++k) {
    const float beta = a.temps[k];
    if (a.order == 1)
      lw += ais_dlw(beta, beta_old, (float)E, n, __popc(word), logp,
                    log1p_, uniform_ref);
    const int32_t* perm =
        a.perm + ((int64_t)k * a.num_instances + inst) * a.max_n;
    const AisThreshold at(beta, scale, lr, uniform_ref);
    SweepEnergy dE;
    uint32_t rnd[4];
    auto turn = [&](int t, int i, float hv, uint32_t x) {
      const bool sb = (word >> i) & 1u;
      const float y = sb ? hv : -hv;
      const float off = sb ? at.up : -at.up;
      float tl, th;
      at.at(x, tl, th);
      bool acc = y >= th + off;
      if (!acc && !(y < tl + off))
        acc = ais_accept(beta, scale * y, sb, lr, uniform_ref, x);
      word ^= acc ? 1u << i : 0u;
      dE.add(acc ? -(scale * y) : 0.0f);
      const float d = acc ? (sb ? -scale : scale) : 0.0f;
      const uint64_t dd = pack2(d, d);
      const uint32_t row = js_addr + (uint32_t)(i * NP * 4);
#pragma unroll
      for (int c = 0; c < NP / 4; ++c) {
        const ulonglong2 j = load_pairs(row + 16 * c);
        H[2 * c] = fma2(dd, j.x, H[2 * c]);
        H[2 * c + 1] = fma2(dd, j.y, H[2 * c + 1]);
      }
    };
    if constexpr (RANDOM) {
#pragma unroll 1
      for (int t = 0; t < n; t += 4) {
        int ids[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) ids[q] = t + q < n ? perm[t + q] : 0;
        draw4(a.seed, TAG_AIS, (uint32_t)inst, (uint32_t)k, (uint32_t)my,
              (uint32_t)(t >> 2), rnd);
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          if (t + q >= n) break;
          const int i = q < 2 ? (q ? ids[1] : ids[0])
                              : (q == 2 ? ids[2] : ids[3]);
          // the spin is the same in every thread: a uniform branch picks its
          // register
          uint64_t pr = 0ull;
          switch (i >> 1) {
#define PYSA_GB_FIELD(c) \
  case c:                \
    if constexpr (c < NP / 2) pr = H[c < NP / 2 ? c : 0]; \
    break;
            PYSA_GB_FIELD(0) PYSA_GB_FIELD(1) PYSA_GB_FIELD(2)
            PYSA_GB_FIELD(3) PYSA_GB_FIELD(4) PYSA_GB_FIELD(5)
            PYSA_GB_FIELD(6) PYSA_GB_FIELD(7) PYSA_GB_FIELD(8)
            PYSA_GB_FIELD(9) PYSA_GB_FIELD(10) PYSA_GB_FIELD(11)
            PYSA_GB_FIELD(12) PYSA_GB_FIELD(13) PYSA_GB_FIELD(14)
            PYSA_GB_FIELD(15)
#undef PYSA_GB_FIELD
            default: break;
          }
          turn(t + q, i, half2(pr, i & 1),
               q < 2 ? (q ? rnd[1] : rnd[0]) : (q == 2 ? rnd[2] : rnd[3]));
        }
      }
    } else {
#pragma unroll
      for (int t = 0; t < NP; ++t) {
        if (t >= n) break;  // uniform
        if ((t & 3) == 0)
          draw4(a.seed, TAG_AIS, (uint32_t)inst, (uint32_t)k, (uint32_t)my,
                (uint32_t)(t >> 2), rnd);
        turn(t, t, half2(H[t >> 1], t & 1), rnd[t & 3]);
      }
    }
    E += dE.value();
    if (a.order == 0)
      lw += ais_dlw(beta, beta_old, (float)E, n, __popc(word), logp,
                    log1p_, uniform_ref);
    beta_old = beta;
  }
  a.log_w[myc] = lw;
  a.energies[myc] = (float)E;
  a.spins[myc * a.words] = word;
}

// Warp per sample keeps the code simple for the small n AIS is used on;
// GW samples per warp amortise the decision shuffles.
template <int NC, int GW>
static cudaError_t launch_ais_t(const AisArgs& a, int64_t max_samples,
                                cudaStream_t st) {
  const int64_t warps = (max_samples + GW - 1) / GW;
  const int64_t blocks = (warps * 32 + 127) / 128;
  dim3 grid((unsigned)(blocks > 0 ? blocks : 1), (unsigned)a.num_instances);
  k_ais<NC, GW><<<grid, 128, 0, st>>>(a);
  return cudaGetLastError();
}

// Widest instance whose couplings the warp-per-sample kernel keeps in shared
// memory (n x 256 floats at n > 128).
constexpr int kTurnMaxN = 220;

template <int NC>
static cudaError_t launch_turn_t(const AisArgs& a, int64_t max_samples,
                                 cudaStream_t st) {
  const bool random = a.update == PYSA_GB_RANDOM;
  const int wpc = NC >= 8 ? 16 : 4;  // samples that share the couplings
  const size_t smem = (size_t)a.max_n * 32 * NC * 4;
  const void* f = random ? (const void*)k_ais_turn<NC, true>
                         : (const void*)k_ais_turn<NC, false>;
  constexpr int widest = 32 * NC < kTurnMaxN ? 32 * NC : kTurnMaxN;
  static std::atomic<uint64_t> allowed[2];
  cudaError_t e =
      allow_smem(f, (size_t)widest * 32 * NC * 4, allowed[random]);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)((max_samples + wpc - 1) / wpc),
            (unsigned)a.num_instances);
  if (random)
    k_ais_turn<NC, true><<<grid, 32 * wpc, smem, st>>>(a);
  else
    k_ais_turn<NC, false><<<grid, 32 * wpc, smem, st>>>(a);
  return cudaGetLastError();
}

template <int NP>
static cudaError_t launch_small_t(const AisArgs& a, int64_t max_samples,
                                  cudaStream_t st) {
  const int64_t blocks = (max_samples + 127) / 128;
  dim3 grid((unsigned)(blocks > 0 ? blocks : 1), (unsigned)a.num_instances);
  if (a.update == PYSA_GB_RANDOM)
    k_ais_small<NP, true><<<grid, 128, 0, st>>>(a);
  else
    k_ais_small<NP, false><<<grid, 128, 0, st>>>(a);
  return cudaGetLastError();
}

// Few samples: a warp each.  Many: threads (n <= 32) or warps holding several
// samples, which need fewer instructions per attempt once the GPU is full.
// A thread a sample takes n attempts one after another whatever the number of
// samples, a warp a sample the same time for any n but more the more samples:
// 200 steps, warp against thread, n = 8, 2000 samples 0.53 and 0.31 ms, n = 16
// 0.56 and 0.62, n = 24, 4000 samples 1.00 and 0.95, n = 31, 4870 samples 1.42
// and 1.42.  Whole calls with 50 steps, warp per sample against several a warp:
// n = 96, 24000 samples 9.5 and 12.1 ms; n = 50, 16000 4.0 and 4.4; n = 200, 16000
// 17.5 and 24.4.
constexpr int64_t kTurnPerSpin = 160;  // n <= 32
constexpr int64_t kTurnSamplesWide = 24576;

cudaError_t launch_ais(const AisArgs& a, int64_t max_samples, cudaStream_t st) {
  const int64_t total = max_samples * a.num_instances;
  const int nc = (a.max_n + 31) / 32;
  if (nc <= 1) {
    if (total <= kTurnPerSpin * (int64_t)a.max_n)
      return launch_turn_t<1>(a, max_samples, st);
    if (a.max_n <= 8) return launch_small_t<8>(a, max_samples, st);
    if (a.max_n <= 16) return launch_small_t<16>(a, max_samples, st);
    if (a.max_n <= 24) return launch_small_t<24>(a, max_samples, st);
    return launch_small_t<32>(a, max_samples, st);
  }
  if (total <= kTurnSamplesWide && a.max_n <= kTurnMaxN) {
    if (nc <= 2) return launch_turn_t<2>(a, max_samples, st);
    if (nc <= 4) return launch_turn_t<4>(a, max_samples, st);
    return launch_turn_t<8>(a, max_samples, st);
  }
  if (nc <= 2) return launch_ais_t<2, 8>(a, max_samples, st);
  if (nc <= 4) return launch_ais_t<4, 8>(a, max_samples, st);
  if (nc <= 8) return launch_ais_t<8, 4>(a, max_samples, st);
  if (nc <= 16) return launch_ais_t<16, 2>(a, max_samples, st);
  if (nc <= 32) return launch_ais_t<32, 1>(a, max_samples, st);
  return cudaErrorInvalidValue;
}

// Fisher-Yates of instance blockIdx.y for sweep blockIdx.x (draws of
// stream PERM, a = sweep), j = floor(x (i+1) / 2^32).
__global__ void k_perm_all(const int32_t* n_tab, int num_instances, int max_n,
                           uint64_t seed, int32_t* out) {
  extern __shared__ int32_t sh[];
  const int inst = blockIdx.y;
  const int n = n_tab[inst];
  const uint32_t sweep = blockIdx.x;
  int32_t* p = sh;
  uint32_t* x = reinterpret_cast<uint32_t*>(sh + max_n);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    p[i] = i;
    x[i] = draw1(seed, TAG_PERM, (uint32_t)inst, sweep, 0u, (uint32_t)i);
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = n - 1; i > 0; --i) {
      const int j = (int)(((uint64_t)x[i] * (uint64_t)(i + 1)) >> 32);
      const int32_t t = p[i];
      p[i] = p[j];
      p[j] = t;
    }
  __syncthreads();
  int32_t* o = out + ((int64_t)sweep * num_instances + inst) * max_n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) o[i] = p[i];
}

cudaError_t launch_perm_all(const int32_t* n_tab, int num_instances, int max_n,
                            int count, uint64_t seed, int32_t* out,
                            cudaStream_t st) {
  if (count <= 0 || num_instances <= 0) return cudaSuccess;
  dim3 grid((unsigned)count, (unsigned)num_instances);
  k_perm_all<<<grid, 256, sizeof(int32_t) * 2 * max_n, st>>>(
      n_tab, num_instances, max_n, seed, out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- log Z
// Thread t of instance b walks Gray codes g(j), j in [t 2^B, (t+1) 2^B):
// fields and energy of the first state from scratch in f64, then one flip
// per step.  Per-thread (max, sum) of exp(-beta E) relative to the max.
__global__ void k_logz(const LogzArgs a) {
  const int inst = blockIdx.y;
  const int n = a.n[inst];
  const int ld = a.ld[inst];
  const float* J = a.J + a.j_off[inst];
  const float* h = a.h + a.h_off[inst];
  const int B = n < a.chunk_bits ? n : a.chunk_bits;
  const uint64_t threads = (uint64_t)1 << (n - B);
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double mx = -INFINITY, sum = 0.0;
  if (t < threads) {
    const bool ising = a.problem_type == PYSA_GB_ISING;
    const double lo = ising ? -1.0 : 0.0;
    double s[32], f[32];
    const uint64_t j0 = t << B;
    const uint64_t g0 = j0 ^ (j0 >> 1);
    for (int i = 0; i < n; ++i) s[i] = ((g0 >> i) & 1u) ? 1.0 : lo;
    double e = 0.0;
    for (int i = 0; i < n; ++i) {
      double acc = 0.0;
      for (int j = 0; j < n; ++j) acc += (double)J[(int64_t)i * ld + j] * s[j];
      f[i] = acc;
      e += s[i] * (0.5 * acc + (double)h[i]);
    }
    const double beta = a.beta;
    const uint64_t steps = (uint64_t)1 << B;
    for (uint64_t q = 0; q < steps; ++q) {
      const double w = -beta * e;
      if (w > mx) {
        sum = sum * exp(mx - w) + 1.0;
        mx = w;
      } else {
        sum += exp(w - mx);
      }
      if (q + 1 == steps) break;
      const int i = __ffsll((long long)(j0 + q + 1)) - 1;
      const double ns = ising ? -s[i] : 1.0 - s[i];
      const double d = ns - s[i];
      e += d * (f[i] + (double)h[i]);
      for (int j = 0; j < n; ++j) f[j] += (double)J[(int64_t)i * ld + j] * d;
      s[i] = ns;
    }
  }
  // block reduction of (max, sum)
  __shared__ double smx[256], ssum[256];
  smx[threadIdx.x] = mx;
  ssum[threadIdx.x] = sum;
  __syncthreads();
  for (int o = blockDim.x >> 1; o; o >>= 1) {
    if (threadIdx.x < o) {
      const double m1 = smx[threadIdx.x], m2 = smx[threadIdx.x + o];
      const double s1 = ssum[threadIdx.x], s2 = ssum[threadIdx.x + o];
      const double m = m1 > m2 ? m1 : m2;
      double v = 0.0;
      if (m1 != -INFINITY) v += s1 * exp(m1 - m);
      if (m2 != -INFINITY) v += s2 * exp(m2 - m);
      smx[threadIdx.x] = m;
      ssum[threadIdx.x] = v;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const int64_t slot = (int64_t)inst * gridDim.x + blockIdx.x;
    a.part_max[slot] = smx[0];
    a.part_sum[slot] = ssum[0];
  }
}

cudaError_t launch_logz(const LogzArgs& a, int max_n, cudaStream_t st) {
  const int B = max_n < a.chunk_bits ? max_n : a.chunk_bits;
  const uint64_t threads = (uint64_t)1 << (max_n - B);
  const uint64_t blocks = (threads + 255) / 256;
  dim3 grid((unsigned)blocks, (unsigned)a.num_instances);
  k_logz<<<grid, 256, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace pysa_gb
