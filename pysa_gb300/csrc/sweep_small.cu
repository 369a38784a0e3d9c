// sweep_small.cu -- many sweeps of small dense instances (n <= 64) in one
// launch, everything resident on the SM.
//
// Same sweeps as pysa/simulation.py:60-76 (sequential) / :41-57 (random
// order) with the rule of pysa/ising.py:40-63 / pysa/qubo.py:40-63, each
// followed by the replica exchange of pysa/utils.py:44-58 and, when enabled,
// the log-omega of pysa/ais.py:79-112.
//
// One CTA per read: its couplings, its chains' fields and spins, the ladder
// and the slot map live in shared memory for the whole launch, so a sweep
// costs no launch, no global memory and no gap.  A warp takes a chain; lane
// l holds visiting positions l and l + 32.  Positions are not tried one
// after another: all are tested against their rejection thresholds at once,
// the first one not certainly rejected is the next decision (the ones before
// it are rejected as the one-by-one rule rejects them, having seen every
// earlier flip), and an accepted flip corrects all fields with one row of
// couplings.  A sweep thus takes its accepted flips + 1 rounds of about 100
// cycles instead of n dependent attempts.  Field updates, energy sums and
// draws are those of the plain sweep kernel, bit for bit.
//
// One more warp works ahead: the next sweep's visiting order and this
// sweep's exchange draws.
//
// Measured (times per sweep with exchange): n = 60, 640 chains, log-omega
// 62 -> 3.3 us; n = 24, 4 chains, random order 20 -> 1.2 us (three launches
// per sweep before).
#include "aux.cuh"
#include "small_api.h"

namespace pysa_gb {

namespace {

constexpr int kMaxSmallWarps = 31;  // chains at a time; one more works ahead

// Shared memory of a CTA, in 4-byte words: fixed part, then per replica.
struct SmallSmem {
  static constexpr int J = 0;                  // [64][64] couplings
  static constexpr int PERM = J + 64 * 64;     // [2][64] visiting orders
  static constexpr int INV = PERM + 2 * 64;    // [2][64] positions of spins
  static constexpr int WORK = INV + 2 * 64;    // [2][64] helper scratch
  static constexpr int FIXED = WORK + 2 * 64;
  static constexpr int PER = 64 + 2 + 14;      // words per replica
  static size_t bytes(int cap) {
    return 4 * ((size_t)FIXED + (size_t)PER * cap);
  }
};

// Fisher-Yates order of one sweep (draws of stream PERM, swaps from n - 1
// down, j = floor(x (i + 1) / 2^32)) by one warp, without replaying the
// swaps: position i ends with what position j_i held before step i.  A
// position a < i holds its own number until some step k > i names it (j_k =
// a), after which it holds what position k held before step k; the latest
// such step is the smallest k.
__device__ void small_order(uint64_t seed, uint32_t inst, uint32_t sweep,
                            int n, int lane, int32_t* js, int32_t* nxt,
                            int32_t* perm, int32_t* inv) {
  if (lane < 16) {
    uint32_t x[4];
    draw4(seed, TAG_PERM, inst, sweep, 0u, (uint32_t)lane, x);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = 4 * lane + k;
      js[i] = (int)(((uint64_t)x[k] * (uint64_t)(i + 1)) >> 32);
    }
  }
  __syncwarp();
  const int a0 = js[lane], a1 = js[lane + 32];
  int n0 = -1, n1 = -1, m0 = -1, m1 = -1;
  for (int k = n - 1; k > 0; --k) {
    const int j = js[k];
    if (j == lane && k > lane) n0 = k;
    if (j == lane + 32 && k > lane + 32) n1 = k;
    if (j == a0 && k > lane) m0 = k;
    if (j == a1 && k > lane + 32) m1 = k;
  }
  nxt[lane] = n0;
  nxt[lane + 32] = n1;
  __syncwarp();
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int i = lane + 32 * half, a = half ? a1 : a0, m = half ? m1 : m0;
    if (i < n) {
      int c = a;
      if (a == i || m >= 0) {
        c = a == i ? i : m;
        for (int k = nxt[c]; k >= 0; k = nxt[c]) c = k;
      }
      perm[i] = c;
      inv[c] = i;
    }
  }
  __syncwarp();
}

}  // namespace

template <bool RANDOM>
__global__ void __launch_bounds__(32 * (kMaxSmallWarps + 1), 1)
    k_sweep_small(const SmallArgs a) {
  extern __shared__ __align__(16) uint32_t sm[];
  const int64_t r = blockIdx.x;
  const int inst = a.p.read_inst[r];
  const int n = a.p.n[inst];
  const bool mine = n <= kSmallMaxN &&
                    !(a.p.csr_row_off && a.p.csr_row_off[inst] >= 0) &&
                    !(a.skip_inst && a.skip_inst[inst]);  // uniform per CTA
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sweep0 = (uint32_t)(*a.s.sweep_counter);
  if (mine) {
    const int NW = (int)(blockDim.x >> 5) - 1;  // warps with chains
    const int R = a.p.replicas[inst];
    const bool fit = R <= a.cap;  // else the state stays in global memory
    const int64_t lread = r - a.p.read_off[inst];
    const int64_t base = a.p.chain_off[inst] + lread * R;
    const int words = (n + 31) >> 5;
    const bool ising = a.p.problem_type == PYSA_GB_ISING;
    const float scale = ising ? 2.0f : 1.0f;
    const float* betas = a.p.ladder + a.p.ladder_off[inst];
    const int32_t* sorted = a.p.ladder_sorted + a.p.ladder_off[inst];
    float* J = reinterpret_cast<float*>(sm + SmallSmem::J);
    int32_t* perm_s = reinterpret_cast<int32_t*>(sm + SmallSmem::PERM);
    int32_t* inv_s = reinterpret_cast<int32_t*>(sm + SmallSmem::INV);
    int32_t* work_s = reinterpret_cast<int32_t*>(sm + SmallSmem::WORK);
    uint32_t* per = sm + SmallSmem::FIXED;
    const int cap = a.cap;
    // per replica; the first six are copies of global state when they fit
    float* Hs = reinterpret_cast<float*>(per);             // [cap][64]
    uint32_t* Ss = per + 64 * cap;                         // [cap][2]
    float* E = fit ? reinterpret_cast<float*>(per + 66 * cap)
                   : a.s.energies + base;
    int32_t* B = fit ? reinterpret_cast<int32_t*>(per + 67 * cap)
                     : a.s.beta_idx + base;
    float* beta_c = fit ? reinterpret_cast<float*>(per + 68 * cap)
                        : a.s.chain_beta + base;
    float* bestE = fit ? reinterpret_cast<float*>(per + 69 * cap)
                       : a.s.best_energy + base;
    const float* Bt = fit ? reinterpret_cast<float*>(per + 70 * cap) : betas;
    float2* dE = reinterpret_cast<float2*>(per + 72 * cap);  // [cap]
    float2* X2 = reinterpret_cast<float2*>(per + 74 * cap);  // draw, log
    float2* E2 = reinterpret_cast<float2*>(per + 76 * cap);  // energy, dbeta
    int32_t* B2 = reinterpret_cast<int32_t*>(per + 78 * cap);
    auto Hc = [&](int c) {
      return fit ? Hs + 64 * c : a.fields + (base + c) * (int64_t)a.field_ld;
    };
    auto Sc = [&](int c) {
      return fit ? Ss + 2 * c : a.s.spins + (base + c) * (int64_t)a.p.words;
    };

    // ---- state in
    {
      const float* Jg = a.p.J + a.p.j_off[inst];
      const int ld = a.p.ld[inst];
      for (int e = tid; e < n * 64; e += blockDim.x) {
        const int i = e >> 6, c = e & 63;
        J[e] = c < n ? Jg[(int64_t)i * ld + c] : 0.0f;
      }
      if (fit) {
        for (int e = tid; e < R * 64; e += blockDim.x) {
          const int c = e >> 6, i = e & 63;
          Hs[e] = i < n ? a.fields[(base + c) * (int64_t)a.field_ld + i]
                        : 0.0f;
        }
        for (int c = tid; c < R; c += blockDim.x) {
          const int64_t g = base + c;
          Ss[2 * c] = a.s.spins[g * a.p.words];
          Ss[2 * c + 1] = words > 1 ? a.s.spins[g * a.p.words + 1] : 0u;
          E[c] = a.s.energies[g];
          B[c] = a.s.beta_idx[g];
          beta_c[c] = a.s.chain_beta[g];
          bestE[c] = a.s.best_energy[g];
          const_cast<float*>(Bt)[c] = betas[c];
        }
      }
      if (RANDOM && warp == NW)
        small_order(a.seed, (uint32_t)inst, sweep0, n, lane, work_s,
                    work_s + 64, perm_s + 64 * (sweep0 & 1),
                    inv_s + 64 * (sweep0 & 1));
    }
    __syncthreads();

    for (int s = 0; s < a.num_sweeps; ++s) {
      const uint32_t sweep = sweep0 + (uint32_t)s;
      const bool xch = a.use_pt && exchange_after(a.exchange_every, sweep);
      if (warp < NW) {
        // ------------------------------------------------------- sweeps
        const int32_t* perm = perm_s + 64 * (sweep & 1);
        const int32_t* inv = inv_s + 64 * (sweep & 1);
        const bool two = n > 32;
        const int k1 = lane + 32;
        const bool in0 = lane < n, in1 = k1 < n;
        const int i0 = in0 ? (RANDOM ? perm[lane] : lane) : 0;
        const int i1 = in1 ? (RANDOM ? perm[k1] : k1) : 0;
        for (int c = warp; c < R; c += NW) {
          float* H = Hc(c);
          uint32_t* S = Sc(c);
          float h0 = in0 ? H[i0] : 0.0f, h1 = in1 ? H[i1] : 0.0f;
          const uint32_t wa = S[0], wb = words > 1 ? S[1] : 0u;
          // the spins by position, as masks (bit l: position l, l + 32)
          uint32_t S0 = __ballot_sync(
              0xffffffffu, in0 && (((i0 < 32 ? wa : wb) >> (i0 & 31)) & 1u));
          uint32_t S1 = __ballot_sync(
              0xffffffffu, in1 && (((i1 < 32 ? wa : wb) >> (i1 & 31)) & 1u));
          const float beta = beta_c[c];
          const uint32_t cl = (uint32_t)(lread * R + c);
          const uint64_t seed =
              chain_seed(a.seed, a.s.stream_key, base + c);
          // draws of quad l in lane l (< 16), one per position by shuffle
          uint32_t x0, x1 = 0u;
          {
            uint32_t x[4];
            draw4(seed, TAG_SWEEP, (uint32_t)inst, sweep, cl,
                  (uint32_t)(lane & 15), x);
            const int src = lane >> 2, q = lane & 3;
            uint32_t v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
              v[k] = __shfl_sync(0xffffffffu, x[k], src);
            x0 = q < 2 ? (q ? v[1] : v[0]) : (q == 2 ? v[2] : v[3]);
            if (two) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                v[k] = __shfl_sync(0xffffffffu, x[k], src + 8);
              x1 = q < 2 ? (q ? v[1] : v[0]) : (q == 2 ? v[2] : v[3]);
            }
          }
          const FieldThreshold ft(beta, scale);
          float tl0, th0, tl1, th1;
          ft.at(x0, tl0, th0);
          ft.at(x1, tl1, th1);
          // sign word of this lane's spins: x = +-h, dn = scale x
          uint32_t g0 = ((S0 >> lane) & 1u) ? 0u : 0x80000000u;
          uint32_t g1 = ((S1 >> lane) & 1u) ? 0u : 0x80000000u;
          uint32_t p0 = __ballot_sync(0xffffffffu, in0);
          uint32_t p1 = __ballot_sync(0xffffffffu, in1);
          float d0 = 0.0f, d1 = 0.0f;  // energy change, 32 positions each
          for (;;) {
            const float y0 = __uint_as_float(__float_as_uint(h0) ^ g0);
            const float y1 = __uint_as_float(__float_as_uint(h1) ^ g1);
            const uint32_t c0 =
                __ballot_sync(0xffffffffu, !(y0 < tl0)) & p0;
            const uint32_t a0 = __ballot_sync(0xffffffffu, y0 >= th0);
            uint32_t c1 = 0u, a1 = 0u;
            if (two) {
              c1 = __ballot_sync(0xffffffffu, !(y1 < tl1)) & p1;
              a1 = __ballot_sync(0xffffffffu, y1 >= th1);
            }
            if ((c0 | c1) == 0u) break;
            // the next decision: position js of half hf
            const bool hf = c0 == 0u;
            const int js = __ffs(hf ? c1 : c0) - 1;
            const uint32_t bit = 1u << js;
            if (hf) {
              p0 = 0u;
              p1 &= ~(bit | (bit - 1u));
            } else {
              p0 &= ~(bit | (bit - 1u));
            }
            const float y = __shfl_sync(0xffffffffu, hf ? y1 : y0, js);
            const int i = RANDOM ? perm[js + (hf ? 32 : 0)]
                                 : js + (hf ? 32 : 0);
            bool acc = ((hf ? a1 : a0) & bit) != 0u;
            if (!acc)  // inside the band: the exact rule
              acc = accept_slow_redraw(scale * y, beta, seed, (uint32_t)inst,
                                       sweep, cl,
                                       (uint32_t)(js + (hf ? 32 : 0)));
            if (acc) {
              const bool sb = ((hf ? S1 : S0) & bit) != 0u;
              const float d = sb ? -scale : scale;
              const float* row = J + 64 * i;
              if (in0) h0 = fmaf(d, row[i0], h0);
              if (in1) h1 = fmaf(d, row[i1], h1);
              const float dn = scale * y;
              if (hf) {
                S1 ^= bit;
                d1 -= dn;
                if (lane == js) g1 ^= 0x80000000u;
              } else {
                S0 ^= bit;
                d0 -= dn;
                if (lane == js) g0 ^= 0x80000000u;
              }
            }
          }
          if (in0) H[i0] = h0;
          if (in1) H[i1] = h1;
          uint32_t na = S0, nb = S1;
          if (RANDOM) {  // spins back in their own order
            const int q0 = in0 ? inv[lane] : 0, q1 = in1 ? inv[k1] : 0;
            na = __ballot_sync(
                0xffffffffu, in0 && (((q0 < 32 ? S0 : S1) >> (q0 & 31)) & 1u));
            nb = __ballot_sync(
                0xffffffffu, in1 && (((q1 < 32 ? S0 : S1) >> (q1 & 31)) & 1u));
          }
          if (lane == 0) {
            S[0] = na;
            if (words > 1) S[1] = nb;
            if (fit) {
              dE[c] = make_float2(d0, d1);
            } else {
              // no room for the pair: the energy now
              E[c] = (float)((double)E[c] + ((double)d0 + (double)d1));
            }
          }
        }
      } else {
        // ---------------------------------------------------- work ahead
        if (fit && xch)
          for (int k = lane; k < R - 1; k += 32) {
            const uint32_t x = draw1(a.seed, TAG_PT, (uint32_t)inst, sweep,
                                     (uint32_t)lread, (uint32_t)k);
            X2[k] = make_float2(__uint_as_float(x), log_uniform_f32(x));
          }
        if (RANDOM && s + 1 < a.num_sweeps) {
          const uint32_t nx = (sweep + 1u) & 1u;
          small_order(a.seed, (uint32_t)inst, sweep + 1u, n, lane, work_s,
                      work_s + 64, perm_s + 64 * nx, inv_s + 64 * nx);
        }
      }
      __syncthreads();

      // ------------------------- energies, best states, exchange: warp 0
      if (warp == 0) {
        for (int c = lane; c < R; c += 32) {
          float e = E[c];
          if (fit) {
            const float2 d = dE[c];
            e = (float)((double)e + ((double)d.x + (double)d.y));
            E[c] = e;
          }
          // strict < (pysa/simulation.py:150-171)
          if (e < bestE[c]) {
            bestE[c] = e;
            const int64_t g = base + c;
            a.s.best_sweep[g] = (int32_t)sweep;
            const uint32_t* S = Sc(c);
            for (int w = 0; w < words; ++w)
              a.s.best_spins[g * a.p.words + w] = S[w];
          }
        }
        __syncwarp();
        if (xch && R > 1) {
          // pairs (R-1, R-2), (R-2, R-3), ... in order: only the replica
          // entering slot k1 carries from pair to pair, so every pair's
          // other replica, its energy and the betas' difference are read up
          // front and the pass keeps the carried one in registers
          if (fit) {
            for (int k = lane; k < R - 1; k += 32) {
              const int t1 = R - k - 1, t2 = R - k - 2;
              const int b2 = B[t2];
              B2[k] = b2;
              E2[k] = make_float2(E[b2], __fsub_rn(Bt[t1], Bt[t2]));
            }
            __syncwarp();
          }
          if (lane == 0) {
            int cb = B[R - 1];
            float ce = E[cb];
            for (int k = 0; k < R - 1; ++k) {
              int b2;
              float2 e2, x2;
              if (fit) {
                b2 = B2[k];
                e2 = E2[k];
                x2 = X2[k];
              } else {
                const int t1 = R - k - 1, t2 = R - k - 2;
                b2 = B[t2];
                e2 = make_float2(E[b2], __fsub_rn(Bt[t1], Bt[t2]));
                const uint32_t x = draw1(a.seed, TAG_PT, (uint32_t)inst,
                                         sweep, (uint32_t)lread, (uint32_t)k);
                x2 = make_float2(__uint_as_float(x), log_uniform_f32(x));
              }
              const float de = __fmul_rn(__fsub_rn(ce, e2.x), e2.y);
              const bool sw = pt_accept_lf(de, x2.y, __float_as_uint(x2.x));
              B[R - k - 1] = sw ? b2 : cb;  // final: no later pair
              cb = sw ? cb : b2;
              ce = sw ? ce : e2.x;
            }
            B[0] = cb;
          }
          __syncwarp();
          for (int k = lane; k < R; k += 32) beta_c[B[k]] = Bt[k];
        }
        if (a.log_omega_stride > 0) {
          // terms of the sorted ladder, f32 products, summed in f64
          __syncwarp();
          double lw = 0.0;
          for (int q = 1 + lane; q < R; q += 32) {
            const float b = Bt[sorted[q]];
            const float old = q > 1 ? Bt[sorted[q - 1]] : 0.0f;
            const float e = E[B[sorted[q]]];
            lw += (double)__fsub_rn(__fmul_rn(-b, e), __fmul_rn(-old, e));
          }
          lw = warp_sum(lw);
          if (lane == 0)
            a.s.log_omega[r * a.log_omega_stride + sweep] = lw;
        }
      }
      __syncthreads();
    }

    // ---- state out
    if (fit) {
      for (int e = tid; e < R * 64; e += blockDim.x) {
        const int c = e >> 6, i = e & 63;
        if (i < n) a.fields[(base + c) * (int64_t)a.field_ld + i] = Hs[e];
      }
      for (int c = tid; c < R; c += blockDim.x) {
        const int64_t g = base + c;
        a.s.spins[g * a.p.words] = Ss[2 * c];
        if (words > 1) a.s.spins[g * a.p.words + 1] = Ss[2 * c + 1];
        a.s.energies[g] = E[c];
        a.s.beta_idx[g] = B[c];
        a.s.chain_beta[g] = beta_c[c];
        a.s.best_energy[g] = bestE[c];
      }
    }
  }
  __syncthreads();
  if (tid == 0 && a.advance) {  // the last CTA advances the sweep counter
    __threadfence();
    const uint32_t t = atomicAdd(a.s.ticket, 1u);
    if (t == gridDim.x - 1) {
      *a.s.ticket = 0u;
      __threadfence();
      *a.s.sweep_counter += a.num_sweeps;
    }
  }
}

cudaError_t launch_small(SmallArgs a, bool random, cudaStream_t st) {
  if (a.p.num_reads <= 0) return cudaSuccess;
  // a warp per replica of an average read; reads with more replicas take
  // turns, and keep their state in global memory
  const int64_t avg = (a.p.num_chains + a.p.num_reads - 1) / a.p.num_reads;
  a.cap = (int32_t)(avg < kMaxReplicas ? (avg > 1 ? avg : 1) : kMaxReplicas);
  a.cap += a.cap & 1;  // pairs of words stay 8-byte aligned
  const int nw = a.cap < kMaxSmallWarps ? a.cap : kMaxSmallWarps;
  const size_t smem = SmallSmem::bytes(a.cap);
  const void* f = random ? (const void*)k_sweep_small<true>
                         : (const void*)k_sweep_small<false>;
  cudaError_t e = cudaFuncSetAttribute(
      f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)a.p.num_reads), block(32 * (nw + 1));
  if (random)
    k_sweep_small<true><<<grid, block, smem, st>>>(a);
  else
    k_sweep_small<false><<<grid, block, smem, st>>>(a);
  return cudaGetLastError();
}

}  // namespace pysa_gb
