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
// couplings.  A sweep thus takes its accepted flips + 1 rounds instead of n
// dependent attempts; a chain whose last sweep flipped many spins takes the
// positions in turn.  Field updates, energy sums and draws are those of the
// plain sweep kernel, bit for bit.
//
// One more warp works ahead where there is something to: the next sweep's
// visiting order and this sweep's exchange draws.  While the reads are fewer than the SMs, a cluster
// of up to 8 CTAs shares a read's chains; energies and new betas cross
// through distributed shared memory.
//
// Measured (times per sweep with exchange): n = 60, 640 chains in 20 reads,
// log-omega 62 -> 8 us (22 on one CTA per read in rounds alone); n = 24, 4
// chains, random order 25 -> 2.5 us (three launches per sweep before).  Many
// reads: rows of 32 columns up to n = 32 and CTAs of as many warps as let an SM
// hold several, n = 24, 8000 reads of 16 chains 245 -> 109 us, n = 40 313 -> 174
// (launches: 148 and 291).
#include <cooperative_groups.h>

#include "aux.cuh"
#include "small_api.h"

namespace pysa_gb {

namespace {

constexpr int kMaxSmallWarps = 31;  // chains at a time; one more works ahead
// A chain is swept position by position after a sweep that flipped more than
// one spin in kDenseFlips (a round of the other form costs about as much as
// five positions), in rounds otherwise.
constexpr int kDenseFlips = 5;

// Shared memory of a CTA, in 4-byte words: fixed part, then per replica.  N:
// columns kept per row, 32 or 64.
template <int N>
struct SmallSmem {
  static constexpr int J = 0;                  // [N][N] couplings
  static constexpr int PERM = J + N * N;       // [2][64] visiting orders
  static constexpr int INV = PERM + 2 * 64;    // [2][64] positions of spins
  static constexpr int WORK = INV + 2 * 64;    // [2][64] helper scratch
  static constexpr int FIXED = WORK + 2 * 64;
  static constexpr int PER = N + 2 + 15;       // words per replica
  static size_t bytes(int cap) {  // and a byte per replica of any read
    return 4 * ((size_t)FIXED + (size_t)PER * cap) + kMaxReplicas;
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

template <bool RANDOM, int N>
__global__ void __launch_bounds__(32 * (kMaxSmallWarps + 1), 1)
    k_sweep_small(const SmallArgs a) {
  using Smem = SmallSmem<N>;
  constexpr bool kTwo = N > 32;  // a second position per lane
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) uint32_t sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  auto sync_read = [&]() {  // every CTA of the read
    if (csize > 1) cl.sync(); else __syncthreads();
  };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sweep0 = (uint32_t)(*a.s.sweep_counter);
  // instances of this launch (uniform per CTA)
  auto wanted = [&](int i) {
    return a.p.n[i] <= kSmallMaxN && a.p.replicas[i] > a.above &&
           a.p.replicas[i] <= a.cap &&
           !(a.p.csr_row_off && a.p.csr_row_off[i] >= 0) &&
           !(a.skip_inst && a.skip_inst[i]);
  };
  bool some = a.above == 0;
  if (a.above > 0) {  // nearly always there is none
    bool own = false;
    for (int i = tid; i < a.p.num_instances; i += blockDim.x)
      own = own || wanted(i);
    some = __syncthreads_or(own);
  }
  for (int64_t r = blockIdx.x / csize; some && r < a.p.num_reads;
       r += gridDim.x / csize) {
    const int inst = a.p.read_inst[r];
    if (!wanted(inst)) continue;
    const int n = a.p.n[inst];
    const int NW = a.warps;  // warps with chains
    const int R = a.p.replicas[inst];
    // this CTA's chains c0 ... c1 - 1; the energies of all, the slot map and
    // the exchange are rank 0's
    const int Rc = (R + csize - 1) / csize;
    const int c0 = rank * Rc < R ? rank * Rc : R;
    const int c1 = c0 + Rc < R ? c0 + Rc : R;
    const int64_t lread = r - a.p.read_off[inst];
    const int64_t base = a.p.chain_off[inst] + lread * R;
    const int words = (n + 31) >> 5;
    const bool ising = a.p.problem_type == PYSA_GB_ISING;
    const float scale = ising ? 2.0f : 1.0f;
    const float* betas = a.p.ladder + a.p.ladder_off[inst];
    const int32_t* sorted = a.p.ladder_sorted + a.p.ladder_off[inst];
    float* J = reinterpret_cast<float*>(sm + Smem::J);
    int32_t* perm_s = reinterpret_cast<int32_t*>(sm + Smem::PERM);
    int32_t* inv_s = reinterpret_cast<int32_t*>(sm + Smem::INV);
    int32_t* work_s = reinterpret_cast<int32_t*>(sm + Smem::WORK);
    uint32_t* per = sm + Smem::FIXED;
    const int cap = a.cap;
    // per replica; the first six are copies of global state
    float* Hs = reinterpret_cast<float*>(per);             // [cap][N]
    uint32_t* Ss = per + N * cap;                          // [cap][2]
    float* E = reinterpret_cast<float*>(per + (N + 2) * cap);
    int32_t* B = reinterpret_cast<int32_t*>(per + (N + 3) * cap);
    float* beta_c = reinterpret_cast<float*>(per + (N + 4) * cap);
    float* bestE = reinterpret_cast<float*>(per + (N + 5) * cap);
    float* Bt = reinterpret_cast<float*>(per + (N + 6) * cap);
    float2* dE = reinterpret_cast<float2*>(per + (N + 8) * cap);  // [cap]
    float2* X2 = reinterpret_cast<float2*>(per + (N + 10) * cap);  // draw, log
    float2* E2 =  // energy, dbeta
        reinterpret_cast<float2*>(per + (N + 12) * cap);
    int32_t* B2 = reinterpret_cast<int32_t*>(per + (N + 14) * cap);
    uint32_t* LT = per + (N + 15) * cap;                     // reject below
    uint8_t* dense = reinterpret_cast<uint8_t*>(per + (N + 16) * cap);  // [R]

    // ---- state in
    {
      const float* Jg = a.p.J + a.p.j_off[inst];
      const int ld = a.p.ld[inst];
      for (int e = tid; e < n * N; e += blockDim.x) {
        const int i = e / N, c = e % N;
        J[e] = c < n ? Jg[(int64_t)i * ld + c] : 0.0f;
      }
      for (int e = N * c0 + tid; e < N * c1; e += blockDim.x) {
        const int c = e / N, i = e % N;
        Hs[e] = i < n ? a.fields[(base + c) * (int64_t)a.field_ld + i] : 0.0f;
      }
      for (int c = tid; c < R; c += blockDim.x) {
        const int64_t g = base + c;
        Ss[2 * c] = a.s.spins[g * a.p.words];
        Ss[2 * c + 1] = words > 1 ? a.s.spins[g * a.p.words + 1] : 0u;
        E[c] = a.s.energies[g];
        B[c] = a.s.beta_idx[g];
        beta_c[c] = a.s.chain_beta[g];
        bestE[c] = a.s.best_energy[g];
        Bt[c] = betas[c];
      }
      for (int c = tid; c < R; c += blockDim.x) dense[c] = 1;
      if (RANDOM && warp == NW)
        small_order(a.seed, (uint32_t)inst, sweep0, n, lane, work_s,
                    work_s + 64, perm_s + 64 * (sweep0 & 1),
                    inv_s + 64 * (sweep0 & 1));
    }
    sync_read();

    for (int s = 0; s < a.num_sweeps; ++s) {
      const uint32_t sweep = sweep0 + (uint32_t)s;
      const bool xch = a.use_pt && exchange_after(a.exchange_every, sweep);
      if (warp < NW) {
        // ------------------------------------------------------- sweeps
        const int32_t* perm = perm_s + 64 * (sweep & 1);
        const int32_t* inv = inv_s + 64 * (sweep & 1);
        const bool two = kTwo && n > 32;
        const int k1 = lane + 32;
        const bool in0 = lane < n, in1 = kTwo && k1 < n;
        const int i0 = in0 ? (RANDOM ? perm[lane] : lane) : 0;
        const int i1 = in1 ? (RANDOM ? perm[k1] : k1) : 0;
        for (int c = c0 + warp; c < c1; c += NW) {
          float* H = Hs + N * c;
          uint32_t* S = Ss + 2 * c;
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
          const uint32_t B0 = S0, B1 = S1;  // spins before the sweep
          // one decision: position js of half hf, signed field y.  The exact
          // rule where the thresholds have no answer.
          auto exact = [&](int t, float y) {
            return accept_slow_redraw(scale * y, beta, seed, (uint32_t)inst,
                                      sweep, cl, (uint32_t)t);
          };
          bool again = !dense[c];
          if (!again) {
            // Flips are common: the positions in turn.  Every row, threshold
            // and the field values after a flip are ready before the
            // decision, which selects: about 60 cycles a position.  No exact
            // rule here: a decision that needs it (once in a few hundred
            // sweeps) has the chain swept again in rounds.
            uint32_t unsure = 0u, f0 = 0u, f1 = 0u;
            auto turn = [&](int t, bool hf) {
              const int js = t & 31;
              const float* row = J + N * (RANDOM ? perm[t] : t);
              const float r0 = row[i0], r1 = kTwo ? row[i1] : 0.0f;
              const float th = __shfl_sync(0xffffffffu, hf ? th1 : th0, js);
              const float tl = __shfl_sync(0xffffffffu, hf ? tl1 : tl0, js);
              const bool sb = (((hf ? S1 : S0) >> js) & 1u) != 0u;
              const float d = sb ? -scale : scale;
              const float v0 = fmaf(d, r0, h0), v1 = fmaf(d, r1, h1);
              const float hv = __shfl_sync(0xffffffffu, hf ? h1 : h0, js);
              const float y = sb ? hv : -hv;
              const bool acc = y >= th;
              unsure |= (!acc && !(y < tl)) ? 1u : 0u;
              h0 = acc ? v0 : h0;
              h1 = acc ? v1 : h1;
              const float de = acc ? scale * y : 0.0f;
              if (hf) {
                f1 |= acc ? 1u << js : 0u;
                d1 -= de;
              } else {
                f0 |= acc ? 1u << js : 0u;
                d0 -= de;
              }
            };
            const int na = n < 32 ? n : 32;
#pragma unroll 4
            for (int t = 0; t < na; ++t) turn(t, false);
#pragma unroll 4
            for (int t = 32; t < n; ++t) turn(t, true);
            again = unsure != 0u;
            if (again) {
              h0 = in0 ? H[i0] : 0.0f;
              h1 = in1 ? H[i1] : 0.0f;
              d0 = d1 = 0.0f;
            } else {
              S0 ^= f0;
              S1 ^= f1;
            }
          }
          if (again) {
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
              acc = exact(js + (hf ? 32 : 0), y);
            if (acc) {
              const bool sb = ((hf ? S1 : S0) & bit) != 0u;
              const float d = sb ? -scale : scale;
              const float* row = J + N * i;
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
            dense[c] = kDenseFlips * (__popc(S0 ^ B0) + __popc(S1 ^ B1)) > n;
            S[0] = na;
            if (words > 1) S[1] = nb;
            dE[c] = make_float2(d0, d1);
          }
        }
      } else {
        // ---------------------------------------------------- work ahead
        if (xch && rank == 0)
          for (int k = lane; k < R - 1; k += 32) {
            const uint32_t x = draw1(a.seed, TAG_PT, (uint32_t)inst, sweep,
                                     (uint32_t)lread, (uint32_t)k);
            // accept a pair at de >= .y, reject it below LT: log u and its
            // band (pt_accept_lf); in between, the exact rule
            const float lf = log_uniform_f32(x);
            const float m = fmaf(2e-6f, fabsf(lf), 3.1e-5f);
            X2[k] = make_float2(__uint_as_float(x), fminf(lf + m, 0.0f));
            LT[k] = __float_as_uint(lf - m);
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
        for (int c = c0 + lane; c < c1; c += 32) {
          const float2 d = dE[c];
          const float e =
              (float)((double)E[c] + ((double)d.x + (double)d.y));
          E[c] = e;
          if (rank != 0) cl.map_shared_rank(E, 0)[c] = e;
          // strict < (pysa/simulation.py:150-171)
          if (e < bestE[c]) {
            bestE[c] = e;
            const int64_t g = base + c;
            a.s.best_sweep[g] = (int32_t)sweep;
            const uint32_t* S = Ss + 2 * c;
            for (int w = 0; w < words; ++w)
              a.s.best_spins[g * a.p.words + w] = S[w];
          }
        }
        __syncwarp();
      }
      if (csize > 1) cl.sync();  // the energies are in rank 0
      if (warp == 0 && rank == 0) {
        if (xch && R > 1) {
          // pairs (R-1, R-2), (R-2, R-3), ... in order: only the replica
          // entering slot k1 carries from pair to pair, so every pair's
          // other replica, its energy and the betas' difference are read up
          // front and the pass keeps the carried one in registers
          for (int k = lane; k < R - 1; k += 32) {
            const int t1 = R - k - 1, t2 = R - k - 2;
            const int b2 = B[t2];
            B2[k] = b2;
            E2[k] = make_float2(E[b2], __fsub_rn(Bt[t1], Bt[t2]));
          }
          __syncwarp();
          if (lane == 0) {
            // without the exact rule; a pair that needs it has the pass made
            // again below
            const int cb0 = B[R - 1];
            const float ce0 = E[cb0];
            int cb = cb0;
            float ce = ce0;
            uint32_t unsure = 0u;
#pragma unroll 4
            for (int k = 0; k < R - 1; ++k) {
              const int b2 = B2[k];
              const float2 e2 = E2[k], x2 = X2[k];
              const float de = __fmul_rn(__fsub_rn(ce, e2.x), e2.y);
              const bool sw = de >= x2.y;
              unsure |= (!sw && !(de < __uint_as_float(LT[k]))) ? 1u : 0u;
              B[R - k - 1] = sw ? b2 : cb;  // final: no later pair
              cb = sw ? cb : b2;
              ce = sw ? ce : e2.x;
            }
            if (unsure) {
              for (int k = 0; k < R - 1; ++k) B[R - k - 2] = B2[k];
              B[R - 1] = cb0;
              cb = cb0;
              ce = ce0;
              for (int k = 0; k < R - 1; ++k) {
                const int t1 = R - k - 1, t2 = R - k - 2, b2 = B[t2];
                const float e2 = E[b2];
                const float de = __fmul_rn(__fsub_rn(ce, e2),
                                           __fsub_rn(Bt[t1], Bt[t2]));
                const bool sw = pt_accept(
                    de, draw1(a.seed, TAG_PT, (uint32_t)inst, sweep,
                              (uint32_t)lread, (uint32_t)k));
                B[t1] = sw ? b2 : cb;
                cb = sw ? cb : b2;
                ce = sw ? ce : e2;
              }
            }
            B[0] = cb;
          }
          __syncwarp();
          for (int k = lane; k < R; k += 32) {
            const int c = B[k], own = csize > 1 ? c / Rc : 0;
            if (own == 0)
              beta_c[c] = Bt[k];
            else
              cl.map_shared_rank(beta_c, own)[c] = Bt[k];
          }
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
      sync_read();
    }

    // ---- state out
    for (int e = N * c0 + tid; e < N * c1; e += blockDim.x) {
      const int c = e / N, i = e % N;
      if (i < n) a.fields[(base + c) * (int64_t)a.field_ld + i] = Hs[e];
    }
    for (int c = c0 + tid; c < c1; c += blockDim.x) {
      const int64_t g = base + c;
      a.s.spins[g * a.p.words] = Ss[2 * c];
      if (words > 1) a.s.spins[g * a.p.words + 1] = Ss[2 * c + 1];
      a.s.energies[g] = E[c];
      a.s.chain_beta[g] = beta_c[c];
      a.s.best_energy[g] = bestE[c];
    }
    if (rank == 0)
      for (int c = tid; c < R; c += blockDim.x) a.s.beta_idx[base + c] = B[c];
    sync_read();  // before the next read's state
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

template <bool RANDOM, int N>
static cudaError_t launch_small_t(const SmallArgs& a, int64_t ctas, int cs,
                                  bool helper, cudaStream_t st) {
  using Smem = SmallSmem<N>;
  const void* f = (const void*)k_sweep_small<RANDOM, N>;
  static std::atomic<uint64_t> allowed;
  cudaError_t e = allow_smem(f, Smem::bytes(kMaxReplicas), allowed);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(32 * (a.warps + (helper ? 1 : 0)));
  cfg.dynamicSmemBytes = Smem::bytes(a.cap);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_sweep_small<RANDOM, N>, a);
}

cudaError_t launch_small(SmallArgs a, bool random, int sms, cudaStream_t st) {
  if (a.p.num_reads <= 0) return cudaSuccess;
  // couplings of up to 32 or 64 columns (instances wider than 64, swept
  // elsewhere, may share the batch)
  const bool narrow = a.p.max_n <= 32;
  auto launch = [&](int64_t ctas, int cs, bool helper) {
    if (narrow)
      return random ? launch_small_t<true, 32>(a, ctas, cs, helper, st)
                    : launch_small_t<false, 32>(a, ctas, cs, helper, st);
    return random ? launch_small_t<true, 64>(a, ctas, cs, helper, st)
                  : launch_small_t<false, 64>(a, ctas, cs, helper, st);
  };
  // The replicas of an average read (of every read in a batch of one
  // instance).  Reads with far more have a launch of their own below.
  const int64_t avg = (a.p.num_chains + a.p.num_reads - 1) / a.p.num_reads;
  const bool mixed = a.p.num_instances > 1;
  const int64_t room = !mixed ? avg : 2 * avg > 32 ? 2 * avg : 32;
  a.above = 0;
  a.cap = (int32_t)(room < kMaxReplicas ? room : kMaxReplicas);
  a.cap += a.cap & 1;  // pairs of words stay 8-byte aligned
  // a cluster per read while the reads leave SMs idle (a sixteenth more CTAs
  // than SMs is still one each for nearly all) and a CTA keeps four chains
  int cs = 1;
  while (cs < 8 && a.p.num_reads * cs * 32 <= sms * 17 &&
         (avg + 1) / (2 * cs) >= 4)
    cs *= 2;
  // warps of a CTA: its chains in equal turns, as few turns as the CTAs that
  // an SM then holds at once (64 registers a thread, shared memory) allow
  // without more rounds of CTAs
  // (a short call's time goes into moving the state, by every warp there is)
  const bool helper = random || (a.use_pt && avg > 1) || a.num_sweeps < 16;
  const int64_t per = (avg + cs - 1) / cs, ctas = a.p.num_reads * cs;
  const int64_t smem = 1024 + (int64_t)(narrow ? SmallSmem<32>::bytes(a.cap)
                                               : SmallSmem<64>::bytes(a.cap));
  double best = 0.0;
  a.warps = 0;
  for (int64_t t = (per + kMaxSmallWarps - 1) / kMaxSmallWarps; t <= per; ++t) {
    const int64_t w = (per + t - 1) / t;
    if (a.warps && w == a.warps) continue;
    int64_t held = 32 / (w + (helper ? 1 : 0));
    if (held > 233472 / smem) held = 233472 / smem;
    if (held < 1) held = 1;
    const int64_t rounds = (ctas + held * sms - 1) / (held * sms);
    const double cost = (double)rounds * ((double)t + 0.5);
    if (a.warps == 0 || cost < best) {
      best = cost;
      a.warps = (int32_t)w;
    }
    if (rounds == 1) break;  // more turns gain nothing
  }
  const int32_t advance = a.advance;
  const bool more = mixed && a.cap < kMaxReplicas;
  a.advance = more ? 0 : advance;
  cudaError_t e = launch(ctas, cs, helper);
  if (e != cudaSuccess || !more) return e;
  // reads of more replicas: an SM each, all its warps
  a.above = a.cap;
  a.cap = kMaxReplicas;
  a.warps = kMaxSmallWarps;
  a.advance = advance;
  return launch(a.p.num_reads < sms ? a.p.num_reads : sms, 1, true);
}

}  // namespace pysa_gb
