// sweep_csr.cu -- the Metropolis sweep for sparse couplings on CUDA cores
// (sm_103a).
//
// Same sweep as pysa/simulation.py:60-76 (sequential) / :41-57 (random
// order) with the rule of pysa/ising.py:40-63 / pysa/qubo.py:40-63, but the
// field of spin i is recomputed from the nonzero couplings of row i instead
// of a dense dot, so an attempt costs O(degree).
//
// A CTA holds 32 chains (lane = chain); shared memory holds their spins as
// one word per spin, bit = chain, so a warp reads a neighbour's spins with
// one broadcast load and its own chain's with a shift by the lane.  The
// visiting positions are cut into quads of four (one Philox draw each), and
// the quads into levels: a quad's level is one more than the largest level of
// the earlier quads that read its spins or hold spins it reads.  Quads of
// one level do not see each other's flips, so the CTA's warps decide them at
// the same time, a barrier apart from the next level, and every attempt reads
// exactly the spins it reads when the positions are visited one by one.  A
// quad is decided in order by one warp; its records and random thresholds
// are fetched before the barrier.  (Where quads tie unrelated positions
// together, as at the row ends of a lattice whose side is no multiple of
// four, the schedule cuts them into shorter units; see k_csr_schedule.)
//
// Bound by instruction issue and, per level, by the latency of one quad's four
// dependent attempts.  Measured against one thread per chain visiting the
// positions one by one (times per sweep with the exchange): 64 x 64 lattice,
// 4000 chains 1.44 -> 0.12 ms in visiting order (79 levels), 1.66 -> 0.21 ms
// in random order (half of it makes the orders and the schedule); ring of 1000,
// every quad a level, 4000 chains 0.36 -> 0.18, 100 000 0.62 -> 0.48; 2000 spins
// with 48 neighbours, 4000 chains 6.7 -> 1.3, 100 000 9.8 -> 8.3.
//
// Row layout: the entries of row i are grouped by column % 8 (ascending
// column inside a group) and rows[9 i + k] .. rows[9 i + k + 1] delimit group
// k; or, when every row has at most 32 entries, each row is a fixed record
// of D = 4, 8, 16 or 32 entries in that order (bit 31 of the column marks
// the last entry of a group, padding entries have value 0), read with
// vector loads all at once.  The field is summed as eight partial sums, one
// per group, added in group order, then h_i: the fixed-order f32 dot of the
// oracle with its zero terms left out (adding a zero product changes no
// partial sum), so trajectories equal the oracle's for any couplings, not
// only integer ones.
#include <type_traits>

#include "common.cuh"
#include "csr_api.h"
#include "sweep_plain.cuh"

namespace pysa_gb {

// --------------------------------------------------------------- schedule
// The level schedule of one visiting order lives in the high halves of the
// order's row of the visiting-order workspace (spins are below 2^16).  With
// nu units in nl levels: entry k < nu the k-th unit by (level, position),
// entries nu ... nu + nl the levels' first places in that list, and the last
// three entries of the row's first n: whether field sums are exact in any
// order, nu, nl.  A unit is quad q, or (when nu > quads) q << 4 | first
// position in it << 2 | positions - 1.  That takes nu + nl + 4 <= n entries,
// which quads fit for n >= 10; below that, and where there is no such
// workspace, every quad is a level of its own.  So it is up to n = 32, and in
// random order to n = 64, where the schedule takes longer than the levels it
// saves (n = 24, 20 000 chains, random order: 52 us a sweep with it, 39 without).
__host__ __device__ constexpr int sched_min_n(bool random) {
  return random ? 65 : 33;
}
constexpr int kSchedThreads = 512;
constexpr int kSchedRounds = 48;
constexpr int kSchedNames = 32768;  // units named by a stretch of units
// Widest instance whose quads may be cut (shared memory, 16 bits per unit).
constexpr int kSchedCutN = 8192;

// Whether a schedule is made by rounds alone (see k_csr_schedule).
__host__ __device__ constexpr bool sched_by_rounds(bool random, int width) {
  return random && (width == 4 || width == 8);
}

// Dynamic shared memory a CTA of these kernels may take (a little is static).
constexpr size_t kCsrSmem = 232448 - 2560;

__host__ __device__ constexpr int csr_quads(int n) { return (n + 3) >> 2; }

// Schedule entries (units, and first places of the levels) the sweep holds:
// at most n - 2 when quads may be cut, else two per quad and one.
__host__ __device__ constexpr int sched_cap(int n) {
  const int cut = (n < kSchedCutN ? n : kSchedCutN) + 1;
  const int whole = 2 * csr_quads(n) + 1;
  return cut > whole ? cut : whole;
}

// Shared memory of k_csr_schedule for up to nu units of n positions.
__host__ __device__ constexpr size_t sched_bytes(int nu, int n, bool random,
                                                 bool cut) {
  return 4 * ((size_t)nu + 1) + 4 * (size_t)nu + 2 * (size_t)nu +
         (random ? 2 * (size_t)n : 0) +
         (cut ? 2 * (size_t)n + 2 * ((size_t)nu + 1) : 0);
}

// CTA per instance.  Units are levelled 512 at a time (earlier ones are
// final), the levels of a chunk raised until none changes.  That takes as many
// rounds as the longest chain of units in the chunk, and a round as long as a
// row, so it is kept for records of 4 entries and, in random order, of 8; other
// rows, and in visiting order a chunk that is not done after kSchedRounds
// rounds, take the units in order (a sweep with its schedule in random order,
// 2000 spins with 32 neighbours 4.03 -> 0.47 ms, 1500 with 100 19.2 -> 3.4).
// Then a counting sort, stable in the position.  When the quads give fewer than
// 8 per level, they are cut between positions that do not touch (neither reads
// the other's spin) and levelled again; the cut schedule is kept when it has
// less than two thirds of the levels.
template <bool RANDOM>
__global__ void __launch_bounds__(kSchedThreads)
    k_csr_schedule(const CsrArgs a) {
  extern __shared__ __align__(16) unsigned char ssm[];
  __shared__ int max_level;
  __shared__ int at_s[kSchedThreads + 1];  // see in_order_grouped
  __shared__ int warp_sum_s[kSchedThreads / 32];
  const int inst = blockIdx.x;
  if (a.p.csr_row_off[inst] < 0) return;  // dense
  const int n = a.p.n[inst], nq = csr_quads(n);
  if (n < sched_min_n(RANDOM)) return;
  const uint32_t sweep = (uint32_t)(*a.s.sweep_counter);
  int32_t* row =
      a.perm + ((int64_t)(RANDOM ? sweep % (uint32_t)a.perm_slots : 0u) *
                    a.p.num_instances + inst) * (int64_t)a.p.max_n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int32_t* rows =
      a.width > 0 ? nullptr : a.p.csr_rows + a.p.csr_row_off[inst] * 9;
  const int32_t* colp = a.p.csr_col + a.p.csr_ent_off[inst];
  const float* valp = a.p.csr_val + a.p.csr_ent_off[inst];
  auto entries = [&](int i, int64_t& e, int64_t& e1) {
    e = (int64_t)a.width * i;
    e1 = e + a.width;
    if (a.width == 0) {
      e = rows[(int64_t)i * 9];
      e1 = rows[(int64_t)i * 9 + 8];
    }
  };
  auto column = [&](int64_t e) { return __ldg(colp + e) & 0x7fffffff; };
  // positions of the spins, and the uncut/cut units' tables behind it
  uint16_t* names = reinterpret_cast<uint16_t*>(ssm);  // see in_order
  uint16_t* inv =                                      // [n], random
      names + (sched_by_rounds(RANDOM, a.width) ? 0 : kSchedNames);
  unsigned char* tab = reinterpret_cast<unsigned char*>(inv) +
                       (RANDOM ? 2 * (((size_t)n + 1) & ~1ull) : 0);
  bool odd = false;  // a coupling that is no integer below 2^18
  for (int t = tid; t < n; t += blockDim.x) {
    if (RANDOM)
      inv[row[t] & 0xFFFF] = (uint16_t)t;
    else
      row[t] = t;
    if (a.width > 0)
      for (int64_t e = (int64_t)a.width * t, e1 = e + a.width; e < e1; ++e) {
        const float v = __ldg(valp + e);
        odd = odd || !(fabsf(v) <= 262144.0f && v == rintf(v));
      }
  }
  // up to 32 such couplings add up without rounding, whatever the order
  const bool any_order = !__syncthreads_or(odd) && a.width > 0;
  auto spin_at = [&](int t) { return RANDOM ? row[t] & 0xFFFF : t; };
  auto pos_of = [&](int i) { return RANDOM ? (int)inv[i] : i; };

  int best_nl = 0;
  for (int cut = 0; cut < 2; ++cut) {
    int nu = nq;
    uint16_t *uid = nullptr, *first = nullptr;
    unsigned char* mem = tab;
    if (cut) {
      // unit of every position: a running count of the unit starts
      uid = reinterpret_cast<uint16_t*>(mem);                    // [n]
      mem += 2 * (((size_t)n + 1) & ~1ull);
      int carry = 0;
      for (int t0 = 0; t0 < n; t0 += blockDim.x) {
        const int t = t0 + tid;
        int start = 0;
        if (t < n) {
          start = 1;
          if (t & 3) {
            const int i = spin_at(t), j = spin_at(t - 1);
            int64_t e, e1;
            for (entries(i, e, e1); e < e1; ++e)
              if (column(e) == j) start = 0;
            for (entries(j, e, e1); e < e1; ++e)
              if (column(e) == i) start = 0;
          }
        }
        int v = start;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o) v += up;
        }
        if (lane == 31) warp_sum_s[warp] = v;
        __syncthreads();
        int before = carry, all = 0;
        for (int w = 0; w < kSchedThreads / 32; ++w) {
          if (w < warp) before += warp_sum_s[w];
          all += warp_sum_s[w];
        }
        if (t < n) uid[t] = (uint16_t)(before + v - 1);
        carry += all;
        __syncthreads();
      }
      nu = carry;
      if (nu == nq) return;  // nothing to cut (uniform)
      first = reinterpret_cast<uint16_t*>(mem);                  // [nu + 1]
      mem += 2 * (((size_t)nu + 2) & ~1ull);
      for (int t = tid; t < n; t += blockDim.x)
        if (t == 0 || uid[t] != uid[t - 1]) first[uid[t]] = (uint16_t)t;
      if (tid == 0) first[nu] = (uint16_t)n;
    }
    uint32_t* cnt = reinterpret_cast<uint32_t*>(mem);            // [nu + 1]
    volatile int32_t* lev =
        reinterpret_cast<volatile int32_t*>(cnt + nu + 1);       // [nu]
    uint16_t* order =
        reinterpret_cast<uint16_t*>(cnt + 2 * nu + 1);           // [nu]
    auto unit_of = [&](int t) { return cut ? (int)uid[t] : t >> 2; };
    if (tid == 0) max_level = 0;
    for (int u = tid; u < nu; u += blockDim.x) lev[u] = 0;
    for (int u = tid; u <= nu; u += blockDim.x) cnt[u] = 0u;
    __syncthreads();
    auto first_of = [&](int u) { return cut ? (int)first[u] : 4 * u; };
    auto end_of = [&](int u) {
      return cut ? (int)first[u + 1] : 4 * u + 4 < n ? 4 * u + 4 : n;
    };
    // Levels of units ub ... ue - 1, one after another (the earlier ones are
    // final).  The CTA gathers the units that a stretch of units names; then
    // one warp goes through them in shared memory.  Fixed records: the next
    // unit's names are on their way (about 150 cycles a unit).
    auto in_order = [&](int ub, int ue) {
      const int per = 4 * a.width, step = kSchedNames / per;
      for (int c0 = ub; c0 < ue; c0 += step) {
        const int c1 = c0 + step < ue ? c0 + step : ue;
        for (int k = tid; k < (c1 - c0) * per; k += blockDim.x) {
          const int u = c0 + k / per, j = k % per;
          const int t = first_of(u) + j / a.width;
          names[k] = (uint16_t)(
              t < end_of(u)
                  ? unit_of(pos_of(
                        column((int64_t)a.width * spin_at(t) + j % a.width)))
                  : u);  // itself: no dependence
        }
        __syncthreads();
        if (warp == 0) {
          int nx[4];
          auto load = [&](int u) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              nx[i] = lane + 32 * i < per
                          ? names[(u - c0) * per + lane + 32 * i]
                          : u;
          };
          load(c0);
          for (int u = c0; u < c1; ++u) {
            int at[4], lv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) at[i] = nx[i];
            const int own = lev[u];
#pragma unroll
            for (int i = 0; i < 4; ++i) lv[i] = lev[at[i]];
            if (u + 1 < c1) load(u + 1);
            int m = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (at[i] < u) m = max(m, lv[i] + 1);
            m = max(__reduce_max_sync(0xffffffffu, m), own);
            if (lane == 0) lev[u] = m;
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (at[i] > u)
                atomicMax(const_cast<int32_t*>(lev) + at[i], m + 1);
            __syncwarp();
          }
        }
        __syncthreads();
      }
    };
    // The same for grouped rows, which may be very uneven: as many units at a
    // time as their entries fit; one that does not fit by itself (four rows of
    // more than kSchedNames entries) is read from the rows.
    auto in_order_grouped = [&]() {
      for (int c0 = 0; c0 < nu;) {
        int len = 0;
        if (c0 + tid < nu)
          for (int t = first_of(c0 + tid), te = end_of(c0 + tid); t < te; ++t) {
            int64_t e, e1;
            entries(spin_at(t), e, e1);
            len += (int)(e1 - e);
          }
        int upto = len;  // entries up to this thread's unit
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += up;
        }
        if (lane == 31) warp_sum_s[warp] = upto;
        __syncthreads();
        for (int w = 0; w < warp; ++w) upto += warp_sum_s[w];
        at_s[tid + 1] = upto;
        if (tid == 0) at_s[0] = 0;
        const int fit =
            __syncthreads_count(c0 + tid < nu && upto <= kSchedNames);
        const int c1 = c0 + (fit > 0 ? fit : 1);
        for (int u = c0 + warp; fit > 0 && u < c1; u += kSchedThreads / 32) {
          uint16_t* name = names + at_s[u - c0];
          for (int t = first_of(u), te = end_of(u); t < te; ++t) {
            int64_t e, e1;
            entries(spin_at(t), e, e1);
            for (int64_t x = e + lane; x < e1; x += 32)
              name[x - e] = (uint16_t)unit_of(pos_of(column(x)));
            name += e1 - e;
          }
        }
        __syncthreads();
        if (warp == 0)
          for (int u = c0; u < c1; ++u) {
            // f(unit named) over the unit's entries, a lane each
            auto each = [&](auto f) {
              if (fit > 0) {
                const int end = at_s[u - c0 + 1];
#pragma unroll 4
                for (int j = at_s[u - c0] + lane; j < end; j += 32)
                  f((int)names[j]);
              } else {
                for (int t = first_of(u), te = end_of(u); t < te; ++t) {
                  int64_t e, e1;
                  entries(spin_at(t), e, e1);
                  for (int64_t x = e + lane; x < e1; x += 32)
                    f(unit_of(pos_of(column(x))));
                }
              }
            };
            int m = 0;
            each([&](int at) {
              const int lv = lev[at];
              if (at < u) m = max(m, lv + 1);
            });
            m = max(__reduce_max_sync(0xffffffffu, m), lev[u]);
            if (lane == 0) lev[u] = m;
            each([&](int at) {
              if (at > u) atomicMax(const_cast<int32_t*>(lev) + at, m + 1);
            });
            __syncwarp();
          }
        __syncthreads();
        c0 = c1;
      }
    };
    for (int u0 = 0; u0 < nu; u0 += blockDim.x) {
      const int u = u0 + tid;
      int tb = 0, te = 0;
      if (u < nu) {
        tb = first_of(u);
        te = end_of(u);
      }
      if (a.width != 4 && !sched_by_rounds(RANDOM, a.width)) {
        if (a.width > 0)
          in_order(0, nu);
        else
          in_order_grouped();
        break;
      }
      // the units of the spins that this one reads, the first kDeps of them
      // kept in registers over the rounds (all for rows of 4 entries)
      constexpr int kDeps = 16;
      int dep[kDeps], nd = 0;
#pragma unroll
      for (int d = 0; d < kDeps; ++d) dep[d] = u;  // itself: no dependence
      if (a.width == 4) {
#pragma unroll
        for (int d = 0; d < kDeps; ++d) {
          const int t = tb + (d >> 2);
          if (t < te)
            dep[d] = unit_of(pos_of(
                column((int64_t)4 * spin_at(t) + (d & 3))));
        }
        nd = kDeps;
      }
      for (int round = 0;; ++round) {
        if (!RANDOM && round == kSchedRounds) {  // uniform
          in_order(u0, u0 + (int)blockDim.x < nu ? u0 + (int)blockDim.x : nu);
          break;
        }
        bool up = false;
        int m = 0;
        auto meet = [&](int uc) {
          if (uc < u) {
            m = max(m, lev[uc] + 1);
          } else if (uc > u && lev[uc] <= lev[u]) {
            // a later unit may flip a spin that this one reads: the rows
            // name it also where the other row lacks the entry
            atomicMax(const_cast<int32_t*>(lev) + uc, lev[u] + 1);
            up = true;
          }
        };
        if (nd) {
          if (u < nu)
#pragma unroll
            for (int d = 0; d < kDeps; ++d) meet(dep[d]);
        } else {
          for (int t = tb; t < te; ++t) {
            int64_t e, e1;
            for (entries(spin_at(t), e, e1); e < e1; ++e)
              meet(unit_of(pos_of(column(e))));
          }
        }
        if (u < nu && m > lev[u]) {
          atomicMax(const_cast<int32_t*>(lev) + u, m);
          up = true;
        }
        if (!__syncthreads_or(up)) break;
      }
    }
    for (int u = tid; u < nu; u += blockDim.x) {
      atomicAdd(&cnt[lev[u] + 1], 1u);
      atomicMax(&max_level, lev[u]);
    }
    __syncthreads();
    const int nl = max_level + 1;
    // the quads' schedule is already written when a cut one is tried
    const bool keep = !cut || (3 * nl < 2 * best_nl && nu + nl + 4 <= n);
    if (!keep) return;  // uniform
    best_nl = nl;
    if (tid < 32) {
      // cnt[l] = first place of level l; cnt[nl] = nu
      uint32_t carry = 0u;
      for (int l0 = 0; l0 <= nl; l0 += 32) {
        uint32_t v = l0 + lane <= nl ? cnt[l0 + lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t up = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o) v += up;
        }
        v += carry;
        if (l0 + lane <= nl) cnt[l0 + lane] = v;
        carry = __shfl_sync(0xffffffffu, v, 31);
      }
    }
    __syncthreads();
    auto put_high = [&](int k, uint32_t v) {
      row[k] = (row[k] & 0xFFFF) | (int32_t)(v << 16);
    };
    for (int l = tid; l <= nl; l += blockDim.x) put_high(nu + l, cnt[l]);
    __syncthreads();
    if (tid < 32) {
      for (int u0 = 0; u0 < nu; u0 += 32) {
        const int u = u0 + lane;
        const uint32_t l = u < nu ? (uint32_t)lev[u] : 0xFFFFFFFFu;
        const uint32_t same = __match_any_sync(0xffffffffu, l);
        const uint32_t base = u < nu ? cnt[l] : 0u;
        __syncwarp();
        if (u < nu) {
          order[base + __popc(same & ((1u << lane) - 1u))] = (uint16_t)u;
          if ((same >> lane) == 1u) cnt[l] = base + __popc(same);
        }
        __syncwarp();
      }
    }
    __syncthreads();
    for (int k = tid; k < nu; k += blockDim.x) {
      const int u = order[k];
      uint32_t code = (uint32_t)u;
      if (cut) {
        const uint32_t t = first[u], len = first[u + 1] - t;
        code = ((t >> 2) << 4) | ((t & 3u) << 2) | (len - 1u);
      }
      put_high(k, code);
    }
    if (tid == 0) {
      put_high(n - 3, any_order ? 1u : 0u);
      put_high(n - 2, (uint32_t)nu);
      put_high(n - 1, (uint32_t)nl);
    }
    // wide enough, or too dear for every sweep (uniform)
    if (n > kSchedCutN || nq >= 8 * nl ||
        (RANDOM && (a.width == 0 || a.width > 8)))
      return;
    __syncthreads();
  }
}

// ------------------------------------------------------------------ sweep
// A quad's four records in the warp's shared memory, each
//   [D entries][D values][h_i][own][pad],
// an entry being the byte offset of its column's spin word (bit 31: end of a
// group, left out when the sums are exact in any order), own that of the
// visited spin.
template <int D>
struct QuadSlab {
  static constexpr int STRIDE = 2 * D + 4;  // words per record
  // words per buffer (grouped rows: 32 entries of one row)
  static constexpr int QUAD = D > 0 ? 4 * STRIDE : 64;
  // 16-byte pieces of columns and values per record, and per lane and quad
  static constexpr int PIECES = D / 2;
  static constexpr int PER_LANE = (4 * PIECES + 31) / 32;
};

// 32 x 32 bit transpose over a warp: lane l's bit b becomes lane b's bit l.
__device__ __forceinline__ uint32_t warp_transpose(uint32_t v, int lane) {
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    const uint32_t m = s == 16  ? 0x0000FFFFu
                       : s == 8 ? 0x00FF00FFu
                       : s == 4 ? 0x0F0F0F0Fu
                       : s == 2 ? 0x33333333u
                                : 0x55555555u;
    const uint32_t o = __shfl_xor_sync(0xffffffffu, v, s);
    v = (lane & s) ? ((o >> s) & m) | (v & ~m) : (v & m) | ((o << s) & ~m);
  }
  return v;
}

template <bool RANDOM, bool ISING, int D>
__global__ void __launch_bounds__(32 * kCsrWarps, 1)
    k_sweep_csr(const CsrArgs a) {
  using Q = QuadSlab<D>;
  extern __shared__ __align__(128) uint32_t smem_u[];
  const SweepItem item = a.items[blockIdx.x];
  const int inst = item.inst;
  const int n = a.p.n[inst], nq = csr_quads(n);
  const int words = (n + 31) >> 5;
  const int W = blockDim.x >> 5;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t* spin_s = smem_u;                                  // [32 words]
  uint32_t* slab = smem_u + words * 32 + warp * 2 * Q::QUAD;  // [W][2][QUAD]
  float2* de_s = reinterpret_cast<float2*>(
      smem_u + words * 32 + W * 2 * Q::QUAD);                 // [W][32]
  uint16_t* sched = reinterpret_cast<uint16_t*>(de_s + W * 32);  // [cap]
  uint16_t* perm_s = sched + sched_cap(n);                    // [n], random
  __shared__ uint8_t imp_s[32];
  const bool valid = lane < item.nchains;
  const int64_t chain = item.chain0 + lane;
  const uint32_t sweep = (uint32_t)(*a.s.sweep_counter);

  const int32_t* row =
      a.perm + ((int64_t)(RANDOM ? sweep % (uint32_t)a.perm_slots : 0u) *
                    a.p.num_instances + inst) * (int64_t)a.p.max_n;
  const bool scheduled = a.perm && n >= sched_min_n(RANDOM);
  if (a.pick != 0) {  // a launch of its own for narrow schedules (launch_csr)
    const bool narrow =
        !scheduled || ((uint32_t)row[n - 2] >> 16) <
                          2u * ((uint32_t)row[n - 1] >> 16);
    if (narrow != (a.pick == 1)) return;
  }
  // spins in, each word's 32 spins x 32 chains transposed
#pragma unroll 4
  for (int w = warp; w < words; w += W)
    spin_s[w * 32 + lane] = warp_transpose(
        valid ? a.s.spins[chain * (int64_t)a.p.words + w] : 0u, lane);
  int nu = nq, nl = nq;
  bool any_order = false;
  if (scheduled) {
    any_order = ((uint32_t)row[n - 3] >> 16) != 0u;
    nu = (int)((uint32_t)row[n - 2] >> 16);
    nl = (int)((uint32_t)row[n - 1] >> 16);
#pragma unroll 2
    for (int k = tid; k <= nu + nl; k += blockDim.x)
      sched[k] = (uint16_t)((uint32_t)row[k] >> 16);
  } else {  // every quad a level of its own
    for (int k = tid; k <= 2 * nq; k += blockDim.x)
      sched[k] = (uint16_t)(k < nq ? k : k - nq);
  }
  const bool cut = nu != nq;  // units are parts of quads
  if (RANDOM)
    for (int t = tid; t < n; t += blockDim.x)
      perm_s[t] = (uint16_t)(row[t] & 0xFFFF);
  __syncthreads();

  const float beta = valid ? a.s.chain_beta[chain] : 0.0f;
  const uint32_t cl = (uint32_t)(chain - a.p.chain_off[inst]);
  const int32_t* rows =
      D > 0 ? nullptr : a.p.csr_rows + a.p.csr_row_off[inst] * 9;
  const int32_t* colp = a.p.csr_col + a.p.csr_ent_off[inst];
  const float* valp = a.p.csr_val + a.p.csr_ent_off[inst];
  const float* h = a.p.h + a.p.h_off[inst];
  constexpr float kScale = ISING ? 2.0f : 1.0f;
  const FieldThreshold ft(beta, kScale);
  // energy change in field units: an exact f32 pair, no f64 in the loop
  float2 dE = make_float2(0.0f, 0.0f);

  auto spin_at = [&](int t) { return RANDOM ? (int)perm_s[t] : t; };
  // records of quad q: 16-byte pieces and h into registers ...
  uint4 rg[Q::PER_LANE > 0 ? Q::PER_LANE : 1];
  float rh = 0.0f;
  // grouped rows: bounds of the next unit's quad, and of the one being decided
  // with the first entries of its four rows
  int rb = 0, re = 0, cb = 0, ce = 0;
  float ch = 0.0f;
  uint32_t cc[4] = {0u, 0u, 0u, 0u};
  float cv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  // the lane's first piece: record pr, columns 4 pk ... or values past them
  const int pr = D > 0 ? lane / (D > 0 ? Q::PIECES : 1) : 0;
  const int pk = D > 0 ? lane % (D > 0 ? Q::PIECES : 1) : 0;
  const bool pcol = 4 * pk < D;
  const uint4* psrc = reinterpret_cast<const uint4*>(
      pcol ? (const void*)(colp + 4 * pk) : (const void*)(valp + 4 * pk - D));
  constexpr int REC_STEP = D > 0 ? 32 / (Q::PIECES > 0 ? Q::PIECES : 1) : 1;
  auto fetch = [&](int q) {
    if constexpr (D > 0) {
#pragma unroll
      for (int e = 0; e < Q::PER_LANE; ++e) {
        const int r = pr + e * REC_STEP, t = 4 * q + r;
        if (r < 4 && t < n) rg[e] = __ldg(psrc + spin_at(t) * (D / 4));
      }
      if (lane < 4 && 4 * q + lane < n) rh = __ldg(h + spin_at(4 * q + lane));
    } else {
      // group starts of position lane / 8, ends and h in lanes 0 .. 3
      const int t = 4 * q + (lane >> 3), te = 4 * q + lane;
      rb = t < n ? __ldg(rows + (int64_t)spin_at(t) * 9 + (lane & 7)) : 0;
      const bool own = lane < 4 && te < n;
      re = own ? __ldg(rows + (int64_t)spin_at(te) * 9 + 8) : 0;
      rh = own ? __ldg(h + spin_at(te)) : 0.0f;
    }
  };
  // 32 entries of a grouped row, one a lane
  auto chunk = [&](int e0, int end, uint32_t& c, float& v) {
    const int e = e0 + lane;
    c = e < end ? 4u * (uint32_t)__ldg(colp + e) : 0u;
    v = e < end ? __ldg(valp + e) : 0.0f;
  };
  // ... and from there into slab buffer b: columns become byte offsets of
  // spin words (times 4; bit 31 kept unless the sums need no groups)
  const uint32_t mul = pcol ? 4u : 1u;
  const uint32_t keep = pcol && !any_order ? 0x80000000u : 0u;
  auto put = [&](int q, int b) {
    if constexpr (D > 0) {
      uint32_t* s = slab + b * Q::QUAD;
#pragma unroll
      for (int e = 0; e < Q::PER_LANE; ++e) {
        const int r = pr + e * REC_STEP;
        uint4 v = rg[e];
        v.x = v.x * mul | (v.x & keep);
        v.y = v.y * mul | (v.y & keep);
        v.z = v.z * mul | (v.z & keep);
        v.w = v.w * mul | (v.w & keep);
        if (r < 4)
          *reinterpret_cast<uint4*>(s + r * Q::STRIDE + 4 * pk) = v;
      }
      if (lane < 4)
        *reinterpret_cast<uint2*>(s + lane * Q::STRIDE + 2 * D) = make_uint2(
            __float_as_uint(rh),
            4 * q + lane < n ? 4u * (uint32_t)spin_at(4 * q + lane) : 0u);
      __syncwarp();
    } else {
      cb = rb;
      ce = re;
      ch = rh;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        chunk(__shfl_sync(0xffffffffu, cb, 8 * k),
              __shfl_sync(0xffffffffu, ce, k), cc[k], cv[k]);
    }
  };
  float tl[4], th[4];
  auto thresholds = [&](int q) {
    uint32_t x[4];
    if (a.s.stream_key)
      draw4(chain_seed(a.seed, valid ? a.s.stream_key : nullptr, chain),
            TAG_SWEEP, (uint32_t)inst, sweep, cl, (uint32_t)q, x);
    else
      draw4_keys(a.keys, TAG_SWEEP, (uint32_t)inst, sweep, cl, (uint32_t)q, x);
#pragma unroll
    for (int k = 0; k < 4; ++k) ft.at(x[k], tl[k], th[k]);
  };
  auto word_at = [&](uint32_t off) {
    return reinterpret_cast<uint32_t*>(
        reinterpret_cast<unsigned char*>(spin_s) + off);
  };
  // a product by a lane constant (the multiply-add pipe; the logic pipe, at
  // half its rate, is the busier one) brings this lane's spin to the sign bit
  const uint32_t to_sign = 0x80000000u >> lane;
  // value of an entry with its spin's sign (Ising), or masked by the spin
  // (QUBO: adding +0 changes no partial sum)
  auto signed_value = [&](uint32_t off, float v) {
    const uint32_t s = *word_at(off) * to_sign;
    return __uint_as_float(ISING
                               ? __float_as_uint(v) ^ (~s & 0x80000000u)
                               : __float_as_uint(v) &
                                     (uint32_t)((int32_t)s >> 31));
  };
  // decides position k of a quad, field f, spin at byte offset `own`.  The
  // fast rule only notes a decision inside the band (`ask`); EXACT decides
  // such a one with the exact rule.
  bool ask = false;
  auto attempt = [&](auto exact_t, int q, int k, float tlk, float thk,
                     uint32_t own, float f) {
    uint32_t* wp = word_at(own);
    const uint32_t w = *wp;
    const float x = __uint_as_float(__float_as_uint(f) ^
                                    (~(w * to_sign) & 0x80000000u));
    bool acc = x >= thk && valid;
    const bool in = valid && !(x >= thk) && !(x < tlk);
    if constexpr (decltype(exact_t)::value) {
      if (in)
        acc = accept_slow_redraw(
            kScale * x, beta, chain_seed(a.seed, a.s.stream_key, chain),
            (uint32_t)inst, sweep, cl, (uint32_t)(4 * q + k));
      __syncwarp();
    } else {
      ask = ask || in;
    }
    const uint32_t flips = __ballot_sync(0xffffffffu, acc);
    if (lane == 0) *wp = w ^ flips;
    const float y = acc ? x : 0.0f;
    const float t1 = dE.x - y;
    const float bb = t1 - dE.x;
    dE.y += (dE.x - (t1 - bb)) - (y + bb);
    dE.x = t1;
    __syncwarp();  // the flips seen by every lane
    return w;
  };
  // position k of quad q, records in slab buffer b; returns the spin word
  // before it
  auto decide = [&](auto any_order_t, auto exact_t, int q, int b, int k,
                    float tlk, float thk) {
    if constexpr (D > 0) {
      const uint32_t* rec = slab + b * Q::QUAD + k * Q::STRIDE;
      float sum = 0.0f, part = 0.0f;
#pragma unroll
      for (int e4 = 0; e4 < D / 4; ++e4) {
        const uint4 c4 = reinterpret_cast<const uint4*>(rec)[e4];
        const float4 v4 = reinterpret_cast<const float4*>(rec + D)[e4];
        const uint32_t cs[4] = {c4.x, c4.y, c4.z, c4.w};
        const float vs[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if constexpr (decltype(any_order_t)::value) {
            sum += signed_value(cs[e], vs[e]);
          } else {
            part += signed_value(cs[e] & 0x7fffffffu, vs[e]);
            const bool last = (int32_t)cs[e] < 0;  // end of its group
            sum = last ? sum + part : sum;
            part = last ? 0.0f : part;
          }
        }
      }
      const uint2 ho = *reinterpret_cast<const uint2*>(rec + 2 * D);
      return attempt(exact_t, q, k, tlk, thk, ho.y,
                     sum + __uint_as_float(ho.x));
    } else {
      // 32 entries at a time, the next ones on their way; a lane each holds
      // the end of a group, where the partial sum joins the total (an empty
      // group adds nothing)
      const int beg = __shfl_sync(0xffffffffu, cb, 8 * k);
      const int end = __shfl_sync(0xffffffffu, ce, k);
      const int start = __shfl_sync(0xffffffffu, cb, 8 * k + (lane & 7));
      const int bound = lane == 8 ? end : start;  // in lanes 1 .. 8
      uint32_t c = k < 2 ? (k ? cc[1] : cc[0]) : (k == 2 ? cc[2] : cc[3]);
      float v = k < 2 ? (k ? cv[1] : cv[0]) : (k == 2 ? cv[2] : cv[3]);
      float sum = 0.0f, part = 0.0f;
      for (int e0 = beg; e0 < end; e0 += 32) {
        uint32_t cn = 0u;
        float vn = 0.0f;
        if (e0 + 32 < end) chunk(e0 + 32, end, cn, vn);
        const int bit = bound - 1 - e0;
        const uint32_t last = __reduce_or_sync(
            0xffffffffu,
            lane >= 1 && lane <= 8 && bit >= 0 && bit < 32 ? 1u << bit : 0u);
        const int m = end - e0 < 32 ? end - e0 : 32;
        // through shared memory: two broadcast loads for four entries
        uint32_t* s = slab + ((e0 - beg) & 32 ? Q::QUAD : 0);
        s[lane] = c | (((last >> lane) & 1u) << 31);
        s[32 + lane] = __float_as_uint(v);
        __syncwarp();
#pragma unroll 2
        for (int j = 0; j < m; j += 4) {
          const uint4 c4 = *reinterpret_cast<const uint4*>(s + j);
          const float4 v4 = *reinterpret_cast<const float4*>(s + 32 + j);
          const uint32_t cs[4] = {c4.x, c4.y, c4.z, c4.w};
          const float vs[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            part += signed_value(cs[i] & 0x7fffffffu, vs[i]);
            const bool end_of_group = (int32_t)cs[i] < 0;
            sum = end_of_group ? sum + part : sum;
            part = end_of_group ? 0.0f : part;
          }
        }
        c = cn;
        v = vn;
      }
      __syncwarp();
      return attempt(exact_t, q, k, tlk, thk,
                     4u * (uint32_t)spin_at(4 * q + k),
                     sum + __shfl_sync(0xffffffffu, ch, k));
    }
  };
  auto pick = [&](const float (&v)[4], int k) {
    return k < 2 ? (k ? v[1] : v[0]) : (k == 2 ? v[2] : v[3]);
  };

  // Two groups of warps take the levels in turn: while one decides a level,
  // the other fetches and draws for the next.  This warp's units: places
  // first(l) + its number in the group, + the group's size, ... of every
  // other level.
  // (Grouped rows may have a lone warp: it takes every level.)
  const int G = D == 0 && W == 1 ? 1 : 2, WG = W / G, wi = warp % WG;
  const int qshift = cut ? 4 : 0;
  const uint16_t* first = sched + nu;
  auto sweep_all = [&](auto any_order_t) {
    int l = warp / WG - G, place = 0, end = 0;
    // on to this warp's next unit
    auto settle = [&]() {
      place += WG;
      while (place >= end) {
        l += G;
        if (l >= nl) return;
        place = (int)first[l] + wi;
        end = (int)first[l + 1];
      }
    };
    settle();
    int unit = 0, b = 0;
    if (l < nl) {
      unit = sched[place];
      fetch(unit >> qshift);
      thresholds(unit >> qshift);
      put(unit >> qshift, 0);
    }
    int done = 0;  // barriers passed: one before every level but the first
    while (l < nl) {
      const int lv = l, u = unit, q = u >> qshift;
      settle();
      if (l < nl) {
        unit = sched[place];
        fetch(unit >> qshift);
      }
      for (; done < lv; ++done) __syncthreads();
      int k0 = cut ? (u >> 2) & 3 : 0;
      const int left = n - 4 * q;
      const int k1 = cut ? k0 + (u & 3) + 1 : left < 4 ? left : 4;
      if (k1 - k0 == 4) {
        // the fast rule for all four; where a lane's decision needed the
        // exact one, the quad is undone and decided again below
        const float2 dE0 = dE;
        uint32_t w0[4];
        ask = false;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          w0[k] = decide(any_order_t, std::false_type{}, q, b, k, tl[k],
                         th[k]);
        if (!__any_sync(0xffffffffu, ask)) {
          k0 = k1;
        } else {
          if (lane == 0) {
#pragma unroll
            for (int k = 3; k >= 0; --k) spin_s[spin_at(4 * q + k)] = w0[k];
          }
          __syncwarp();
          dE = dE0;
        }
      }
#pragma unroll 1
      for (int k = k0; k < k1; ++k)
        decide(any_order_t, std::true_type{}, q, b, k, pick(tl, k),
               pick(th, k));
      if (l != lv && lv + 1 < nl) {  // this warp is through with the level
        ++done;
        __syncthreads();
      }
      b ^= 1;
      if (l < nl) {
        thresholds(unit >> qshift);
        put(unit >> qshift, b);
      }
    }
    for (; done < nl; ++done) __syncthreads();
  };
  if constexpr (D > 0) {
    if (any_order)
      sweep_all(std::true_type{});
    else
      sweep_all(std::false_type{});
  } else {
    sweep_all(std::false_type{});
  }

  // energies and the per-chain best (strict <, pysa/simulation.py:150-171)
  de_s[warp * 32 + lane] = dE;
  __syncthreads();
  if (warp == 0) {
    bool improved = false;
    if (valid) {
      double d = 0.0;
      for (int w = 0; w < W; ++w) {
        const float2 v = de_s[w * 32 + lane];
        d += fabsf(v.x) < INFINITY ? (double)v.x + (double)v.y : (double)v.x;
      }
      const float e_new =
          (float)((double)a.s.energies[chain] + (double)kScale * d);
      a.s.energies[chain] = e_new;
      if (e_new < a.s.best_energy[chain]) {
        improved = true;
        a.s.best_energy[chain] = e_new;
        a.s.best_sweep[chain] = (int32_t)sweep;
      }
    }
    imp_s[lane] = improved ? 1 : 0;
  }
  __syncthreads();
  const bool keep_best = imp_s[lane] != 0;
#pragma unroll 4
  for (int w = warp; w < words; w += W) {
    const uint32_t v = warp_transpose(spin_s[w * 32 + lane], lane);
    const int64_t off = chain * (int64_t)a.p.words + w;
    if (valid) {
      a.s.spins[off] = v;
      if (keep_best) a.s.best_spins[off] = v;
    }
  }
}

template <bool RANDOM, bool ISING, int D>
static cudaError_t launch_csr_t(const CsrArgs& a, int W, cudaStream_t st) {
  const int n = a.p.max_n;
  auto bytes = [&](int w) {
    return (size_t)((n + 31) / 32) * 128 +
           (size_t)w * (2 * QuadSlab<D>::QUAD * 4 + 256) +
           2 * (size_t)sched_cap(n) + (RANDOM ? 2 * (size_t)n : 0);
  };
  while (W > 2 && bytes(W) > kCsrSmem) W /= 2;
  const size_t smem = bytes(W);
  static std::atomic<uint64_t> allowed;
  cudaError_t e = allow_smem((const void*)k_sweep_csr<RANDOM, ISING, D>,
                             kCsrSmem, allowed);
  if (e != cudaSuccess) return e;
  k_sweep_csr<RANDOM, ISING, D><<<a.num_items, 32 * W, smem, st>>>(a);
  return cudaGetLastError();
}

template <bool RANDOM, bool ISING>
static cudaError_t launch_csr_w(const CsrArgs& a, int W, cudaStream_t st) {
  switch (a.width) {
    case 4: return launch_csr_t<RANDOM, ISING, 4>(a, W, st);
    case 8: return launch_csr_t<RANDOM, ISING, 8>(a, W, st);
    case 16: return launch_csr_t<RANDOM, ISING, 16>(a, W, st);
    case 32: return launch_csr_t<RANDOM, ISING, 32>(a, W, st);
    default: return launch_csr_t<RANDOM, ISING, 0>(a, W, st);
  }
}

cudaError_t launch_csr_schedule(const CsrArgs& a, bool random,
                                cudaStream_t st) {
  if (a.num_items <= 0 || !a.perm || a.p.max_n < sched_min_n(random))
    return cudaSuccess;
  // the larger of all quads and, up to kSchedCutN, as many units as spins
  const int n = a.p.max_n, nc = n < kSchedCutN ? n : kSchedCutN;
  const size_t whole = sched_bytes(csr_quads(n), n, random, false);
  const size_t parts = sched_bytes(nc, nc, random, true);
  // (no more than needed: the L1 cache keeps the rest)
  const size_t smem =
      (sched_by_rounds(random, a.width) ? 0 : 2 * (size_t)kSchedNames) +
      (whole > parts ? whole : parts) + 16;
  const void* f = random ? (const void*)k_csr_schedule<true>
                         : (const void*)k_csr_schedule<false>;
  static std::atomic<uint64_t> allowed[2];
  cudaError_t e = allow_smem(f, kCsrSmem, allowed[random]);
  if (e != cudaSuccess) return e;
  if (random)
    k_csr_schedule<true><<<a.p.num_instances, kSchedThreads, smem, st>>>(a);
  else
    k_csr_schedule<false><<<a.p.num_instances, kSchedThreads, smem, st>>>(a);
  return cudaGetLastError();
}

// Warps of a CTA.  A level holds a few to a few dozen units, more of them the
// wider the instance, so while every SM has at most one CTA it gets the most
// that have work.  Beyond that CTAs share an SM's 32 warps (64 registers a
// thread): narrow schedules, whose levels hold a unit or two, in CTAs of few
// warps, so that all are resident; wide ones in larger CTAs.  Which one an
// instance has, the device knows: both are launched, and a CTA of the other
// kind leaves at once.  Measured, us a sweep at 2 / 4 / 8 / 16 / 32 warps: ring
// of 1000, 100 000 chains 482 / 564 / 912 / 1605 / 3020 (one thread per chain 622),
// 20 000 chains 205 / 197 / 333 / 469 / 755 (393); 64 x 64 lattice, 100 000 chains
// 3457 / 2027 / 1852 / 1885 / 2019 (3385), 20 000 1077 / 616 / 575 / 482 / 488
// (1558), 4000 1007 / 507 / 261 / 155 / 119.
cudaError_t launch_csr(CsrArgs a, bool random, cudaStream_t st) {
  if (a.num_items <= 0) return cudaSuccess;
  const bool ising = a.p.problem_type == PYSA_GB_ISING;
  auto launch = [&](int W) {
    if (random)
      return ising ? launch_csr_w<true, true>(a, W, st)
                   : launch_csr_w<true, false>(a, W, st);
    return ising ? launch_csr_w<false, true>(a, W, st)
                 : launch_csr_w<false, false>(a, W, st);
  };
  const int n = a.p.max_n;
  const int most = n <= 512 ? 8 : n <= 2048 ? 16 : kCsrWarps;
  if (a.num_items <= a.sms) return launch(most);
  auto fit = [&](int warps, int least) {  // a power of two
    int w = most;
    while (w > least && w > warps) w /= 2;
    return w;
  };
  const int share = (a.num_items + a.sms - 1) / a.sms;  // CTAs an SM gets
  const int few = fit(32 / share, a.width == 0 ? 1 : 2);
  if (n <= 512) return launch(a.width == 0 ? few : 4);
  a.pick = 1;
  cudaError_t e = launch(few);
  if (e != cudaSuccess) return e;
  a.pick = 2;
  return launch(fit(160 / (a.num_items / a.sms), 4));
}

}  // namespace pysa_gb
