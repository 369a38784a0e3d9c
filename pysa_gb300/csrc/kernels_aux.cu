// kernels_aux.cu -- the kernels around the sweep: coupling packing, field and
// energy preparation, replica exchange + log-omega, visiting orders, f64
// energies and spin unpacking.
#include <cooperative_groups.h>

#include "aux.cuh"
#include "sweep_plain.cuh"

namespace pysa_gb {

// ------------------------------------------------------------ J packing
// packed[i][l * LS + m] = J[i][32 m + l] (0 outside the instance); blockIdx.y
// instances at even steps.
__global__ void k_pack_rows(const float* J, int ld, int n, int nc, int ls,
                            float* packed, int64_t j_step, int64_t p_step) {
  J += blockIdx.y * j_step;
  packed += blockIdx.y * p_step;
  const int row_len = 32 * ls;
  const int64_t total = (int64_t)n * row_len;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / row_len), r = (int)(e % row_len);
    const int l = r / ls, m = r % ls;
    const int col = 32 * m + l;
    packed[e] = (m < nc && col < n) ? J[(int64_t)i * ld + col] : 0.0f;
  }
}

void launch_pack_rows(const float* J, int ld, int n, int nc, int ls,
                      float* packed, int count, int64_t j_step,
                      int64_t p_step, cudaStream_t st) {
  const int64_t total = (int64_t)n * 32 * ls;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 4096) blocks = 4096;
  k_pack_rows<<<dim3(blocks, count), 256, 0, st>>>(J, ld, n, nc, ls, packed,
                                                   j_step, p_step);
}

// -------------------------------------------------- fields and energies
// F_i = sum_j J_ij s_j from f32 partial sums over 32 rows (the products
// J_ij s_j are exact in f32), the partial sums accumulated as an exact f32
// pair; H_i = F_i + h_i rounded once to f32; E = sum_i s_i (F_i / 2 + h_i)
// (pysa/ising.py:37, pysa/qubo.py:37) in the same pairs, reduced over lanes,
// column groups and cluster ranks in a fixed order, so the result does not
// depend on timing.
constexpr int kFieldWarps = 8;

// Instance of chain c: binary search over chain_off.
__device__ __forceinline__ int chain_instance(const pysa_gb_problems& p,
                                              int64_t c) {
  int lo = 0, hi = p.num_instances - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (p.chain_off[mid] <= c) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// s + e = a + b exactly (Knuth's two-sum).
__device__ __forceinline__ float two_sum(float a, float b, float& e) {
  const float s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
  return s;
}

// Three f32 a value: the sum to 2^-72 of its largest term.
struct Triple {
  float a, b, c;
  __device__ __forceinline__ void add(float x) {
    float e, f;
    a = two_sum(a, x, e);
    b = two_sum(b, e, f);
    c += f;
  }
  __device__ __forceinline__ float rounded() const {
    float e;
    const float s = two_sum(a, b, e);
    return s + (e + c);
  }
};

// Sparse instances: the terms J_ij s_j of row i's stored entries in order (the
// products are exact; padding entries have value 0), each given to `add`, from
// the fixed records (width > 0: entries csr_ent_off + width i ...) or the
// grouped rows (csr_rows, 9 offsets per row).
template <typename Add>
__device__ __forceinline__ void csr_row_terms(const pysa_gb_problems& p,
                                              int inst, int i,
                                              const uint32_t* sw, bool ising,
                                              Add add) {
  const int64_t eo = p.csr_ent_off[inst];
  int64_t beg, end;
  if (p.csr_width > 0) {
    beg = eo + (int64_t)p.csr_width * i;
    end = beg + p.csr_width;
  } else {
    const int32_t* r = p.csr_rows + 9 * (p.csr_row_off[inst] + i);
    beg = eo + r[0];
    end = eo + r[8];
  }
  for (int64_t e = beg; e < end; ++e) {
    const int j = p.csr_col[e] & 0x7fffffff;
    const float sj = ((sw[j >> 5] >> (j & 31)) & 1u) ? 1.0f
                                                     : (ising ? -1.0f : 0.0f);
    add(p.csr_val[e] * sj);
  }
}
__device__ __forceinline__ double csr_row_dot(const pysa_gb_problems& p,
                                              int inst, int i,
                                              const uint32_t* sw,
                                              bool ising) {
  double f = 0.0;
  csr_row_terms(p, inst, i, sw, ising, [&](float x) { f += (double)x; });
  return f;
}

__device__ __forceinline__ bool is_sparse_inst(const pysa_gb_problems& p,
                                               int inst) {
  return p.csr_row_off && p.csr_row_off[inst] >= 0;
}

// CTA per chain, thread per row.  Sums in triples of f32 (f64 instructions run
// at 1/64 of the rate; they took most of 417 us for 4000 chains of 4096 spins
// with 4 couplings each, 146 so); a field or energy that leaves the f32
// range is added in f64.
__global__ void __launch_bounds__(32 * kFieldWarps)
    k_fields_csr(const PrepArgs a) {
  __shared__ Triple e_s[kFieldWarps];
  __shared__ double d_s[kFieldWarps];
  const int64_t c = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarps = blockDim.x >> 5;
  const int inst = chain_instance(a.p, c);
  if (!is_sparse_inst(a.p, inst)) return;  // uniform per CTA
  const int n = a.p.n[inst];
  const bool ising = a.p.problem_type == PYSA_GB_ISING;
  const float* h = a.p.h + a.p.h_off[inst];
  const uint32_t* sw = a.s.spins + c * a.p.words;
  auto spin = [&](int i) {
    return ((sw[i >> 5] >> (i & 31)) & 1u) ? 1.0f : (ising ? -1.0f : 0.0f);
  };
  Triple e = {0.0f, 0.0f, 0.0f};  // sum_i s_i (f_i + 2 h_i)
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    Triple f = {0.0f, 0.0f, 0.0f};
    csr_row_terms(a.p, inst, i, sw, ising, [&](float x) { f.add(x); });
    const float hi = h[i], si = spin(i);
    e.add(si * f.a);
    e.add(si * f.b);
    e.add(si * f.c);
    e.add(si * (2.0f * hi));
    f.add(hi);
    float H = f.rounded();
    if (!(fabsf(H) < INFINITY))
      H = (float)(csr_row_dot(a.p, inst, i, sw, ising) + (double)hi);
    a.fields[c * a.field_ld + i] = H;
  }
  if (!a.set_energies) return;
  const bool bad = __syncthreads_or(!(fabsf(e.a) < INFINITY));
  if (!bad) {
    for (int o = 16; o; o >>= 1) {
      const Triple u = {__shfl_xor_sync(0xffffffffu, e.a, o),
                        __shfl_xor_sync(0xffffffffu, e.b, o),
                        __shfl_xor_sync(0xffffffffu, e.c, o)};
      e.add(u.a);
      e.add(u.b);
      e.add(u.c);
    }
    if (lane == 0) e_s[warp] = e;
  } else {
    double d = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      d += (double)spin(i) * (0.5 * csr_row_dot(a.p, inst, i, sw, ising) +
                              (double)h[i]);
    d = warp_sum(d);
    if (lane == 0) d_s[warp] = d;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    if (bad) {
      for (int w = 0; w < nwarps; ++w) t += d_s[w];
    } else {
      Triple s = e_s[0];
      for (int w = 1; w < nwarps; ++w) {
        s.add(e_s[w].a);
        s.add(e_s[w].b);
        s.add(e_s[w].c);
      }
      t = 0.5 * ((double)s.a + ((double)s.b + (double)s.c));
      if (!(fabsf(s.a) < INFINITY)) {  // the warps' sum left the range
        t = 0.0;
        for (int i = 0; i < n; ++i)
          t += (double)spin(i) * (0.5 * csr_row_dot(a.p, inst, i, sw, ising) +
                                  (double)h[i]);
      }
    }
    a.s.energies[c] = (float)t;
  }
}

// ---- dense instances
// A CTA of 8 warps holds CH chains x W columns in registers (a warp: 8 chains
// x 32 TC columns) and walks the n rows 32 at a time: the J tile (cp.async,
// double-buffered) is read once per CH chains instead of once per chain, and
// the chains' spins become +-1 / 0 multipliers in shared memory, so a row is
// one shared load and two broadcasts per 8 TC multiply-adds, done two at a
// time (f32x2 over pairs of chains: half the issue slots, which were two
// thirds taken).  Bound by the shared loads (three 16-byte ones per 16 paired
// multiply-adds) and the multiply-adds themselves; a warp of f64
// instructions takes about 64 times the cycles of an f32 one on this GPU, so
// f64 is kept out of the loop by adding each 32-row partial sum into an f32
// pair with an exact two-sum.  The pair holds the sum of the partial sums to
// 2^-48 of its largest term, and exactly when the sum's bits span fewer than
// 48 places: fields and energies equal those of the f64 accumulation bit for
// bit on every size measured (normal couplings, and ones spread over nine
// decades).  A cluster of up to 8 CTAs splits the columns while there are too
// few chains to fill the GPU; its energies meet in rank 0 through distributed
// shared memory.
// Measured: n = 2048, 8192 chains 2.6 -> 1.87 ms; n = 1024, 16384 chains
// 1.3 -> 0.96; n = 512, 65536 chains 1.19 -> 0.95 (single multiply-adds before;
// one CTA per chain with f64 accumulation took 14.2 ms at n = 2048, 9728
// chains, this tile 2.7 with single multiply-adds).

// Pair (hi, lo) + x.
__device__ __forceinline__ void pair_add(float2& p, float x) {
  float e;
  p.x = two_sum(p.x, x, e);
  p.y += e;
}

// The same for two pairs at once: hi, lo and x hold two f32 each.  The
// differences are multiply-adds by -1 (the product is exact).
__device__ __forceinline__ uint64_t two_sum2(uint64_t a, uint64_t b,
                                             uint64_t& e) {
  const uint64_t m1 = pack2(-1.0f, -1.0f);
  const uint64_t s = add2(a, b);
  const uint64_t bb = fma2(a, m1, s);
  const uint64_t ea = fma2(fma2(bb, m1, s), m1, a);
  e = add2(ea, fma2(bb, m1, b));
  return s;
}
__device__ __forceinline__ void pair_add2(uint64_t& hi, uint64_t& lo,
                                          uint64_t x) {
  uint64_t e;
  hi = two_sum2(hi, x, e);
  lo = add2(lo, e);
}
// Three f32 a value: the sum to 2^-72 of its largest term.
struct Triple2 {
  uint64_t a, b, c;
  __device__ __forceinline__ void add(uint64_t x) {
    uint64_t e, f;
    a = two_sum2(a, x, e);
    b = two_sum2(b, e, f);
    c = add2(c, f);
  }
  __device__ __forceinline__ void add(const Triple2& t) {
    add(t.a);
    add(t.b);
    add(t.c);
  }
};
__device__ __forceinline__ void lane_sum(Triple2& t) {
  for (int o = 16; o; o >>= 1) {
    const Triple2 u = {__shfl_xor_sync(0xffffffffu, t.a, o),
                       __shfl_xor_sync(0xffffffffu, t.b, o),
                       __shfl_xor_sync(0xffffffffu, t.c, o)};
    t.add(u);
  }
}

// Field of one column in f64, for the columns whose f32 pair left the finite
// range (infinite or NaN couplings, or sums past f32).
static __device__ __noinline__ double field_f64(const float* J, int ld, int n,
                                                const uint32_t* sw, bool ising,
                                                int col) {
  double F = 0.0;
  float part = 0.0f;
  for (int j = 0; j < n; ++j) {
    const uint32_t bit = (sw[j >> 5] >> (j & 31)) & 1u;
    if (bit)
      part += J[(int64_t)j * ld + col];
    else if (ising)
      part -= J[(int64_t)j * ld + col];
    if ((j & 31) == 31 || j == n - 1) {
      F += (double)part;
      part = 0.0f;
    }
  }
  return F;
}

__device__ __forceinline__ void cp_async_zfill16(void* dst, const void* src,
                                                 int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_zfill4(void* dst, const void* src,
                                                int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}

template <int TC, int CG>
struct FieldTile {
  static constexpr int CH = 8 * (kFieldWarps / CG);  // chains per CTA
  static constexpr int W = 32 * TC * CG;             // columns per pass
  static constexpr size_t J_BYTES = (size_t)32 * W * 4;
  static constexpr size_t M_BYTES = (size_t)32 * CH * 4;
  static constexpr size_t E_BYTES = (size_t)CG * CH * 8;
  static constexpr size_t P_BYTES = (size_t)8 * 32 * kFieldWarps * 8;
  static constexpr size_t BYTES = 2 * (J_BYTES + M_BYTES) + E_BYTES + P_BYTES;
};

template <int TC, int CG>
__global__ void __launch_bounds__(32 * kFieldWarps, 2)
    k_fields(const PrepArgs a) {
  using T = FieldTile<TC, CG>;
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char fsm[];
  float* jt = reinterpret_cast<float*>(fsm);                   // [2][32][W]
  float* mt = reinterpret_cast<float*>(fsm + 2 * T::J_BYTES);  // [2][32][CH]
  float2* es =                                                 // [CG][CH]
      reinterpret_cast<float2*>(fsm + 2 * (T::J_BYTES + T::M_BYTES));
  // this thread's energy pairs of its warp's 8 chains, a row of 256 apart
  // (16 registers that the loop over the rows needs)
  float2* eps = es + T::E_BYTES / 8 + threadIdx.x;
  cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wc = warp % CG, wg = warp / CG;
  const int64_t tile0 = (int64_t)(blockIdx.x / csize) * T::CH;
  const int64_t tile1 = tile0 + T::CH < a.p.num_chains ? tile0 + T::CH
                                                       : a.p.num_chains;
  const bool ising = a.p.problem_type == PYSA_GB_ISING;
  const bool vec_out = TC == 4 && a.field_ld % 4 == 0 &&
                       reinterpret_cast<uintptr_t>(a.fields) % 16 == 0;
  // the tile's chains, one instance at a time
  for (int64_t c0 = tile0; c0 < tile1;) {
    const int inst = chain_instance(a.p, c0);
    int64_t c1 = inst + 1 < a.p.num_instances ? a.p.chain_off[inst + 1]
                                              : (int64_t)a.p.num_chains;
    c1 = c1 < tile1 ? (c1 > c0 ? c1 : c0 + 1) : tile1;
    if (is_sparse_inst(a.p, inst)) {  // k_fields_csr's
      c0 = c1;
      continue;
    }
    const int n = a.p.n[inst], ld = a.p.ld[inst];
    const float* J = a.p.J + a.p.j_off[inst];
    const float* h = a.p.h + a.p.h_off[inst];
    const bool vec_in =
        ld % 4 == 0 && reinterpret_cast<uintptr_t>(J) % 16 == 0;
    const int nt = (n + 31) >> 5;
    const int64_t cw = c0 + 8 * wg;  // this warp's first chain
    for (int g = 0; g < 8; ++g)
      eps[g * 32 * kFieldWarps] = make_float2(0.0f, 0.0f);

    for (int base = rank * T::W; base < n; base += csize * T::W) {
      auto stage = [&](int t, int buf) {  // rows 32 t ... of J
        float* dst = jt + buf * (32 * T::W);
        if (vec_in) {
          for (int e = tid; e < 32 * T::W / 4; e += blockDim.x) {
            const int r = e / (T::W / 4), q = 4 * (e % (T::W / 4));
            const int row = 32 * t + r, col = base + q;
            const int left = row < n ? n - col : 0;
            const int bytes = left >= 4 ? 16 : left > 0 ? 4 * left : 0;
            cp_async_zfill16(dst + r * T::W + q,
                             bytes ? J + (int64_t)row * ld + col : J, bytes);
          }
        } else {
          for (int e = tid; e < 32 * T::W; e += blockDim.x) {
            const int r = e / T::W, q = e % T::W;
            const int row = 32 * t + r, col = base + q;
            const bool in = row < n && col < n;
            cp_async_zfill4(dst + r * T::W + q,
                            in ? J + (int64_t)row * ld + col : J, in ? 4 : 0);
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      // word t of this thread's chain; its multipliers, [row][chain]
      constexpr int RPT = T::CH / 8;  // rows per thread: 32 CH / 256
      const int mc = tid % T::CH, mr = (tid / T::CH) * RPT;
      auto word = [&](int t) {
        return c0 + mc < c1 ? a.s.spins[(c0 + mc) * a.p.words + t] : 0u;
      };
      auto put_mult = [&](uint32_t w, int buf) {
#pragma unroll
        for (int r = 0; r < RPT; ++r)
          mt[buf * (32 * T::CH) + (mr + r) * T::CH + mc] =
              ((w >> (mr + r)) & 1u) ? 1.0f : (ising ? -1.0f : 0.0f);
      };
      stage(0, 0);
      put_mult(word(0), 0);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();

      uint64_t Fh[4][TC], Fl[4][TC];  // chains 2 q, 2 q + 1
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int k = 0; k < TC; ++k) Fh[q][k] = Fl[q][k] = 0ull;
      for (int t = 0; t < nt; ++t) {
        const int buf = t & 1;
        uint32_t wn = 0u;
        if (t + 1 < nt) {
          stage(t + 1, buf ^ 1);
          wn = word(t + 1);
        }
        uint64_t part[4][TC];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int k = 0; k < TC; ++k) part[q][k] = 0ull;
        const float* jr = jt + buf * (32 * T::W) + (wc * 32 + lane) * TC;
        const float* mr8 = mt + buf * (32 * T::CH) + 8 * wg;
        // rows past n are zero in the tile: they add +-0
#pragma unroll 4
        for (int r = 0; r < 32; ++r) {
          float v[TC];
          if constexpr (TC == 4) {
            const float4 x = *reinterpret_cast<const float4*>(jr + r * T::W);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
          } else {
#pragma unroll
            for (int k = 0; k < TC; ++k) v[k] = jr[r * T::W + k];
          }
          const ulonglong2 m0 =
              *reinterpret_cast<const ulonglong2*>(mr8 + r * T::CH);
          const ulonglong2 m1 =
              *reinterpret_cast<const ulonglong2*>(mr8 + r * T::CH + 4);
          const uint64_t m[4] = {m0.x, m0.y, m1.x, m1.y};
#pragma unroll
          for (int k = 0; k < TC; ++k) {
            const uint64_t vv = pack2(v[k], v[k]);
#pragma unroll
            for (int q = 0; q < 4; ++q) part[q][k] = fma2(m[q], vv, part[q][k]);
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int k = 0; k < TC; ++k)
            pair_add2(Fh[q][k], Fl[q][k], part[q][k]);
        if (t + 1 < nt) {
          put_mult(wn, buf ^ 1);
          asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
      }

      // fields out, energy terms s (F / 2 + h)
      const int col0 = base + (wc * 32 + lane) * TC;
      float hc[TC];
#pragma unroll
      for (int k = 0; k < TC; ++k) hc[k] = col0 + k < n ? h[col0 + k] : 0.0f;
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        const int64_t c = cw + g;
        if (c >= c1 || col0 >= n) continue;
        const uint32_t* sw = a.s.spins + c * a.p.words;
        const uint32_t wv = sw[col0 >> 5];  // TC divides 32: one word
        float H[TC];
        float2 ep = eps[g * 32 * kFieldWarps];
#pragma unroll
        for (int k = 0; k < TC; ++k) {
          const float hi = half2(Fh[g >> 1][k], g & 1);
          const float lo = half2(Fl[g >> 1][k], g & 1);
          float e1, e2, e3;
          const float s1 = two_sum(hi, hc[k], e1);
          const float t1 = two_sum(e1, lo, e2);
          const float r1 = two_sum(s1, t1, e3);
          H[k] = r1 + (e3 + e2);
          const float half = 0.5f * hi;
          const bool up = (wv >> ((col0 + k) & 31)) & 1u;
          const float sg = up ? 1.0f : (ising ? -1.0f : 0.0f);
          if (fabsf(hi) < INFINITY && fabsf(s1) < INFINITY) {
            const float s2 = two_sum(half, hc[k], e1);
            pair_add(ep, sg * s2);
            ep.y += sg * (e1 + 0.5f * lo);
          } else if (col0 + k < n) {
            H[k] = (float)(field_f64(J, ld, n, sw, ising, col0 + k) +
                           (double)hc[k]);
            ep.x = __int_as_float(0x7fc00000);  // energy in f64 below
          }
        }
        eps[g * 32 * kFieldWarps] = ep;
        float* out = a.fields + c * a.field_ld + col0;
        if (vec_out && col0 + TC <= n) {
          if constexpr (TC == 4)
            *reinterpret_cast<float4*>(out) =
                make_float4(H[0], H[1], H[2], H[3]);
        } else {
#pragma unroll
          for (int k = 0; k < TC; ++k)
            if (col0 + k < n) out[k] = H[k];
        }
      }
    }  // column passes

    if (a.set_energies) {
      // lane sums of the pairs: three halving steps leave chain 4 b4 + 2 b3
      // + b2 (bits of the lane) in every lane, two more finish the sum
      float2 ep[8];
#pragma unroll
      for (int g = 0; g < 8; ++g) ep[g] = eps[g * 32 * kFieldWarps];
#pragma unroll
      for (int o = 4; o; o >>= 1) {
        const bool up = lane & (4 * o);
#pragma unroll
        for (int g = 0; g < o; ++g) {
          const float2 mine = up ? ep[g + o] : ep[g];
          const float2 give = up ? ep[g] : ep[g + o];
          ep[g] = mine;
          const float gx = __shfl_xor_sync(0xffffffffu, give.x, 4 * o);
          const float gy = __shfl_xor_sync(0xffffffffu, give.y, 4 * o);
          pair_add(ep[g], gx);
          ep[g].y += gy;
        }
      }
#pragma unroll
      for (int o = 2; o; o >>= 1) {
        const float gx = __shfl_xor_sync(0xffffffffu, ep[0].x, o);
        const float gy = __shfl_xor_sync(0xffffffffu, ep[0].y, o);
        pair_add(ep[0], gx);
        ep[0].y += gy;
      }
      if ((lane & 3) == 0) es[wc * T::CH + 8 * wg + (lane >> 2)] = ep[0];
      if (csize > 1) cl.sync(); else __syncthreads();
      if (rank == 0 && tid < T::CH && c0 + tid < c1) {
        double t = 0.0;
        bool fin = true;
        for (int r = 0; r < csize; ++r) {
          const float2* er = csize > 1 ? cl.map_shared_rank(es, r) : es;
          for (int w = 0; w < CG; ++w) {
            const float2 v = er[w * T::CH + tid];
            fin = fin && fabsf(v.x) < INFINITY;
            t += (double)v.x + (double)v.y;
          }
        }
        if (!fin) {
          const uint32_t* sw = a.s.spins + (c0 + tid) * a.p.words;
          t = 0.0;
          for (int col = 0; col < n; ++col) {
            const double si = ((sw[col >> 5] >> (col & 31)) & 1u)
                                  ? 1.0 : (ising ? -1.0 : 0.0);
            t += si * (0.5 * field_f64(J, ld, n, sw, ising, col) +
                       (double)h[col]);
          }
        }
        a.s.energies[c0 + tid] = (float)t;
      }
      if (csize > 1) cl.sync(); else __syncthreads();
    }
    c0 = c1;
  }
}

template <int TC, int CG>
static cudaError_t launch_fields_t(const PrepArgs& a, int csize,
                                   cudaStream_t st) {
  using T = FieldTile<TC, CG>;
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr[dev]) {
    cudaError_t e = cudaFuncSetAttribute(
        k_fields<TC, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
        (int)T::BYTES);
    if (e != cudaSuccess) return e;
    attr[dev] = true;
  }
  const int64_t tiles = ((int64_t)a.p.num_chains + T::CH - 1) / T::CH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * csize));
  cfg.blockDim = dim3(32 * kFieldWarps);
  cfg.dynamicSmemBytes = T::BYTES;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)csize;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_fields<TC, CG>, a);
}

// The tile by size: 256 columns x 32 chains (4 columns a lane) when that
// still gives every SM work; up to 128 columns, 64 chains; up to 32 columns,
// one column a lane.  Few chains, or few per instance (a tile's chains are
// done one instance after another), take 8 chains x 256 columns, the columns
// split over a cluster.  The wider tiles also split their columns, by up to 4
// and evenly, while there are fewer than 8 waves of them: the last wave is
// then shorter (n = 2048, 256 tiles: 2.21 ms at 1, 2.16 at 2, 1.87 at 4, 2.00
// at 8; n = 1024, 512 tiles: 1.10, 0.96, 0.96; 13 waves of n = 64 .. 1536:
// 6.5, 7.0, 8.6).
static cudaError_t launch_fields(const PrepArgs& a, int sms,
                                 cudaStream_t st) {
  const int64_t chains = a.p.num_chains;
  const int64_t per = chains / (a.p.num_instances > 0 ? a.p.num_instances : 1);
  const int n = a.p.max_n;
  const int64_t fill = 2 * sms;  // CTAs that keep the GPU busy
  if (per >= 64 && n <= 32 && chains / 64 >= fill)
    return launch_fields_t<1, 1>(a, 1, st);
  if (per >= 64 && n <= 128 && chains / 64 >= fill)
    return launch_fields_t<4, 1>(a, 1, st);
  const int passes = (n + 255) / 256;
  if (per >= 32 && chains / 32 * passes >= fill) {
    const int64_t tiles = chains / 32;
    int cs = 1;
    while (cs < 8 && cs < passes &&
           (tiles * cs < fill ||
            (cs < 4 && tiles < 8 * fill && passes % (2 * cs) == 0)))
      cs *= 2;
    return launch_fields_t<4, 2>(a, cs, st);
  }
  int cs = 1;
  while (cs < 8 && cs < passes && (chains + 7) / 8 * cs < fill) cs *= 2;
  return launch_fields_t<1, 8>(a, cs, st);
}

// CTA per read, thread per replica: the slot betas and the initial best.
__global__ void k_read_init(const PrepArgs a) {
  const int64_t r = blockIdx.x;
  const int inst = a.p.read_inst[r];
  const int R = a.p.replicas[inst];
  const int64_t base = a.p.chain_off[inst] + (r - a.p.read_off[inst]) * R;
  const float* betas = a.p.ladder + a.p.ladder_off[inst];
  for (int k = threadIdx.x; k < R; k += blockDim.x) {
    a.s.chain_beta[base + a.s.beta_idx[base + k]] = betas[k];
    if (a.init_best) {
      const int64_t c = base + k;
      a.s.best_energy[c] = a.best_global ? __int_as_float(0x7f800000)
                                         : a.s.energies[c];
      a.s.best_sweep[c] = 0;
      for (int w = 0; w < a.p.words; ++w)
        a.s.best_spins[c * a.p.words + w] = a.s.spins[c * a.p.words + w];
    }
  }
}

cudaError_t launch_prepare(const PrepArgs& a, int sms, cudaStream_t st) {
  if (a.p.num_chains > 0 && a.p.num_instances > 0) {
    const cudaError_t e = launch_fields(a, sms, st);
    if (e != cudaSuccess) return e;
    if (a.p.csr_row_off) {
      int warps = (a.p.max_n + 255) / 256;
      warps = warps < 1 ? 1 : warps > kFieldWarps ? kFieldWarps : warps;
      k_fields_csr<<<(unsigned)a.p.num_chains, warps * 32, 0, st>>>(a);
    }
  }
  if (a.p.num_reads > 0)
    k_read_init<<<(unsigned)a.p.num_reads, 128, 0, st>>>(a);
  return cudaGetLastError();
}

// ------------------------------------------------------ replica exchange
// Warp per read.  pysa/utils.py:44-58: pairs (R-1,R-2), (R-2,R-3), ... in
// order; swap beta_idx when de >= 0 or u < exp(de), de in f32.  Then the
// per-replica betas of the next sweep and, if requested, get_log_omega
// (pysa/ais.py:79-112) in f64.  The last block to finish advances the sweep
// counter.
constexpr int kXWarps = 4;


__global__ void k_exchange(const XArgs a) {
  __shared__ float E_s[kXWarps][kMaxReplicas];
  __shared__ int32_t B_s[kXWarps][kMaxReplicas];
  __shared__ uint32_t X_s[kXWarps][kMaxReplicas];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t r = (int64_t)blockIdx.x * kXWarps + warp;
  const uint32_t sweep = (uint32_t)(*a.s.sweep_counter);
  const bool xch = a.use_pt && exchange_after(a.exchange_every, sweep);
  if (r < a.p.num_reads) {
    const int inst = a.p.read_inst[r];
    const int R = a.p.replicas[inst];
    const int64_t lread = r - a.p.read_off[inst];
    const int64_t base = a.p.chain_off[inst] + lread * R;
    const float* betas = a.p.ladder + a.p.ladder_off[inst];
    float* E = E_s[warp];
    int32_t* B = B_s[warp];
    uint32_t* X = X_s[warp];
    for (int k = lane; k < R; k += 32) {
      E[k] = a.s.energies[base + k];
      B[k] = a.s.beta_idx[base + k];
      if (xch && k < R - 1)
        X[k] = draw1(a.seed, TAG_PT, (uint32_t)inst, sweep, (uint32_t)lread,
                     (uint32_t)k);
    }
    __syncwarp();
    if (xch && R > 1 && lane == 0) {
      for (int k = 0; k < R - 1; ++k) {
        const int k1 = R - k - 1, k2 = R - k - 2;
        const int b1 = B[k1], b2 = B[k2];
        const float de = __fmul_rn(__fsub_rn(E[b1], E[b2]),
                                   __fsub_rn(betas[k1], betas[k2]));
        if (pt_accept(de, X[k])) {
          B[k1] = b2;
          B[k2] = b1;
        }
      }
    }
    __syncwarp();
    for (int k = lane; k < R; k += 32) {
      a.s.beta_idx[base + k] = B[k];
      a.s.chain_beta[base + B[k]] = betas[k];
    }
    if (a.log_omega_stride > 0 && lane == 0) {
      const int32_t* sorted = a.p.ladder_sorted + a.p.ladder_off[inst];
      double lw = 0.0;
      float beta_old = 0.0f;
      for (int q = 1; q < R; ++q) {
        const float b = betas[sorted[q]];
        const float e = E[B[sorted[q]]];
        const float t1 = __fmul_rn(-b, e), t2 = __fmul_rn(-beta_old, e);
        lw += (double)__fsub_rn(t1, t2);
        beta_old = b;
      }
      a.s.log_omega[r * a.log_omega_stride + sweep] = lw;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const uint32_t t = atomicAdd(a.s.ticket, 1u);
    if (t == gridDim.x - 1) {
      *a.s.ticket = 0u;
      __threadfence();
      *a.s.sweep_counter += 1;
    }
  }
}

void launch_exchange(const XArgs& a, cudaStream_t st) {
  const int64_t blocks = (a.p.num_reads + kXWarps - 1) / kXWarps;
  k_exchange<<<(unsigned)(blocks > 0 ? blocks : 1), kXWarps * 32, 0, st>>>(a);
}

// ---------------------------------------------------- visiting orders
// Fisher-Yates for (instance, sweep): for i from n - 1 down to 1 swap places i
// and j_i = floor(x_i (i + 1) / 2^32).  Block per instance.
//
// The swaps run in rounds instead of one after another: in a round every
// swap still to do claims its two places, the one that comes first in the
// sequence (the largest i) winning each, and the swaps holding both claims
// are done.  A swap waits exactly for the earlier ones that share a place
// with it, so the order is the sequential one; the rounds are about 3 log2 n
// (Shun, Gu, Blelloch, Fineman and Gibbons, "Sequential random permutation,
// list contraction and tree contraction are highly parallel", SODA 2015).
// Claims of a round outrank those of earlier ones, so none is cleared.
// Measured (one thread swapping before): n = 1024, 16 orders 38 -> 12 us; n =
// 4096 150 -> 20 us.
constexpr int kPermSmem = 232448;

__global__ void __launch_bounds__(1024) k_perm(const PermArgs a) {
  extern __shared__ uint32_t sh[];
  const int inst = blockIdx.x;
  const int n = a.p.n[inst];
  // grid row y: the sweep y after the current one (orders made ahead)
  const uint32_t sweep = (uint32_t)(*a.sweep_counter) + blockIdx.y;
  uint32_t* claim = sh;                                           // [max_n]
  uint16_t* p = reinterpret_cast<uint16_t*>(claim + a.p.max_n);   // [max_n]
  uint16_t* js = p + a.p.max_n;                                   // [max_n]
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const uint32_t x =
        draw1(a.seed, TAG_PERM, (uint32_t)inst, sweep, 0u, (uint32_t)i);
    p[i] = (uint16_t)i;
    js[i] = (uint16_t)(((uint64_t)x * (uint64_t)(i + 1)) >> 32);
    claim[i] = 0u;
  }
  __syncthreads();
  // bit k of todo: swap threadIdx.x + k blockDim.x is still to do
  uint32_t todo = 0u;
  for (int k = 0; k < 32; ++k) {
    const int i = (int)threadIdx.x + k * (int)blockDim.x;
    if (i > 0 && i < n) todo |= 1u << k;
  }
  for (uint32_t round = 1;; ++round) {
    for (uint32_t b = todo; b; b &= b - 1u) {
      const int i = (int)threadIdx.x + (__ffs(b) - 1) * (int)blockDim.x;
      const uint32_t c = (round << 16) | (uint32_t)i;
      atomicMax(claim + i, c);
      atomicMax(claim + js[i], c);
    }
    __syncthreads();
    for (uint32_t b = todo; b; b &= b - 1u) {
      const int k = __ffs(b) - 1;
      const int i = (int)threadIdx.x + k * (int)blockDim.x, j = js[i];
      const uint32_t c = (round << 16) | (uint32_t)i;
      if (claim[i] == c && claim[j] == c) {
        const uint16_t t = p[i];
        p[i] = p[j];
        p[j] = t;
        todo &= ~(1u << k);
      }
    }
    if (!__syncthreads_or(todo != 0u)) break;
  }
  int32_t* out = a.perm + ((int64_t)(sweep % (uint32_t)a.perm_slots) *
                               a.p.num_instances + inst) * (int64_t)a.p.max_n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = p[i];
}

// The same orders for instances too wide for k_perm's shared memory (up to
// 65536 spins), one swap after another: the draws are staged in the output
// row, the positions held as 16-bit values in shared memory.
__global__ void k_perm_wide(const PermArgs a) {
  extern __shared__ uint16_t pw[];
  const int inst = blockIdx.x;
  const int n = a.p.n[inst];
  const uint32_t sweep = (uint32_t)(*a.sweep_counter) + blockIdx.y;
  int32_t* out = a.perm + ((int64_t)(sweep % (uint32_t)a.perm_slots) *
                               a.p.num_instances + inst) * (int64_t)a.p.max_n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    pw[i] = (uint16_t)i;
    out[i] = (int32_t)draw1(a.seed, TAG_PERM, (uint32_t)inst, sweep, 0u,
                            (uint32_t)i);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = n - 1; i > 0; --i) {
      const uint32_t xi = (uint32_t)__ldcg(out + i);
      const int j = (int)(((uint64_t)xi * (uint64_t)(i + 1)) >> 32);
      const uint16_t t = pw[i];
      pw[i] = pw[j];
      pw[j] = t;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = (int32_t)pw[i];
}

void launch_perm(const PermArgs& a, cudaStream_t st, int count) {
  // claims, places and partners: 8 bytes per spin, up to n = 29 056 (and 32
  // swaps per thread)
  const size_t sm = 8 * (size_t)a.p.max_n;
  dim3 grid((unsigned)a.p.num_instances, (unsigned)(count > 0 ? count : 1));
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr[dev]) {
    cudaFuncSetAttribute(k_perm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kPermSmem);
    cudaFuncSetAttribute(k_perm_wide,
                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(uint16_t) * PYSA_GB_MAX_N));
    attr[dev] = true;
  }
  if (sm <= (size_t)kPermSmem) {
    k_perm<<<grid, a.p.max_n <= 2048 ? 512 : 1024, sm, st>>>(a);
    return;
  }
  const size_t smw = sizeof(uint16_t) * (size_t)a.p.max_n;  // <= 128 KB
  k_perm_wide<<<grid, 256, smw, st>>>(a);
}

// ----------------------------------------------------------- f64 energy
// CTA per state, warp per row i (rows warp, warp + 8, ...), lanes over the
// columns: f_i = sum_j J_ij s_j, E = sum_i s_i (f_i / 2 + h_i) in f64,
// reduced in a fixed order (lanes, then rows of a warp, then warps).
template <typename T>
__device__ __forceinline__ void energy64_body(
    int ptype, int n, int ld, const T* J, const T* h, const uint32_t* spins,
    int words, int64_t c, double* out) {
  __shared__ double e_s[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t* sw = spins + c * words;
  const bool ising = ptype == PYSA_GB_ISING;
  double e = 0.0;
  for (int i = warp; i < n; i += 8) {
    const double si =
        ((sw[i >> 5] >> (i & 31)) & 1u) ? 1.0 : (ising ? -1.0 : 0.0);
    if (si == 0.0) continue;  // warp-uniform
    const T* row = J + (int64_t)i * ld;
    double f = 0.0;
    for (int j = lane; j < n; j += 32) {
      const double sj =
          ((sw[j >> 5] >> (j & 31)) & 1u) ? 1.0 : (ising ? -1.0 : 0.0);
      f += (double)row[j] * sj;
    }
    f = warp_sum(f);
    e += si * (0.5 * f + (double)h[i]);
  }
  if (lane == 0) e_s[warp] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += e_s[w];
    out[c] = t;
  }
}

__global__ void __launch_bounds__(256) k_energy64(
    int ptype, int n, int ld, const double* J, const double* h,
    const uint32_t* spins, int words, double* out) {
  energy64_body<double>(ptype, n, ld, J, h, spins, words, blockIdx.x, out);
}

// ---- the same with instance inst's f32 couplings of the problem tables
// Dense instances: a cluster takes 4 states, its warps (32 columns x 128
// rows) units of their sum s (J s + 2 h).  f64 instructions run at 1/64 of the
// f32 rate and one state's n^2 of them took nearly all of the time, so every
// lane adds its products, which are exact, into triples of f32 (two states at
// a time) that carry 72 bits, more than the f64 sum they stand in for, and
// converts once at the end, after the lanes and warps have been added.  Bound by
// their 14 paired f32 instructions a product and two states.  QUBO, 128 states,
// n = 912: 335 us with f64, 103 so; n = 1284: 602 and 192.  A state whose sum
// leaves the f32 range (or meets an infinity or NaN) is added in f64.
constexpr int kE64Chunk = 1024;  // rows whose multipliers are staged
constexpr int kE64Rows = 128;    // rows of a unit

__global__ void __launch_bounds__(256) k_energy64_dense(
    const pysa_gb_problems p, int inst, const uint32_t* spins, int words,
    int64_t count, double* out) {
  namespace cg = cooperative_groups;
  __shared__ ulonglong2 mult[kE64Chunk];  // [row]: the 4 states' s
  __shared__ Triple2 e_s[2][8];  // [states 2 q, 2 q + 1][warp]
  __shared__ int bad_s[4];
  if (is_sparse_inst(p, inst)) return;  // k_energy64_tables'
  cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t c0 = 4 * (int64_t)(blockIdx.x / csize);
  const bool ising = p.problem_type == PYSA_GB_ISING;
  const int n = p.n[inst], ld = p.ld[inst];
  const float* J = p.J + p.j_off[inst];
  const float* h = p.h + p.h_off[inst];
  const float down = ising ? -1.0f : 0.0f;
  auto spin = [&](int64_t c, int i) {  // 0 past the last state
    return c >= count ? 0.0f
           : (spins[c * words + (i >> 5)] >> (i & 31)) & 1u ? 1.0f : down;
  };
  Triple2 E[2] = {};
  const int nt = (n + 31) >> 5;
  for (int r0 = 0; r0 < n; r0 += kE64Chunk) {
    const int rows = n - r0 < kE64Chunk ? n - r0 : kE64Chunk;
    __syncthreads();
    for (int i = tid; i < rows; i += 256)
      mult[i] = make_ulonglong2(
          pack2(spin(c0, r0 + i), spin(c0 + 1, r0 + i)),
          pack2(spin(c0 + 2, r0 + i), spin(c0 + 3, r0 + i)));
    __syncthreads();
    const int units = nt * ((rows + kE64Rows - 1) / kE64Rows);
    for (int u = rank * 8 + warp; u < units; u += 8 * csize) {
      const int b = u / nt, col = 32 * (u - b * nt) + lane;
      const bool in = col < n;
      const int i1 = (b + 1) * kE64Rows < rows ? (b + 1) * kE64Rows : rows;
      const float* Jc = J + (int64_t)r0 * ld + (in ? col : 0);
      Triple2 F[2] = {};
#pragma unroll 4
      for (int i = b * kE64Rows; i < i1; ++i) {
        const float v = in ? Jc[(int64_t)i * ld] : 0.0f;
        const uint64_t vv = pack2(v, v);
        const ulonglong2 m = mult[i];
        F[0].add(mul2(vv, m.x));
        F[1].add(mul2(vv, m.y));
      }
      const float h2 = in && r0 == 0 && b == 0 ? 2.0f * h[col] : 0.0f;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint64_t s =
            in ? pack2(spin(c0 + 2 * q, col), spin(c0 + 2 * q + 1, col))
               : 0ull;
        E[q].add(mul2(F[q].a, s));
        E[q].add(mul2(F[q].b, s));
        E[q].add(mul2(F[q].c, s));
        E[q].add(mul2(pack2(h2, h2), s));
      }
    }
  }
  // lanes, then the cluster's warps (two a lane), still as triples
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    lane_sum(E[q]);
    if (lane == 0) e_s[q][warp] = E[q];
  }
  cl.sync();
  if (rank == 0) {
    if (warp < 2) {
      Triple2 t = {};
      for (int i = lane; i < 8 * csize; i += 32)
        t.add(*cl.map_shared_rank(&e_s[warp][i & 7], i >> 3));
      lane_sum(t);
      if (lane < 2) {
        const bool hi = lane;
        const int64_t c = c0 + 2 * warp + lane;
        const float a = half2(t.a, hi);
        const bool bad = !(fabsf(a) < INFINITY) && c < count;
        bad_s[2 * warp + lane] = bad;
        if (!bad && c < count)
          out[c] = 0.5 * ((double)a + ((double)half2(t.b, hi) +
                                       (double)half2(t.c, hi)));
      }
    }
    __syncthreads();
    for (int q = 0; q < 4; ++q) {
      if (!bad_s[q]) continue;  // uniform
      energy64_body<float>(p.problem_type, n, ld, J, h, spins, words, c0 + q,
                           out);
      __syncthreads();
    }
  }
  cl.sync();
}

// Sparse instances from their stored rows: a CTA per state, thread per row,
// fixed reduction order.
__global__ void __launch_bounds__(256) k_energy64_tables(
    const pysa_gb_problems p, int inst, const uint32_t* spins, int words,
    double* out) {
  if (!is_sparse_inst(p, inst)) return;  // k_energy64_dense's
  __shared__ double e_s[8];
  const int64_t c = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t* sw = spins + c * words;
  const bool ising = p.problem_type == PYSA_GB_ISING;
  const int n = p.n[inst];
  const float* h = p.h + p.h_off[inst];
  double e = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double si =
        ((sw[i >> 5] >> (i & 31)) & 1u) ? 1.0 : (ising ? -1.0 : 0.0);
    if (si != 0.0) e += si * (0.5 * csr_row_dot(p, inst, i, sw, ising) +
                              (double)h[i]);
  }
  e = warp_sum(e);
  if (lane == 0) e_s[warp] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += e_s[w];
    out[c] = t;
  }
}

void launch_energy64(int ptype, int n, int ld, const double* J,
                     const double* h, const uint32_t* spins, int words,
                     int64_t count, double* out, cudaStream_t st) {
  if (count > 0)
    k_energy64<<<(unsigned)count, 256, 0, st>>>(ptype, n, ld, J, h, spins,
                                                words, out);
}

void launch_energy64_tables(const pysa_gb_problems& p, int inst,
                            const uint32_t* spins, int words, int64_t count,
                            double* out, cudaStream_t st) {
  if (count <= 0) return;
  // as many CTAs a cluster as have a unit for each of their warps
  const int64_t nt = ((int64_t)p.max_n + 31) / 32;
  const int64_t units = nt * ((p.max_n + kE64Rows - 1) / kE64Rows);
  int cs = 1;
  while (cs < 8 && units > 8 * cs) cs *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((count + 3) / 4 * cs));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_energy64_dense, p, inst, spins, words, count,
                     out);
  if (p.csr_row_off)
    k_energy64_tables<<<(unsigned)count, 256, 0, st>>>(p, inst, spins, words,
                                                       out);
}

// ---------------------------------------------------------------- unpack
__global__ void k_unpack(int ptype, int n, const uint32_t* spins, int words,
                         int64_t count, float* out, int out_ld) {
  const int64_t total = count * n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = e / n;
    const int j = (int)(e % n);
    const uint32_t bit = (spins[c * words + (j >> 5)] >> (j & 31)) & 1u;
    out[c * out_ld + j] = bit ? 1.0f : (ptype == PYSA_GB_ISING ? -1.0f : 0.0f);
  }
}

void launch_unpack(int ptype, int n, const uint32_t* spins, int words,
                   int64_t count, float* out, int out_ld, cudaStream_t st) {
  const int64_t total = count * n;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 65535) blocks = 65535;
  if (blocks > 0)
    k_unpack<<<(unsigned)blocks, 256, 0, st>>>(ptype, n, spins, words, count,
                                               out, out_ld);
}

// Float states (+-1 or 0/1) -> bit-packed words: a warp per (state, word),
// one ballot per word.  The bit is x > 0 (Ising) or x != 0 (QUBO), the rule
// of the host-side packing.
__global__ void k_pack(int ptype, int n, const float* x, int x_ld,
                       int64_t count, uint32_t* spins, int words) {
  const int lane = threadIdx.x & 31;
  const int64_t total = count * words;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t e = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
       e < total; e += nw) {
    const int64_t c = e / words;
    const int w = (int)(e % words);
    const int j = 32 * w + lane;
    bool b = false;
    if (j < n) {
      const float v = x[c * x_ld + j];
      b = ptype == PYSA_GB_ISING ? v > 0.0f : v != 0.0f;
    }
    const uint32_t bits = __ballot_sync(0xffffffffu, b);
    if (lane == 0) spins[c * words + w] = bits;
  }
}

void launch_pack(int ptype, int n, const float* x, int x_ld, int64_t count,
                 uint32_t* spins, int words, cudaStream_t st) {
  const int64_t warps = count * words;
  int64_t blocks = (warps + 7) / 8;
  if (blocks > 65535) blocks = 65535;
  if (blocks > 0)
    k_pack<<<(unsigned)blocks, 256, 0, st>>>(ptype, n, x, x_ld, count, spins,
                                             words);
}

// A dense symmetric problem matrix P (n x n, row stride p_ld) of instance
// inst split as the reference's Solver does (pysa/sa.py:66-69): couplings =
// P with a zero diagonal, stored transposed (row j = column j of P), and
// local fields = diag(P).
__global__ void k_load_problem(const pysa_gb_problems p, int inst,
                               const float* P, int p_ld) {
  const int n = p.n[inst];
  const int ld = p.ld[inst];
  // the tables' J and h are const for the sweeps; this kernel refills them
  float* Jt = const_cast<float*>(p.J) + p.j_off[inst];
  float* h = const_cast<float*>(p.h) + p.h_off[inst];
  const int64_t total = (int64_t)n * ld;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int j = (int)(e / ld), i = (int)(e % ld);
    float v = 0.0f;
    if (i < n && i != j) v = P[(int64_t)i * p_ld + j];
    Jt[e] = v;
    if (i == j) h[j] = P[(int64_t)j * p_ld + j];
  }
}

void launch_load_problem(const pysa_gb_problems& p, int inst, int n, int ld,
                         const float* P, int p_ld, cudaStream_t st) {
  const int64_t total = (int64_t)n * ld;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 65535) blocks = 65535;
  if (blocks > 0)
    k_load_problem<<<(unsigned)blocks, 256, 0, st>>>(p, inst, P, p_ld);
}

}  // namespace pysa_gb
