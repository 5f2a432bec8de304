// Tabulated se_e2_a embedding fused with the G^T.R contraction (sm_103a):
// the operator-contract kernels behind deepmd::tabulate_fusion_se_a.
//
// out[i, m, k] = sum_j w_j em[i, j, m] P_k(x_ij), P_k the fifth-order
// polynomial of table row locate(x_ij).  The nloc x nnei x M embedding is
// never materialised.  Reference semantics: source/lib/src/tabulate.cc:80-384
// (CPU, the oracle) and source/lib/src/gpu/tabulate.cu:196-503.
//
// Work split.  A warp takes its neighbours 32 at a time: each lane locates
// one neighbour's table row (the two divisions once per neighbour instead of
// once per lane) and stages its env row, weight and in-row offset in shared
// memory; then
//   forward / grad-grad (k_tab_sum): lanes over the outputs k in full
//     32-wide chunks, neighbours sequential, the coefficients kept while the
//     next neighbour is on the same row; the leftover outputs run several
//     neighbours per instruction (100 outputs: 3 chunks and a tail of
//     4, not 4 chunks);
//   grad (k_tab_grad): G lanes per neighbour, 32 / G neighbours per
//     instruction, dy in registers, the five sums of a neighbour reduced over
//     its G lanes by a reduce-scatter.
// With S = 4 the four warps of a CTA share one atom's neighbours (small
// batches: as many warps in flight with a quarter of the serial walk).
// What bounds them: FP32, the L1 wavefronts of the 24-byte coefficient stride
// and the issue slots (12,288 atoms, 92 slots, 100 outputs: forward 105 ->
// 72 us, grad 187 -> 121 us against one lane-redundant location per
// neighbour, four chunks and separate value and slope polynomials; 1,536
// atoms, 46 slots: grad-grad 27 -> 14.5 us); FP64, the FP64 pipe (771 atoms,
// 92 slots: forward 257 -> 103 us, grad 507 -> 211 us; the pipe's floor for
// the 9 and 18 FMAs of an output is 64 and 128 us).
// The padding fold (tabulate.cc:108-155): with is_sorted, the first slot
// whose x equals the last slot's x and whose em[1:4] are zero stands for all
// remaining slots (weight nnei - j) and ends the sum; slots after it get no
// gradient.
#include "common.cuh"

namespace gbdp {
namespace {

constexpr int kTabWarps = 4;

template <typename T>
struct alignas(16) Row4 {
  T v[4];
};

// one row of 4 values; vec: 16-byte aligned rows
__device__ __forceinline__ Row4<float> ld_row(const float* p, bool vec) {
  Row4<float> r;
  if (vec) {
    const float4 u = __ldg(reinterpret_cast<const float4*>(p));
    r.v[0] = u.x;
    r.v[1] = u.y;
    r.v[2] = u.z;
    r.v[3] = u.w;
  } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) r.v[m] = __ldg(p + m);
  }
  return r;
}
__device__ __forceinline__ Row4<double> ld_row(const double* p, bool vec) {
  Row4<double> r;
  if (vec) {
    const double2 u = __ldg(reinterpret_cast<const double2*>(p));
    const double2 w = __ldg(reinterpret_cast<const double2*>(p) + 1);
    r.v[0] = u.x;
    r.v[1] = u.y;
    r.v[2] = w.x;
    r.v[3] = w.y;
  } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) r.v[m] = __ldg(p + m);
  }
  return r;
}
__device__ __forceinline__ void st_row(float* p, const Row4<float>& r, bool vec) {
  if (vec) {
    *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) p[m] = r.v[m];
  }
}
__device__ __forceinline__ void st_row(double* p, const Row4<double>& r, bool vec) {
  if (vec) {
    reinterpret_cast<double2*>(p)[0] = make_double2(r.v[0], r.v[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(r.v[2], r.v[3]);
  } else {
#pragma unroll
    for (int m = 0; m < 4; ++m) p[m] = r.v[m];
  }
}

// First fold slot of atom i (nnei if none), found by the whole warp: four
// 32-slot groups per round trip.
template <typename T>
__device__ __forceinline__ int fold_point(const T* __restrict__ em_x, const T* __restrict__ em,
                                          int i, int nnei, bool is_sorted, bool vec) {
  if (!is_sorted) return nnei;
  const int lane = threadIdx.x & 31;
  const T* xi = em_x + (size_t)i * nnei;
  const T* ei = em + (size_t)i * nnei * 4;
  const T last = xi[nnei - 1];
  for (int b = 0; b < nnei; b += 128) {
    bool hit[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = b + 32 * u + lane;
      hit[u] = false;
      if (j < nnei) {
        const Row4<T> e = ld_row(ei + 4 * (size_t)j, vec);
        hit[u] = xi[j] == last && e.v[1] == T(0) && e.v[2] == T(0) && e.v[3] == T(0);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned m = __ballot_sync(kFull, hit[u]);
      if (m) return b + 32 * u + __ffs(m) - 1;
    }
  }
  return nnei;
}

template <typename T>
__device__ __forceinline__ void load_coef(Coef<T>& c, const T* __restrict__ row, int k) {
  using P = typename TabVec<T>::v2;
  const P* p = reinterpret_cast<const P*>(row + 6 * k);
#pragma unroll
  for (int q = 0; q < 3; ++q) c.p[q] = __ldg(p + q);
}

// e . d over the four env columns
__device__ __forceinline__ float dot4(const Row4<float>& e, const float* d) {
  const float2 h = __ffma2_rn(make_float2(e.v[2], e.v[3]), make_float2(d[2], d[3]),
                              __fmul2_rn(make_float2(e.v[0], e.v[1]), make_float2(d[0], d[1])));
  return h.x + h.y;
}
__device__ __forceinline__ double dot4(const Row4<double>& e, const double* d) {
  return e.v[0] * d[0] + e.v[1] * d[1] + e.v[2] * d[2] + e.v[3] * d[3];
}

// the neighbours of warp `warp` of the S that share jend neighbours:
// contiguous, so that neighbours on the same table row stay together
template <int S>
__device__ __forceinline__ void warp_range(int jend, int warp, int& lo, int& hi) {
  if (S == 1) {
    lo = 0;
    hi = jend;
    return;
  }
  const int per = (jend + S - 1) / S;
  lo = min(jend, warp * per);
  hi = min(jend, lo + per);
}

// ------------------------------------------------- forward and grad-grad --
// forward:   out[m][k] = sum_j w em[j][m] P_k(x_j)
// grad-grad: out[m][k] = sum_j w (dz_dem[j][m] P_k + em[j][m] dz_dem_x[j] P'_k)
// NQF: full 32-wide output chunks; tail_w (0..31) outputs after them run
// 2^tail_lg >= tail_w lanes per neighbour.
template <typename T, int NQF, bool GG, int S>
__global__ void __launch_bounds__(kTabWarps * 32)
    k_tab_sum(T* __restrict__ out, const T* __restrict__ table, TableInfo<T> ti,
              const T* __restrict__ em_x, const T* __restrict__ em,
              const T* __restrict__ dz_dem_x, const T* __restrict__ dz_dem, int nloc, int nnei,
              int M, int k_base, int tail_w, int tail_lg, bool is_sorted, bool vec) {
  constexpr int NA = NQF + 1;
  constexpr int NB = GG ? 2 : 1;
  __shared__ Row4<T> s_row[kTabWarps][NB][32];
  __shared__ T s_x[kTabWarps][32];
  __shared__ int s_idx[kTabWarps][32];
  __shared__ T s_red[S > 1 ? S : 1][S > 1 ? 4 * 128 : 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = S == 1 ? blockIdx.x * kTabWarps + warp : blockIdx.x;
  if (S == 1 && i >= nloc) return;  // uniform over the warp; no CTA-wide barrier at S = 1
  const int bp = fold_point(em_x, em, i, nnei, is_sorted, vec);
  int lo, hi;
  warp_range<S>(bp < nnei ? bp + 1 : nnei, warp, lo, hi);
  T acc[NA][4];
#pragma unroll
  for (int q = 0; q < NA; ++q)
#pragma unroll
    for (int m = 0; m < 4; ++m) acc[q][m] = T(0);
  Coef<T> c[NQF > 0 ? NQF : 1];
  int prev = -1;
  const int tw = 1 << tail_lg, tn = lane >> tail_lg, tt = lane & (tw - 1);
  for (int j0 = lo; j0 < hi; j0 += 32) {
    const int cnt = min(32, hi - j0);
    if (lane < cnt) {
      const int j = j0 + lane;
      const size_t ij = (size_t)i * nnei + j;
      T x = em_x[ij];
      Row4<T> e = ld_row(em + ij * 4, vec);
      const T w = j == bp ? T(nnei - j) : T(1);
      if (GG) {
        Row4<T> h = ld_row(dz_dem + ij * 4, vec);
        const T g = w * dz_dem_x[ij];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          h.v[m] *= w;
          e.v[m] *= g;
        }
        s_row[warp][NB - 1][lane] = e;
        s_row[warp][0][lane] = h;
      } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) e.v[m] *= w;
        s_row[warp][0][lane] = e;
      }
      s_idx[warp][lane] = locate_row(ti, x);
      s_x[warp][lane] = x;
    }
    __syncwarp();
    if (NQF > 0) {
      for (int jj = 0; jj < cnt; ++jj) {
        const int idx = s_idx[warp][jj];
        const XPow<T> xp(s_x[warp][jj]);
        const Row4<T> a = s_row[warp][0][jj];
        if (idx != prev) {  // uniform over the warp
          prev = idx;
          const T* row = table + (size_t)idx * M * 6;
#pragma unroll
          for (int q = 0; q < NQF; ++q) load_coef<T>(c[q], row, k_base + q * 32 + lane);
        }
#pragma unroll
        for (int q = 0; q < NQF; ++q) {
          if (GG) {
            const Row4<T> b = s_row[warp][NB - 1][jj];
            T v, d;
            tab_val_slope(c[q], xp, v, d);
#pragma unroll
            for (int m = 0; m < 4; ++m) acc[q][m] += v * a.v[m] + d * b.v[m];
          } else {
            const T v = tab_val(c[q], xp);
#pragma unroll
            for (int m = 0; m < 4; ++m) acc[q][m] += v * a.v[m];
          }
        }
      }
    }
    if (tail_w > 0) {
      for (int jt = 0; jt < cnt; jt += 32 >> tail_lg) {
        const int jj = jt + tn;
        if (jj < cnt && tt < tail_w) {
          const XPow<T> xp(s_x[warp][jj]);
          const Row4<T> a = s_row[warp][0][jj];
          Coef<T> ct;
          load_coef<T>(ct, table + (size_t)s_idx[warp][jj] * M * 6, k_base + NQF * 32 + tt);
          if (GG) {
            const Row4<T> b = s_row[warp][NB - 1][jj];
            T v, d;
            tab_val_slope(ct, xp, v, d);
#pragma unroll
            for (int m = 0; m < 4; ++m) acc[NQF][m] += v * a.v[m] + d * b.v[m];
          } else {
            const T v = tab_val(ct, xp);
#pragma unroll
            for (int m = 0; m < 4; ++m) acc[NQF][m] += v * a.v[m];
          }
        }
      }
    }
    __syncwarp();
  }
  if (tail_w > 0)
    for (int o = tw; o < 32; o <<= 1)
#pragma unroll
      for (int m = 0; m < 4; ++m) acc[NQF][m] += __shfl_xor_sync(kFull, acc[NQF][m], o);
  const int w = NQF * 32 + tail_w;
  if (S == 1) {
#pragma unroll
    for (int q = 0; q < NA; ++q) {
      const int k = q * 32 + lane;
      if (k < w)
#pragma unroll
        for (int m = 0; m < 4; ++m) out[((size_t)i * 4 + m) * M + k_base + k] = acc[q][m];
    }
  } else {
#pragma unroll
    for (int q = 0; q < NA; ++q) {
      const int k = q * 32 + lane;
      if (k < w)
#pragma unroll
        for (int m = 0; m < 4; ++m) s_red[warp][m * 128 + k] = acc[q][m];
    }
    __syncthreads();
    const int k = threadIdx.x;
    if (k < w)
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        T t = s_red[0][m * 128 + k];
#pragma unroll
        for (int u = 1; u < S; ++u) t += s_red[u][m * 128 + k];
        out[((size_t)i * 4 + m) * M + k_base + k] = t;
      }
  }
}

// ---------------------------------------------------------------- grad --
// G lanes per neighbour (lane t of a group owns outputs t + G q, q < NK),
// 32 / G neighbours per instruction: dy_dem[m] = sum_k P_k dy[m][k] and
// dy_dem_x = sum_k P'_k (em . dy[., k]).  FP32 G = 16; FP64 G = 8, where the
// pipe-bound kernel gains from the narrower last step (100 outputs: 104
// lanes' worth instead of 112) and the shorter reduction.
template <typename T>
struct TabGroup {
  static constexpr int G = sizeof(T) == 4 ? 16 : 8;
};

template <typename T, int NK, int S>
__global__ void __launch_bounds__(kTabWarps * 32)
    k_tab_grad(T* __restrict__ dy_dem_x, T* __restrict__ dy_dem, const T* __restrict__ table,
               TableInfo<T> ti, const T* __restrict__ em_x, const T* __restrict__ em,
               const T* __restrict__ dy, int nloc, int nnei, int M, int k_base, bool accumulate,
               bool is_sorted, bool vec) {
  constexpr int G = TabGroup<T>::G, NG = 32 / G;
  __shared__ Row4<T> s_row[kTabWarps][32];  // env rows, then dy_dem
  __shared__ T s_x[kTabWarps][32];          // offsets, then dy_dem_x
  __shared__ int s_idx[kTabWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = S == 1 ? blockIdx.x * kTabWarps + warp : blockIdx.x;
  if (i >= nloc) return;  // uniform over the warp; no CTA-wide barrier below
  const int n = lane / G, t = lane & (G - 1);
  const int Mc = min(M - k_base, G * NK);
  T g[NK][4];
#pragma unroll
  for (int q = 0; q < NK; ++q) {
    const int k = t + G * q;
#pragma unroll
    for (int m = 0; m < 4; ++m)
      g[q][m] = k < Mc ? dy[((size_t)i * 4 + m) * M + k_base + k] : T(0);
  }
  const int bp = fold_point(em_x, em, i, nnei, is_sorted, vec);
  const int jend = bp < nnei ? bp + 1 : nnei;
  // slots after the fold point get no gradient (tabulate.cc:166-170, :251-256)
  if (!accumulate) {
    const Row4<T> z{{T(0), T(0), T(0), T(0)}};
    for (int j = jend + (S == 1 ? lane : (int)threadIdx.x); j < nnei; j += S == 1 ? 32 : S * 32) {
      const size_t ij = (size_t)i * nnei + j;
      dy_dem_x[ij] = T(0);
      st_row(dy_dem + ij * 4, z, vec);
    }
  }
  int lo, hi;
  warp_range<S>(jend, warp, lo, hi);
  for (int j0 = lo; j0 < hi; j0 += 32) {
    const int cnt = min(32, hi - j0);
    if (lane < cnt) {
      const size_t ij = (size_t)i * nnei + j0 + lane;
      T x = em_x[ij];
      s_row[warp][lane] = ld_row(em + ij * 4, vec);
      s_idx[warp][lane] = locate_row(ti, x);
      s_x[warp][lane] = x;
    }
    __syncwarp();
    for (int jt = 0; jt < cnt; jt += NG) {
      // a group past the end re-evaluates slot jt; its sums are dropped
      const int jj = jt + n < cnt ? jt + n : jt;
      const T* row = table + (size_t)s_idx[warp][jj] * M * 6 + 6 * k_base;
      const XPow<T> xp(s_x[warp][jj]);
      const Row4<T> e = s_row[warp][jj];
      T p[4] = {T(0), T(0), T(0), T(0)}, px = T(0);
      // no branch between the steps, so that several steps' loads are in
      // flight: a lane past the width (in the last step) reads the last
      // output and drops it (against dy = 0 alone an infinite one would be
      // 0 inf = NaN)
#pragma unroll
      for (int q = 0; q < NK; ++q) {
        Coef<T> c;
        load_coef<T>(c, row, min(t + G * q, Mc - 1));
        T v, d;
        tab_val_slope(c, xp, v, d);
        if (q == NK - 1 && t + G * q >= Mc) v = d = T(0);
#pragma unroll
        for (int m = 0; m < 4; ++m) p[m] += v * g[q][m];
        px += d * dot4(e, g[q]);
      }
      // reduce-scatter over the group: the upper half of the G lanes takes
      // components 2, 3 and the lower half 0, 1, then one component each
      // (the slope sum is added in full beside them), and at the next level
      // the pairs split into component and slope sum
      const bool hb = (t & (G / 2)) != 0, hq = (t & (G / 4)) != 0;
      const T r0 = __shfl_xor_sync(kFull, hb ? p[0] : p[2], G / 2);
      const T r1 = __shfl_xor_sync(kFull, hb ? p[1] : p[3], G / 2);
      px += __shfl_xor_sync(kFull, px, G / 2);
      const T a0 = (hb ? p[2] : p[0]) + r0, a1 = (hb ? p[3] : p[1]) + r1;
      const T b = (hq ? a1 : a0) + __shfl_xor_sync(kFull, hq ? a0 : a1, G / 4);
      px += __shfl_xor_sync(kFull, px, G / 4);
      const bool hx = (t & (G / 8)) != 0;  // this lane ends with the slope sum
      T r = (hx ? px : b) + __shfl_xor_sync(kFull, hx ? b : px, G / 8);
      if (G == 16) r += __shfl_xor_sync(kFull, r, 1);
      if (jt + n < cnt && (t & (G / 8 - 1)) == 0) {
        if (!hx)
          s_row[warp][jt + n].v[t / (G / 4)] = r;
        else if (t == G / 8)
          s_x[warp][jt + n] = r;
      }
    }
    __syncwarp();
    if (lane < cnt) {
      const int j = j0 + lane;
      const size_t ij = (size_t)i * nnei + j;
      const T w = j == bp ? T(nnei - j) : T(1);
      Row4<T> r = s_row[warp][lane];
      T rx = s_x[warp][lane] * w;
#pragma unroll
      for (int m = 0; m < 4; ++m) r.v[m] *= w;
      if (accumulate) {
        rx += dy_dem_x[ij];
#pragma unroll
        for (int m = 0; m < 4; ++m) r.v[m] += dy_dem[ij * 4 + m];
      }
      dy_dem_x[ij] = rx;
      st_row(dy_dem + ij * 4, r, vec);
    }
    __syncwarp();
  }
}

template <typename T>
int check_common(const T* table, const T* table_info, const T* em_x, const T* em, int nloc,
                 int nnei, int M) {
  GBDP_REQUIRE(nloc >= 0 && nnei >= 0, "tabulate_fusion_se_a: negative nloc/nnei");
  GBDP_REQUIRE(M > 0 && M <= 1024, "tabulate_fusion_se_a: last_layer_size %d not in [1,1024]",
               M);
  GBDP_REQUIRE(table_info != nullptr, "tabulate_fusion_se_a: table_info (host) is null");
  GBDP_REQUIRE(nloc == 0 || nnei == 0 || (table && em_x && em),
               "tabulate_fusion_se_a: null device pointer");
  GBDP_REQUIRE(((uintptr_t)table & 15) == 0,
               "tabulate_fusion_se_a: table must be 16-byte aligned");
  GBDP_REQUIRE(table_info[3] > 0 && table_info[4] > 0,
               "tabulate_fusion_se_a: table strides must be positive");
  return GBDP_OK;
}

inline bool rows_aligned(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Below these numbers of atoms the four warps of a CTA share one atom: with
// few atoms an SM, a warp per atom leaves the schedulers short of warps and
// the kernel waits for the serial walk over the neighbours; above, the
// repeated fold search (and dy loads) of the four warps cost more.  Measured
// on the H section of water (92 slots, 100 outputs), shared / own, us:
//   FP32 sum   192: 10.4 / 17.9   1536: 19.2 / 18.8   3072: 28.9 / 26.6
//   FP32 grad  192: 12.3 / 24.7   3072: 43.3 / 46.2   4500: 58.4 / 53.2
//   FP64 sum   192: 37.1 / 75.1   3072:  335 /  355   4500:  476 /  463
//   FP64 grad  192: 76.5 /  160   4500:  991 / 1062   6144: 1328 / 1324
template <typename T>
constexpr int kTabShareSum = 152 * (sizeof(T) == 4 ? 10 : 24);
template <typename T>
constexpr int kTabShareGrad = 152 * (sizeof(T) == 4 ? 20 : 32);

template <typename T, bool GG, int S>
void launch_sum(int nqf, cudaStream_t st, T* out, const T* table, const TableInfo<T>& ti,
                const T* em_x, const T* em, const T* dzx, const T* dzm, int nloc, int nnei, int M,
                int kb, int tail_w, int tail_lg, bool sorted, bool vec) {
  const dim3 grid(S == 1 ? (nloc + kTabWarps - 1) / kTabWarps : nloc), block(kTabWarps * 32);
#define GBDP_TAB_CASE(N)                                                                        \
  case N:                                                                                       \
    k_tab_sum<T, N, GG, S><<<grid, block, 0, st>>>(out, table, ti, em_x, em, dzx, dzm, nloc,    \
                                                   nnei, M, kb, tail_w, tail_lg, sorted, vec);  \
    break;
  switch (nqf) {
    GBDP_TAB_CASE(0)
    GBDP_TAB_CASE(1)
    GBDP_TAB_CASE(2)
    GBDP_TAB_CASE(3)
    GBDP_TAB_CASE(4)
  }
#undef GBDP_TAB_CASE
}

template <typename T, bool GG>
void tab_sum(T* out, const T* table, const T* info, const T* em_x, const T* em, const T* dzx,
             const T* dzm, int nloc, int nnei, int M, int is_sorted, cudaStream_t st) {
  const TableInfo<T> ti = make_table_info(info);
  const bool vec = rows_aligned(em) && (!GG || rows_aligned(dzm));
  // outputs 128 at a time: full 32-wide chunks, then the tail
  for (int kb = 0; kb < M; kb += 128) {
    const int w = M - kb < 128 ? M - kb : 128;
    const int tail_w = w & 31;
    int lg = 0;
    while ((1 << lg) < tail_w) ++lg;
    if (nloc < kTabShareSum<T>)
      launch_sum<T, GG, 4>(w / 32, st, out, table, ti, em_x, em, dzx, dzm, nloc, nnei, M, kb,
                           tail_w, lg, is_sorted != 0, vec);
    else
      launch_sum<T, GG, 1>(w / 32, st, out, table, ti, em_x, em, dzx, dzm, nloc, nnei, M, kb,
                           tail_w, lg, is_sorted != 0, vec);
  }
}

template <typename T>
int tab_fwd(T* out, const T* table, const T* info, const T* em_x, const T* em, int nloc,
            int nnei, int M, int is_sorted, cudaStream_t st) {
  int rc = check_common(table, info, em_x, em, nloc, nnei, M);
  if (rc) return rc;
  if (nloc == 0) return GBDP_OK;
  if (nnei == 0)
    cudaMemsetAsync(out, 0, sizeof(T) * (size_t)nloc * 4 * M, st);
  else
    tab_sum<T, false>(out, table, info, em_x, em, nullptr, nullptr, nloc, nnei, M, is_sorted, st);
  GBDP_CHECK_LAUNCH("tabulate_fusion_se_a");
  return GBDP_OK;
}

template <typename T>
int tab_grad_grad(T* dz_dy, const T* table, const T* info, const T* em_x, const T* em,
                  const T* dzx, const T* dzm, int nloc, int nnei, int M, int is_sorted,
                  cudaStream_t st) {
  int rc = check_common(table, info, em_x, em, nloc, nnei, M);
  if (rc) return rc;
  if (nloc == 0) return GBDP_OK;
  if (nnei == 0) {
    cudaMemsetAsync(dz_dy, 0, sizeof(T) * (size_t)nloc * 4 * M, st);
    GBDP_CHECK_LAUNCH("tabulate_fusion_se_a_grad_grad");
    return GBDP_OK;
  }
  GBDP_REQUIRE(dzx && dzm, "tabulate_fusion_se_a_grad_grad: null dz pointers");
  tab_sum<T, true>(dz_dy, table, info, em_x, em, dzx, dzm, nloc, nnei, M, is_sorted, st);
  GBDP_CHECK_LAUNCH("tabulate_fusion_se_a_grad_grad");
  return GBDP_OK;
}

template <typename T, int NK>
void launch_grad(cudaStream_t st, T* dy_dem_x, T* dy_dem, const T* table, const TableInfo<T>& ti,
                 const T* em_x, const T* em, const T* dy, int nloc, int nnei, int M, int kb,
                 bool sorted, bool vec) {
  const dim3 block(kTabWarps * 32);
  if (nloc < kTabShareGrad<T>)
    k_tab_grad<T, NK, 4><<<dim3(nloc), block, 0, st>>>(dy_dem_x, dy_dem, table, ti, em_x, em, dy,
                                                        nloc, nnei, M, kb, kb > 0, sorted, vec);
  else
    k_tab_grad<T, NK, 1><<<dim3((nloc + kTabWarps - 1) / kTabWarps), block, 0, st>>>(
        dy_dem_x, dy_dem, table, ti, em_x, em, dy, nloc, nnei, M, kb, kb > 0, sorted, vec);
}

template <typename T>
int tab_grad(T* dy_dem_x, T* dy_dem, const T* table, const T* info, const T* em_x, const T* em,
             const T* dy, int nloc, int nnei, int M, int is_sorted, cudaStream_t st) {
  int rc = check_common(table, info, em_x, em, nloc, nnei, M);
  if (rc) return rc;
  if (nloc == 0 || nnei == 0) return GBDP_OK;
  GBDP_REQUIRE(dy && dy_dem_x && dy_dem, "tabulate_fusion_se_a_grad: null pointer");
  const TableInfo<T> ti = make_table_info(info);
  const bool vec = rows_aligned(em) && rows_aligned(dy_dem);
  constexpr int G = TabGroup<T>::G;
  // outputs 128 at a time; later chunks accumulate
  for (int kb = 0; kb < M; kb += 128) {
    const int w = M - kb < 128 ? M - kb : 128, nk = (w + G - 1) / G;
#define GBDP_TAB_GRAD(N)                                                                       \
  launch_grad<T, N>(st, dy_dem_x, dy_dem, table, ti, em_x, em, dy, nloc, nnei, M, kb,          \
                    is_sorted != 0, vec)
#define GBDP_TAB_GRAD2(N)              \
  case N: GBDP_TAB_GRAD(N); break;     \
  case N + 1: GBDP_TAB_GRAD(N + 1); break;
    switch (nk) {
      GBDP_TAB_GRAD2(1)
      GBDP_TAB_GRAD2(3)
      GBDP_TAB_GRAD2(5)
      GBDP_TAB_GRAD2(7)
      default:
        if constexpr (G == 8) switch (nk) {
            GBDP_TAB_GRAD2(9)
            GBDP_TAB_GRAD2(11)
            GBDP_TAB_GRAD2(13)
            GBDP_TAB_GRAD2(15)
          }
    }
#undef GBDP_TAB_GRAD2
#undef GBDP_TAB_GRAD
  }
  GBDP_CHECK_LAUNCH("tabulate_fusion_se_a_grad");
  return GBDP_OK;
}

}  // namespace
}  // namespace gbdp

using namespace gbdp;

#define GBDP_TAB_ENTRY(T, SFX)                                                                  \
  extern "C" int gbdp_tabulate_fusion_se_a_##SFX(T* out, const T* table, const T* table_info,   \
                                                 const T* em_x, const T* em, int nloc,         \
                                                 int nnei, int last_layer_size, int is_sorted, \
                                                 gbdp_stream stream) {                         \
    return tab_fwd<T>(out, table, table_info, em_x, em, nloc, nnei, last_layer_size,           \
                      is_sorted, (cudaStream_t)stream);                                        \
  }                                                                                             \
  extern "C" int gbdp_tabulate_fusion_se_a_grad_##SFX(                                          \
      T* dy_dem_x, T* dy_dem, const T* table, const T* table_info, const T* em_x, const T* em, \
      const T* dy, int nloc, int nnei, int last_layer_size, int is_sorted,                     \
      gbdp_stream stream) {                                                                     \
    return tab_grad<T>(dy_dem_x, dy_dem, table, table_info, em_x, em, dy, nloc, nnei,          \
                       last_layer_size, is_sorted, (cudaStream_t)stream);                      \
  }                                                                                             \
  extern "C" int gbdp_tabulate_fusion_se_a_grad_grad_##SFX(                                     \
      T* dz_dy, const T* table, const T* table_info, const T* em_x, const T* em,               \
      const T* dz_dy_dem_x, const T* dz_dy_dem, int nloc, int nnei, int last_layer_size,       \
      int is_sorted, gbdp_stream stream) {                                                      \
    return tab_grad_grad<T>(dz_dy, table, table_info, em_x, em, dz_dy_dem_x, dz_dy_dem, nloc,  \
                            nnei, last_layer_size, is_sorted, (cudaStream_t)stream);           \
  }

GBDP_TAB_ENTRY(float, f32)
GBDP_TAB_ENTRY(double, f64)
