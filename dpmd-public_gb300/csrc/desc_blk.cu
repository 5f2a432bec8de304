// Fused compressed se_e2_a descriptor in FP32 on blocked tables (sm_103a).
//
// Tables.  A row holds blocks of 32 outputs, 768 bytes each; block b holds
// three 256-byte planes c, plane c the 16-byte pieces
//   {a_2c[k], a_2c[k + 16], a_2c+1[k], a_2c+1[k + 16]},  k = 32 b + t, t < 16
// (zeros past M).  A 16-lane group reads a plane with one contiguous 16-byte
// load a lane, and every coefficient arrives beside that of output k + 16 in
// a register pair, as the packed FP32x2 FMAs take them: no move between load
// and Horner sweep, and offsets that do not depend on M.  (From the k-planar
// rows of fused.cu the same packed sweep spends as many moves as FMAs.)
//
// k_fwd_blk.  As k_desc_fwd, with a neighbour's blocks two at a time over the
// half-warps (100 outputs: blocks 0, 1, then 2, 3), the coefficients kept
// while the next neighbour is on the same row; no tail pass.
//
// k_bwd_blk.  As k_desc_bwd: 16 lanes per neighbour, U x 2 neighbours in
// flight per warp; dE/dD is read once, coalesced, for both products of dX.
//
// Both run one warp per atom, or (S = 4 and, forward, 8: small batches) the
// warps of a CTA on one atom's neighbours, so that the serial walk over the
// neighbours is that much shorter and a few hundred atoms still fill the SMs.
//
// Bounds and measurements (water, M = 100; against the k-planar kernels).
// 125,000 atoms in 160 frames: forward 1,178 -> 1,008 us (L1: without the kept
// coefficients 1,303 us; 36 resident warps at 56 registers 1,238 us), backward
// 2,256 -> 1,717 us (28 resident warps 1,781, 20 warps 1,731; a branch on M
// between the steps costs 20 %, since it keeps a step's loads behind the
// previous step's sums).  12,288 atoms: 125 -> 111 and 258 -> 195 us.  192
// atoms: 34 -> 18 and 63 -> 28 us.
#include "fused.cuh"

namespace gbdp {
namespace {

constexpr int kBlk = 192;  // floats per 32-output block of a row

__device__ __forceinline__ float4 ld_tab4(const float* p) {
  float4 v;
  asm("ld.global.nc.L1::evict_last.v4.f32 {%0, %1, %2, %3}, [%4];"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p));
  return v;
}

// the warps of one atom
template <int S>
__device__ __forceinline__ void atom_sync() {
  if constexpr (S == 1)
    __syncwarp();
  else
    __syncthreads();
}

// warp w's part of n neighbours shared by S warps (contiguous; even bounds,
// as the backward takes them two by two)
template <int S>
__device__ __forceinline__ void atom_range(int n, int w, int& lo, int& hi) {
  if constexpr (S == 1) {
    lo = 0;
    hi = n;
  } else {
    const int per = ((n + S - 1) / S + 1) & ~1;
    lo = min(n, w * per);
    hi = min(n, lo + per);
  }
}

__device__ __forceinline__ float dot44(const float4& a, const float4& b) {
  const float2 h = __ffma2_rn(hi2(a), hi2(b), __fmul2_rn(lo2(a), lo2(b)));
  return h.x + h.y;
}

// a slot's env row, and its in-row offset with the table row's index
struct SlotArr {
  float4* em;
  float2* xi;
  int* cnt;   // [kMaxTypes] slots of each section
  int* fold;  // [kMaxTypes] S > 1: fold point of each section
};
__host__ __device__ constexpr size_t slot_bytes(int nnei) {
  return ((size_t)nnei * 24 + 8 * kMaxTypes + 31) & ~(size_t)31;
}
__device__ __forceinline__ SlotArr carve(unsigned char* b, int nnei) {
  SlotArr s;
  s.em = reinterpret_cast<float4*>(b);
  s.xi = reinterpret_cast<float2*>(b + (size_t)nnei * 16);
  s.cnt = reinterpret_cast<int*>(b + (size_t)nnei * 24);
  s.fold = s.cnt + kMaxTypes;
  return s;
}

// ---------------------------------------------------------------- forward --
// S = 1: the slots, then X^T over them; S > 1: the slots, then the warps'
// partial sums over them, and X^T
template <int S>
__host__ __device__ constexpr size_t fwd_bytes(int nnei, int M) {
  const size_t sl = slot_bytes(nnei), xt = (size_t)M * 16;
  if (S == 1) return sl > xt ? sl : xt;
  return (sl > S * xt ? sl : S * xt) + xt;
}

template <int NS, int W, int S>
__global__ void __launch_bounds__(W * 32, 32 / W)
    k_fwd_blk(const __grid_constant__ DescFwdArgs p, const __grid_constant__ TabSet<float> ts,
              int nloc, int M) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  grid_wait();
  grid_release();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = S == 1 ? blockIdx.x * W + warp : blockIdx.x;
  if (i >= nloc) return;  // S = 1: uniform over the warp; S > 1: the grid is exact
  const int w = S == 1 ? 0 : warp;
  const int nnei = ts.sec[ts.ntypes];
  unsigned char* base = smem_raw + (S == 1 ? (size_t)warp * fwd_bytes<S>(nnei, M) : 0);
  const SlotArr sl = carve(base, nnei);
  float4* xT = reinterpret_cast<float4*>(S == 1 ? base : base + fwd_bytes<S>(nnei, M) - M * 16);
  const int NB = (M + 31) >> 5, rs = NB * kBlk;
  const int half = lane >> 4, t16 = lane & 15;
  // this lane's piece of step s: block 2 s + half, output 32 b + t16 (a lane
  // past M, or a half without a block, repeats a valid piece; its sums are
  // not stored)
  int loff[NS], k0[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const int b = min(2 * s + half, NB - 1), lim = min(16, M - 32 * b);
    loff[s] = b * kBlk + 4 * min(t16, lim - 1);
    k0[s] = 2 * s + half < NB && t16 < lim ? 32 * b + t16 : M;
  }
  float2 acc[NS][4];
#pragma unroll
  for (int s = 0; s < NS; ++s)
#pragma unroll
    for (int m = 0; m < 4; ++m) acc[s][m] = make_float2(0.f, 0.f);
  const int ti = p.atype[i];
  if (ti >= 0) {
    // ---- prepass: fold point, rows and env rows per section, the fold slot
    //      with the weight of the slots it stands for (tabulate.cc:108-115)
    if (S > 1) {
      if (threadIdx.x < ts.ntypes)
        sl.fold[threadIdx.x] = ts.sec[threadIdx.x + 1] - ts.sec[threadIdx.x];
      __syncthreads();
    }
    int chunk = 0;
    for (int t = 0; t < ts.ntypes; ++t) {
      const int s0 = ts.sec[t], ns = ts.sec[t + 1] - s0;
      int bp = ns;
      if (ns > 0) {
        const TableInfo<float> inf = ts.info[tab_index(ts, t, ti)];
        const float* e0 = p.em + ((size_t)i * nnei + s0) * 4;
        const float last = e0[(ns - 1) * 4];
        for (int b = 0; b < ns; b += 32, ++chunk) {
          if (S > 1 && chunk % S != w) continue;
          const int j = b + lane;
          bool hit = false;
          if (j < ns) {
            const float4 e = ld_prev4(e0 + 4 * j);
            hit = e.x == last && e.y == 0.f && e.z == 0.f && e.w == 0.f;
            float x = e.x;
            const int idx = locate_row(inf, x);
            sl.em[s0 + j] = e;
            sl.xi[s0 + j] = make_float2(x, __int_as_float(idx));
          }
          const unsigned mk = __ballot_sync(kFull, hit);
          if (mk) {
            bp = b + __ffs(mk) - 1;
            if (S == 1) break;
            if (lane == 0) atomicMin(&sl.fold[t], bp);
          }
        }
      }
      if (S == 1) {
        __syncwarp();
        if (lane == 0) {
          if (bp < ns) {
            const float f = (float)(ns - bp);
            float4 e = sl.em[s0 + bp];
            sl.em[s0 + bp] = make_float4(e.x * f, e.y * f, e.z * f, e.w * f);
          }
          sl.cnt[t] = bp < ns ? bp + 1 : ns;
        }
      }
    }
    atom_sync<S>();
    if (S > 1) {
      if (threadIdx.x < ts.ntypes) {
        const int t = threadIdx.x, s0 = ts.sec[t], ns = ts.sec[t + 1] - s0, bp = sl.fold[t];
        if (bp < ns) {
          const float f = (float)(ns - bp);
          float4 e = sl.em[s0 + bp];
          sl.em[s0 + bp] = make_float4(e.x * f, e.y * f, e.z * f, e.w * f);
        }
        sl.cnt[t] = bp < ns ? bp + 1 : ns;
      }
      __syncthreads();
    }
    // ---- main: the section's slots are in ascending distance, so
    //      neighbours that look up the same table row are consecutive (about
    //      a third of them on water): their coefficients stay in registers
    for (int t = 0; t < ts.ntypes; ++t) {
      int lo, hi;
      atom_range<S>(sl.cnt[t], w, lo, hi);
      const int s0 = ts.sec[t];
      const float* tab = ts.table[tab_index(ts, t, ti)];
      float4 c[NS][3];
      int prev = -1;
      for (int j = lo; j < hi; ++j) {
        const float4 e = sl.em[s0 + j];
        const float2 xi = sl.xi[s0 + j];
        const int idx = __float_as_int(xi.y);
        if (idx != prev) {  // uniform over the warp
          prev = idx;
          const float* row = tab + (size_t)idx * rs;
#pragma unroll
          for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int u = 0; u < 3; ++u) c[s][u] = ld_tab4(row + loff[s] + 64 * u);
        }
        const float2 X = dup2(xi.x);
#pragma unroll
        for (int s = 0; s < NS; ++s) {
          float2 V = hi2(c[s][2]);
          V = __ffma2_rn(V, X, lo2(c[s][2]));
          V = __ffma2_rn(V, X, hi2(c[s][1]));
          V = __ffma2_rn(V, X, lo2(c[s][1]));
          V = __ffma2_rn(V, X, hi2(c[s][0]));
          V = __ffma2_rn(V, X, lo2(c[s][0]));
          acc[s][0] = __ffma2_rn(V, dup2(e.x), acc[s][0]);
          acc[s][1] = __ffma2_rn(V, dup2(e.y), acc[s][1]);
          acc[s][2] = __ffma2_rn(V, dup2(e.z), acc[s][2]);
          acc[s][3] = __ffma2_rn(V, dup2(e.w), acc[s][3]);
        }
      }
    }
  }
  // ---- X^T = sum / nnei; X
  const float inv = 1.f / (float)nnei;
  atom_sync<S>();  // the slots are read
  if constexpr (S == 1) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const int k = k0[s];
      if (k < M) {
        xT[k] = make_float4(acc[s][0].x * inv, acc[s][1].x * inv, acc[s][2].x * inv,
                            acc[s][3].x * inv);
        if (k + 16 < M)
          xT[k + 16] = make_float4(acc[s][0].y * inv, acc[s][1].y * inv, acc[s][2].y * inv,
                                   acc[s][3].y * inv);
      }
    }
    __syncwarp();
  } else {
    float4* red = reinterpret_cast<float4*>(base);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const int k = k0[s];
      if (k < M) {
        red[w * M + k] = make_float4(acc[s][0].x, acc[s][1].x, acc[s][2].x, acc[s][3].x);
        if (k + 16 < M)
          red[w * M + k + 16] = make_float4(acc[s][0].y, acc[s][1].y, acc[s][2].y, acc[s][3].y);
      }
    }
    __syncthreads();
    const int k = threadIdx.x;
    if (k < M) {
      float4 v = red[k];
#pragma unroll
      for (int u = 1; u < S; ++u) {
        const float4 q = red[u * M + k];
        v.x += q.x;
        v.y += q.y;
        v.z += q.z;
        v.w += q.w;
      }
      xT[k] = make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv);
    }
    __syncthreads();
  }
  constexpr int NT = S == 1 ? 32 : S * 32;
  const int tid = S == 1 ? lane : threadIdx.x;
  float* Xi = p.X + (size_t)i * 4 * M;
  for (int k = tid; k < M; k += NT) {
    const float4 v = xT[k];
    Xi[k] = v.x;
    Xi[M + k] = v.y;
    Xi[2 * M + k] = v.z;
    Xi[3 * M + k] = v.w;
  }
  // ---- D[k, a] = X_k . X_a, a < 16: a thread's four columns a are the same
  //      on every pass, their X_a stay in registers
  const size_t r = p.drow ? (size_t)p.drow[i] : (size_t)i;
  const int a0 = 4 * (tid & 3);
  float4 xa[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) xa[c] = xT[a0 + c];
  if (p.D_lo) {
    // split for the tensor-core fitting: FP16 hi / lo of c D, c = 2^s from
    // |D_ka| <= |X_k| |X_a| (Cauchy-Schwarz over the 4 rows of X)
    float nk = 0.f, na = 0.f;
    for (int k = lane; k < M; k += 32) {
      const float4 v = xT[k];
      const float q = v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
      nk = fmaxf(nk, q);
      if (k < kAxis) na = fmaxf(na, q);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      nk = fmaxf(nk, __shfl_xor_sync(kFull, nk, o));
      na = fmaxf(na, __shfl_xor_sync(kFull, na, o));
    }
    const float sc = f16_scale_for(sqrtf(nk * na) * 1.0001f);
    __half* dh = static_cast<__half*>(p.D) + r * M * kAxis;
    __half* dl = static_cast<__half*>(p.D_lo) + r * M * kAxis;
    for (int e = 4 * tid; e < M * kAxis; e += 4 * NT) {
      const float4 xk = xT[e >> 4];
      const float v[4] = {dot44(xk, xa[0]), dot44(xk, xa[1]), dot44(xk, xa[2]), dot44(xk, xa[3])};
      st_split4_f16(dh + e, dl + e, v, sc);
    }
    if (tid == 0) p.D_rs[r] = 1.f / sc;
    return;
  }
  float* d = static_cast<float*>(p.D) + r * M * kAxis;
  for (int e = 4 * tid; e < M * kAxis; e += 4 * NT) {
    const float4 xk = xT[e >> 4];
    *reinterpret_cast<float4*>(d + e) =
        make_float4(dot44(xk, xa[0]), dot44(xk, xa[1]), dot44(xk, xa[2]), dot44(xk, xa[3]));
  }
}

// --------------------------------------------------------------- backward --
// dy [M] and X^T [M] while dX is formed (and the S warps' parts of dD^T X),
// then the slots over them (dy is in registers by then)
template <int S>
__host__ __device__ constexpr size_t bwd_bytes(int nnei, int M) {
  const size_t sl = slot_bytes(nnei), dx = (size_t)M * 32 + (S > 1 ? S * 256 : 0);
  return sl > dx ? sl : dx;
}

// Phase-1 sums of one neighbour over a lane's outputs (16 lanes a
// neighbour): p[m] = sum_k P_k dy[m][k], p[4] = sum_k P'_k (e . dy[., k]).
// Full blocks in packed FMAs over the pair k, k + 16; a last block of at
// most 16 outputs (NK odd) by even and odd coefficients.
template <int NK>
__device__ __forceinline__ void bwd_sums(float* p, const float* __restrict__ row, int loff,
                                         int loff_last, float x, const float4& e,
                                         const float (&dr)[NK][4]) {
  constexpr int NP = NK / 2;
  const float2 X = dup2(x);
  const float2 E[4] = {dup2(e.x), dup2(e.y), dup2(e.z), dup2(e.w)};
  float2 P[4], PX = make_float2(0.f, 0.f);
#pragma unroll
  for (int m = 0; m < 4; ++m) P[m] = make_float2(0.f, 0.f);
#pragma unroll
  for (int b = 0; b < NP; ++b) {
    const float* r = row + (b == NP - 1 && !(NK & 1) ? loff_last : loff) + b * kBlk;
    float4 c[3];
#pragma unroll
    for (int u = 0; u < 3; ++u) c[u] = ld_tab4(r + 64 * u);
    float2 V = hi2(c[2]), D = V;
    V = __ffma2_rn(V, X, lo2(c[2]));
    D = __ffma2_rn(D, X, V);
    V = __ffma2_rn(V, X, hi2(c[1]));
    D = __ffma2_rn(D, X, V);
    V = __ffma2_rn(V, X, lo2(c[1]));
    D = __ffma2_rn(D, X, V);
    V = __ffma2_rn(V, X, hi2(c[0]));
    D = __ffma2_rn(D, X, V);
    V = __ffma2_rn(V, X, lo2(c[0]));
    float2 Y = make_float2(0.f, 0.f);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const float2 d = make_float2(dr[2 * b][m], dr[2 * b + 1][m]);
      P[m] = __ffma2_rn(V, d, P[m]);
      Y = m == 0 ? __fmul2_rn(E[m], d) : __ffma2_rn(E[m], d, Y);
    }
    PX = __ffma2_rn(D, Y, PX);
  }
  if (NK & 1) {
    const float* r = row + loff_last + NP * kBlk;
    Coef<float> c;
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const float4 q = ld_tab4(r + 64 * u);
      c.p[u] = make_float2(q.x, q.z);
    }
    const XPow<float> xp(x);
    float v, d;
    tab_val_slope(c, xp, v, d);
    const float* g = dr[NK - 1];
#pragma unroll
    for (int m = 0; m < 4; ++m) P[m].x = fmaf(v, g[m], P[m].x);
    PX.x = fmaf(d, e.x * g[0] + e.y * g[1] + e.z * g[2] + e.w * g[3], PX.x);
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) p[m] = P[m].x + P[m].y;
  p[4] = PX.x + PX.y;
}

constexpr int bwd_warps(int U) { return U == 1 ? 24 : 16; }  // resident warps an SM

template <int NK, int W, int S, int U>
__global__ void __launch_bounds__(W * 32, bwd_warps(U) / W)
    k_bwd_blk(const __grid_constant__ DescBwdArgs p, const __grid_constant__ TabSet<float> ts,
              int nloc, int M, float inv_rw, int pf_dist) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  grid_wait();
  grid_release();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = S == 1 ? blockIdx.x * W + warp : blockIdx.x;
  if (i >= nloc) return;  // S = 1: uniform over the warp; S > 1: the grid is exact
  const int w = S == 1 ? 0 : warp;
  const int nnei = ts.sec[ts.ntypes];
  if (S == 1) {
    // the atom pf_dist ahead (about one wave of resident warps later): its
    // dE/dD row, X and env rows prefetched into L2, so that the warp that
    // takes it finds its first loads in L2 rather than in DRAM
    const int ip = i + pf_dist;
    if (pf_dist > 0 && ip < nloc) {
      const size_t rp = p.drow ? (size_t)p.drow[ip] : (size_t)ip;
      const char* pd = reinterpret_cast<const char*>(p.dD + rp * M * kAxis);
      const char* px = reinterpret_cast<const char*>(p.X + (size_t)ip * 4 * M);
      const char* pe = reinterpret_cast<const char*>(p.em + (size_t)ip * nnei * 4);
      const int ld = (4 * M * kAxis + 127) / 128, lx = (16 * M + 127) / 128,
                le = (16 * nnei + 127) / 128;
      for (int l = lane; l < ld + lx + le; l += 32)
        prefetch_l2(l < ld        ? pd + 128 * l
                    : l < ld + lx ? px + 128 * (l - ld)
                                  : pe + 128 * (l - ld - lx));
    }
  }
  const int ti = p.atype[i];
  if (ti < 0) return;  // uniform over the atom's warps
  unsigned char* base = smem_raw + (S == 1 ? (size_t)warp * bwd_bytes<S>(nnei, M) : 0);
  float4* dyT = reinterpret_cast<float4*>(base);
  float4* xT = dyT + M;
  float* dys = reinterpret_cast<float*>(dyT);
  constexpr int NT = S == 1 ? 32 : S * 32;
  const int tid = S == 1 ? lane : threadIdx.x;
  {
    const float* Xi = p.X + (size_t)i * 4 * M;
    constexpr int NX = (16 * NK + NT - 1) / NT;  // every load before the first store
    float4 v[NX];
#pragma unroll
    for (int u = 0; u < NX; ++u) {
      const int k = tid + NT * u;
      if (k < M)
        v[u] = make_float4(ld_prev(Xi + k), ld_prev(Xi + M + k), ld_prev(Xi + 2 * M + k),
                           ld_prev(Xi + 3 * M + k));
    }
#pragma unroll
    for (int u = 0; u < NX; ++u) {
      const int k = tid + NT * u;
      if (k < M) xT[k] = v[u];
    }
  }
  atom_sync<S>();
  // ---- dX = dD X[:, :A] + (dD^T X)[:A].  Lanes walk the row of dD in 16-byte
  //      pieces, coalesced: piece q of output k (a = 4 q ..) is lane q of a
  //      quad.  It adds its four columns to the first product (summed over
  //      the quad: lane q ends with component m = q of dX[k]), and its
  //      part of the second, which stays in registers over all k.
  {
    const int q = lane & 3;
    const size_t r = p.drow ? (size_t)p.drow[i] : (size_t)i;
    const float* g_i = p.dD + r * M * kAxis;
    float2 xa[4][2];  // X[m][4 q + 0, 1], X[m][4 q + 2, 3]
    {
      float4 v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) v[c] = xT[4 * q + c];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        xa[0][h] = make_float2(v[2 * h].x, v[2 * h + 1].x);
        xa[1][h] = make_float2(v[2 * h].y, v[2 * h + 1].y);
        xa[2][h] = make_float2(v[2 * h].z, v[2 * h + 1].z);
        xa[3][h] = make_float2(v[2 * h].w, v[2 * h + 1].w);
      }
    }
    float2 sa[4][2];  // [c][m pair]
#pragma unroll
    for (int c = 0; c < 4; ++c) sa[c][0] = sa[c][1] = make_float2(0.f, 0.f);
    constexpr int BT = S == 1 ? 7 : 4;  // loads in flight
    const int nit = (M + 7) >> 3;
    for (int it0 = w; it0 < nit; it0 += S * BT) {
      float4 g[BT];
#pragma unroll
      for (int u = 0; u < BT; ++u) {
        const int k = (it0 + S * u) * 8 + (lane >> 2);
        g[u] = k < M ? ld_prev4(g_i + k * kAxis + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < BT; ++u) {
        const int k = (it0 + S * u) * 8 + (lane >> 2);
        if ((it0 + S * u) * 8 >= M) break;  // uniform
        float d[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const float2 h = __ffma2_rn(hi2(g[u]), xa[m][1], __fmul2_rn(lo2(g[u]), xa[m][0]));
          d[m] = h.x + h.y;
        }
        halve<2>(d, 2, (lane & 2) != 0);
        halve<1>(d, 1, (lane & 1) != 0);
        if (k < M) dys[4 * k + q] = d[0];
        const float4 xk = xT[min(k, M - 1)];
        const float gc[4] = {g[u].x, g[u].y, g[u].z, g[u].w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          sa[c][0] = __ffma2_rn(dup2(gc[c]), lo2(xk), sa[c][0]);
          sa[c][1] = __ffma2_rn(dup2(gc[c]), hi2(xk), sa[c][1]);
        }
      }
    }
    float s[16];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        s[4 * c + 2 * h] = sa[c][h].x;
        s[4 * c + 2 * h + 1] = sa[c][h].y;
      }
    halve<8>(s, 16, (lane & 16) != 0);
    halve<4>(s, 8, (lane & 8) != 0);
    halve<2>(s, 4, (lane & 4) != 0);
    // column a = 4 q + c, components m, m + 1
    const int c = (lane & 16 ? 2 : 0) + (lane & 8 ? 1 : 0), m = lane & 4 ? 2 : 0;
    const int at = 4 * (4 * q + c) + m;
    atom_sync<S>();
    if (S == 1) {
      dys[at] += s[0];
      dys[at + 1] += s[1];
      __syncwarp();
    } else {
      float* part = reinterpret_cast<float*>(xT + M);  // [S][64]
      part[64 * w + at] = s[0];
      part[64 * w + at + 1] = s[1];
      __syncthreads();
      if (threadIdx.x < 64) {
        float v = part[threadIdx.x];
#pragma unroll
        for (int u = 1; u < S; ++u) v += part[64 * u + threadIdx.x];
        dys[threadIdx.x] += v;
      }
      __syncthreads();
    }
  }
  // phase 1 mapping: 16 lanes per neighbour; lane t16 owns outputs
  // k = t16 + 16 q and keeps their dy = dX / nnei in registers
  const int n = lane >> 4, t16 = lane & 15;
  const float inv = 1.f / (float)nnei;
  float dr[NK][4];
#pragma unroll
  for (int q = 0; q < NK; ++q) {
    const int k = t16 + 16 * q;
    const float4 d = k < M ? dyT[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    dr[q][0] = d.x * inv;
    dr[q][1] = d.y * inv;
    dr[q][2] = d.z * inv;
    dr[q][3] = d.w * inv;
  }
  atom_sync<S>();

  // ---- prepass over filled slots (the slots replace dy and X^T)
  const SlotArr sl = carve(base, nnei);
  const int* nl_i = p.nlist_ext + (size_t)i * nnei;
  {
    int chunk = 0;
    for (int t = 0; t < ts.ntypes; ++t) {
      const int s0 = ts.sec[t], ns = ts.sec[t + 1] - s0;
      const int nv = filled_prefix(nl_i + s0, ns);
      const TableInfo<float> inf = ts.info[tab_index(ts, t, ti)];
      for (int b = 0; b < nv; b += 32, ++chunk) {
        if (S > 1 && chunk % S != w) continue;
        const int j = b + lane;
        if (j < nv) {
          const float4 e = ld_prev4(p.em + ((size_t)i * nnei + s0 + j) * 4);
          float x = e.x;
          const int idx = locate_row(inf, x);
          sl.em[s0 + j] = e;
          sl.xi[s0 + j] = make_float2(x, __int_as_float(idx));
        }
      }
      if (tid == 0) sl.cnt[t] = nv;
    }
  }
  atom_sync<S>();

  // ---- phase 1: tabulation gradient, 16 lanes per neighbour
  {
    const int rs = ((M + 31) >> 5) * kBlk;
    // the lane's piece in a full block, and in the last one (a lane past M
    // repeats a valid piece against dy = 0)
    const int loff = 4 * t16, lim = min(16, M - 32 * ((NK - 1) / 2)),
              loff_last = 4 * min(t16, lim - 1);
    for (int t = 0; t < ts.ntypes; ++t) {
      int lo, hi;
      atom_range<S>(sl.cnt[t], w, lo, hi);
      const int s0 = ts.sec[t];
      const float* tab = ts.table[tab_index(ts, t, ti)];
      for (int j0 = lo; j0 < hi; j0 += 2 * U) {
        float s[U][5];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          // a slot past the end re-evaluates slot j0 (always filled); its
          // sums are dropped
          const int j = j0 + n + 2 * u, js = s0 + (j < hi ? j : j0);
          const float2 xi = sl.xi[js];
          bwd_sums<NK>(s[u], tab + (size_t)__float_as_int(xi.y) * rs, loff, loff_last, xi.x,
                       sl.em[js], dr);
        }
        // dE/d em[j, :] = (p0 + p4, p1, p2, p3) (em_x is em[:, 0]) summed over
        // the 16-lane group by a reduce-scatter: lane t16 ends with
        // component t16 >> 2
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float v[4] = {s[u][0] + s[u][4], s[u][1], s[u][2], s[u][3]};
          halve<2>(v, 8, (t16 & 8) != 0);
          halve<1>(v, 4, (t16 & 4) != 0);
          v[0] += __shfl_xor_sync(kFull, v[0], 2);
          v[0] += __shfl_xor_sync(kFull, v[0], 1);
          const int j = j0 + n + 2 * u;
          if ((t16 & 3) == 0 && j < hi) reinterpret_cast<float*>(&sl.em[s0 + j])[t16 >> 2] = v[0];
        }
      }
    }
  }
  atom_sync<S>();

  // ---- phase 2: threads over filled slots: env-matrix derivative row
  //      d em / d x_i (env_mat.cc:157-204) / std, force and virial scatter
  const int f = p.geo.atom_frame[i];
  const int aoff = p.geo.frame_aoff[f];
  const float* xc = p.ext_coord + 3 * (size_t)p.geo.frame_eoff[f];
  const int* emap = p.ext_map + p.geo.frame_eoff[f];
  const int il = i - aoff;
  const float xi = xc[3 * il], yi = xc[3 * il + 1], zi = xc[3 * il + 2];
  const float* isd = p.inv_std + (size_t)ti * nnei * 4;
  float v[16];  // virial (9), centre force (3)
#pragma unroll
  for (int q = 0; q < 16; ++q) v[q] = 0.f;
  for (int t = 0; t < ts.ntypes; ++t) {
    const int s0 = ts.sec[t], nv = sl.cnt[t];
    for (int jj = tid; jj < nv; jj += NT) {
      const int s = s0 + jj;
      const int je = nl_i[s];
      const float rr[3] = {xc[3 * je] - xi, xc[3 * je + 1] - yi, xc[3 * je + 2] - zi};
      const float nr2 = rr[0] * rr[0] + rr[1] * rr[1] + rr[2] * rr[2];
      const float inr = rsqrtf(nr2);
      const float nr = nr2 * inr;
      const float inr2 = inr * inr;
      const float inr4 = inr2 * inr2;
      const float inr3 = inr4 * nr;
      // the switch (switcher.h:60-83) and its slope
      float sw = 1.f, dsw = 0.f;
      if (nr >= p.rmin) {
        const float u = (nr - p.rmin) * inv_rw;
        const float c = -6.f * u * u + 15.f * u - 10.f;
        sw = u * u * u * c + 1.f;
        dsw = (3.f * u * u * c + u * u * u * (-12.f * u + 15.f)) * inv_rw;
        if (!(nr < p.rmax)) sw = dsw = 0.f;
      }
      const float ev[4] = {inr, rr[0] * inr2, rr[1] * inr2, rr[2] * inr2};
      const float4 net = sl.em[s];
      const float4 sd = ld_row4(isd + (size_t)s * 4);
      const float gw[4] = {net.x * sd.x, net.y * sd.y, net.z * sd.z, net.w * sd.w};
      float v3[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        float a = gw[0] * (rr[d] * inr3 * sw - ev[0] * dsw * rr[d] * inr);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float tt = 2.f * rr[c] * rr[d] * inr4;
          if (c == d) tt -= inr2;
          a += gw[1 + c] * (tt * sw - ev[1 + c] * dsw * rr[d] * inr);
        }
        v3[d] = a;
      }
      const size_t jl = (size_t)(aoff + emap[je]) * 3;
      if (p.force_fx)
        fx_add3(p.force_fx + jl, v3, FxScale<float>::force);
      else
        scatter3(p.force + jl, v3);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int b = 0; b < 3; ++b) v[a * 3 + b] += v3[a] * rr[b];
        v[9 + a] += v3[a];
      }
    }
  }
  halve<8>(v, 16, (lane & 16) != 0);
  halve<4>(v, 8, (lane & 8) != 0);
  halve<2>(v, 4, (lane & 4) != 0);
  halve<1>(v, 2, (lane & 2) != 0);
  v[0] += __shfl_xor_sync(kFull, v[0], 1);
  const int q = lane >> 1;  // the value this lane holds
  if (lane & 1) return;
  if (q < 9) {
    double* va = p.vir_acc + f * 9 + q;
    if (p.force_fx)  // the accumulator holds fixed-point sums in this mode
      fx_add(reinterpret_cast<long long*>(va), v[0], FxScale<float>::virial);
    else
      atomicAdd(va, (double)v[0]);
  } else if (q < 12) {
    const size_t at = (size_t)i * 3 + (q - 9);
    if (p.force_fx)
      fx_add(p.force_fx + at, -v[0], FxScale<float>::force);
    else
      atomicAdd(p.force + at, -v[0]);
  }
}

// ------------------------------------------------------------- host side --
// Below these numbers of atoms the four warps of a CTA share one atom: with
// few atoms an SM, a warp per atom is a serial walk over ~85 neighbours with
// too few warps to hide its loads; above, the repeated location of the
// slots, the barriers and the sums across warps cost more.  Measured on
// water, shared / own, us: forward 192 atoms 18.4 / 24.4, 1200: 24.4 / 30.5,
// 1800: 36.7 / 31.3; backward 192: 31.7 / 48.1, 768: 39.9 / 50.1, 1200: 52.2
// / 52.2, 1800: 58.3 / 54.2.  The forward takes eight warps an atom while all
// CTAs are resident at once, four an SM (eight / four, us: 48 atoms 14.5 /
// 19.0, 192: 14.5 / 18.6, 600: 16.6 / 20.5, 1200: 27.0 / 24.5; the backward,
// two CTAs an SM, would gain under 1 us up to 300 atoms and lose 6 at 600).
// The line is on the number of atoms alone, never on the tuner's choice: an
// atom's sums are grouped by the warps that share it.
constexpr int kShareFwd8 = 152 * 4, kShareFwd = 152 * 10, kShareBwd = 152 * 8;

// shared memory of a launch, and the smallest shared-memory carveout that
// holds the resident CTAs: the rest of the unified L1 caches table rows
template <typename K>
void set_smem(K kern, size_t smem, int ctas_sm) {
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int per_sm = ctas_sm * (int)(smem + 1024);
  cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                       per_sm >= 228 * 1024 ? 100 : (per_sm * 100 + 228 * 1024 - 1) / (228 * 1024));
}

template <int NS, int W, int S>
void launch_fwd(const DescFwdArgs& a, const TabSet<float>& ts, int nloc, int M, cudaStream_t st) {
  auto kern = k_fwd_blk<NS, W, S>;
  const int nnei = ts.sec[ts.ntypes];
  const size_t smem = (S == 1 ? W : 1) * fwd_bytes<S>(nnei, M);
  set_smem(kern, smem, 32 / W);
  launch_dep(kern, dim3((unsigned)(S == 1 ? (nloc + W - 1) / W : nloc)), dim3(W * 32), smem, st, a,
             ts, nloc, M);
}

template <int NS>
void fwd_width(const DescFwdArgs& a, const TabSet<float>& ts, int nloc, int M, int W,
               cudaStream_t st) {
  if (nloc <= kShareFwd8)
    launch_fwd<NS, 8, 8>(a, ts, nloc, M, st);
  else if (nloc < kShareFwd)
    launch_fwd<NS, 4, 4>(a, ts, nloc, M, st);
  else if (W == 1)
    launch_fwd<NS, 1, 1>(a, ts, nloc, M, st);
  else if (W == 2)
    launch_fwd<NS, 2, 1>(a, ts, nloc, M, st);
  else
    launch_fwd<NS, 4, 1>(a, ts, nloc, M, st);
}

template <int NK, int W, int S, int U>
void launch_bwd(const DescBwdArgs& a, const TabSet<float>& ts, int nloc, int M, cudaStream_t st) {
  auto kern = k_bwd_blk<NK, W, S, U>;
  const int nnei = ts.sec[ts.ntypes];
  const size_t smem = (S == 1 ? W : 1) * bwd_bytes<S>(nnei, M);
  set_smem(kern, smem, bwd_warps(U) / W);
  // prefetch distance: the warps resident on the device at once (queried
  // again only when the device or the shared-memory size changes)
  thread_local int c_dev = -1, c_pf = 0;
  thread_local size_t c_smem = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev != c_dev || smem != c_smem) {
    int sms = 0, ctas = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, kern, W * 32, smem);
    c_dev = dev;
    c_smem = smem;
    c_pf = sms * ctas * W;
  }
  launch_dep(kern, dim3((unsigned)(S == 1 ? (nloc + W - 1) / W : nloc)), dim3(W * 32), smem, st, a,
             ts, nloc, M, 1.f / (a.rmax - a.rmin), c_pf);
}

template <int NK, int U>
void bwd_width(const DescBwdArgs& a, const TabSet<float>& ts, int nloc, int M, int W,
               cudaStream_t st) {
  if (nloc < kShareBwd)
    launch_bwd<NK, 4, 4, U>(a, ts, nloc, M, st);
  else if (W == 1)
    launch_bwd<NK, 1, 1, U>(a, ts, nloc, M, st);
  else if (W == 2)
    launch_bwd<NK, 2, 1, U>(a, ts, nloc, M, st);
  else
    launch_bwd<NK, 4, 1, U>(a, ts, nloc, M, st);
}

__global__ void k_table_blocked(float* __restrict__ dst, const float* __restrict__ src, int nrow,
                                int M) {
  const int rs = ((M + 31) >> 5) * kBlk;
  const size_t n = (size_t)nrow * rs;
  for (size_t u = (size_t)blockIdx.x * blockDim.x + threadIdx.x; u < n;
       u += (size_t)gridDim.x * blockDim.x) {
    const size_t r = u / rs;
    const int rem = (int)(u - r * rs), b = rem / kBlk, w = rem - b * kBlk;
    const int c = w >> 6, t = (w >> 2) & 15, h = w & 3;
    const int k = 32 * b + t + 16 * (h & 1), a = 2 * c + (h >> 1);
    dst[u] = k < M ? src[r * 6 * M + 6 * k + a] : 0.f;
  }
}

}  // namespace

int desc_fwd_share(int nloc) { return nloc <= kShareFwd8 ? 8 : nloc < kShareFwd ? 4 : 1; }
int desc_bwd_share(int nloc) { return nloc < kShareBwd ? 4 : 1; }

int desc_fwd_blk(const DescFwdArgs& a, const TabSet<float>& ts, int nloc, int M, int W,
                 cudaStream_t st) {
  if (M <= 64)
    fwd_width<1>(a, ts, nloc, M, W, st);
  else
    fwd_width<2>(a, ts, nloc, M, W, st);
  GBDP_CHECK_LAUNCH("se_a_descriptor_fwd_blk");
  return GBDP_OK;
}

int desc_bwd_blk(const DescBwdArgs& a, const TabSet<float>& ts, int nloc, int M, int W, int U,
                 cudaStream_t st) {
#define GBDP_BLK_CASE(N)                      \
  case N:                                     \
    if (U == 2)                               \
      bwd_width<N, 2>(a, ts, nloc, M, W, st); \
    else                                      \
      bwd_width<N, 1>(a, ts, nloc, M, W, st); \
    break;
  switch ((M + 15) / 16) {
    GBDP_BLK_CASE(1)
    GBDP_BLK_CASE(2)
    GBDP_BLK_CASE(3)
    GBDP_BLK_CASE(4)
    GBDP_BLK_CASE(5)
    GBDP_BLK_CASE(6)
    GBDP_BLK_CASE(7)
    GBDP_BLK_CASE(8)
  }
#undef GBDP_BLK_CASE
  GBDP_CHECK_LAUNCH("se_a_descriptor_bwd_blk");
  return GBDP_OK;
}

}  // namespace gbdp

using namespace gbdp;

extern "C" size_t gbdp_table_blocked_row_elems(int last_layer_size) {
  return last_layer_size < 1 ? 0 : (size_t)((last_layer_size + 31) / 32) * kBlk;
}

extern "C" int gbdp_table_to_blocked_f32(float* dst, const float* src, int nrow,
                                         int last_layer_size, gbdp_stream stream) {
  const int M = last_layer_size;
  GBDP_REQUIRE(M >= 1 && M <= 4096 && nrow >= 0, "table_to_blocked: nrow %d, M %d", nrow, M);
  if (nrow == 0) return GBDP_OK;
  GBDP_REQUIRE(dst && src, "table_to_blocked: null pointer");
  GBDP_REQUIRE(((uintptr_t)dst & 127) == 0, "table_to_blocked: dst not 128-byte aligned");
  const size_t n = (size_t)nrow * gbdp_table_blocked_row_elems(M);
  const unsigned blocks = (unsigned)((n + 255) / 256 < 152 * 16 ? (n + 255) / 256 : 152 * 16);
  k_table_blocked<<<blocks, 256, 0, (cudaStream_t)stream>>>(dst, src, nrow, M);
  GBDP_CHECK_LAUNCH("table_to_blocked");
  return GBDP_OK;
}
