// What the fused descriptor kernels share (fused.cu: k-planar tables;
// desc_blk.cu: blocked FP32 tables).
#pragma once

#include "common.cuh"

namespace gbdp {

// One call's arguments of the descriptor on blocked tables.
struct DescFwdArgs {
  float* X;
  void* D;      // FP32, or the FP16 hi part with D_lo
  void* D_lo;   // optional FP16 lo part
  float* D_rs;  // with D_lo: inverse row scales
  const float* em;
  const int *atype, *drow;
};
struct BwdGeom {
  const int* atom_frame;   // [nloc_total] frame of each centre
  const int* frame_aoff;   // [nframes] first local atom of each frame
  const int* frame_eoff;   // [nframes] first extended slot of each frame
};
struct DescBwdArgs {
  float* force;
  double* vir_acc;
  long long* force_fx;
  const float *X, *dD;
  const int* drow;
  const float* em;
  const int* nlist_ext;
  const float* ext_coord;
  const int *ext_map, *atype;
  const float* inv_std;
  BwdGeom geo;
  float rmin, rmax;
};

constexpr int kMaxTab = 16;
constexpr int kMaxTypes = 4;
constexpr int kAxis = 16;

template <typename T>
struct TabSet {
  const T* table[kMaxTab];
  TableInfo<T> info[kMaxTab];
  int ntypes;
  int one_side;  // 1: table per neighbour type; 0: per (neighbour, centre)
  int ps;        // plane pitch of the k-planar tables (elements)
  int sec[kMaxTab + 1];
};

template <typename T>
__device__ __forceinline__ int tab_index(const TabSet<T>& ts, int tj, int ti) {
  return ts.one_side ? tj : tj * ts.ntypes + ti;
}

// plane pitch of the k-planar layout: 2 M elements rounded up to 128 bytes
template <typename T>
__host__ __device__ constexpr int kp_pitch(int M) {
  return sizeof(T) == 4 ? (2 * M + 31) & ~31 : (2 * M + 15) & ~15;
}

template <typename T>
struct Vec;
template <>
struct Vec<float> {
  using v2 = float2;
  using v4 = float4;
};
struct alignas(32) dbl4 {
  double x, y, z, w;
};
template <>
struct Vec<double> {
  using v2 = double2;
  using v4 = dbl4;
};
template <typename T>
using V4 = typename Vec<T>::v4;

// L1 policy.  The table rows are the only data the kernels re-read across
// atoms; everything per atom (env rows, X, dE/dD) streams through once or
// twice.  Table loads carry L1::evict_last, per-atom rows L1::no_allocate
// (read once) or L1::evict_first (read twice), so that the hot band of
// table rows stays resident in L1.
__device__ __forceinline__ float2 ld_tab2(const float2* p) {
  float2 v;
  asm("ld.global.nc.L1::evict_last.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 ld_tab2(const double2* p) {
  double2 v;
  asm("ld.global.nc.L1::evict_last.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

// a non-binding prefetch of the 128-byte line holding p into L2
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// one row of 4 values (16-byte aligned), not allocated in L1
__device__ __forceinline__ float4 ld_stream4(const float* p) {
  float4 v;
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p));
  return v;
}
__device__ __forceinline__ dbl4 ld_stream4(const double* p) {
  dbl4 v;
  asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.z), "=d"(v.w) : "l"(p + 2));
  return v;
}
__device__ __forceinline__ float ld_stream(const float* p) {
  float v;
  asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_stream(const double* p) {
  double v;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// The same for data of the kernel launched directly before (dependent
// launches): plain loads, after the wait.
__device__ __forceinline__ float4 ld_prev4(const float* p) {
  float4 v;
  asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ float ld_prev(const float* p) {
  float v;
  asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

// a row of 4 values read twice by the same warp: first out of L1
__device__ __forceinline__ float4 ld_first4(const float* p) {
  float4 v;
  asm("ld.global.nc.L1::evict_first.v4.f32 {%0, %1, %2, %3}, [%4];"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p));
  return v;
}
__device__ __forceinline__ dbl4 ld_first4(const double* p) {
  dbl4 v;
  asm("ld.global.nc.L1::evict_first.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  asm("ld.global.nc.L1::evict_first.v2.f64 {%0, %1}, [%2];" : "=d"(v.z), "=d"(v.w) : "l"(p + 2));
  return v;
}
__device__ __forceinline__ float ld_first(const float* p) {
  float v;
  asm("ld.global.nc.L1::evict_first.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_first(const double* p) {
  double v;
  asm("ld.global.nc.L1::evict_first.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// one row of 4 values through the default path (16-byte aligned)
__device__ __forceinline__ float4 ld_row4(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}
__device__ __forceinline__ dbl4 ld_row4(const double* p) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p));
  const double2 b = __ldg(reinterpret_cast<const double2*>(p) + 1);
  return dbl4{a.x, a.y, b.x, b.y};
}

__device__ __forceinline__ void st_row4(float* p, const float4& v) {
  *reinterpret_cast<float4*>(p) = v;
}
__device__ __forceinline__ void st_row4(double* p, const dbl4& v) {
  reinterpret_cast<double2*>(p)[0] = double2{v.x, v.y};
  reinterpret_cast<double2*>(p)[1] = double2{v.z, v.w};
}

// --------------------------------------------------------------- backward --
template <typename T>
__device__ __forceinline__ void spline5_d(T& vv, T& dd, T xx, T rmin, T rmax) {
  if (xx < rmin) {
    dd = T(0);
    vv = T(1);
  } else if (xx < rmax) {
    T uu = (xx - rmin) / (rmax - rmin);
    T du = T(1) / (rmax - rmin);
    vv = uu * uu * uu * (T(-6) * uu * uu + T(15) * uu - T(10)) + T(1);
    dd = (T(3) * uu * uu * (T(-6) * uu * uu + T(15) * uu - T(10)) +
          uu * uu * uu * (T(-12) * uu + T(15))) *
         du;
  } else {
    dd = T(0);
    vv = T(0);
  }
}

__device__ __forceinline__ float rsqrt_t(float x) { return rsqrtf(x); }
__device__ __forceinline__ double rsqrt_t(double x) { return rsqrt(x); }

// Number of filled slots of a section: the env kernel fills each type
// section from its start, so the filled slots are a prefix.
__device__ __forceinline__ int filled_prefix(const int* __restrict__ nl, int ns) {
  const int lane = threadIdx.x & 31;
  int n = 0;
  for (int b = 0; b < ns; b += 32) {
    const bool ok = b + lane < ns && nl[b + lane] >= 0;
    n += __popc(__ballot_sync(kFull, ok));
  }
  return n;
}


// desc_blk.cu: the descriptor on blocked tables, warps per CTA W (1, 2 or 4,
// one atom each; without meaning where warps share an atom), U neighbours in
// flight per group; and the warps that share an atom, by the number of atoms
int desc_fwd_share(int nloc);
int desc_bwd_share(int nloc);
int desc_fwd_blk(const DescFwdArgs& a, const TabSet<float>& ts, int nloc, int M, int W,
                 cudaStream_t st);
int desc_bwd_blk(const DescBwdArgs& a, const TabSet<float>& ts, int nloc, int M, int W, int U,
                 cudaStream_t st);

}  // namespace gbdp
