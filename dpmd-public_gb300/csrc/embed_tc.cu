// Embedding net of the uncompressed se_e2_a descriptor on the 5th-generation
// tensor cores (sm_103a), fused with the G^T R contraction so that the
// nloc x nnei x M embedding never reaches HBM.
//
// Reference semantics: DescrptBlockSeA.forward
// (deepmd/pt/model/descriptor/se_a.py:750-866) with EmbeddingNet /
// MLPLayer (deepmd/pt/model/network/mlp.py:188-219): per neighbour-type
// section t (and centre type when !type_one_side), s = em[..., 0],
// G = net(s) with 1 -> N1 -> N2 -> N3 tanh layers (identity or [x, x]
// skips), X = sum_j em[j, :]^T G[j, :] / nnei; D = X^T X[:, :A].
//
// Precision: layers 2 and 3 are BF16 tcgen05.mma (kind::f16, FP32
// accumulation in tensor memory); layer 1, the activations (tanh.approx),
// the skips, G^T R and D are FP32.
//
// A tile is 128 rows, one thread each (thread r <-> TMEM lane r), 32 a warp;
// the rows of a warp are its own atom's (see the row mapping below); one
// warpgroup per CTA, three CTAs per SM forward and two backward.
//   layer 1 (SIMT)  -> A (bf16, 128 x 64, SW128 K-major, shared)
//   MMA  D2 = A W2   (N 64)
//   epilogue 2       -> A (bf16), the layer-2 output in FP32 registers
//   MMA  D3 = A W3   (N 128)
//   epilogue 3       -> G, 32 columns at a time through the warp's part of A
//   G^T R            -> X of the warp's atom (FP32, registers, lane = column)
// With two atoms' sections concatenated over tiles, both nets restaged for
// every pair of atoms, padding rows evaluated one by one and G of 128 rows in
// shared memory (8 warps an SM), 6,141 atoms took 342 us forward and 306 us
// backward; now 151 and 176 us, same bits.
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"

namespace gbdp {
namespace {

// ----------------------------------------------------- per-net parameters --
// One block of kNetBytes per embedding net (built on the host): the weight
// images in the exact shared-memory layout the MMAs read (bf16, K-major,
// 128-byte swizzle: 16-byte piece p of row n at piece p ^ (n & 7), rows of
// 128 B, K beyond 64 in further [rows x 128 B] chunks), then FP32 params.
constexpr int kNetB2 = 0;       // W2^T  [64 n][64 k]       8 KiB
constexpr int kNetB3 = 8192;    // W3^T  [128 n][64 k]     16 KiB
constexpr int kNetPar = 24576;  // w1[64] b1[64] b2[64] b3[128] (FP32)
constexpr int kNetB3T = 26624;  // W3    [64 n][128 k]     16 KiB (backward)
constexpr int kNetB2T = 43008;  // W2    [64 n][64 k]       8 KiB (backward)
constexpr int kNetBytes = 51200;
constexpr int kNetFwdBytes = kNetPar + 320 * 4;  // what the forward stages
constexpr int kParW1 = 0, kParB1 = 64, kParB2 = 128, kParB3 = 192;

constexpr int kRows = 128;
constexpr int kSlot = 26624;   // one staged net, forward part (1024-aligned)
constexpr size_t kFwdBytes = 2 * kSlot + 16384 + kRows * 16 + 64;  // the forward's shared memory
constexpr int kMaxTypes = 8;

struct EmbArgs {
  float* X;           // [nloc, 4, N3]
  void* D;            // [rows, N3 * A]: FP32, or FP16 hi with D_lo
  void* D_lo;         // optional FP16 lo part (split for the tensor-core fitting)
  float* D_rs;        // with D_lo: [rows] inverse scale of each D row
  const int* drow;    // D row of each atom (null: the atom index)
  const float* em;    // [nloc, nnei, 4]
  const int* units;   // [nunits, 2] atom pairs of one centre type (-1: none)
  const int* atype;   // [nloc]
  const unsigned char* nets;
  int* status;
  int nunits, ntypes, type_one_side, nloc, nnei, A;
  int sec[kMaxTypes + 1];
};

// ------------------------------------------------------------------ PTX --
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);  // start address
  d |= (uint64_t)1 << 16;                    // leading byte offset (unused with swizzle)
  d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset: 8 rows x 128 B
  d |= (uint64_t)1 << 46;                    // descriptor version (sm_100 family)
  d |= (uint64_t)2 << 61;                    // 128-byte swizzle
  return d;
}

// kind::f16 with BF16 A and B, FP32 D, both K-major, M = 128
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                          uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

// the same load without the wait: several may be in flight before one
// tcgen05.wait::ld (tmem_wait) makes all their registers valid
__device__ __forceinline__ void tmem_ld16_nw(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// one row's 16-byte piece u (columns 8u..8u+7) of a [128 x 64] bf16 SW128 tile
__device__ __forceinline__ void st_piece(unsigned char* tile, int r, int u, const float* v8) {
  uint4 w;
  w.x = pack_bf16(v8[0], v8[1]);
  w.y = pack_bf16(v8[2], v8[3]);
  w.z = pack_bf16(v8[4], v8[5]);
  w.w = pack_bf16(v8[6], v8[7]);
  *reinterpret_cast<uint4*>(tile + r * 128 + ((u ^ (r & 7)) << 4)) = w;
}

// Half G0 (pieces 4 G0 .. 4 G0 + 3, columns 32 G0 .. 32 G0 + 31) of a tile
// row from the NV activations h (zero beyond NV); G0 is
// compile-time so that h is indexed statically.
template <int NV, int G0>
__device__ __forceinline__ void st_half(unsigned char* tile, int r, const float* h) {
#pragma unroll
  for (int uu = 0; uu < 4; ++uu) {
    const int u8 = G0 * 4 + uu;
    float v8[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int j = u8 * 8 + c;
      v8[c] = j < NV ? h[j < NV ? j : 0] : 0.f;
    }
    st_piece(tile, r, u8, v8);
  }
}

// skip of a layer from width NI to NO: identity, [x, x] or none
template <int NI, int NO>
struct Skip {
  static constexpr int kind = NI == NO ? 1 : (NO == 2 * NI ? 2 : 0);
  __device__ static __forceinline__ float at(const float* x, int j) {
    if (kind == 1) return x[j];
    if (kind == 2) return x[j < NI ? j : j - NI];
    return 0.f;
  }
};

// ------------------------------------------------------------ row mapping --
// A tile's 128 rows are four slabs of 32, one per warp, each from that warp's
// own atom: a CTA takes two units (four atoms) at a time, section by section,
// and a warp walks its atom's section 32 rows a tile.  Padding slots repeat
// one env row, and equal rows give equal embeddings: the rows from the first
// of the equal ones at a section's end to its last slot are evaluated once
// (water: some 30 and 60 of 46 and 92 rows).
//
// rows of section [s0, s0 + ns) of an atom to evaluate: 1 + the last row that
// differs from the section's last row, plus one for the equal rest (NaN
// differs from itself: every row)
__device__ __forceinline__ int distinct_rows(const float4* em, int ns) {
  const int lane = threadIdx.x & 31;
  const float4 last = em[ns - 1];
  int top = -1;
  for (int b = 0; b < ns; b += 128) {
    bool ne[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = b + 32 * u + lane;
      ne[u] = false;
      if (j < ns) {
        const float4 e = em[j];
        ne[u] = !(e.x == last.x && e.y == last.y && e.z == last.z && e.w == last.w);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned m = __ballot_sync(kFull, ne[u]);
      if (m) top = b + 32 * u + 31 - __clz(m);
    }
  }
  return min(ns, top + 2);
}

// the group's units that share nets: both in one pass, or (nets per centre
// type and types differ) one pass each
struct Group {
  int atom;    // this warp's atom (-1: none)
  int ti[2];   // centre type of each unit
  bool both;
};
__device__ __forceinline__ Group load_group(const int* __restrict__ units,
                                            const int* __restrict__ atype, int nunits, int g,
                                            int warp, bool one_side, bool split = false) {
  Group r;
  if (split) {  // warps 0 and 2: the unit's first atom, 1 and 3: its second
    r.atom = units[2 * g + (warp & 1)];
    r.ti[0] = r.ti[1] = atype[units[2 * g]];
    r.both = true;
    return r;
  }
  const int u0 = 2 * g, u1 = u0 + 1;
  const int mine = u0 + (warp >> 1);
  r.atom = mine < nunits ? units[2 * mine + (warp & 1)] : -1;
  r.ti[0] = atype[units[2 * u0]];
  r.ti[1] = u1 < nunits ? atype[units[2 * u1]] : r.ti[0];
  r.both = one_side || r.ti[0] == r.ti[1];
  return r;
}

// 16 columns of a parameter row, read as float4 broadcasts
__device__ __forceinline__ void par16(const float* par, float* v) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 u = reinterpret_cast<const float4*>(par)[q];
    v[4 * q] = u.x;
    v[4 * q + 1] = u.y;
    v[4 * q + 2] = u.z;
    v[4 * q + 3] = u.w;
  }
}

// Columns 32 C .. 32 C + 31 of epilogue 3: G = tanh(D3 + b3) + skip(h2) of
// this lane's row into the warp's [32 rows][32 columns] buffer, 16-byte piece
// p of row r at piece p ^ (r & 7) (stores of a row by its lane and loads of a
// column by its lane both without bank conflicts)
template <int N2, int N3, int C>
__device__ __forceinline__ void epi3(uint32_t trow, const float* par, const float* h2,
                                     float* gbuf) {
  constexpr int NC = N3 - 32 * C >= 32 ? 2 : (N3 - 32 * C + 15) / 16;
  const int lane = threadIdx.x & 31;
  uint32_t v[NC][16];
#pragma unroll
  for (int c = 0; c < NC; ++c) tmem_ld16_nw(trow + 32 * C + 16 * c, v[c]);
  tmem_wait();
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    float b[16], gv[16];
    par16(par + kParB3 + 32 * C + 16 * c, b);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int m = 32 * C + 16 * c + k;
      gv[k] = m < N3 ? tanh_fast(__uint_as_float(v[c][k]) + b[k]) +
                           Skip<N2, N3>::at(h2, m < N3 ? m : 0)
                     : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<float4*>(gbuf + lane * 32 + (((4 * c + q) ^ (lane & 7)) << 2)) =
          make_float4(gv[4 * q], gv[4 * q + 1], gv[4 * q + 2], gv[4 * q + 3]);
  }
}

// ---------------------------------------------------------------- kernel --
// G^T R keeps the order of the sums of a 128-row tile of two concatenated
// atoms: rows in ascending order in one chain of FMAs per column, broken
// where (member of the unit) sel + row is a multiple of 128 (X feeds BF16
// operands in the backward: another grouping would move their rounding).
// SPLIT: one unit a CTA, for calls of up to a wave of units, whose time is the
// chain of slabs: an atom's slabs go to two warps (0 and 2, 1 and 3), which
// evaluate them side by side and then sum the rows of both in slab order,
// one warp the even 32-column chunks, the other the odd ones (the same sums
// bit for bit).
template <int N1, int N2, int N3, bool SPLIT>
__global__ void __launch_bounds__(128, 3) k_emb_fwd(const __grid_constant__ EmbArgs p) {
  static_assert(N1 <= 32 && N2 <= 64 && N3 <= 128 && N3 >= 1, "embedding widths");
  constexpr int NCH = (N3 + 31) / 32;  // 32-column chunks
  grid_wait();
  grid_release();
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* slots = sm;                  // two staged nets: section t in slot t & 1
  unsigned char* atile = sm + 2 * kSlot;      // A operand, 16 KiB; a warp's quarter is its buffer
  float4* rsm = reinterpret_cast<float4*>(atile + 16384);  // [128] env rows
  uint64_t* bar = reinterpret_cast<uint64_t*>(rsm + kRows);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  int* cached = reinterpret_cast<int*>(tslot + 1);  // [2] net held by each slot
  int* nslab = cached + 2;                          // [4 warps] slabs of the section
  float* odd = reinterpret_cast<float*>(sm + kFwdBytes);  // SPLIT: [4 warps] odd chunks

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = tid;  // this thread's tile row = TMEM lane

  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
    cached[0] = cached[1] = -1;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(
                     smem_addr(tslot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;  // D2 in columns 0 .. 63, then D3 in 0 .. 127
  const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
  const uint32_t aaddr = smem_addr(atile);
  float* gbuf = reinterpret_cast<float*>(atile + warp * 4096);
  unsigned phase = 0;
  bool alive = true;
  const float inv_nnei = 1.f / (float)p.nnei;
  const int ngroups = SPLIT ? p.nunits : (p.nunits + 1) >> 1;
  // the pair of warps of one atom (SPLIT); this one's slabs are s0, s0 + ss, ..
  constexpr int ss = SPLIT ? 2 : 1, NOWN = SPLIT ? (NCH + 1) / 2 : NCH;
  const int s0 = SPLIT ? warp >> 1 : 0;
  auto pair_sync = [&]() {
    asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 1)) : "memory");
  };

  for (int g = blockIdx.x; g < ngroups && alive; g += gridDim.x) {
    const Group gr = load_group(p.units, p.atype, p.nunits, g, warp, p.type_one_side, SPLIT);
    // this lane's columns of X (sums), components (0, 1), (2, 3): of chunk c,
    // or (SPLIT) of chunk 2 c + s0
    float2 xt[NOWN][2];
#pragma unroll
    for (int c = 0; c < NOWN; ++c) xt[c][0] = xt[c][1] = make_float2(0.f, 0.f);
    for (int pass = 0; pass < (gr.both ? 1 : 2) && alive; ++pass) {
      const bool act = gr.atom >= 0 && (gr.both || (warp >> 1) == pass);
      for (int tj = 0; tj < p.ntypes && alive; ++tj) {
        const int sel = p.sec[tj + 1] - p.sec[tj];
        if (sel == 0) continue;
        const int net = p.type_one_side ? tj : tj * p.ntypes + gr.ti[pass];
        unsigned char* slot = slots + (tj & 1) * kSlot;
        const float4* em = reinterpret_cast<const float4*>(p.em) +
                           (size_t)(act ? gr.atom : 0) * p.nnei + p.sec[tj];
        const int neff = act ? distinct_rows(em, sel) : 0;
        if (lane == 0) nslab[warp] = (neff + 31) >> 5;
        __syncthreads();
        const int nsl =
            (max(max(nslab[0], nslab[1]), max(nslab[2], nslab[3])) + ss - 1) / ss;
        if (cached[tj & 1] != net) {  // uniform: stage this net's weights and params
          const uint4* src = reinterpret_cast<const uint4*>(p.nets + (size_t)net * kNetBytes);
          uint4* dst = reinterpret_cast<uint4*>(slot);
          for (int k = tid; k < kNetFwdBytes / 16; k += 128) dst[k] = __ldg(src + k);
          fence_proxy_async_smem();
          __syncthreads();
          if (tid == 0) cached[tj & 1] = net;
        }
        __syncthreads();  // nslab and cached read before they change again
        const float* par = reinterpret_cast<const float*>(slot + kNetPar);
        const uint32_t b2 = smem_addr(slot + kNetB2), b3 = smem_addr(slot + kNetB3);
        float2 acc[NOWN][2];
#pragma unroll
        for (int c = 0; c < NOWN; ++c) acc[c][0] = acc[c][1] = make_float2(0.f, 0.f);
        auto flush = [&](int c) {
          xt[c][0] = make_float2(xt[c][0].x + acc[c][0].x, xt[c][0].y + acc[c][0].y);
          xt[c][1] = make_float2(xt[c][1].x + acc[c][1].x, xt[c][1].y + acc[c][1].y);
          acc[c][0] = acc[c][1] = make_float2(0.f, 0.f);
        };
        float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
        if (32 * s0 + lane < neff) e = em[32 * s0 + lane];
        for (int sl = 0; sl < nsl && alive; ++sl) {
          rsm[r] = e;
          // ---- layer 1 (FP32): h1 = tanh(s w1 + b1), all N1 columns per thread
          float h1[N1];
#pragma unroll
          for (int j = 0; j < N1; ++j)
            h1[j] = tanh_fast(fmaf(e.x, par[kParW1 + j], par[kParB1 + j]));
          st_half<N1, 0>(atile, r, h1);
          st_half<N1, 1>(atile, r, h1);
          // the next slab's row
          const int jn = 32 * (ss * (sl + 1) + s0) + lane;
          e = jn < neff ? em[jn] : make_float4(0.f, 0.f, 0.f, 0.f);
          fence_proxy_async_smem();
          tc_fence_before();
          __syncthreads();
          if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_bf16(tmem, sdesc_sw128(aaddr + kk * 32), sdesc_sw128(b2 + kk * 32),
                        idesc_bf16(64), kk > 0);
            umma_commit(bar);
          }
          alive = __syncthreads_and(mbar_wait_bounded(bar, phase, p.status));
          phase ^= 1u;
          if (!alive) break;
          tc_fence_after();
          // ---- epilogue 2: h2 = tanh(D2 + b2) + skip(h1), all N2 columns
          float h2[N2];
          {
            constexpr int NC = (N2 + 15) / 16;
            uint32_t v[NC][16];
#pragma unroll
            for (int c = 0; c < NC; ++c) tmem_ld16_nw(trow + c * 16, v[c]);
            tmem_wait();
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              float b[16];
              par16(par + kParB2 + 16 * c, b);
#pragma unroll
              for (int k = 0; k < 16; ++k) {
                const int j = c * 16 + k;
                if (j < N2)
                  h2[j] = tanh_fast(__uint_as_float(v[c][k]) + b[k]) + Skip<N1, N2>::at(h1, j);
              }
            }
          }
          // MMA 2 is done with A and a warp rewrites only its own rows; the
          // barrier orders every warp's D2 loads and A stores before MMA 3
          st_half<N2, 0>(atile, r, h2);
          st_half<N2, 1>(atile, r, h2);
          fence_proxy_async_smem();
          tc_fence_before();
          __syncthreads();
          if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_bf16(tmem, sdesc_sw128(aaddr + kk * 32), sdesc_sw128(b3 + kk * 32),
                        idesc_bf16(128), kk > 0);
            umma_commit(bar);
          }
          alive = __syncthreads_and(mbar_wait_bounded(bar, phase, p.status));
          phase ^= 1u;
          if (!alive) break;
          tc_fence_after();
          // ---- epilogue 3 and G^T R, 32 columns at a time: a lane per column
          //      over a slab's rows, through the warp's quarter of A (MMA 3 is
          //      done with it)
          // rows of slab `s` (G chunk in G, env rows in R) onto the owned
          // chunk c, up to the row that stands for the equal rest
          auto add_slab = [&](int c, int s, const float* G, const float4* R, float& gt) {
            const int nrow = min(32, neff - 32 * s);
            const int pos = (warp & 1) * sel + 32 * s;
            const int brk = (128 - (pos & 127)) & 127;  // row before which the chain breaks
            const int plain = 32 * s + nrow == neff ? nrow - 1 : nrow;
            auto rows = [&](int lo, int hi) {
#pragma unroll 4
              for (int rr = lo; rr < hi; ++rr) {
                const float gv = G[rr * 32 + ((((lane >> 2) ^ (rr & 7)) << 2) | (lane & 3))];
                const float4 q = R[rr];
                acc[c][0] = __ffma2_rn(lo2(q), dup2(gv), acc[c][0]);
                acc[c][1] = __ffma2_rn(hi2(q), dup2(gv), acc[c][1]);
              }
            };
            if (brk < plain) {
              rows(0, brk);
              flush(c);
              rows(brk, plain);
            } else {
              rows(0, plain);
            }
            const int rr = nrow - 1;
            gt = G[rr * 32 + ((((lane >> 2) ^ (rr & 7)) << 2) | (lane & 3))];
          };
          // the last row of slab `s` for itself and the equal rest
          auto add_rest = [&](int s, const float4* R, const float* gt) {
            const float4 q = R[neff - 32 * s - 1];
            // a padding row; 0 G is no 0 where G is not finite
            bool one = q.y == 0.f && q.z == 0.f && q.w == 0.f;
#pragma unroll
            for (int c = 0; c < NOWN; ++c) one = one && fabsf(gt[c]) < INFINITY;
            int at = (warp & 1) * sel + neff - 1;
            for (int left = sel - neff + 1; left > 0;) {
              if ((at & 127) == 0)
#pragma unroll
                for (int c = 0; c < NOWN; ++c) flush(c);
              const int n = min(left, 128 - (at & 127));
              if (one) {
                for (int k = 0; k < n; ++k)
#pragma unroll
                  for (int c = 0; c < NOWN; ++c) acc[c][0].x = fmaf(q.x, gt[c], acc[c][0].x);
              } else {
                for (int k = 0; k < n; ++k)
#pragma unroll
                  for (int c = 0; c < NOWN; ++c) {
                    acc[c][0] = __ffma2_rn(lo2(q), dup2(gt[c]), acc[c][0]);
                    acc[c][1] = __ffma2_rn(hi2(q), dup2(gt[c]), acc[c][1]);
                  }
              }
              at += n;
              left -= n;
            }
          };
          if constexpr (!SPLIT) {
            const int nrow = min(32, neff - 32 * sl);  // live rows of this warp
            if (nrow > 0) {  // uniform over the warp
              const float4* R = rsm + warp * 32;
              float gt[NCH];
              __syncwarp();
              epi3<N2, N3, 0>(trow, par, h2, gbuf);
              __syncwarp();
              add_slab(0, sl, gbuf, R, gt[0]);
              if constexpr (NCH > 1) {
                __syncwarp();
                epi3<N2, N3, 1>(trow, par, h2, gbuf);
                __syncwarp();
                add_slab(1, sl, gbuf, R, gt[1]);
              }
              if constexpr (NCH > 2) {
                __syncwarp();
                epi3<N2, N3, 2>(trow, par, h2, gbuf);
                __syncwarp();
                add_slab(2, sl, gbuf, R, gt[2]);
              }
              if constexpr (NCH > 3) {
                __syncwarp();
                epi3<N2, N3, 3>(trow, par, h2, gbuf);
                __syncwarp();
                add_slab(3, sl, gbuf, R, gt[3]);
              }
              if (32 * sl + nrow == neff) add_rest(sl, R, gt);
              __syncwarp();
            }
          } else if (32 * ss * sl < neff) {  // uniform over the pair
            const int w0 = warp & 1, w1 = w0 + 2, sE = 2 * sl, sO = sE + 1;
            const bool two = 32 * sO < neff;
            // even chunks in a warp's quarter of A, odd ones in its odd buffer
            const float* b0 = s0 ? odd + w0 * 1024 : reinterpret_cast<float*>(atile + w0 * 4096);
            const float* b1 = s0 ? odd + w1 * 1024 : reinterpret_cast<float*>(atile + w1 * 4096);
            float gt[NOWN] = {};
            epi3<N2, N3, 0>(trow, par, h2, gbuf);
            if constexpr (NCH > 1) epi3<N2, N3, 1>(trow, par, h2, odd + warp * 1024);
            pair_sync();
            if (s0 < NCH) {
              add_slab(0, sE, b0, rsm + w0 * 32, gt[0]);
              if (two) add_slab(0, sO, b1, rsm + w1 * 32, gt[0]);
            }
            if constexpr (NCH > 2) {
              pair_sync();
              epi3<N2, N3, 2>(trow, par, h2, gbuf);
              if constexpr (NCH > 3) epi3<N2, N3, 3>(trow, par, h2, odd + warp * 1024);
              pair_sync();
              if (2 + s0 < NCH) {
                add_slab(1, sE, b0, rsm + w0 * 32, gt[1]);
                if (two) add_slab(1, sO, b1, rsm + w1 * 32, gt[1]);
              }
            }
            if (32 * (two ? sO : sE) + 32 >= neff)
              add_rest(two ? sO : sE, rsm + (two ? w1 : w0) * 32, gt);
            pair_sync();  // the buffers read before they are filled again
          }
          tc_fence_before();
        }
#pragma unroll
        for (int c = 0; c < NOWN; ++c) flush(c);
      }
    }
    if (!alive) break;
    // ---- X and D of this warp's atom
    if (gr.atom >= 0) {
      const size_t row = p.drow ? (size_t)p.drow[gr.atom] : (size_t)gr.atom;
      // (SPLIT: the pair shares xT and the rows of D)
      float4* xT = reinterpret_cast<float4*>(atile + (SPLIT ? warp & 1 : warp) * 4096);
      float nk = 0.f, na = 0.f;
      __syncwarp();
#pragma unroll
      for (int c = 0; c < NOWN; ++c) {
        const int m = 32 * (ss * c + s0) + lane;
        if (m < N3) {
          const float4 x = make_float4(xt[c][0].x * inv_nnei, xt[c][0].y * inv_nnei,
                                       xt[c][1].x * inv_nnei, xt[c][1].y * inv_nnei);
          xT[m] = x;
          float* Xa = p.X + (size_t)gr.atom * 4 * N3 + m;
          Xa[0] = x.x;
          Xa[N3] = x.y;
          Xa[2 * N3] = x.z;
          Xa[3 * N3] = x.w;
          const float q = x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
          nk = fmaxf(nk, q);
          if (m < p.A) na = fmaxf(na, q);
        }
      }
      if constexpr (SPLIT)
        pair_sync();
      else
        __syncwarp();
      if constexpr (SPLIT)
        for (int m = lane; m < N3; m += 32) {
          const float4 x = xT[m];
          const float q = x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
          nk = fmaxf(nk, q);
          if (m < p.A) na = fmaxf(na, q);
        }
      auto dval = [&](int m, int a) {
        const float4 u = xT[m], w = xT[a];
        return fmaf(u.w, w.w, fmaf(u.z, w.z, fmaf(u.y, w.y, fmaf(u.x, w.x, 0.f))));
      };
      if (p.D_lo) {
        // split for the tensor-core fitting: FP16 hi / lo of c D, c = 2^s
        // from |D_ka| <= |X_k| |X_a| (Cauchy-Schwarz over the 4 rows of X)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          nk = fmaxf(nk, __shfl_xor_sync(kFull, nk, o));
          na = fmaxf(na, __shfl_xor_sync(kFull, na, o));
        }
        const float sc = f16_scale_for(sqrtf(nk * na) * 1.0001f);
        __half* dh = static_cast<__half*>(p.D) + row * (size_t)N3 * p.A;
        __half* dl = static_cast<__half*>(p.D_lo) + row * (size_t)N3 * p.A;
        for (int at = 4 * (lane + 32 * s0); at < N3 * p.A; at += 128 * ss) {
          const int m = at / p.A, a = at - m * p.A;
          const float v[4] = {dval(m, a), dval(m, a + 1), dval(m, a + 2), dval(m, a + 3)};
          st_split4_f16(dh + at, dl + at, v, sc);
        }
        if (lane == 0 && s0 == 0) p.D_rs[row] = 1.f / sc;
      } else {
        float* d = static_cast<float*>(p.D) + row * (size_t)N3 * p.A;
        for (int at = lane + 32 * s0; at < N3 * p.A; at += 32 * ss) {
          const int m = at / p.A;
          d[at] = dval(m, at - m * p.A);
        }
      }
      if constexpr (SPLIT)
        pair_sync();
      else
        __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(tmem) : "memory");
}

// ------------------------------------------------------------- backward --
// dX (gradient wrt the un-normalised sums X * nnei) of every atom from dE/dD:
// D[m][a] = sum_c X[c][m] X[c][a] (a < A), so
//   dX[c][m] = sum_a dD[m][a] X[c][a] + [m < A] sum_m' dD[m'][m] X[c][m'].
// One CTA per atom: threads over m for the first term, threads over (c, a)
// for the second (4 A sums of N3 terms), combined through shared memory.
__global__ void k_emb_dx(float* __restrict__ dxs, const float* __restrict__ dD,
                         const float* __restrict__ X, const int* __restrict__ drow, int N3, int A,
                         float inv_nnei) {
  extern __shared__ float sh[];
  float* xs = sh;                // [4][N3]
  const int As = A + 1;          // odd row stride: threads over m hit distinct banks
  float* dds = sh + 4 * N3;      // [N3][As]
  float* t2 = dds + N3 * As;     // [4][A] second term
  const int atom = blockIdx.x;
  const size_t row = drow ? (size_t)drow[atom] : (size_t)atom;
  for (int k = threadIdx.x; k < 4 * N3; k += blockDim.x) xs[k] = X[(size_t)atom * 4 * N3 + k];
  {  // warps over rows m, lanes over columns a: no division by A
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const float* src = dD + row * N3 * A;
    for (int m = w; m < N3; m += nw)
      for (int a = lane; a < A; a += 32) dds[m * As + a] = src[m * A + a];
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 4 * A; k += blockDim.x) {
    const int c = k / A, a = k - c * A;
    float o = 0.f;
    for (int m2 = 0; m2 < N3; ++m2) o = fmaf(dds[m2 * As + a], xs[c * N3 + m2], o);
    t2[k] = o;
  }
  __syncthreads();
  for (int m = threadIdx.x; m < N3; m += blockDim.x) {
    float o[4] = {0.f, 0.f, 0.f, 0.f};
    for (int a = 0; a < A; ++a) {
      const float w = dds[m * As + a];
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] = fmaf(w, xs[c * N3 + a], o[c]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (m < A) o[c] += t2[c * A + m];
      dxs[((size_t)atom * 4 + c) * N3 + m] = o[c] * inv_nnei;
    }
  }
}

// The same for 16 axis columns (same sums in the same order, the same bits:
// dX is rounded to BF16 operands later), a warp per atom: the row of dD by
// coalesced 16-byte loads, 24 atoms in flight per SM (six CTAs by shared
// memory, 33.6 KB each at 100 columns) instead of a CTA each (6,141 atoms: 70
// -> 26 us).
constexpr int kDxWarps = 4;
__host__ __device__ constexpr size_t dx16_warp_bytes(int N3) {
  return (size_t)N3 * 16 + ((size_t)N3 * 17 * 4 + 15) / 16 * 16;  // X^T, then dD (odd row stride)
}
__global__ void __launch_bounds__(kDxWarps * 32)
    k_emb_dx16(float* __restrict__ dxs, const float* dD, const float* X,
               const int* __restrict__ drow, int nloc, int N3, float inv_nnei) {
  grid_wait();
  grid_release();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int atom = blockIdx.x * kDxWarps + warp;
  if (atom >= nloc) return;  // uniform over the warp; no CTA-wide barrier below
  float4* xT = reinterpret_cast<float4*>(smem_raw + warp * dx16_warp_bytes(N3));
  float* dds = reinterpret_cast<float*>(xT + N3);
  const float* Xi = X + (size_t)atom * 4 * N3;
  const float4* g_i =
      reinterpret_cast<const float4*>(dD + (drow ? (size_t)drow[atom] : (size_t)atom) * N3 * 16);
  for (int m = lane; m < N3; m += 32)
    xT[m] = make_float4(Xi[m], Xi[N3 + m], Xi[2 * N3 + m], Xi[3 * N3 + m]);
  constexpr int BT = 8;  // loads in flight
  for (int u0 = 0; u0 < 4 * N3; u0 += 32 * BT) {
    float4 g[BT];
#pragma unroll
    for (int u = 0; u < BT; ++u) {
      const int at = u0 + 32 * u + lane;
      if (at < 4 * N3) g[u] = __ldcs(g_i + at);
    }
#pragma unroll
    for (int u = 0; u < BT; ++u) {
      const int at = u0 + 32 * u + lane;
      if (at < 4 * N3) {
        float* p = dds + (at >> 2) * 17 + (at & 3) * 4;
        p[0] = g[u].x;
        p[1] = g[u].y;
        p[2] = g[u].z;
        p[3] = g[u].w;
      }
    }
  }
  __syncwarp();
  // second sum: lane a (mod 16) takes components (0, 1) or (2, 3)
  float2 t2 = make_float2(0.f, 0.f);
  {
    const int a = lane & 15, h = lane >> 4;
    const float2* x2 = reinterpret_cast<const float2*>(xT);
#pragma unroll 4
    for (int m = 0; m < N3; ++m) t2 = __ffma2_rn(dup2(dds[m * 17 + a]), x2[2 * m + h], t2);
  }
  float* out = dxs + (size_t)atom * 4 * N3;
  for (int m0 = 0; m0 < N3; m0 += 32) {
    const int m = m0 + lane;
    float2 o01 = make_float2(0.f, 0.f), o23 = o01;
    if (m < N3) {
#pragma unroll
      for (int a = 0; a < 16; ++a) {
        const float2 w = dup2(dds[m * 17 + a]);
        const float4 x = xT[a];
        o01 = __ffma2_rn(w, lo2(x), o01);
        o23 = __ffma2_rn(w, hi2(x), o23);
      }
    }
    if (m0 == 0) {  // columns m < 16 take the second sum from the lanes that hold it
      const float2 a01 = make_float2(__shfl_sync(kFull, t2.x, lane & 15),
                                     __shfl_sync(kFull, t2.y, lane & 15));
      const float2 a23 = make_float2(__shfl_sync(kFull, t2.x, 16 + (lane & 15)),
                                     __shfl_sync(kFull, t2.y, 16 + (lane & 15)));
      if (lane < 16) {
        o01 = make_float2(o01.x + a01.x, o01.y + a01.y);
        o23 = make_float2(o23.x + a23.x, o23.y + a23.y);
      }
    }
    if (m < N3) {
      out[m] = o01.x * inv_nnei;
      out[N3 + m] = o01.y * inv_nnei;
      out[2 * N3 + m] = o23.x * inv_nnei;
      out[3 * N3 + m] = o23.y * inv_nnei;
    }
  }
}

struct EmbBwdArgs {
  float* net;          // [nloc, nnei, 4] dE/d(env matrix)
  const float* dxs;    // [nloc, 4, N3] from k_emb_dx
  const float* em;     // [nloc, nnei, 4]
  const int* units;
  const int* atype;
  const unsigned char* nets;
  int* status;
  int nunits, ntypes, type_one_side, nloc, nnei;
  int sec[kMaxTypes + 1];
};

constexpr int kBwdSlot = kNetBytes;  // the whole net block (forward and transposed images)

// Backward epilogue 3 over one half of the D3 columns (G0 compile-time, so
// that every register array is indexed statically): G (recomputed) and the
// incoming dG = R . dX give dR, the skip gradient of dG into sk (the layer
// 2 -> 3 skip: identity or [x, x]) and dZ3 = dG (1 - t3^2) -> the K = 128 A
// operand (bf16, chunk G0).
template <int N1, int N2, int N3, int G0>
__device__ __forceinline__ void bepi3(uint32_t trow, const float* par, const float* t2,
                                      const float* h1, bool live, float4 R, const float4* dx,
                                      float* sk, unsigned char* atile, int r, float* dr) {
  unsigned char* chunk = atile + G0 * 16384;
#pragma unroll
  for (int c16 = 0; c16 < 4; ++c16) {
    const int m0 = G0 * 64 + c16 * 16;
    float dz[16];
    if (m0 >= N3) {
#pragma unroll
      for (int k = 0; k < 16; ++k) dz[k] = 0.f;
    } else {
      float v[16];
      tmem_ld16(trow + 128 + m0, v);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const int m = m0 + k;
        float z = 0.f;
        if (m < N3 && live) {
          const float t3 = tanh_fast(v[k] + par[kParB3 + m]);
          float gv = t3;
          if (Skip<N2, N3>::kind != 0) {  // h2 at the skip index, from t2 and h1
            const int j = m < N2 ? m : m - N2;
            gv += t2[j] + Skip<N1, N2>::at(h1, j);
          }
          const float4 q = dx[m];
          const float d0 = q.x, d1 = q.y, d2 = q.z, d3 = q.w;
          const float dg = R.x * d0 + R.y * d1 + R.z * d2 + R.w * d3;
          dr[0] = fmaf(gv, d0, dr[0]);
          dr[1] = fmaf(gv, d1, dr[1]);
          dr[2] = fmaf(gv, d2, dr[2]);
          dr[3] = fmaf(gv, d3, dr[3]);
          if (Skip<N2, N3>::kind == 1) sk[m] += dg;
          if (Skip<N2, N3>::kind == 2) sk[m < N2 ? m : m - N2] += dg;
          z = dg * (1.f - t3 * t3);
        }
        dz[k] = z;
      }
    }
    st_piece(chunk, r, c16 * 2, dz);
    st_piece(chunk, r, c16 * 2 + 1, dz + 8);
  }
}

// SPLIT as in k_emb_fwd: every row's gradient is its own, so the warps of an
// atom need nothing of each other.
template <int N1, int N2, int N3, bool SPLIT>
__global__ void __launch_bounds__(128, 2) k_emb_bwd(const __grid_constant__ EmbBwdArgs p) {
  grid_wait();
  grid_release();
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* slot = sm;                      // one staged net (all images)
  unsigned char* atile = sm + kBwdSlot;          // A operand, 2 chunks of 16 KiB
  float4* dxsm = reinterpret_cast<float4*>(atile + 32768);  // [4 warps][128]: dX^T of its atom
  uint64_t* bar = reinterpret_cast<uint64_t*>(dxsm + 4 * 128);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  int* cached = reinterpret_cast<int*>(tslot + 1);
  int* nslab = cached + 1;  // [4 warps] slabs of the section

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = tid;  // this thread's tile row = TMEM lane

  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
    cached[0] = -1;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(
                     smem_addr(tslot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
  unsigned phase = 0;
  bool alive = true;

  const uint32_t aaddr = smem_addr(atile);
  float4* dx = dxsm + warp * 128;
  const int ngroups = SPLIT ? p.nunits : (p.nunits + 1) >> 1;
  // this warp's slabs of its atom's section: s0, s0 + ss, ..
  constexpr int ss = SPLIT ? 2 : 1;
  const int s0 = SPLIT ? warp >> 1 : 0;

  for (int tj = 0; tj < p.ntypes && alive; ++tj) {
    const int sel = p.sec[tj + 1] - p.sec[tj];
    if (sel == 0) continue;
    for (int g = blockIdx.x; g < ngroups && alive; g += gridDim.x) {
      const Group gr = load_group(p.units, p.atype, p.nunits, g, warp, p.type_one_side, SPLIT);
      for (int pass = 0; pass < (gr.both ? 1 : 2) && alive; ++pass) {
        const bool act = gr.atom >= 0 && (gr.both || (warp >> 1) == pass);
        const int net = p.type_one_side ? tj : tj * p.ntypes + gr.ti[pass];
        const size_t row0 = (size_t)(act ? gr.atom : 0) * p.nnei + p.sec[tj];
        const float4* em = reinterpret_cast<const float4*>(p.em) + row0;
        float4* out = reinterpret_cast<float4*>(p.net) + row0;
        const int neff = act ? distinct_rows(em, sel) : 0;
        if (lane == 0) nslab[warp] = (neff + 31) >> 5;
        if (act)
          for (int m = lane; m < N3; m += 32) {
            const float* d = p.dxs + (size_t)gr.atom * 4 * N3 + m;
            dx[m] = make_float4(d[0], d[N3], d[2 * N3], d[3 * N3]);
          }
        __syncthreads();  // (and the previous group is done with the shared buffers)
        const int nsl =
            (max(max(nslab[0], nslab[1]), max(nslab[2], nslab[3])) + ss - 1) / ss;
        if (cached[0] != net) {
          const uint4* src = reinterpret_cast<const uint4*>(p.nets + (size_t)net * kNetBytes);
          uint4* dst = reinterpret_cast<uint4*>(slot);
          for (int k = tid; k < kNetBytes / 16; k += 128) dst[k] = __ldg(src + k);
          fence_proxy_async_smem();
          __syncthreads();
          if (tid == 0) cached[0] = net;
        }
        __syncthreads();  // nslab and cached read before they change again
        const float* par = reinterpret_cast<const float*>(slot + kNetPar);
        const uint32_t b2 = smem_addr(slot + kNetB2), b3 = smem_addr(slot + kNetB3);
        const uint32_t b3t = smem_addr(slot + kNetB3T), b2t = smem_addr(slot + kNetB2T);
        float4 en = make_float4(0.f, 0.f, 0.f, 0.f);
        if (32 * s0 + lane < neff) en = em[32 * s0 + lane];
        for (int sl = 0; sl < nsl && alive; ++sl) {
          const int slab = ss * sl + s0;
          const int j = 32 * slab + lane;
          const bool live = j < neff;
          const float4 e = en;
          en = j + 32 * ss < neff ? em[j + 32 * ss] : make_float4(0.f, 0.f, 0.f, 0.f);
          // ---- forward recompute: layer 1, MMA 2, epilogue 2, MMA 3
          float h1[N1];
  #pragma unroll
          for (int j = 0; j < N1; ++j) h1[j] = tanh_fast(fmaf(e.x, par[kParW1 + j], par[kParB1 + j]));
          st_half<N1, 0>(atile, r, h1);
          st_half<N1, 1>(atile, r, h1);
          fence_proxy_async_smem();
          tc_fence_before();
          __syncthreads();
          if (tid == 0) {
            tc_fence_after();
  #pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_bf16(tmem, sdesc_sw128(aaddr + kk * 32), sdesc_sw128(b2 + kk * 32),
                        idesc_bf16(64), kk > 0);
            umma_commit(bar);
          }
          alive = __syncthreads_and(mbar_wait_bounded(bar, phase, p.status));
          phase ^= 1u;
          if (!alive) break;
          tc_fence_after();
          float t2[N2];
  #pragma unroll
          for (int c16 = 0; c16 < (N2 + 15) / 16; ++c16) {
            float v[16];
            tmem_ld16(trow + c16 * 16, v);
  #pragma unroll
            for (int k = 0; k < 16; ++k) {
              const int j = c16 * 16 + k;
              if (j < N2) t2[j] = tanh_fast(v[k] + par[kParB2 + j]);
            }
          }
          tc_fence_before();
          __syncthreads();
          {
            float h2[N2];
  #pragma unroll
            for (int j = 0; j < N2; ++j) h2[j] = t2[j] + Skip<N1, N2>::at(h1, j);
            st_half<N2, 0>(atile, r, h2);
            st_half<N2, 1>(atile, r, h2);
          }
          fence_proxy_async_smem();
          __syncthreads();
          if (tid == 0) {
            tc_fence_after();
  #pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_bf16(tmem + 128, sdesc_sw128(aaddr + kk * 32), sdesc_sw128(b3 + kk * 32),
                        idesc_bf16(128), kk > 0);
            umma_commit(bar);
          }
          alive = __syncthreads_and(mbar_wait_bounded(bar, phase, p.status));
          phase ^= 1u;
          if (!alive) break;
          tc_fence_after();
          // ---- backward epilogue 3: dG, dR, the skip gradient, dZ3 -> A (K = 128)
          float dr[4] = {0.f, 0.f, 0.f, 0.f};
          float sk[N2];
  #pragma unroll
          for (int j = 0; j < N2; ++j) sk[j] = 0.f;
          bepi3<N1, N2, N3, 0>(trow, par, t2, h1, live, e, dx, sk, atile, r, dr);
          bepi3<N1, N2, N3, 1>(trow, par, t2, h1, live, e, dx, sk, atile, r, dr);
          fence_proxy_async_smem();
          tc_fence_before();
          __syncthreads();
          if (tid == 0) {  // dH2 (partial) = dZ3 W3: K = 128 in two 64-column chunks
            tc_fence_after();
  #pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
              const uint32_t ca = aaddr + (kk >> 2) * 16384 + (kk & 3) * 32;
              const uint32_t cb = b3t + (kk >> 2) * 8192 + (kk & 3) * 32;
              umma_bf16(tmem, sdesc_sw128(ca), sdesc_sw128(cb), idesc_bf16(64), kk > 0);
            }
            umma_commit(bar);
          }
          alive = __syncthreads_and(mbar_wait_bounded(bar, phase, p.status));
          phase ^= 1u;
          if (!alive) break;
          tc_fence_after();
          // ---- epilogue 4: dH2 = dZ3 W3 + skip(dG), dZ2 = dH2 (1 - t2^2)
          float sb1[N1];  // t2 becomes dZ2 in place
          {
            float dh2[N2];
  #pragma unroll
            for (int c16 = 0; c16 < (N2 + 15) / 16; ++c16) {
              float v[16];
              tmem_ld16(trow + c16 * 16, v);
  #pragma unroll
              for (int k = 0; k < 16; ++k) {
                const int j = c16 * 16 + k;
                if (j < N2) {
                  dh2[j] = v[k] + sk[j];
                  t2[j] = dh2[j] * (1.f - t2[j] * t2[j]);
                }
              }
            }
  #pragma unroll
            for (int j = 0; j < N1; ++j) {
              float sk = 0.f;
              if (Skip<N1, N2>::kind == 1) sk = dh2[j];
              if (Skip<N1, N2>::kind == 2) sk = dh2[j] + dh2[j + N1];
              sb1[j] = sk;
            }
          }
          tc_fence_before();
          __syncthreads();  // MMA 4 done with A; every lane has read D4
          st_half<N2, 0>(atile, r, t2);
          st_half<N2, 1>(atile, r, t2);
          fence_proxy_async_smem();
          __syncthreads();
          if (tid == 0) {  // dH1 (partial) = dZ2 W2
            tc_fence_after();
  #pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_bf16(tmem + 64, sdesc_sw128(aaddr + kk * 32), sdesc_sw128(b2t + kk * 32),
                        idesc_bf16(64), kk > 0);
            umma_commit(bar);
          }
          alive = __syncthreads_and(mbar_wait_bounded(bar, phase, p.status));
          phase ^= 1u;
          if (!alive) break;
          tc_fence_after();
          // ---- epilogue 5: dZ1, ds, and the env-matrix gradient of the row
          float ds = 0.f;
  #pragma unroll
          for (int c16 = 0; c16 < (N1 + 15) / 16; ++c16) {
            float v[16];
            tmem_ld16(trow + 64 + c16 * 16, v);
  #pragma unroll
            for (int k = 0; k < 16; ++k) {
              const int j = c16 * 16 + k;
              if (j < N1) {
                const float dz1 = (v[k] + sb1[j]) * (1.f - h1[j] * h1[j]);
                ds = fmaf(dz1, par[kParW1 + j], ds);
              }
            }
          }
          {
            const float4 o = make_float4(ds + dr[0], dr[1], dr[2], dr[3]);
            if (live) out[j] = o;
            // the last row's gradient is that of the equal rows after it too
            const int tl = neff - 1 - 32 * slab;
            if (tl >= 0 && tl < 32) {  // uniform over the warp
              const float4 q = make_float4(
                  __shfl_sync(kFull, o.x, tl), __shfl_sync(kFull, o.y, tl),
                  __shfl_sync(kFull, o.z, tl), __shfl_sync(kFull, o.w, tl));
              for (int k = neff + lane; k < sel; k += 32) out[k] = q;
            }
          }
          tc_fence_before();
          __syncthreads();  // every lane has read D5 before the next tile
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
}

// A unit a CTA while all of them are resident at once, two an SM (forward and
// backward, 120 atoms: 70 us with two units a CTA, 56 so; 450 atoms: 78, 66).
// Above that two units a CTA: half the tiles are then taken per SM and the
// warps' work, not the chain, bounds the call.
inline bool split_units(int nunits, int& sms) {
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return nunits <= 2 * sms;
}

// 92 KiB: two CTAs per SM (2 x 256 TMEM columns)
template <int N3>
constexpr size_t bwd_smem() {
  return 1024 + kBwdSlot + 32768 + 4 * 128 * 16 + 64;
}

template <int N1, int N2, int N3, bool SPLIT>
int emb_bwd_launch(const EmbBwdArgs& a, int sms, cudaStream_t st) {
  auto kern = k_emb_bwd<N1, N2, N3, SPLIT>;
  constexpr size_t smem = bwd_smem<N3>();
  static const cudaError_t attr = [&] {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    return e;
  }();
  if (attr != cudaSuccess) return cuda_status(attr, "embed_bwd_tc attribute");
  // two CTAs per SM: registers by __launch_bounds__(128, 2), shared memory
  // below half an SM's
  static_assert(2 * (smem + 1024) <= 228 * 1024, "two CTAs per SM");
  const int grid = std::max(1, SPLIT ? a.nunits : std::min(2 * sms, (a.nunits + 1) / 2));
  launch_dep(kern, dim3(grid), dim3(128), smem, st, a);
  GBDP_CHECK_LAUNCH("embed_bwd_tc");
  return GBDP_OK;
}

// 72 KiB: three CTAs per SM (3 x 128 TMEM columns)
// (SPLIT: 16 KiB more, two an SM)
template <bool SPLIT>
constexpr size_t fwd_smem() { return 1024 + kFwdBytes + (SPLIT ? 16384 : 0); }

template <int N1, int N2, int N3, bool SPLIT>
int emb_fwd_launch(const EmbArgs& a, int sms, cudaStream_t st) {
  auto kern = k_emb_fwd<N1, N2, N3, SPLIT>;
  constexpr size_t smem = fwd_smem<SPLIT>();
  // the largest shared-memory carveout, so that three CTAs fit an SM
  static const cudaError_t attr = [&] {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
    return e;
  }();
  if (attr != cudaSuccess) return cuda_status(attr, "embed_fwd_tc attribute");
  // three CTAs per SM: registers by __launch_bounds__(128, 3), shared memory
  // below a third of an SM's
  static_assert((SPLIT ? 2 : 3) * (smem + 1024) <= 228 * 1024, "CTAs per SM");
  const int grid = std::max(1, SPLIT ? a.nunits : std::min(3 * sms, (a.nunits + 1) / 2));
  launch_dep(kern, dim3(grid), dim3(128), smem, st, a);
  GBDP_CHECK_LAUNCH("embed_fwd_tc");
  return GBDP_OK;
}

}  // namespace
}  // namespace gbdp

using namespace gbdp;

extern "C" size_t gbdp_embed_tc_net_bytes(void) { return (size_t)kNetBytes; }

extern "C" int gbdp_embed_fwd_tc_bf16(float* X, void* D, void* D_lo, float* D_rscale,
                                      const int* drow, const float* em, const int* atype,
                                      const int* units, int nunits, const void* nets, int ntypes,
                                      const int* sel, int type_one_side, int nloc, int nnei,
                                      int n1, int n2, int n3, int axis, int* status,
                                      gbdp_stream stream) {
  GBDP_REQUIRE(ntypes >= 1 && ntypes <= kMaxTypes, "embed_fwd_tc: ntypes %d not in [1, %d]",
               ntypes, kMaxTypes);
  GBDP_REQUIRE(nloc >= 0 && nunits >= 0 && nnei > 0, "embed_fwd_tc: bad sizes");
  GBDP_REQUIRE(axis >= 1 && axis <= n3, "embed_fwd_tc: axis_neuron %d not in [1, %d]", axis, n3);
  GBDP_REQUIRE(X && D && em && atype && units && nets && status,
               "embed_fwd_tc: null pointer");
  GBDP_REQUIRE(((uintptr_t)em & 15) == 0 && ((uintptr_t)nets & 15) == 0,
               "embed_fwd_tc: em and nets must be 16-byte aligned");
  GBDP_REQUIRE(!D_lo || (D_rscale && axis % 4 == 0 && ((uintptr_t)D & 7) == 0 &&
                          ((uintptr_t)D_lo & 7) == 0),
               "embed_fwd_tc: the split D needs D_rscale, axis_neuron %% 4 == 0 and 8-byte "
               "aligned parts");
  EmbArgs a{};
  a.X = X;
  a.D = D;
  a.D_lo = D_lo;
  a.D_rs = D_rscale;
  a.drow = drow;
  a.em = em;
  a.units = units;
  a.atype = atype;
  a.nets = static_cast<const unsigned char*>(nets);
  a.status = status;
  a.nunits = nunits;
  a.ntypes = ntypes;
  a.type_one_side = type_one_side;
  a.nloc = nloc;
  a.nnei = nnei;
  a.A = axis;
  a.sec[0] = 0;
  for (int t = 0; t < ntypes; ++t) {
    GBDP_REQUIRE(sel[t] >= 0, "embed_fwd_tc: negative sel");
    a.sec[t + 1] = a.sec[t] + sel[t];
  }
  GBDP_REQUIRE(a.sec[ntypes] == nnei, "embed_fwd_tc: sum(sel) %d != nnei %d", a.sec[ntypes], nnei);
  if (nunits == 0) return GBDP_OK;
  const cudaStream_t st = (cudaStream_t)stream;
  int sms = 0;
  const bool split = split_units(nunits, sms);
  if (n1 == 25 && n2 == 50 && n3 == 100)
    return split ? emb_fwd_launch<25, 50, 100, true>(a, sms, st)
                 : emb_fwd_launch<25, 50, 100, false>(a, sms, st);
  if (n1 == 3 && n2 == 6 && n3 == 12)
    return split ? emb_fwd_launch<3, 6, 12, true>(a, sms, st)
                 : emb_fwd_launch<3, 6, 12, false>(a, sms, st);
  set_error("embed_fwd_tc: embedding widths %d-%d-%d not built (25-50-100, 3-6-12)", n1, n2, n3);
  return GBDP_ERR_INVALID;
}

extern "C" int gbdp_embed_bwd_tc_bf16(float* net_deriv, float* dx_work, const float* dD,
                                      const float* X, const int* drow, const float* em,
                                      const int* atype, const int* units, int nunits,
                                      const void* nets, int ntypes, const int* sel,
                                      int type_one_side, int nloc, int nnei, int n1, int n2,
                                      int n3, int axis, int* status, gbdp_stream stream) {
  GBDP_REQUIRE(ntypes >= 1 && ntypes <= kMaxTypes, "embed_bwd_tc: ntypes %d not in [1, %d]",
               ntypes, kMaxTypes);
  GBDP_REQUIRE(nloc >= 0 && nunits >= 0 && nnei > 0, "embed_bwd_tc: bad sizes");
  GBDP_REQUIRE(axis >= 1 && axis <= n3, "embed_bwd_tc: axis_neuron %d not in [1, %d]", axis, n3);
  GBDP_REQUIRE(net_deriv && dx_work && dD && X && em && atype && units && nets && status,
               "embed_bwd_tc: null pointer");
  GBDP_REQUIRE(((uintptr_t)em & 15) == 0 && ((uintptr_t)net_deriv & 15) == 0 &&
                   ((uintptr_t)nets & 15) == 0,
               "embed_bwd_tc: em, net_deriv and nets must be 16-byte aligned");
  EmbBwdArgs a{};
  a.net = net_deriv;
  a.dxs = dx_work;
  a.em = em;
  a.units = units;
  a.atype = atype;
  a.nets = static_cast<const unsigned char*>(nets);
  a.status = status;
  a.nunits = nunits;
  a.ntypes = ntypes;
  a.type_one_side = type_one_side;
  a.nloc = nloc;
  a.nnei = nnei;
  a.sec[0] = 0;
  for (int t = 0; t < ntypes; ++t) {
    GBDP_REQUIRE(sel[t] >= 0, "embed_bwd_tc: negative sel");
    a.sec[t + 1] = a.sec[t] + sel[t];
  }
  GBDP_REQUIRE(a.sec[ntypes] == nnei, "embed_bwd_tc: sum(sel) %d != nnei %d", a.sec[ntypes], nnei);
  if (nloc == 0 || nunits == 0) return GBDP_OK;
  const cudaStream_t st = (cudaStream_t)stream;
  const bool w25 = n1 == 25 && n2 == 50 && n3 == 100, w3 = n1 == 3 && n2 == 6 && n3 == 12;
  if (!w25 && !w3) {
    set_error("embed_bwd_tc: embedding widths %d-%d-%d not built (25-50-100, 3-6-12)", n1, n2, n3);
    return GBDP_ERR_INVALID;
  }
  const size_t shm = sizeof(float) * (size_t)(4 * n3 + n3 * (axis + 1) + 4 * axis);
  GBDP_REQUIRE(shm <= 48 * 1024, "embed_bwd_tc: N3 * axis too large");
  if (axis == 16 && ((uintptr_t)dD & 15) == 0 && kDxWarps * dx16_warp_bytes(n3) <= 48 * 1024)
    launch_dep(k_emb_dx16, dim3((unsigned)((nloc + kDxWarps - 1) / kDxWarps)), dim3(kDxWarps * 32),
               kDxWarps * dx16_warp_bytes(n3), st, dx_work, dD, X, drow, nloc, n3,
               1.f / (float)nnei);
  else
    k_emb_dx<<<nloc, 128, shm, st>>>(dx_work, dD, X, drow, n3, axis, 1.f / (float)nnei);
  GBDP_CHECK_LAUNCH("embed_dx");
  int sms = 0;
  const bool split = split_units(nunits, sms);
  if (w25)
    return split ? emb_bwd_launch<25, 50, 100, true>(a, sms, st)
                 : emb_bwd_launch<25, 50, 100, false>(a, sms, st);
  return split ? emb_bwd_launch<3, 6, 12, true>(a, sms, st)
               : emb_bwd_launch<3, 6, 12, false>(a, sms, st);
}
