// Dense min-plus (tropical) GEMM  C[i,j] = min_k A[i,k] + B[k,j]  and the
// APSP repeated-squaring driver.
//
// Tensor cores cannot evaluate (min,+), so the math runs on the CUDA cores:
//   int32 : one DPX __viaddmin_s32 (add + min fused) per (i,j,k) pair;
//   fp32  : two additions (or one packed addition) and a three-input min.f32
//           per two pairs.
// Two kernels share that arithmetic and 8 x 8 outputs per thread:
//   k_minplus_tma : 128 x 128 tiles, each k tile of A (128 rows x 32 k, 128-byte
//                   swizzle) and B (32 k x 128 cols) brought in by TMA
//                   (cp.async.bulk.tensor, mbarrier transaction counts, three
//                   stages, one issuing thread);
//   k_minplus_cp  : 128 x 128 or 64 x 64 tiles filled by cp.async, which takes
//                   any leading dimension and base, with k split over the blocks
//                   of a cluster where the tiles alone would leave SMs idle.
// pick_shape() chooses between them by size and alignment.
//
// Semantics follow minplus_kernel_f32 (HIP_kernel/minplus_mm/src/minplus_hip.cpp:13-118):
// accumulators start at +inf and a NaN candidate never replaces the
// accumulator.  The int32 twin (no reference counterpart) starts at
// INT32_MAX/2 = 1073741823 (the "missing" sentinel), so results are clamped to
// it; inputs must lie in [-2^30, 2^30-1] so no sum overflows.
// Fill values never enter a minimum: k_minplus_tma bounds the loop of a partial
// k tile, k_minplus_cp pads it with A = +inf (missing) and B = 0.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "b2_common.cuh"
#include "b2_internal.hpp"

namespace b2 {
namespace {

constexpr int BM = 128, BN = 128, BK = 32, STAGES = 3, NT = 256;
constexpr int A_TILE = BM * BK;   // elements
constexpr int B_TILE = BK * BN;
constexpr int kMissing = 1073741823;
constexpr int kMaxSplit = 8;      // portable cluster size
typedef unsigned long long Pair;   // two k-adjacent 32-bit operands

// Set by a bounded mbarrier wait that gave up.  One word per device: every
// product clears it in stream order before its launch (clear_mp_error), APSP
// reads it back after its last product, and b2_minplus_status reads it for
// the asynchronous GEMM.  Products that overlap on different streams of one
// device share the word.
__device__ uint32_t g_mp_error;

template <typename T>
struct MP;
template <>
struct MP<float> {
  __device__ __forceinline__ static float init() { return __int_as_float(0x7f800000); }
  // acc = min(acc, a + b0, a + b1)
  __device__ __forceinline__ static float step2(float acc, float a0, float b0, float a1, float b1) {
    const float x = a0 + b0, y = a1 + b1;
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(acc), "f"(x), "f"(y));
    return r;
  }
  __device__ __forceinline__ static float step1(float acc, float a, float b) { return fminf(acc, a + b); }
  __device__ __forceinline__ static float vmin(float x, float y) { return fminf(x, y); }
  // acc = min(acc, a.lo + b.lo, a.hi + b.hi): both sums in one packed addition
  __device__ __forceinline__ static float pair(float acc, Pair a, Pair b) {
    Pair s;
    float x, y, r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(s) : "l"(a), "l"(b));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(s));
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(acc), "f"(x), "f"(y));
    return r;
  }
  static constexpr bool kTwoPerMin = true;   // one 3-input min per two pairs
};
template <>
struct MP<int> {
  __device__ __forceinline__ static int init() { return kMissing; }
  __device__ __forceinline__ static int step2(int acc, int a0, int b0, int a1, int b1) {
    return __viaddmin_s32(a1, b1, __viaddmin_s32(a0, b0, acc));
  }
  __device__ __forceinline__ static int step1(int acc, int a, int b) { return __viaddmin_s32(a, b, acc); }
  __device__ __forceinline__ static int vmin(int x, int y) { return min(x, y); }
  __device__ __forceinline__ static int pair(int acc, Pair a, Pair b) {
    return step2(acc, (int)(uint32_t)a, (int)(uint32_t)b, (int)(a >> 32), (int)(b >> 32));
  }
  static constexpr bool kTwoPerMin = false;  // one fused add+min per pair
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after ~2^22 polls (each poll may suspend), records the
// failure and lets the kernel run to completion instead of hanging.
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < (1u << 22); ++i)
    if (mbar_try_wait(bar, parity)) return;
  atomicExch(&g_mp_error, 1u);
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(smem_dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// Tile order: groups of 8 tile-rows share B panels in L2.
__device__ __forceinline__ void tile_coords(int tiles_m, int tiles_n, int& tm, int& tn) {
  const int id = blockIdx.x;
  const int group = 8;
  const int per_group = group * tiles_n;
  const int g = id / per_group;
  const int first_m = g * group;
  const int gsz = min(tiles_m - first_m, group);
  const int in = id - g * per_group;
  tm = first_m + in % gsz;
  tn = in / gsz;
}

// Compute one k-tile held in shared memory (A swizzled, B plain).  A is read
// as k-pairs (8-byte loads inside the swizzled 16-byte chunk), B as two
// 16-byte vectors per k row.
__device__ __forceinline__ void load_b8(const int* Bs, int k, int tx, int (&b)[8]) {
  const int4 p0 = *reinterpret_cast<const int4*>(Bs + k * BN + tx * 4);
  const int4 p1 = *reinterpret_cast<const int4*>(Bs + k * BN + 64 + tx * 4);
  const int pp[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) b[j] = pp[j];
}

template <bool FULL>
__device__ __forceinline__ void mma_tile(const int* __restrict__ As, const int* __restrict__ Bs, int kvalid, int tx,
                                         int ty, int (&acc)[8][8]) {
  const int sw = ty & 7;
#pragma unroll
  for (int k = 0; k < BK; k += 2) {
    if (!FULL && k >= kvalid) break;
    int a0[8], a1[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = ty + 16 * i;
      const int2 v = *reinterpret_cast<const int2*>(As + r * BK + (((k >> 2) ^ sw) << 2) + (k & 2));
      a0[i] = v.x;
      a1[i] = v.y;
    }
    int b0[8], b1[8];
    load_b8(Bs, k, tx, b0);
    if (FULL || k + 1 < kvalid) {
      load_b8(Bs, k + 1, tx, b1);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = MP<int>::step2(acc[i][j], a0[i], b0[j], a1[i], b1[j]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = MP<int>::step1(acc[i][j], a0[i], b0[j]);
    }
  }
}

__device__ __forceinline__ void store_tile(int* C, int M, int N, int ldc, int m0, int n0, int tx, int ty,
                                           const int (&acc)[8][8], const int* Aold, int lda, uint32_t* changed) {
  bool diff = false;
  const bool vec = ((ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = m0 + ty + 16 * i;
    if (r >= M) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c0 = n0 + h * 64 + tx * 4;
      if (vec && c0 + 3 < N) {
        int4 v;
        v.x = acc[i][h * 4 + 0];
        v.y = acc[i][h * 4 + 1];
        v.z = acc[i][h * 4 + 2];
        v.w = acc[i][h * 4 + 3];
        *reinterpret_cast<int4*>(C + (size_t)r * ldc + c0) = v;
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (c0 + q < N) C[(size_t)r * ldc + c0 + q] = acc[i][h * 4 + q];
      }
      if (Aold) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (c0 + q < N) {
            const int o = Aold[(size_t)r * lda + c0 + q];
            diff |= (o != acc[i][h * 4 + q]);
          }
      }
    }
  }
  if (Aold && __any_sync(0xffffffffu, diff) && (threadIdx.x & 31) == 0) atomicExch(changed, 1u);
}

// TMA pipeline kernel.  `Aold` (nullable): compare results against it and set
// *changed (APSP squaring, where C <= A elementwise because diag(A) = 0).
// `previous` (nullable): the last squaring's word; where it is 0 that squaring
// changed nothing and there is nothing left to do.
__global__ void __launch_bounds__(NT, 2)
    k_minplus_tma(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int* C, int M,
                  int N, int K, int ldc, const int* Aold, int lda, uint32_t* changed, const uint32_t* previous) {
  if (previous && *previous == 0u) return;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  int* As = reinterpret_cast<int*>(base);
  int* Bs = As + STAGES * A_TILE;
  uint64_t* full = reinterpret_cast<uint64_t*>(Bs + STAGES * B_TILE);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  int tm, tn;
  tile_coords((M + BM - 1) / BM, (N + BN - 1) / BN, tm, tn);
  const int m0 = tm * BM, n0 = tn * BN;
  const int KT = (K + BK - 1) / BK;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tid == 0) {
    for (int s = 0; s < STAGES && s < KT; ++s) {
      mbar_expect_tx(&full[s], (A_TILE + B_TILE) * sizeof(int));
      tma_load_2d(As + s * A_TILE, &mapA, s * BK, m0, &full[s]);
      tma_load_2d(Bs + s * B_TILE, &mapB, n0, s * BK, &full[s]);
    }
  }
  int acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = MP<int>::init();
  for (int kt = 0; kt < KT; ++kt) {
    const int s = kt % STAGES;
    mbar_wait(&full[s], (kt / STAGES) & 1);
    const int kvalid = min(BK, K - kt * BK);
    if (kvalid == BK) mma_tile<true>(As + s * A_TILE, Bs + s * B_TILE, BK, tx, ty, acc);
    else mma_tile<false>(As + s * A_TILE, Bs + s * B_TILE, kvalid, tx, ty, acc);
    __syncthreads();   // every thread is done with stage s
    if (tid == 0 && kt + STAGES < KT) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&full[s], (A_TILE + B_TILE) * sizeof(int));
      tma_load_2d(As + s * A_TILE, &mapA, (kt + STAGES) * BK, m0, &full[s]);
      tma_load_2d(Bs + s * B_TILE, &mapB, n0, (kt + STAGES) * BK, &full[s]);
    }
  }
  store_tile(C, M, N, ldc, m0, n0, tx, ty, acc, Aold, lda, changed);
}

// ---- cp.async kernel --------------------------------------------------------
// Bound by instruction issue and register reads, like k_minplus_tma; what it is
// for is everything that keeps that kernel from its rate: operands TMA cannot
// describe (each B word is copied by itself, A 16 bytes at a time where its rows
// allow it), and products with too few 128 x 128 tiles for the GPU.  B's tile is
// stored with each pair of k rows interleaved, [k/2][n][2] (free, since every
// word is placed by its own copy), so that both operands come as k-adjacent
// register pairs and two additions are one add.f32x2.  A cluster of up to 8
// blocks splits k and takes the minimum of its partial tiles through
// distributed shared memory (minima are exact in any order).
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

template <typename T>
struct Operands {
  const T* A;
  const T* B;
  T* C;
  int M, N, K, lda, ldb, ldc;
  const T* Aold;             // APSP: the result is compared with it ...
  uint32_t* changed;         // ... and any difference sets this word
  const uint32_t* previous;  // APSP: as in k_minplus_tma
  int a_vec;                 // A rows start on 16 bytes
  int c_vec;                 // 4: C rows start on 16 bytes, 2: on 8, 1: neither
};

template <int NTX, int NTY, int BK_>
struct Tile {
  static constexpr int NT = NTX * NTY, BM = 8 * NTY, BN = 8 * NTX, BK = BK_;
  static constexpr int kA = BM * BK, kB = BK * BN;   // elements per stage
  static constexpr size_t kSmem = (size_t)STAGES * (kA + kB) * 4;
  static_assert(kSmem >= (size_t)BM * BN * 4, "a partial tile reuses the pipeline's memory");
  // Thread column tx owns columns 4 tx .. 4 tx + 3 of each half of the tile
  // (16-byte stores).  B's columns are permuted in shared memory so that its q-th
  // pair of columns sits at 2 NTX q + 2 tx: the 16-byte reads of 8 neighbouring
  // threads are contiguous.
  __device__ __forceinline__ static int column(int tx, int q) { return 4 * NTX * (q >> 1) + 4 * tx + 2 * (q & 1); }
  __device__ __forceinline__ static int b_position(int n) {
    const int r = n % (4 * NTX);
    return 2 * NTX * (2 * (n / (4 * NTX)) + ((r >> 1) & 1)) + 2 * (r >> 2) + (r & 1);
  }
  // 16-byte chunk of A row r that holds k .. k+3 (chunk c = k / 4): rows read
  // by one warp at the same k fall into different banks
  __device__ __forceinline__ static int a_index(int r, int c) {
    const int f = BK == 32 ? (r & 7) : ((r >> 1) & 3);
    return r * BK + ((c ^ f) << 2);
  }
};

// Start the copies of k tile `kt` into one stage.
template <typename T, class TL>
__device__ __forceinline__ void load_stage(const Operands<T>& P, T* As, T* Bs, int m0, int n0, int kt) {
  const int tid = threadIdx.x;
  const int k0 = kt * TL::BK;
  if (P.a_vec) {
    constexpr int CH = TL::BK / 4, RP = TL::NT / CH;
    const int c = tid % CH, r0 = tid / CH;
    const int k = k0 + 4 * c;
    const T* src = P.A + (size_t)(m0 + r0) * P.lda + k;
    if (k + 4 <= P.K) {
#pragma unroll
      for (int p = 0; p < TL::BM / RP; ++p, src += (size_t)RP * P.lda)
        if (m0 + r0 + p * RP < P.M) cp_async16(smem_u32(As + TL::a_index(r0 + p * RP, c)), src);
    } else {   // the chunk crosses K: pad it
      for (int p = 0; p < TL::BM / RP; ++p, src += (size_t)RP * P.lda)
        for (int q = 0; q < 4; ++q)
          As[TL::a_index(r0 + p * RP, c) + q] =
              (k + q < P.K && m0 + r0 + p * RP < P.M) ? src[q] : MP<T>::init();
    }
  } else {
    constexpr int RP = TL::NT / TL::BK;
    const int k = tid % TL::BK, r0 = tid / TL::BK;
    const T* src = P.A + (size_t)(m0 + r0) * P.lda + k0 + k;
    if (k0 + k < P.K) {
#pragma unroll
      for (int p = 0; p < TL::BM / RP; ++p, src += (size_t)RP * P.lda)
        if (m0 + r0 + p * RP < P.M) cp_async4(smem_u32(As + TL::a_index(r0 + p * RP, k >> 2) + (k & 3)), src);
    } else {
      for (int p = 0; p < TL::BM / RP; ++p) As[TL::a_index(r0 + p * RP, k >> 2) + (k & 3)] = MP<T>::init();
    }
  }
  {
    constexpr int KP = TL::NT / TL::BN;   // k rows per pass
    const int n = tid % TL::BN, kk = tid / TL::BN;
    const T* src = P.B + (size_t)(k0 + kk) * P.ldb + n0 + n;
    const int pos = TL::b_position(n);
    if (k0 + TL::BK <= P.K) {
      if (n0 + n < P.N) {
#pragma unroll
        for (int p = 0; p < TL::BK / KP; ++p, src += (size_t)KP * P.ldb) {
          const int k = kk + p * KP;
          cp_async4(smem_u32(Bs + ((k >> 1) * TL::BN + pos) * 2 + (k & 1)), src);
        }
      }
    } else {
      for (int p = 0; p < TL::BK / KP; ++p, src += (size_t)KP * P.ldb) {
        const int k = kk + p * KP;
        T* dst = Bs + ((k >> 1) * TL::BN + pos) * 2 + (k & 1);
        if (k0 + k < P.K && n0 + n < P.N) cp_async4(smem_u32(dst), src);
        else *dst = T(0);
      }
    }
  }
}

// Two k steps: A as one pair per row (8-byte loads, a warp reads four rows), B
// as 16-byte vectors (two columns' pairs).  Loading A 16 bytes at a time would
// halve its loads but needs 16 more registers than two blocks per SM leave.
template <typename T, class TL>
__device__ __forceinline__ void two_k(const T* As, const T* Bs, int k2, int tx, int ty, T (&acc)[8][8]) {
  constexpr int NTY = TL::BM / 8, NTX = TL::BN / 8;
  Pair a[8], b[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    a[i] = *reinterpret_cast<const Pair*>(As + TL::a_index(ty + NTY * i, k2 >> 1) + 2 * (k2 & 1));
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const ulonglong2 v =
        *reinterpret_cast<const ulonglong2*>(Bs + ((size_t)k2 * TL::BN + 2 * tx + 2 * NTX * q) * 2);
    b[2 * q] = v.x;
    b[2 * q + 1] = v.y;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = MP<T>::pair(acc[i][j], a[i], b[j]);
}

template <typename T, class TL>
__global__ void __launch_bounds__(TL::NT, TL::NT == 256 ? 2 : 8)
    k_minplus_cp(const Operands<T> P, int splits) {
  extern __shared__ __align__(16) unsigned char cp_smem[];
  if (P.previous && *P.previous == 0u) return;   // the whole cluster
  T* As = reinterpret_cast<T*>(cp_smem);
  T* Bs = As + STAGES * TL::kA;
  constexpr int NTX = TL::BN / 8, NTY = TL::BM / 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (lane & 7) + 8 * (warp % (NTX / 8)), ty = (lane >> 3) + 4 * (warp / (NTX / 8));
  // tile order: groups of 8 tile rows share B panels in L2
  const int tiles_m = (P.M + TL::BM - 1) / TL::BM, tiles_n = (P.N + TL::BN - 1) / TL::BN;
  const int tile = blockIdx.x / splits, part = blockIdx.x - tile * splits;   // the cluster's blocks are the k parts
  const int g = tile / (8 * tiles_n), first_m = g * 8;
  const int gsz = min(tiles_m - first_m, 8), in = tile - g * 8 * tiles_n;
  const int m0 = (first_m + in % gsz) * TL::BM, n0 = (in / gsz) * TL::BN;
  const int KT = (P.K + TL::BK - 1) / TL::BK;
  const int kt0 = (int)((int64_t)KT * part / splits), kt1 = (int)((int64_t)KT * (part + 1) / splits);

  T acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = MP<T>::init();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (kt0 + s < kt1) load_stage<T, TL>(P, As + s * TL::kA, Bs + s * TL::kB, m0, n0, kt0 + s);
    cp_async_commit();
  }
  int s = 0;
  for (int kt = kt0; kt < kt1; ++kt) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();   // stage s has landed for everyone; everyone is done with the stage refilled next
    {
      const int nx = s == 0 ? STAGES - 1 : s - 1;
      if (kt + STAGES - 1 < kt1) load_stage<T, TL>(P, As + nx * TL::kA, Bs + nx * TL::kB, m0, n0, kt + STAGES - 1);
      cp_async_commit();
    }
    const T* as = As + s * TL::kA;
    const T* bs = Bs + s * TL::kB;
    if (kt * TL::BK + TL::BK <= P.K) {
#pragma unroll
      for (int k2 = 0; k2 < TL::BK / 2; ++k2) two_k<T, TL>(as, bs, k2, tx, ty, acc);
    } else {
      const int n2 = (P.K - kt * TL::BK + 1) / 2;
      for (int k2 = 0; k2 < n2; ++k2) two_k<T, TL>(as, bs, k2, tx, ty, acc);
    }
    s = s == STAGES - 1 ? 0 : s + 1;
  }

  bool diff = false;
  if (splits == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = m0 + ty + NTY * i;
      if (r >= P.M) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = n0 + TL::column(tx, 2 * h);
        int* dst = reinterpret_cast<int*>(P.C) + (size_t)r * P.ldc + c;
        int v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = *reinterpret_cast<const int*>(&acc[i][4 * h + e]);
        if (P.c_vec == 4 && c + 3 < P.N) {
          *reinterpret_cast<int4*>(dst) = make_int4(v[0], v[1], v[2], v[3]);
        } else if (P.c_vec == 2 && c + 3 < P.N) {
          reinterpret_cast<int2*>(dst)[0] = make_int2(v[0], v[1]);
          reinterpret_cast<int2*>(dst)[1] = make_int2(v[2], v[3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (c + e < P.N) dst[e] = v[e];
        }
        if (P.Aold) {
          const int* old = reinterpret_cast<const int*>(P.Aold) + (size_t)r * P.lda + c;
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (c + e < P.N) diff |= old[e] != v[e];
        }
      }
    }
  } else {
    // partial tile -> own shared memory; then part p reduces rows
    // [p BM / splits, (p + 1) BM / splits) over all the cluster's blocks
    cp_async_wait<0>();
    __syncthreads();
    T* mine = reinterpret_cast<T*>(cp_smem);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        mine[(ty + NTY * i) * TL::BN + TL::column(tx, j >> 1) + (j & 1)] = acc[i][j];
    cluster_sync();
    const int rows = TL::BM / splits;
    const uint32_t base = smem_u32(mine);
    for (int idx = tid; idx < rows * TL::BN; idx += TL::NT) {
      const int lr = part * rows + idx / TL::BN, lc = idx % TL::BN;
      const int r = m0 + lr, c = n0 + lc;
      if (r >= P.M || c >= P.N) continue;
      const uint32_t at = base + (uint32_t)(lr * TL::BN + lc) * 4u;
      T v = MP<T>::init();
      for (int p = 0; p < splits; ++p) {
        int w;
        asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(w) : "r"(cluster_map(at, (uint32_t)p)) : "memory");
        v = MP<T>::vmin(v, *reinterpret_cast<const T*>(&w));
      }
      P.C[(size_t)r * P.ldc + c] = v;
      if (P.Aold) {
        const T o = P.Aold[(size_t)r * P.lda + c];
        diff |= *reinterpret_cast<const int*>(&o) != *reinterpret_cast<const int*>(&v);
      }
    }
    cluster_sync();   // nobody leaves while a peer may still read its tile
  }
  if (P.Aold && __any_sync(0xffffffffu, diff) && lane == 0) *(volatile uint32_t*)P.changed = 1u;
}

// ---- host ----------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

bool make_map(CUtensorMap* map, const int* ptr, int rows, int cols, int ld, int box_cols, int box_rows, bool swz) {
  auto fn = encode_fn();
  if (!fn) return false;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) || ((size_t)ld * sizeof(int)) % 16) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(int)};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<int*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swz ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

constexpr size_t kTmaSmem = (size_t)STAGES * (A_TILE + B_TILE) * 4 + STAGES * 8 + 1024;

// Host-side state kept per device: the TMA kernels' dynamic shared-memory
// attribute is a per-device setting, and the error word's device address is
// looked up with that device current.
constexpr int kMaxDevices = 64;
struct Capacity {
  int sms = 0;
  int big[4] = {}, small[4] = {};   // blocks, then clusters of 2, 4, 8, that fit the device at once
};
struct DeviceState {
  Capacity f32, i32;
  uint32_t* err = nullptr;
  bool tma_used = false;   // a kernel that can set the error word has run on this device
};
std::mutex g_dev_mu;
DeviceState g_dev[kMaxDevices];

cudaError_t current_state(DeviceState** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  *out = &g_dev[dev];
  return cudaSuccess;
}

using Big = Tile<16, 16, 32>;
using Small = Tile<8, 8, 16>;

template <class TL>
cudaLaunchConfig_t cp_config(int64_t tiles, int splits, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * splits));
  cfg.blockDim = dim3(TL::NT);
  cfg.dynamicSmemBytes = TL::kSmem;
  cfg.stream = st;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = (unsigned)splits;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  return cfg;
}

// Per-device facts of one k_minplus_cp instance: its shared-memory attribute
// is made and the clusters that fit the device at once are counted.
template <typename T, class TL>
cudaError_t prepare_cp(int sms, int (&fit)[4]) {
  cudaError_t e =
      cudaFuncSetAttribute(k_minplus_cp<T, TL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TL::kSmem);
  int per = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_minplus_cp<T, TL>, TL::NT, TL::kSmem);
  fit[0] = per * sms;
  for (int i = 1; i < 4 && e == cudaSuccess; ++i) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = cp_config<TL>(1, 1 << i, nullptr, &attr);
    e = cudaOccupancyMaxActiveClusters(&fit[i], k_minplus_cp<T, TL>, &cfg);
  }
  return e;
}

template <typename T>
cudaError_t ensure_kernels(const Capacity** cap) {
  DeviceState* d = nullptr;
  cudaError_t e = current_state(&d);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_dev_mu);
  Capacity& c = std::is_same<T, float>::value ? d->f32 : d->i32;
  if (!c.sms) {
    int dev = 0, sms = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess && std::is_same<T, int>::value)
      e = cudaFuncSetAttribute(k_minplus_tma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTmaSmem);
    if (e == cudaSuccess) e = prepare_cp<T, Big>(sms, c.big);
    if (e == cudaSuccess) e = prepare_cp<T, Small>(sms, c.small);
    if (e != cudaSuccess) return e;
    c.sms = sms;
  }
  *cap = &c;
  return cudaSuccess;
}

enum Kernel { kTma, kBig, kSmall };
struct Shape {
  Kernel kernel;
  int splits;
};

// The kernel, tile and k split with the least estimated time.  Blocks run in
// rounds of as many as fit the device; a round lasts as long as its fullest SM
// needs for its pairs, at about 115 G pairs/s with 8 resident warps or more (a
// 128 x 128 tile's block brings 8, a 64 x 64 tile's 2) and proportionally
// longer with fewer.  Every round adds the fill of the pipeline, a split the
// exchange of partial tiles (both in pairs at the full rate).
// Relative cost of a pair, measured at 4736 x 4096 x 4736: int32 17.0 T pairs/s
// by TMA, 16.4 by the 128-tile cp.async kernel; fp32 16.6 and 17.0, so that
// fp32 has no TMA instance.  The 64-tile kernel reaches 13.7 (2048^3): it
// reads and copies twice the operand bytes per pair.
Shape pick_shape(int M, int N, int K, const Capacity& cap, bool tma, bool is_int) {
  Shape best{kBig, 1};
  double least = 1e300;
  for (int kern = tma && is_int ? kTma : kBig; kern <= kSmall; ++kern) {
    const int bm = kern == kSmall ? Small::BM : Big::BM, bk = kern == kSmall ? Small::BK : Big::BK;
    const int warps = kern == kSmall ? 2 : 8;
    const double cost = kern == kTma ? 1.0 : kern == kBig ? (is_int ? 1.037 : 1.0) : 1.25;
    const int64_t tiles = (int64_t)((M + bm - 1) / bm) * ((N + bm - 1) / bm);
    const int kt = (K + bk - 1) / bk;
    const int most = kern == kTma ? 1 : kMaxSplit;
    for (int i = 0; (1 << i) <= most && (1 << i) <= kt; ++i) {
      const int s = 1 << i;
      const int64_t fit = kern == kSmall ? cap.small[i] : cap.big[i];   // clusters at once
      if (fit < 1) continue;
      const double work = (double)bm * bm * ((kt + s - 1) / s) * bk * cost;   // of one block
      const double fill = 200000.0 + (s > 1 ? 150000.0 + 60.0 * bm * bm : 0.0);
      auto round = [&](int64_t clusters) {
        const int64_t per_sm = (clusters * s + cap.sms - 1) / cap.sms;
        return work * per_sm / std::min(1.0, per_sm * warps / 8.0) + fill;
      };
      double t = 0.0;
      if (tiles / fit) t += (double)(tiles / fit) * round(fit);
      if (tiles % fit) t += round(tiles % fit);
      if (t < least) {
        least = t;
        best = Shape{(Kernel)kern, s};
      }
    }
  }
  return best;
}

// Device address of g_mp_error on the current device.
cudaError_t mp_error_ptr(uint32_t** out) {
  DeviceState* d = nullptr;
  cudaError_t e = current_state(&d);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_dev_mu);
  if (!d->err) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_mp_error);
    if (e != cudaSuccess) return e;
    d->err = (uint32_t*)p;
  }
  *out = d->err;
  return cudaSuccess;
}

// Only k_minplus_tma waits on barriers and can set the error word.  Until it has
// run on a device the word is 0, and the calls below skip their memset and copy.
cudaError_t mark_tma_used() {
  DeviceState* d = nullptr;
  cudaError_t e = current_state(&d);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_dev_mu);
  d->tma_used = true;
  return cudaSuccess;
}
cudaError_t tma_used(bool* used) {
  DeviceState* d = nullptr;
  cudaError_t e = current_state(&d);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(g_dev_mu);
  *used = d->tma_used;
  return cudaSuccess;
}

// Stream-ordered clear of the error word (allocates nothing).
cudaError_t clear_mp_error(cudaStream_t st) {
  bool used = false;
  cudaError_t e = tma_used(&used);
  if (e != cudaSuccess || !used) return e;
  uint32_t* p = nullptr;
  e = mp_error_ptr(&p);
  if (e != cudaSuccess) return e;
  return cudaMemsetAsync(p, 0, sizeof(uint32_t), st);
}

// Wait for the stream, then read the error word: B2_TIMEOUT when a wait of a
// product issued since the last clear gave up.
b2_status read_mp_error(cudaStream_t st) {
  bool used = false;
  B2_CUDA_TRY(tma_used(&used));
  uint32_t err = 0;
  if (used) {
    uint32_t* p = nullptr;
    B2_CUDA_TRY(mp_error_ptr(&p));
    B2_CUDA_TRY(cudaMemcpyAsync(&err, p, sizeof(err), cudaMemcpyDeviceToHost, st));
  }
  B2_CUDA_TRY(cudaStreamSynchronize(st));
  return err ? B2_TIMEOUT : B2_SUCCESS;
}

template <typename T, class TL>
cudaError_t launch_cp(const Operands<T>& P, int splits, cudaStream_t st) {
  const int64_t tiles = (int64_t)((P.M + TL::BM - 1) / TL::BM) * ((P.N + TL::BN - 1) / TL::BN);
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cp_config<TL>(tiles, splits, st, &attr);
  return cudaLaunchKernelEx(&cfg, k_minplus_cp<T, TL>, P, splits);
}

template <typename T>
bool tma_can_read(const T* p, int ld) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && (ld & 3) == 0;
}

cudaError_t launch_tma(const int* A, const int* B, int* C, int M, int N, int K, int lda, int ldb, int ldc,
                       cudaStream_t st, const int* Aold, uint32_t* changed, const uint32_t* previous, bool* launched) {
  CUtensorMap ma, mb;
  *launched = make_map(&ma, A, M, K, lda, BK, BM, true) && make_map(&mb, B, K, N, ldb, BN, BK, false);
  if (!*launched) return cudaSuccess;
  const cudaError_t e = mark_tma_used();
  if (e != cudaSuccess) return e;
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  k_minplus_tma<<<tiles, NT, kTmaSmem, st>>>(ma, mb, C, M, N, K, ldc, Aold, lda, changed, previous);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_minplus(const T* A, const T* B, T* C, int M, int N, int K, int lda, int ldb, int ldc,
                           cudaStream_t st, const T* Aold = nullptr, uint32_t* changed = nullptr,
                           const uint32_t* previous = nullptr) {
  const Capacity* cap = nullptr;
  cudaError_t e = ensure_kernels<T>(&cap);
  if (e != cudaSuccess) return e;
  const bool a_vec = tma_can_read(A, lda);
  Shape sh = pick_shape(M, N, K, *cap, a_vec && tma_can_read(B, ldb), std::is_same<T, int>::value);
  if constexpr (std::is_same<T, int>::value) {
    if (sh.kernel == kTma) {
      bool launched = false;
      e = launch_tma(A, B, C, M, N, K, lda, ldb, ldc, st, Aold, changed, previous, &launched);
      if (launched || e != cudaSuccess) return e;
      sh = Shape{kBig, 1};   // no tensor map (driver entry point missing)
    }
  }
  Operands<T> P;
  P.A = A;
  P.B = B;
  P.C = C;
  P.M = M;
  P.N = N;
  P.K = K;
  P.lda = lda;
  P.ldb = ldb;
  P.ldc = ldc;
  P.Aold = Aold;
  P.changed = changed;
  P.previous = previous;
  P.a_vec = a_vec;
  const uintptr_t c = reinterpret_cast<uintptr_t>(C);
  P.c_vec = (c & 15) == 0 && (ldc & 3) == 0 ? 4 : (c & 7) == 0 && (ldc & 1) == 0 ? 2 : 1;
  return sh.kernel == kBig ? launch_cp<T, Big>(P, sh.splits, st) : launch_cp<T, Small>(P, sh.splits, st);
}

template <typename T>
b2_status gemm(const T* A, const T* B, T* C, int M, int N, int K, int lda, int ldb, int ldc, b2_stream s) {
  // argument rules of minplus_gemm_f32 (minplus_hip.cpp:132-142)
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0 || lda < K || ldb < N || ldc < N) return B2_INVALID_ARGUMENT;
  B2_CUDA_TRY(clear_mp_error((cudaStream_t)s));
  return from_cuda(launch_minplus<T>(A, B, C, M, N, K, lda, ldb, ldc, (cudaStream_t)s));
}

// D <- tmp where the last squaring changed something (an unchanged or skipped
// one leaves the same matrix in both).
__global__ void k_copy_if(const uint32_t* changed, size_t n, const uint32_t* __restrict__ src,
                          uint32_t* __restrict__ dst) {
  if (*changed == 0u) return;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

constexpr int kMaxSquarings = 31;   // ceil(log2(N - 1)) for any int N

// Repeated squaring between D and tmp.  Every product that may be needed is
// queued at once; the device stops by itself: a product sets its word of `flags`
// when it changes an entry, and a product whose predecessor's word is 0 returns
// at once (about 2 us), so the host waits once, not after every product.
template <typename T>
b2_status square_until_fixed(T* D, T* tmp, uint32_t* flags, int N, cudaStream_t st, int* done) {
  int maxsq = 0;
  while ((1ll << maxsq) < (long long)(N - 1)) ++maxsq;   // ceil(log2(N-1)) products reach N-1 hops
  const size_t words = (size_t)std::max(maxsq, 1);
  B2_CUDA_TRY(clear_mp_error(st));
  B2_CUDA_TRY(cudaMemsetAsync(flags, 0, words * sizeof(uint32_t), st));
  T* cur = D;
  T* nxt = tmp;
  for (int it = 0; it < maxsq; ++it) {
    B2_CUDA_TRY(launch_minplus<T>(cur, cur, nxt, N, N, N, N, N, N, st, cur, flags + it,
                                  it ? flags + it - 1 : nullptr));
    std::swap(cur, nxt);
  }
  if (cur != D) {
    k_copy_if<<<1184, 256, 0, st>>>(flags + maxsq - 1, (size_t)N * N, (const uint32_t*)tmp, (uint32_t*)D);
    B2_CUDA_TRY(cudaGetLastError());
  }
  uint32_t h[kMaxSquarings] = {};
  B2_CUDA_TRY(cudaMemcpyAsync(h, flags, words * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  const b2_status r = read_mp_error(st);
  if (r != B2_SUCCESS) return r;
  *done = maxsq;
  for (int it = 0; it < maxsq; ++it)
    if (h[it] == 0) {   // D unchanged: fixpoint reached
      *done = it + 1;
      break;
    }
  return B2_SUCCESS;
}

// The second matrix and the flags come from the library's stream-ordered pool
// up to this size (a cudaMalloc and cudaFree of it cost 1-2 ms, as much as all
// the products of a 1000-vertex graph); past it from cudaMalloc, so that the
// pool's cache stays small.
constexpr size_t kApspPoolMax = (size_t)256 << 20;

template <typename T>
b2_status apsp(T* D, int N, b2_stream s, int32_t* squarings) {
  if (!D || N <= 0) return B2_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)s;
  if (squarings) *squarings = 0;
  if (N == 1) return B2_SUCCESS;
  const size_t matrix = ((size_t)N * N * sizeof(T) + 255) & ~(size_t)255;
  const size_t bytes = matrix + 256;
  const bool pooled = bytes <= kApspPoolMax;
  unsigned char* buf = nullptr;
  if (pooled) {
    cudaMemPool_t pool;
    B2_CUDA_TRY(scratch_pool(&pool));
    B2_CUDA_TRY(cudaMallocFromPoolAsync((void**)&buf, bytes, pool, st));
  } else {
    B2_CUDA_TRY(cudaMalloc((void**)&buf, bytes));
  }
  int done = 0;
  const b2_status r = square_until_fixed<T>(D, (T*)buf, (uint32_t*)(buf + matrix), N, st, &done);
  if (pooled) cudaFreeAsync(buf, st);
  else cudaFree(buf);
  if (squarings) *squarings = done;
  return r;
}

// ---- ALU peak calibration (roofline denominator for min-plus) -------------
// Updates of an 8 x 8 accumulator tile per thread on registers only (int32: the
// GEMMs' one __viaddmin_s32 per pair; fp32: two additions and one three-input min
// per two pairs), with no shared-memory or global traffic.  The A operand of row i
// at step k is an accumulator of that row (acc[i][(i + k) & 7], a register chosen at
// compile time), so every sum is a new value and no sum can be folded or shared
// between pairs; B is 8 (16 for fp32) runtime constants.  fp32 reads 21.5 T pairs/s;
// the packed addition and three-input min of k_minplus_cp read 18.7 in registers,
// in the order that the compiler gives them, and loops whose additions share an
// operand reached 26.8, so this is a measure, not a bound.
template <typename T>
__global__ void __launch_bounds__(256) k_calibrate(int iters, T seed, T step, T* sink) {
  T acc[8][8];
  T b0[8], b1[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    b0[j] = step + (T)j;
    b1[j] = step + (T)(j + 8);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = seed + (T)(threadIdx.x + 8 * i + j);
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const T a0 = acc[i][(i + k) & 7];
        const T a1 = acc[i][(i + k + 3) & 7];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (sizeof(T) == 4 && MP<T>::kTwoPerMin) acc[i][j] = MP<T>::step2(acc[i][j], a0, b0[j], a1, b1[j]);
          else acc[i][j] = MP<T>::step1(acc[i][j], a0, b0[j]);
        }
      }
    }
  }
  T r = acc[0][0];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) r = r < acc[i][j] ? r : acc[i][j];
  if (r == (T)-12345) sink[0] = r;
}

}  // namespace
}  // namespace b2

using namespace b2;

extern "C" b2_status b2_minplus_gemm_f32(const float* dA, const float* dB, float* dC, int32_t M, int32_t N,
                                         int32_t K, int32_t lda, int32_t ldb, int32_t ldc, b2_stream stream) {
  return gemm<float>(dA, dB, dC, M, N, K, lda, ldb, ldc, stream);
}

extern "C" b2_status b2_minplus_gemm_i32(const int32_t* dA, const int32_t* dB, int32_t* dC, int32_t M, int32_t N,
                                         int32_t K, int32_t lda, int32_t ldb, int32_t ldc, b2_stream stream) {
  return gemm<int>(dA, dB, dC, M, N, K, lda, ldb, ldc, stream);
}

extern "C" b2_status b2_apsp_f32(float* d_D, int32_t N, b2_stream stream, int32_t* sq) {
  return apsp<float>(d_D, N, stream, sq);
}

extern "C" b2_status b2_apsp_i32(int32_t* d_D, int32_t N, b2_stream stream, int32_t* sq) {
  return apsp<int>(d_D, N, stream, sq);
}

extern "C" b2_status b2_minplus_status(b2_stream stream) {
  return read_mp_error((cudaStream_t)stream);
}

extern "C" b2_status b2_minplus_calibrate(int32_t is_float, double* pairs_per_second) {
  if (!pairs_per_second) return B2_INVALID_ARGUMENT;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int threads = 256, blocks = sms * 4, iters = 1 << 12;
  void* sink = nullptr;
  B2_CUDA_TRY(cudaMalloc(&sink, 16));
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  for (int rep = 0; rep < 4; ++rep) {
    cudaEventRecord(e0);
    if (is_float) k_calibrate<float><<<blocks, threads>>>(iters, 0.5f, 0.25f, (float*)sink);
    else k_calibrate<int><<<blocks, threads>>>(iters, 3, 1, (int*)sink);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    if (rep > 0) best = std::min(best, ms);
  }
  cudaError_t e = cudaGetLastError();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(sink);
  if (e != cudaSuccess) return from_cuda(e);
  // per thread and iteration: 8 k steps x 64 updates; an fp32 update is two pairs
  const double pairs = (double)blocks * threads * iters * 8.0 * 64.0 * (is_float ? 2.0 : 1.0);
  *pairs_per_second = pairs / (best * 1e-3);
  return B2_SUCCESS;
}

// ---- allocation-free APSP --------------------------------------------------
// Some callers cannot allocate device memory while they run:
//   * a plugin inside a host whose device memory is owned by another
//     allocator (a framework's caching pool), where a cudaMalloc would
//     fragment or exceed that pool's budget;
//   * a latency-bound serving loop with a fixed memory budget, where
//     cudaMalloc / cudaFree would synchronize the device and add jitter;
//   * code running while a device-wide allocation freeze is in effect.
// b2_apsp_f32_noalloc runs the same repeated squaring as b2_apsp_f32, but its
// ping-pong matrix and change flags live in the fixed array below instead of a
// cudaMalloc'd buffer.  Limits and rules:
//   * N * N * 4 bytes must fit in the array (N <= 2048); larger N is rejected
//     with B2_NOT_SUPPORTED before anything runs;
//   * the array is a module global: every GPU that loads this library holds
//     its 16 MiB until the process exits;
//   * every call on a device shares the one array, and it keeps the previous
//     call's contents (the change flags are cleared at the start of a call): calls
//     that overlap on the GPU (different streams or threads) race and must be
//     serialized by the caller;
//   * the first call on each device looks up the array's device address
//     (cudaGetSymbolAddress) with that device current; make that first call
//     before any stream capture.
namespace b2 {
namespace {
constexpr size_t kNoAllocScratchBytes = (size_t)16 << 20;   // 16 MiB: 2048 x 2048 floats
// scratch matrix, then the squarings' change flags in the last 256 bytes
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes + 256];

std::mutex g_noalloc_mu;
void* g_noalloc_ptr[64] = {};

// Device address of g_noalloc_scratch for the current device (looked up once
// per device; the host-side symbol itself is not a device address).
cudaError_t noalloc_scratch(unsigned char** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_noalloc_ptr[dev] = p;
  }
  *out = (unsigned char*)g_noalloc_ptr[dev];
  return cudaSuccess;
}
}  // namespace
}  // namespace b2

extern "C" b2_status b2_apsp_f32_noalloc(float* d_D, int32_t N, b2_stream stream, int32_t* squarings) {
  using namespace b2;
  if (!d_D || N <= 0) return B2_INVALID_ARGUMENT;
  if ((size_t)N * (size_t)N * sizeof(float) > kNoAllocScratchBytes) return B2_NOT_SUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  if (squarings) *squarings = 0;
  if (N == 1) return B2_SUCCESS;
  unsigned char* base = nullptr;
  B2_CUDA_TRY(noalloc_scratch(&base));
  int done = 0;
  const b2_status r =
      square_until_fixed<float>(d_D, (float*)base, (uint32_t*)(base + kNoAllocScratchBytes), N, st, &done);
  if (squarings) *squarings = done;
  return r;
}
