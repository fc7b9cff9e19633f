// CSR x CSR min-plus product  C = A (min,+) B  (fp32 and int32).
//
// Semantics follow minplus_sparse::minplus_spgemm_csr_f32
// (HIP_kernel/minplus_mm/src/minplus_sparse_hip.hpp:64-150,
// minplus_sparse_hip.cpp:93-99, 170-398): absent entries are +inf; explicit
// +inf and NaN entries of A, and +inf / NaN candidates a + b, are skipped;
// duplicate columns are min-reduced; a bad row pointer or column index makes
// the call fail.  Outputs are allocated here and owned by the caller.
// Unlike the reference (per-row shared-memory hash with a fixed capacity and
// unsorted output) rows have no size limit and output columns are sorted.
//
// Plan (one pass over the expansion for ordinary rows):
//   1. k_row_bound : candidates per row (sum of |B row k| over A's row);
//                    validates A's and B's row pointers and A's columns and
//                    lists the rows of more than 128 and of more than 512
//                    candidates;
//   2. scan        : candidate offsets (CUB) = each row's slot in a scratch
//                    array sized by the bound;
//   3. k_rows      : half a warp per row of up to 128 candidates, a warp per row
//                    of up to 512: gather, sort (column, slot) keys in
//                    registers, write each column's minimum to the row's
//                    scratch slot;
//   4. long rows   : k_rows_dense accumulates them in shared memory, one word
//                    per column (in passes over a wide matrix's columns); rows
//                    too short for their passes are expanded, sorted and
//                    compressed (k_expand, CUB segmented sort, k_compress) into
//                    the same scratch slots;
//   5. scan of the counts (CUB) -> C.rowptr, then k_compact copies every row
//      from its scratch slot to the exact-size outputs: memory this call
//      allocates (the reference's one-call form), or the caller's own buffers
//      (b2_minplus_spgemm_plan / _fill, which need no output allocation here).
// Scratch arrays come from a library-owned stream-ordered memory pool that
// keeps up to 4 GiB cached between calls (no cudaMalloc / cudaFree on the
// critical path after the first call).
// The int32 twin treats values >= INT32_MAX/2 as absent and drops sums that
// reach it.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "b2_common.cuh"
#include "b2_internal.hpp"
#include "b2_relax.cuh"

namespace b2 {
namespace {

constexpr int32_t kMiss32 = 1073741823;
constexpr int32_t kDropCol = 0x7fffffff;   // sorts after every real column
constexpr int kWarpRowMax = 512;           // candidates of a row sorted in one warp's registers
constexpr int kSmallRowMax = 128;          // candidates of a row sorted in half a warp's registers
constexpr int kRowWarps = 8;               // warps per block of k_rows

// Long rows: k_rows_dense takes a row of a matrix of up to kDenseCols columns
// (192 KB of shared memory), and of a wider one in passes over its columns if the
// row has enough candidates for them.  A pass costs its scan of the columns (about
// 6 us) whatever the row holds; expanding and sorting costs by the candidate, more
// so once CUB no longer sorts a segment in one block (5000 candidates, and again
// about 20000) and where the expansion does not fit the memory that the pool keeps.
// So rows of under kDensePerPass candidates a pass are sorted, rows of sorted_max()
// or more accumulated densely, and those between as sort_between() says.  2^13 rows
// of 3000 candidates in 150000 columns (four passes) 2.64 ms densely and 1.42
// sorted, of 8000 3.93 and 3.91; of 16000 in 600000 columns (13 passes) 16.4 and
// 7.1, of 24000 21 and 34; 100 rows of 8000 in 300000 columns 0.28 and 0.53.  90000
// rows of 2025 in 90000 columns (3 GB of expansion) 15 ms densely and 28 to 65
// sorted, RMAT-18 of edge factor 2 18 and 25 to 38; below kDensePerPass, 250000 rows
// of 576 in 250000 columns 60 and 19.
constexpr int kDenseCols = 49152;
constexpr int kDensePasses = 16;
constexpr unsigned long long kDensePerPass = 640;
constexpr int64_t kSortRows = 512;   // fewer rows leave the sort's one block each waiting for the longest
unsigned long long sorted_max(unsigned long long passes) {
  return passes < 4 ? 5120 : std::min(20000ull, 8192 + 5800 * (passes - 4));
}
constexpr unsigned long long kHeavyRow = 32768;   // dealt first, so that none starts last
constexpr int kDenseThreads = 1024;               // largest block of k_rows_dense
// Candidates of a row are counted in 32 bits, and the index that walks them must
// not wrap in its last step of up to kDenseThreads; longer rows are refused.
constexpr unsigned long long kDenseRowMax = 0xFFFFFFFFull - kDenseThreads;

enum SpStatus : uint32_t { kSpOk = 0, kSpBadIndex = 1, kSpBadRowptr = 2 };

template <typename T>
struct SpVal;
template <>
struct SpVal<float> {
  __device__ __forceinline__ static bool present(float a) { return a == a && a != __int_as_float(0x7f800000); }
  __device__ __forceinline__ static bool combine(float a, float b, float& out) {
    out = a + b;
    return present(out);
  }
  __device__ __forceinline__ static float vmin(float x, float y) { return y < x ? y : x; }
};
template <>
struct SpVal<int32_t> {
  __device__ __forceinline__ static bool present(int32_t a) { return a < kMiss32; }
  __device__ __forceinline__ static bool combine(int32_t a, int32_t b, int32_t& out) {
    if (b >= kMiss32) return false;
    const long long s = (long long)a + (long long)b;
    out = (int32_t)s;
    return s < kMiss32;
  }
  __device__ __forceinline__ static int32_t vmin(int32_t x, int32_t y) { return y < x ? y : x; }
};

// Order-preserving 32-bit encodings of the values (sorting (column, key)
// pairs puts each column's minimum first).
template <typename T>
struct VKey;
template <>
struct VKey<float> {
  __device__ __forceinline__ static uint32_t enc(float v) { return f32_to_key(v); }
  __device__ __forceinline__ static float dec(uint32_t k) { return key_to_f32(k); }
};
template <>
struct VKey<int32_t> {
  __device__ __forceinline__ static uint32_t enc(int32_t v) { return (uint32_t)v ^ 0x80000000u; }
  __device__ __forceinline__ static int32_t dec(uint32_t k) { return (int32_t)(k ^ 0x80000000u); }
};

// Device counters read back in one copy after k_row_bound.
struct SpCounters {
  unsigned long long heavy, lng, mid, wide;   // entries of the four row lists
  unsigned long long between;                 // rows of `wide` that may as well be accumulated densely
  unsigned long long split[2];                // cursors of k_split
  uint32_t status;
  uint32_t too_long;   // a row of more than kDenseRowMax candidates
};

// Candidates per row, validation, and the lists of the rows that need
// more than half a warp.  Two arrays of M entries hold four lists, one from each
// end: mid_rows the rows of up to kWarpRowMax candidates (front) and the long rows
// to expand and sort (back); long_rows the long rows to accumulate densely, those
// of at least `dense_from` candidates, the ones of kHeavyRow or more from the front
// and the others from the back.  LANES lanes per row (bound_lanes), list appends
// aggregated per warp.
template <int LANES>
__global__ void k_row_bound(int64_t M, int64_t K, int64_t annz, int64_t bnnz, const int64_t* __restrict__ arp,
                            const int32_t* __restrict__ aci, const int64_t* __restrict__ brp,
                            unsigned long long* __restrict__ ub, SpCounters* cnt, int64_t* __restrict__ long_rows,
                            int64_t* __restrict__ mid_rows, unsigned long long dense_from,
                            unsigned long long dense_slots) {
  const uint32_t lane = threadIdx.x & 31u, sub = lane & (LANES - 1);
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  constexpr int kRpw = 32 / LANES;
  for (int64_t base = warp * kRpw; base < M; base += nwarps * kRpw) {
    const int64_t i = base + lane / LANES;
    unsigned long long s = 0;
    if (i < M) {
      const int64_t a0 = arp[i], a1 = arp[i + 1];
      if (a0 < 0 || a1 < a0 || a1 > annz) {
        if (sub == 0) atomicCAS(&cnt->status, kSpOk, (uint32_t)kSpBadRowptr);
      } else {
        for (int64_t p = a0 + sub; p < a1; p += LANES) {
          const int32_t k = aci[p];
          if (k < 0 || (int64_t)k >= K) {
            atomicCAS(&cnt->status, kSpOk, (uint32_t)kSpBadIndex);
            continue;
          }
          const int64_t b0 = brp[k], b1 = brp[k + 1];
          if (b0 < 0 || b1 < b0 || b1 > bnnz) {
            atomicCAS(&cnt->status, kSpOk, (uint32_t)kSpBadRowptr);
            continue;
          }
          s += (unsigned long long)(b1 - b0);
        }
      }
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const bool lead = sub == 0 && i < M;
    const bool is_long = lead && s > (unsigned long long)kWarpRowMax;
    const bool is_dense = is_long && s >= dense_from;
    const bool is_heavy = is_dense && s >= kHeavyRow;
    const bool is_mid = lead && !is_long && s > (unsigned long long)kSmallRowMax;
    if (is_dense && s > kDenseRowMax) cnt->too_long = 1u;
    if (lead) ub[i] = is_dense && s > dense_slots ? dense_slots : s;
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t bh = __ballot_sync(0xffffffffu, is_heavy);
    const uint32_t bl = __ballot_sync(0xffffffffu, is_dense && !is_heavy);
    const uint32_t bm = __ballot_sync(0xffffffffu, is_mid);
    const uint32_t bw = __ballot_sync(0xffffffffu, is_long && !is_dense);
    if (bh | bl | bm | bw) {
      unsigned long long ph = 0, pl = 0, pm = 0, pw = 0;
      if (lane == 0) {
        if (bh) ph = atomicAdd(&cnt->heavy, (unsigned long long)__popc(bh));
        if (bl) pl = atomicAdd(&cnt->lng, (unsigned long long)__popc(bl));
        if (bm) pm = atomicAdd(&cnt->mid, (unsigned long long)__popc(bm));
        if (bw) pw = atomicAdd(&cnt->wide, (unsigned long long)__popc(bw));
      }
      ph = __shfl_sync(0xffffffffu, ph, 0);
      pl = __shfl_sync(0xffffffffu, pl, 0);
      pm = __shfl_sync(0xffffffffu, pm, 0);
      pw = __shfl_sync(0xffffffffu, pw, 0);
      if (is_heavy) long_rows[ph + __popc(bh & below)] = i;
      else if (is_dense) long_rows[M - 1 - (int64_t)(pl + __popc(bl & below))] = i;
      else if (is_long) mid_rows[M - 1 - (int64_t)(pw + __popc(bw & below))] = i;
      else if (is_mid) mid_rows[pm + __popc(bm & below)] = i;
    }
  }
}

// A row of A rarely has more than eight entries, and a warp for each leaves most
// lanes idle (2^20 rows of 8: 0.14 ms with a warp, 0.07 with eight lanes; even for
// rows of 384 the two are alike).  Where the rows are so few that a warp for each is
// at hand anyway, the longest of them is what counts (the call for 8192 rows of 3000
// entries, 3000 columns: 0.83 ms with eight lanes, 0.67 with a warp; for one row of
// 10^6 entries 32.3 and 11.7).
int bound_lanes(int64_t M) { return M <= 8192 ? 32 : 8; }

template <typename T>
struct RowArgs {
  int64_t M, N;
  const int64_t* __restrict__ arp;
  const int32_t* __restrict__ aci;
  const T* __restrict__ av;
  const int64_t* __restrict__ brp;
  const int32_t* __restrict__ bci;
  const T* __restrict__ bv;
  const unsigned long long* __restrict__ off;
  int32_t* __restrict__ tcol;
  T* __restrict__ tval;
  int64_t* __restrict__ cnt;
  uint32_t* status;
};

// ---- ordinary rows: a warp or half a warp, registers ------------------------
// A row of up to 128 candidates takes half a warp (two rows' gathers in flight
// per warp), one of up to 512 a whole warp.  The lanes of a row gather its
// candidates, sort them by column in registers and write each column's minimum.
//
// What is sorted is (column, slot), not (column, value): with the column in the
// upper bits of a 32-bit word and the candidate's slot in the lower ones a
// compare-exchange is one shuffle and one minimum or maximum, where 64-bit
// (column, value) keys took two shuffles, a two-word comparison and two
// selects.  Values wait in shared memory under their slot.  Matrices whose
// columns do not fit beside the slot (2^25 columns for half a warp, 2^23 for a
// whole one) use the same code with 64-bit words.
//
// Every comparison of the network is ascending, so padding never moves and a row
// takes as many registers a lane as it needs, not a power of two: 70 candidates
// on 16 lanes sort 5 registers.  Candidates land in registers directly, all
// their loads in flight at once, when the row of A has at most one entry per
// lane; longer ones go through shared memory.
//
// Bound by instruction issue (0.75 per cycle and scheduler).  A (x) A, 2^20 rows
// of 8 (67 M candidates), int32: row kernels 2.41 ms with 64-bit (column, value)
// keys -> 0.77 ms; the call 2.90 -> 1.19 ms.
template <typename K>
struct RowKey;
template <>
struct RowKey<uint32_t> {
  __device__ __forceinline__ static uint32_t shfl_xor(uint32_t x, int m) { return __shfl_xor_sync(0xffffffffu, x, m); }
};
template <>
struct RowKey<unsigned long long> {
  __device__ __forceinline__ static unsigned long long shfl_xor(unsigned long long x, int m) {
    return __shfl_xor_sync(0xffffffffu, x, m);
  }
};

// Batcher's odd-even merge sort of key[0 .. PR) in one lane's registers.  Every
// comparison puts the smaller key at the lower index, so the network of the next
// power of two serves any PR.  The comparisons are listed at compile time: as
// nested loops the compiler left those of 16 registers rolled and indexed the
// registers by selection, five times the instructions (int32, 2^16 rows of 400
// candidates: the call 1.42 ms, with the list 0.61; rows of 361 0.51 either way).
template <int PR>
struct Network {
  int n = 0, lo[64] = {}, hi[64] = {};
  constexpr Network() {
    const int w = PR <= 4 ? 4 : PR <= 8 ? 8 : 16;
    for (int p = 1; p < w; p *= 2)
      for (int k = p; k >= 1; k /= 2)
        for (int x = 0; x < PR - k; ++x)
          if (x >= k % p && (x - k % p) % (2 * k) < k && x / (2 * p) == (x + k) / (2 * p)) {
            lo[n] = x;
            hi[n++] = x + k;
          }
  }
};
template <int A, int B, typename K, int P>
__device__ __forceinline__ void order(K (&key)[P]) {
  const K lo = key[A], hi = key[B];
  key[A] = min(lo, hi);
  key[B] = max(lo, hi);
}
template <int PR, typename K, int P, size_t... I>
__device__ __forceinline__ void apply_network(K (&key)[P], std::index_sequence<I...>) {
  constexpr Network<PR> net;
  (order<net.lo[I], net.hi[I]>(key), ...);
}
template <typename K, int PR, int P>
__device__ __forceinline__ void sort_lane(K (&key)[P]) {
  constexpr Network<PR> net;
  apply_network<PR>(key, std::make_index_sequence<net.n>());
}

// Ascending sort of the first PR registers of each group of LANES lanes, element
// e = lane * PR + r: lanes sort their own registers, then runs of 2, 4, ... lanes
// merge (mirrored comparison, half-cleaners across lanes, sort within lanes).
// Ten steps of a 16-lane sort need shuffles; with elements dealt to the lanes in
// turn 25 would.  The merges are one loop, not unrolled: with a fully unrolled
// network per PR, warps of different PR evicted each other's instructions
// (no-instruction stalls 27 of 33 cycles per issue, 2.25 ms).
template <typename K, int LANES, int PR, int P>
__device__ __forceinline__ void sort_keys(K (&key)[P], uint32_t hl) {
#pragma unroll 1
  for (int run = 1;; run *= 2) {   // lanes per sorted run
    sort_lane<K, PR>(key);
    if (run == LANES) break;
    const bool lower = (hl & (uint32_t)run) == 0;
#pragma unroll
    for (int r = 0; r < (PR + 1) / 2; ++r) {
      const K x = RowKey<K>::shfl_xor(key[PR - 1 - r], 2 * run - 1);
      const K y = RowKey<K>::shfl_xor(key[r], 2 * run - 1);
      key[r] = lower ? min(key[r], x) : max(key[r], x);
      if (r != PR - 1 - r) key[PR - 1 - r] = lower ? min(key[PR - 1 - r], y) : max(key[PR - 1 - r], y);
    }
#pragma unroll 1
    for (int j = run / 2; j > 0; j /= 2) {
      const bool low = (hl & (uint32_t)j) == 0;
#pragma unroll
      for (int r = 0; r < PR; ++r) {
        const K o = RowKey<K>::shfl_xor(key[r], j);
        key[r] = low ? min(key[r], o) : max(key[r], o);
      }
    }
  }
}

// Sort and leave the keys in order in skey[0 .. LANES * regs).  True if some
// lane's keys are all of one column, as every run of 2 PR - 1 or more has a lane's
// (not asked for half warps, whose runs are short enough to walk).
template <typename K, int LANES, int PR, int SB, int P>
__device__ __forceinline__ bool sort_to_shared(K (&key)[P], uint32_t hl, K* skey) {
  sort_keys<K, LANES, PR>(key, hl);
  __syncwarp();   // staged keys have been read
#pragma unroll
  for (int r = 0; r < PR; ++r) skey[hl * PR + r] = key[r];
  if (LANES < 32) return false;
  return __any_sync(0xffffffffu, key[PR - 1] != ~(K)0 && (key[0] >> SB) == (key[PR - 1] >> SB));
}

// One lane's share of a chunk of up to LANES entries of a row of A.
template <typename T, typename K>
struct Entry {
  // an index into B, in 32 bits where the keys are (only used with nnz(B) < 2^31)
  typedef typename std::conditional<sizeof(K) == 4, int32_t, long long>::type Index;
  T a;
  Index base;        // candidate slot sl of this entry is base + sl
  uint32_t excl, len;
};

// Load the chunk and lay its B ranges out one after the other; entries without
// candidates are moved out of the way, so that range starts are distinct.
// Returns the chunk's candidates (per row).
template <typename T, typename K, int LANES>
__device__ __forceinline__ uint32_t load_entries(const RowArgs<T>& R, int64_t p, bool in, uint32_t hl, uint32_t shift,
                                                 Entry<T, K>& e) {
  typedef typename Entry<T, K>::Index Index;
  Index b0 = 0;
  e.a = T(0);
  e.len = 0;
  if (in) {
    const int32_t k = R.aci[p];
    e.a = R.av[p];
    const int64_t x = R.brp[k], y = R.brp[k + 1];
    if (SpVal<T>::present(e.a)) {
      b0 = (Index)x;
      e.len = (uint32_t)(y - x);
    }
  }
  constexpr uint32_t kAll = LANES == 32 ? 0xffffffffu : (1u << (LANES & 31)) - 1u;
  const uint32_t some = (__ballot_sync(0xffffffffu, e.len > 0) >> shift) & kAll;
  if (!__all_sync(0xffffffffu, (some & (some + 1)) == 0)) {   // a gap: compact
    const uint32_t n = __popc(some);
    const uint32_t src = hl < n ? nth_set_bit(some, hl) : 0u;
    e.a = __shfl_sync(0xffffffffu, e.a, src, LANES);
    b0 = __shfl_sync(0xffffffffu, b0, src, LANES);
    const uint32_t l = __shfl_sync(0xffffffffu, e.len, src, LANES);
    e.len = hl < n ? l : 0u;
  }
  uint32_t incl = e.len;
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o, LANES);
    if (hl >= (uint32_t)o) incl += y;
  }
  e.excl = incl - e.len;
  e.base = b0 - (Index)e.excl;
  return __shfl_sync(0xffffffffu, incl, LANES - 1, LANES);
}

// Owner of slot w0 + hl: the ranges that start at or before it, counted from
// the bits of this window's starts; `started` counts those of earlier windows.
template <typename T, typename K, int LANES>
__device__ __forceinline__ uint32_t slot_owner(const Entry<T, K>& e, uint32_t w0, uint32_t hl, uint32_t shift,
                                               uint32_t& started) {
  const uint32_t d = e.excl - w0;
  const uint32_t bit = (e.len > 0 && d < (uint32_t)LANES) ? 1u << (d + shift) : 0u;
  uint32_t starts = __reduce_or_sync(0xffffffffu, bit) >> shift;
  if (LANES < 32) starts &= (1u << (LANES & 31)) - 1u;
  const uint32_t own = started + __popc(starts & (0xffffffffu >> (31u - hl))) - 1u;
  started += __popc(starts);
  return own & (LANES - 1);
}

// Key of candidate `slot`, its value left in sval[slot]; ~0 for none.
template <typename T, typename K, int SB>
__device__ __forceinline__ K make_key(const RowArgs<T>& R, T a, T b, int32_t j, uint32_t slot, uint32_t* sval,
                                      bool& bad) {
  T c = T(0);
  bool ok = SpVal<T>::combine(a, b, c);
  if ((uint32_t)j >= (uint32_t)R.N) {   // N < 2^31
    bad = true;
    ok = false;
  }
  sval[slot] = VKey<T>::enc(c);
  return ok ? ((K)(uint32_t)j << SB) | (K)slot : ~(K)0;
}

// First key of a column's run among the sorted keys.
template <typename K, int SB>
__device__ __forceinline__ bool is_head(K me, K before) {
  return me != ~(K)0 && ((before >> SB) != (me >> SB) || before == ~(K)0);
}

// Lower each run's first value to the run's minimum, every member for itself, in a
// row of a whole warp.  Short runs are walked by their head, which spares rows of
// few duplicates this pass (it cost the rows of half a warp, whose longest run is
// 128, 7 % and gained a narrow result's 14 %); walked so, 2^16 rows of 512
// candidates in one column took 1.44 ms a call instead of 0.70.
template <typename K, int SB>
__device__ __forceinline__ void lower_heads(const K* skey, uint32_t* sval, int regs, uint32_t lane) {
  constexpr uint32_t kMask = (uint32_t)(((K)1 << SB) - 1);
  uint32_t newest = 0;   // the last head so far
#pragma unroll 1
  for (int r = 0; r < regs; ++r) {
    const uint32_t e = (uint32_t)r * 32u + lane;
    const K me = skey[e], before = e ? skey[e - 1] : ~(K)0;
    const bool head = is_head<K, SB>(me, before);
    const uint32_t heads = __ballot_sync(0xffffffffu, head);
    if (me != ~(K)0 && !head) {
      const uint32_t at = heads & ((1u << lane) - 1u);
      const uint32_t first = at ? (uint32_t)r * 32u + 31u - __clz(at) : newest;
      atomicMin(&sval[(uint32_t)skey[first] & kMask], sval[(uint32_t)me & kMask]);
    }
    if (heads) newest = (uint32_t)r * 32u + 31u - __clz(heads);
  }
  __syncwarp();
}

// One row per group of LANES lanes, of at most LANES * regs candidates (regs <= P).
template <typename T, typename K, int LANES, int P>
__device__ __forceinline__ void do_row(const RowArgs<T>& R, int64_t i, bool mine, unsigned long long o0, int64_t a0,
                                       int64_t alen, int regs, uint32_t hl, uint32_t shift, K* skey,
                                       uint32_t* sval) {
  constexpr int SB = sizeof(K) == 8 ? 32 : (LANES == 16 ? 7 : 9);   // slot bits
  constexpr K kMask = ((K)1 << SB) - 1;
  constexpr uint32_t kAll = LANES == 32 ? 0xffffffffu : (1u << (LANES & 31)) - 1u;
  typedef typename Entry<T, K>::Index Index;
  K key[P];
  uint32_t n;   // candidates of this row
  bool bad = false;
  if (__all_sync(0xffffffffu, alen <= LANES)) {
    Entry<T, K> e;
    n = load_entries<T, K, LANES>(R, a0 + hl, (int64_t)hl < alen, hl, shift, e);
    int32_t j[P];
    T a[P], b[P];
    uint32_t started = 0;
#pragma unroll
    for (int r = 0; r < P; ++r) {
      if (r >= 4 && r >= regs) break;
      const uint32_t sl = (uint32_t)(r * LANES) + hl;
      const uint32_t t = slot_owner<T, K, LANES>(e, (uint32_t)(r * LANES), hl, shift, started);
      a[r] = __shfl_sync(0xffffffffu, e.a, t, LANES);
      const Index q = __shfl_sync(0xffffffffu, e.base, t, LANES) + (Index)sl;
      j[r] = 0;
      b[r] = T(0);
      if (sl < n) {
        j[r] = R.bci[q];
        b[r] = R.bv[q];
      }
    }
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const uint32_t sl = (uint32_t)(r * LANES) + hl;
      key[r] = ~(K)0;
      if (r >= 4 && r >= regs) continue;
      if (sl < n) key[r] = make_key<T, K, SB>(R, a[r], b[r], j[r], sl, sval, bad);
    }
  } else {
    int64_t most = alen;
    if (LANES < 32) most = max(most, (int64_t)__shfl_xor_sync(0xffffffffu, (long long)most, 16));
    n = 0;
    for (int64_t pa = 0; pa < most; pa += LANES) {
      Entry<T, K> e;
      const uint32_t total =
          load_entries<T, K, LANES>(R, a0 + pa + hl, pa + (int64_t)hl < alen, hl, shift, e);
      uint32_t longest = total;
      if (LANES < 32) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, 16));
      uint32_t started = 0;
      for (uint32_t w0 = 0; w0 < longest; w0 += LANES) {
        const uint32_t sl = w0 + hl;
        const uint32_t t = slot_owner<T, K, LANES>(e, w0, hl, shift, started);
        const T a = __shfl_sync(0xffffffffu, e.a, t, LANES);
        const Index q = __shfl_sync(0xffffffffu, e.base, t, LANES) + (Index)sl;
        if (sl < total) skey[n + sl] = make_key<T, K, SB>(R, a, R.bv[q], R.bci[q], n + sl, sval, bad);
      }
      n += total;
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const uint32_t sl = (uint32_t)(r * LANES) + hl;
      key[r] = sl < n ? skey[sl] : ~(K)0;
    }
  }
  if (__any_sync(0xffffffffu, bad) && bad) atomicCAS(R.status, kSpOk, (uint32_t)kSpBadIndex);
  bool long_run;
  if (P == 8) {
    if (regs <= 4) long_run = sort_to_shared<K, LANES, 4, SB>(key, hl, skey);
    else if (regs == 5) long_run = sort_to_shared<K, LANES, 5, SB>(key, hl, skey);
    else if (regs == 6) long_run = sort_to_shared<K, LANES, 6, SB>(key, hl, skey);
    else if (regs == 7) long_run = sort_to_shared<K, LANES, 7, SB>(key, hl, skey);
    else long_run = sort_to_shared<K, LANES, 8, SB>(key, hl, skey);
  } else {
    if (regs <= 8) long_run = sort_to_shared<K, LANES, 8, SB>(key, hl, skey);
    else if (regs <= 12) long_run = sort_to_shared<K, LANES, 12 <= P ? 12 : P, SB>(key, hl, skey);
    else long_run = sort_to_shared<K, LANES, P, SB>(key, hl, skey);
  }
  __syncwarp();   // sorted keys and all values are in shared memory
  if (long_run) lower_heads<K, SB>(skey, sval, regs, hl);
  // heads of column runs, in order
  int32_t* tc = R.tcol + o0;
  T* tv = R.tval + o0;
  uint32_t kept = 0;
#pragma unroll 1
  for (int r = 0; r < regs; ++r) {
    const uint32_t e = (uint32_t)(r * LANES) + hl;
    const K me = skey[e], before = e ? skey[e - 1] : ~(K)0;
    const bool head = is_head<K, SB>(me, before);
    const uint32_t bal = __ballot_sync(0xffffffffu, head);
    if (head) {
      uint32_t v = sval[(uint32_t)(me & kMask)];
      for (uint32_t q = e + 1; !long_run && q < (uint32_t)(regs * LANES); ++q) {
        const K other = skey[q];
        if ((other >> SB) != (me >> SB) || other == ~(K)0) break;
        v = min(v, sval[(uint32_t)(other & kMask)]);
      }
      const uint32_t pos = kept + __popc((bal >> shift) & ((1u << hl) - 1u));
      tc[pos] = (int32_t)(me >> SB);
      tv[pos] = VKey<T>::dec(v);
    }
    kept += __popc((bal >> shift) & kAll);
  }
  if (mine && hl == 0) R.cnt[i] = kept;
  __syncwarp();
}

// LANES = 16: every row of up to kSmallRowMax candidates, two per warp.
// LANES = 32: the listed rows.
template <typename T, typename K, int LANES>
__global__ void __launch_bounds__(kRowWarps * 32)
    k_rows(const RowArgs<T> R, const int64_t* __restrict__ rows, int64_t nrows) {
  constexpr int kRpw = 32 / LANES, kCap = LANES == 16 ? kSmallRowMax : kWarpRowMax;
  __shared__ K s_key[kRowWarps][kRpw][kCap];
  __shared__ uint32_t s_val[kRowWarps][kRpw][kCap];
  const uint32_t lane = threadIdx.x & 31u, hl = lane & (LANES - 1), grp = lane / LANES, shift = lane - hl;
  K* skey = s_key[threadIdx.x >> 5][grp];
  uint32_t* sval = s_val[threadIdx.x >> 5][grp];
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t x = warp * kRpw; x < nrows; x += nwarps * kRpw) {
    const bool in = x + grp < nrows;
    const int64_t i = in ? (rows ? rows[x + grp] : x + grp) : 0;
    unsigned long long o0 = 0, ub = 0;
    int64_t a0 = 0, alen = 0;
    if (in) {
      o0 = R.off[i];
      ub = R.off[i + 1] - o0;
      a0 = R.arp[i];
      alen = R.arp[i + 1] - a0;
    }
    const bool mine = in && ub <= (unsigned long long)kCap;
    if (!mine || ub == 0) {
      ub = 0;
      alen = 0;
    }
    uint32_t most = (uint32_t)ub;
    if (LANES < 32) most = max(most, __shfl_xor_sync(0xffffffffu, most, 16));
    const uint32_t regs = (most + LANES - 1) / LANES;
    if (regs == 0) {
      if (mine && hl == 0) R.cnt[i] = 0;
      continue;
    }
    do_row<T, K, LANES, kCap / LANES>(R, i, mine, o0, a0, alen, (int)regs, hl, shift, skey, sval);
  }
}

// ---- long rows of matrices with few columns: dense accumulation --------------
// A block takes a row.  Its candidates go into an array of one 32-bit word per
// column in shared memory (order-preserving value bits, atomicMin), which is
// then read in column order: no expansion to memory, no sort, no limit on the
// row's candidates.  Up to kDenseCols columns fit one pass; wider matrices take
// one pass over the row for each.  Bound by the gather from L2 and shared-memory
// atomics.
// RMAT scale 14, edge factor 8: 21.5 ms per call with the rows expanded, sorted
// by CUB and reduced by one warp each -> 0.82 ms.  RMAT 17 (131072 columns, three
// passes), edge factor 2: 27.1 -> 6.0 ms.
template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_rows_dense(const RowArgs<T> R, const int64_t* __restrict__ rows, int64_t nheavy,
                                                   int64_t nlong, int cap, unsigned long long* next) {
  static_assert(NT <= kDenseThreads, "kDenseRowMax leaves room for a step of the largest block");
  extern __shared__ uint32_t s_acc[];   // cap words
  __shared__ uint32_t s_excl[NT + 1];
  __shared__ long long s_base[NT];
  __shared__ T s_a[NT];
  __shared__ uint32_t s_warp[NT / 32];
  __shared__ unsigned long long s_item;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
  for (int c = (int)tid; c < cap; c += NT) s_acc[c] = 0xFFFFFFFFu;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_item = atomicAdd(next, 1ull);
    __syncthreads();
    const int64_t item = (int64_t)s_item;
    if (item >= nheavy + nlong) break;
    const int64_t i = item < nheavy ? rows[item] : rows[R.M - 1 - (item - nheavy)];
    const int64_t a0 = R.arp[i], a1 = R.arp[i + 1];
    const unsigned long long o0 = R.off[i];
    uint32_t kept = 0;
    for (int64_t c0 = 0; c0 < R.N; c0 += cap) {
      const uint32_t cols = (uint32_t)min((int64_t)cap, R.N - c0);
      for (int64_t pa = a0; pa < a1; pa += NT) {
        // this chunk's entries and the block-wide offsets of their B ranges
        uint32_t len = 0;
        long long b0 = 0;
        T a = T(0);
        if (pa + tid < a1) {
          const int32_t k = R.aci[pa + tid];
          a = R.av[pa + tid];
          b0 = R.brp[k];   // (of absent entries too: their B rows' columns are checked)
          len = (uint32_t)(R.brp[k + 1] - b0);
        }
        const uint32_t incl = warp_incl_scan(len);
        if (lane == 31) s_warp[w] = incl;
        __syncthreads();
        if (w == 0) {
          const uint32_t x = lane < NT / 32 ? s_warp[lane] : 0u;
          const uint32_t y = warp_incl_scan(x);
          if (lane < NT / 32) s_warp[lane] = y - x;
          if (lane == 31) s_excl[NT] = y;
        }
        __syncthreads();
        const uint32_t excl = s_warp[w] + incl - len;
        s_excl[tid] = excl;
        s_base[tid] = b0 - (long long)excl;
        s_a[tid] = a;
        __syncthreads();
        const uint32_t total = s_excl[NT];
#pragma unroll 4
        for (uint32_t sl = tid; sl < total; sl += NT) {
          uint32_t t = 0;   // the last entry whose range starts at or before sl
#pragma unroll
          for (uint32_t step = NT / 2; step >= 1; step >>= 1)
            if (s_excl[t + step] <= sl) t += step;
          const long long q = s_base[t] + sl;
          const int32_t j = R.bci[q];
          T c = T(0);
          const bool ok = SpVal<T>::present(s_a[t]) && SpVal<T>::combine(s_a[t], R.bv[q], c);
          if (j < 0 || (int64_t)j >= R.N) atomicCAS(R.status, kSpOk, (uint32_t)kSpBadIndex);
          else if (ok && (uint32_t)(j - c0) < cols) atomicMin(&s_acc[(uint32_t)(j - c0)], VKey<T>::enc(c));
        }
        __syncthreads();   // the chunk's entries have been used
      }
      // columns in order: each warp owns a range of them; count, then write and clear
      const uint32_t per = (((cols + NT / 32 - 1) / (NT / 32)) + 31u) & ~31u;
      const uint32_t lo = min(w * per, cols), hi = min(lo + per, cols);
      __syncthreads();
      uint32_t mine = 0;
      for (uint32_t c = lo + lane; c < hi; c += 32) mine += s_acc[c] != 0xFFFFFFFFu ? 1u : 0u;
      mine = __reduce_add_sync(0xffffffffu, mine);
      if (lane == 0) s_warp[w] = mine;
      __syncthreads();
      uint32_t before = 0, all = 0;
      for (uint32_t x = 0; x < NT / 32; ++x) {
        const uint32_t y = s_warp[x];
        before += x < w ? y : 0u;
        all += y;
      }
      unsigned long long pos = o0 + kept + before;
      for (uint32_t c = lo; c < hi; c += 32) {
        const bool in = c + lane < hi;
        const uint32_t v = in ? s_acc[c + lane] : 0xFFFFFFFFu;
        const bool have = v != 0xFFFFFFFFu;
        const uint32_t bal = __ballot_sync(0xffffffffu, have);
        if (have) {
          const unsigned long long at = pos + __popc(bal & ((1u << lane) - 1u));
          R.tcol[at] = (int32_t)(c0 + c + lane);
          R.tval[at] = VKey<T>::dec(v);
          s_acc[c + lane] = 0xFFFFFFFFu;
        }
        pos += __popc(bal);
      }
      kept += all;
      __syncthreads();
    }
    if (tid == 0) R.cnt[i] = kept;
  }
}

template <typename T, int NT>
cudaError_t launch_dense(const RowArgs<T>& R, const int64_t* rows, int64_t nheavy, int64_t nlong, int cap, int sms,
                         unsigned long long* next, cudaStream_t st) {
  const size_t smem = (size_t)cap * 4;
  cudaError_t e = cudaFuncSetAttribute(k_rows_dense<T, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kDenseCols * 4);
  int per = 0;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rows_dense<T, NT>, NT, smem);
  if (e != cudaSuccess) return e;
  if (per < 1) return cudaErrorInvalidConfiguration;
  const int64_t blocks = std::min<int64_t>(nheavy + nlong, (int64_t)per * sms);
  k_rows_dense<T, NT><<<(int)blocks, NT, smem, st>>>(R, rows, nheavy, nlong, cap, next);
  return cudaGetLastError();
}

// ---- long rows of wide matrices: expand-sort-compress over a row list --------
// A warp per row, 32 entries of A at a time: a lane loads an entry, and the warp
// walks the slots of all their B rows (entry by entry, a row of many entries of few
// candidates was one chain of loads: 2^13 rows of 1500 entries of 2 candidates, the
// call 3.00 ms, now 1.59).
template <typename T>
__global__ void k_expand(int64_t L, const int64_t* __restrict__ rows, int64_t N, const int64_t* __restrict__ arp,
                         const int32_t* __restrict__ aci, const T* __restrict__ av, const int64_t* __restrict__ brp,
                         const int32_t* __restrict__ bci, const T* __restrict__ bv,
                         const unsigned long long* __restrict__ off, int32_t* __restrict__ ccol,
                         T* __restrict__ cval, uint32_t* status) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = threadIdx.x & 31u;
  for (int64_t r = warp; r < L; r += nwarps) {
    const int64_t i = rows[r];
    unsigned long long pos = off[r];
    const int64_t end = arp[i + 1];
    for (int64_t p0 = arp[i]; p0 < end; p0 += 32) {
      const int64_t p = p0 + lane;
      T a = T(0);
      long long b0 = 0;
      uint32_t len = 0;   // (all of a sort's items together are fewer than 2^31)
      if (p < end) {
        const int32_t k = aci[p];
        a = av[p];
        b0 = brp[k];
        len = (uint32_t)(brp[k + 1] - b0);
      }
      const uint32_t incl = warp_incl_scan(len), excl = incl - len;
      const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
      const long long base = b0 - (long long)excl;
#pragma unroll 2
      for (uint32_t s0 = 0; s0 < total; s0 += 32) {
        const uint32_t sl = s0 + lane;
        uint32_t t = 0;   // the last entry whose range starts at or before slot sl
#pragma unroll
        for (uint32_t step = 16; step >= 1; step >>= 1)
          if (__shfl_sync(0xffffffffu, excl, t + step) <= sl) t += step;
        const T at = __shfl_sync(0xffffffffu, a, t);
        const long long q = __shfl_sync(0xffffffffu, base, t) + sl;
        if (sl < total) {
          const int32_t j = bci[q];
          T c = T(0);
          bool ok = SpVal<T>::present(at) && SpVal<T>::combine(at, bv[q], c);
          if (j < 0 || (int64_t)j >= N) {
            atomicCAS(status, kSpOk, (uint32_t)kSpBadIndex);
            ok = false;
          }
          ccol[pos + sl] = ok ? j : kDropCol;
          cval[pos + sl] = c;
        }
      }
      pos += total;
    }
  }
}

// Heads of column runs of each listed row's sorted segment -> the row's
// scratch slot (tcol / tval at slot[row]) and its count.
template <typename T>
__global__ void k_compress(int64_t L, const int64_t* __restrict__ rows, const unsigned long long* __restrict__ off,
                           const int32_t* __restrict__ scol, const T* __restrict__ sval,
                           const unsigned long long* __restrict__ slot, int32_t* __restrict__ tcol,
                           T* __restrict__ tval, int64_t* __restrict__ cnt) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = threadIdx.x & 31u;
  for (int64_t rr = warp; rr < L; rr += nwarps) {
    const int64_t i = rows[rr];
    const unsigned long long b = off[rr], e = off[rr + 1];
    const unsigned long long dst = slot[i];
    int64_t outpos = 0;
    for (unsigned long long base = b; base < e; base += 32) {
      const unsigned long long q = base + lane;
      const bool in = q < e;
      const int32_t j = in ? scol[q] : kDropCol;
      const bool head = in && j != kDropCol && (q == b || scol[q - 1] != j);
      const uint32_t hm = __ballot_sync(0xffffffffu, head);
      if (head) {
        // min over the run of column j (runs may cross the 32-entry window)
        T m = sval[q];
        for (unsigned long long r = q + 1; r < e && scol[r] == j; ++r) m = SpVal<T>::vmin(m, sval[r]);
        const int64_t w = outpos + __popc(hm & ((1u << lane) - 1u));
        tcol[dst + w] = j;
        tval[dst + w] = m;
      }
      outpos += __popc(hm);
    }
    if (lane == 0) cnt[i] = outpos;
  }
}

// Candidates of the listed rows, and how many have between_from or more.
__global__ void k_long_bounds(int64_t L, const int64_t* __restrict__ rows, const unsigned long long* __restrict__ off,
                              unsigned long long* __restrict__ lub, unsigned long long between_from,
                              unsigned long long* between) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < L; r += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long s = off[rows[r] + 1] - off[rows[r]];
    lub[r] = s;
    if (s >= between_from) atomicAdd(between, 1ull);
  }
}

// The listed rows of between_from candidates or more to one list, the others to another.
__global__ void k_split(int64_t L, const int64_t* __restrict__ rows, const unsigned long long* __restrict__ off,
                        unsigned long long between_from, unsigned long long* cursor, int64_t* __restrict__ more,
                        int64_t* __restrict__ fewer) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < L; r += (int64_t)gridDim.x * blockDim.x) {
    const bool m = off[rows[r] + 1] - off[rows[r]] >= between_from;
    (m ? more : fewer)[atomicAdd(&cursor[m ? 0 : 1], 1ull)] = rows[r];
  }
}

// scratch slots -> exact-size outputs (one warp per row)
template <typename T>
__global__ void k_compact(int64_t M, const unsigned long long* __restrict__ slot, const int64_t* __restrict__ crp,
                          const int32_t* __restrict__ tcol, const T* __restrict__ tval, int32_t* __restrict__ cci,
                          T* __restrict__ cv) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lane = threadIdx.x & 31u;
  for (int64_t i = warp; i < M; i += nwarps) {
    const unsigned long long s0 = slot[i];
    const int64_t c0 = crp[i], c = crp[i + 1] - c0;
    for (int64_t q = lane; q < c; q += 32) {
      cci[c0 + q] = tcol[s0 + q];
      cv[c0 + q] = tval[s0 + q];
    }
  }
}

int grid_rows(int64_t rows) {
  int64_t b = (rows * 32 + 255) / 256;
  if (b < 1) b = 1;
  if (b > 148 * 16) b = 148 * 16;
  return (int)b;
}

// Library-owned stream-ordered pool for scratch arrays, one per device; it
// keeps up to kPoolKeep bytes cached after a call returns.
constexpr uint64_t kPoolKeep = 4ull << 30;
}  // namespace

cudaError_t scratch_pool(cudaMemPool_t* out) {
  static std::mutex mu;
  static std::map<int, cudaMemPool_t> pools;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  auto it = pools.find(dev);
  if (it != pools.end()) {
    *out = it->second;
    return cudaSuccess;
  }
  cudaMemPoolProps props;
  memset(&props, 0, sizeof(props));
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t p;
  e = cudaMemPoolCreate(&p, &props);
  if (e != cudaSuccess) return e;
  uint64_t keep = kPoolKeep;
  cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
  pools[dev] = p;
  *out = p;
  return cudaSuccess;
}

namespace {

// Scratch array from the pool, released (stream-ordered) on scope exit.
template <typename T>
struct DBuf {
  T* p = nullptr;
  cudaStream_t st = nullptr;
  ~DBuf() { if (p) cudaFreeAsync(p, st); }
  cudaError_t alloc(size_t n, cudaStream_t s) {
    st = s;
    cudaMemPool_t pool;
    cudaError_t e = scratch_pool(&pool);
    if (e != cudaSuccess) return e;
    return cudaMallocFromPoolAsync((void**)&p, std::max<size_t>(n, 1) * sizeof(T), pool, s);
  }
  T* release() {
    T* q = p;
    p = nullptr;
    return q;
  }
};

}  // namespace

// A computed product waiting for its outputs: every row's result sits in a
// scratch slot (off[i] .. off[i] + cnt[i]) and crp holds C's row pointers.
struct SpPlan {
  int64_t M = 0;
  int64_t nnz = 0;
  int wt = B2_W_F32;
  int64_t* crp = nullptr;            // pool memory
  unsigned long long* off = nullptr; // pool memory
  int32_t* tcol = nullptr;           // pool memory
  void* tval = nullptr;              // pool memory
  cudaStream_t st = nullptr;
  void release() {
    if (crp) cudaFreeAsync(crp, st);
    if (off) cudaFreeAsync(off, st);
    if (tcol) cudaFreeAsync(tcol, st);
    if (tval) cudaFreeAsync(tval, st);
    crp = nullptr;
    off = nullptr;
    tcol = nullptr;
    tval = nullptr;
  }
};

namespace {

// Whether long rows of a wide matrix that either way suits (see kDensePerPass) are
// sorted: there are rows enough, and the expansion (two pairs of a column and a
// value per candidate) and the result slots fit what the pool keeps, with room for
// the sort's own scratch.
bool sort_between(int64_t rows, unsigned long long candidates, unsigned long long slots) {
  return rows >= kSortRows && candidates <= 0x7fffffffull && candidates * 16 + slots * 8 <= kPoolKeep / 4 * 3;
}

// Steps 1-5 up to C's row pointers; one host synchronization for the scratch
// size (two or three when rows are expanded) and one for nnz(C).
template <typename T>
b2_status compute(const b2_csr* A, const b2_csr* B, cudaStream_t st, SpPlan& plan) {
  if (!A || !B) return B2_INVALID_ARGUMENT;
  if (A->rows < 0 || A->cols < 0 || A->nnz < 0 || B->rows < 0 || B->cols < 0 || B->nnz < 0) return B2_INVALID_ARGUMENT;
  if (A->cols != B->rows) return B2_INVALID_ARGUMENT;
  if (A->cols > 0x7fffffffLL || B->cols > 0x7fffffffLL) return B2_INVALID_ARGUMENT;
  if (A->rowptr_bits != 64 || B->rowptr_bits != 64 || !A->on_device || !B->on_device) return B2_INVALID_ARGUMENT;
  if (!A->rowptr || !B->rowptr) return B2_INVALID_ARGUMENT;
  if ((A->nnz > 0 && (!A->colind || !A->values)) || (B->nnz > 0 && (!B->colind || !B->values)))
    return B2_INVALID_ARGUMENT;
  const int64_t M = A->rows, K = A->cols, N = B->cols;
  const int64_t* arp = (const int64_t*)A->rowptr;
  const int64_t* brp = (const int64_t*)B->rowptr;
  plan.M = M;
  plan.st = st;
  DBuf<int64_t> crp;
  if (crp.alloc((size_t)M + 1, st) != cudaSuccess) return B2_OUT_OF_MEMORY;
  if (M == 0 || K == 0 || A->nnz == 0 || B->nnz == 0) {
    B2_CUDA_TRY(cudaMemsetAsync(crp.p, 0, (size_t)(M + 1) * sizeof(int64_t), st));
    plan.crp = crp.release();
    plan.nnz = 0;
    return B2_SUCCESS;
  }
  DBuf<unsigned long long> ub, off;
  DBuf<int64_t> lrows, mrows;
  DBuf<SpCounters> counters;
  DBuf<unsigned char> tmp;
  if (ub.alloc((size_t)M + 1, st) != cudaSuccess || off.alloc((size_t)M + 1, st) != cudaSuccess ||
      counters.alloc(1, st) != cudaSuccess || lrows.alloc((size_t)M, st) != cudaSuccess ||
      mrows.alloc((size_t)M, st) != cudaSuccess)
    return B2_OUT_OF_MEMORY;
  // a densely accumulated row needs at most N result slots (kept past the ordinary
  // rows' limit, by which the row kernels tell them apart)
  const unsigned long long passes = (unsigned long long)((N + kDenseCols - 1) / kDenseCols);
  // (a matrix without columns takes no pass: the expansion checks its entries' columns)
  const bool can_pass = passes > 0 && passes <= (unsigned long long)kDensePasses;
  const unsigned long long between_from = can_pass && passes > 1 ? passes * kDensePerPass : ~0ull;
  const unsigned long long dense_from = !can_pass ? ~0ull
                                        : passes == 1 ? 0ull
                                        : M < kSortRows ? between_from
                                                        : sorted_max(passes);
  const unsigned long long dense_slots =
      std::max<unsigned long long>((unsigned long long)N, (unsigned long long)kWarpRowMax + 1);
  cudaError_t e = cudaMemsetAsync(counters.p, 0, sizeof(SpCounters), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(ub.p + M, 0, 8, st);
  if (e == cudaSuccess) {
    const int lanes = bound_lanes(M);
    auto* bound = lanes == 32 ? k_row_bound<32> : k_row_bound<8>;
    bound<<<grid_rows((M * lanes + 31) / 32), 256, 0, st>>>(M, K, A->nnz, B->nnz, arp, A->colind, brp, ub.p, counters.p,
                                                            lrows.p, mrows.p, dense_from, dense_slots);
    e = cudaGetLastError();
  }
  size_t tb = 0;
  if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(nullptr, tb, ub.p, off.p, M + 1, st);
  if (e == cudaSuccess) e = tmp.alloc(tb, st);
  if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp.p, tb, ub.p, off.p, M + 1, st);
  unsigned long long U = 0;   // result slots
  SpCounters hc = {};
  if (e == cudaSuccess) e = cudaMemcpyAsync(&U, off.p + M, 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&hc, counters.p, sizeof(hc), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return from_cuda(e);
  if (hc.status == kSpBadIndex) return B2_INVALID_INDEX;
  if (hc.status == kSpBadRowptr) return B2_INVALID_ROWPTR;
  if (hc.too_long) return B2_NOT_SUPPORTED;
  const int64_t nheavy = (int64_t)hc.heavy, nlong = (int64_t)hc.lng, nmid = (int64_t)hc.mid;
  int64_t L = (int64_t)hc.wide;   // rows to expand and sort: the last L entries of mrows
  const int64_t* wrows = mrows.p + (M - L);
  uint32_t* const status = &counters.p->status;
  DBuf<int32_t> tcol;
  DBuf<T> tval;
  DBuf<int64_t> cnt;
  if (tcol.alloc(U, st) != cudaSuccess || tval.alloc(U, st) != cudaSuccess ||
      cnt.alloc((size_t)M + 1, st) != cudaSuccess)
    return B2_OUT_OF_MEMORY;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const RowArgs<T> R = {M,      N,     arp,    A->colind, (const T*)A->values, brp,   B->colind, (const T*)B->values,
                        off.p, tcol.p, tval.p, cnt.p,     status};
  auto dense = [&](const int64_t* rows, int64_t front, int64_t back) -> b2_status {   // k_rows_dense's lists
    DBuf<unsigned long long> next;
    if (next.alloc(1, st) != cudaSuccess) return B2_OUT_OF_MEMORY;
    const int cap = (int)std::min<int64_t>((N + 31) / 32 * 32, kDenseCols);
    cudaError_t x = cudaMemsetAsync(next.p, 0, 8, st);
    // 512 threads while two blocks or more fit an SM, else 1024
    if (x == cudaSuccess)
      x = cap <= 24576 ? launch_dense<T, 512>(R, rows, front, back, cap, sms, next.p, st)
                       : launch_dense<T, kDenseThreads>(R, rows, front, back, cap, sms, next.p, st);
    return from_cuda(x);
  };
  if (U > 0) {
    if (nheavy + nlong > 0) {   // first: the longest of them take longest
      const b2_status d = dense(lrows.p, nheavy, nlong);
      if (d != B2_SUCCESS) return d;
    }
    const bool b32 = B->nnz < (1ll << 31);   // 32-bit indices into B beside the 32-bit keys
    auto blocks = [&](int64_t warps, int per_sm) {
      return (int)std::max<int64_t>(1, std::min<int64_t>((warps + kRowWarps - 1) / kRowWarps, (int64_t)sms * per_sm));
    };
    if (e == cudaSuccess) {
      const int g = blocks((M + 1) / 2, 16);
      if (N < (1ll << 25) && b32) k_rows<T, uint32_t, 16><<<g, kRowWarps * 32, 0, st>>>(R, nullptr, M);
      else k_rows<T, unsigned long long, 16><<<g, kRowWarps * 32, 0, st>>>(R, nullptr, M);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && nmid > 0) {
      const int g = blocks(nmid, 16);
      if (N < (1ll << 23) && b32) k_rows<T, uint32_t, 32><<<g, kRowWarps * 32, 0, st>>>(R, mrows.p, nmid);
      else k_rows<T, unsigned long long, 32><<<g, kRowWarps * 32, 0, st>>>(R, mrows.p, nmid);
      e = cudaGetLastError();
    }
  } else {
    e = cudaMemsetAsync(cnt.p, 0, (size_t)M * sizeof(int64_t), st);
  }
  // long rows: expand, segmented sort, compress into their scratch slots
  DBuf<unsigned long long> lub, loff;
  DBuf<int64_t> more, fewer;
  DBuf<int32_t> col0, col1;
  DBuf<T> val0, val1;
  DBuf<unsigned char> tmp2, tmp3;
  unsigned long long LU = 0;   // candidates of the rows to sort
  if (e == cudaSuccess && L > 0) {
    if (lub.alloc((size_t)L + 1, st) != cudaSuccess || loff.alloc((size_t)L + 1, st) != cudaSuccess)
      return B2_OUT_OF_MEMORY;
    size_t tb1 = 0;
    e = cub::DeviceScan::ExclusiveSum(nullptr, tb1, lub.p, loff.p, L + 1, st);
    if (e == cudaSuccess) e = tmp2.alloc(tb1, st);
    unsigned long long between = 0;
    auto bounds = [&]() {
      const int g = (int)std::min<int64_t>((L + 255) / 256, 1184);
      cudaError_t x = cudaMemsetAsync(lub.p + L, 0, 8, st);
      if (x == cudaSuccess) {
        k_long_bounds<<<g, 256, 0, st>>>(L, wrows, off.p, lub.p, between_from, &counters.p->between);
        x = cudaGetLastError();
      }
      if (x == cudaSuccess) x = cub::DeviceScan::ExclusiveSum(tmp2.p, tb1, lub.p, loff.p, L + 1, st);
      if (x == cudaSuccess) x = cudaMemcpyAsync(&LU, loff.p + L, 8, cudaMemcpyDeviceToHost, st);
      if (x == cudaSuccess) x = cudaMemcpyAsync(&between, &counters.p->between, 8, cudaMemcpyDeviceToHost, st);
      if (x == cudaSuccess) x = cudaStreamSynchronize(st);
      return x;
    };
    if (e == cudaSuccess) e = bounds();
    if (e != cudaSuccess) return from_cuda(e);
    if (between > 0 && !sort_between((int64_t)between, LU, U)) {
      if (more.alloc((size_t)between, st) != cudaSuccess || fewer.alloc((size_t)L, st) != cudaSuccess)
        return B2_OUT_OF_MEMORY;
      k_split<<<(int)std::min<int64_t>((L + 255) / 256, 1184), 256, 0, st>>>(L, wrows, off.p, between_from,
                                                                            counters.p->split, more.p, fewer.p);
      e = cudaGetLastError();
      if (e != cudaSuccess) return from_cuda(e);
      const b2_status d = dense(more.p, (int64_t)between, 0);
      if (d != B2_SUCCESS) return d;
      L -= (int64_t)between;
      wrows = fewer.p;
      if (L > 0) e = bounds();   // (none of these is counted again)
      if (e != cudaSuccess) return from_cuda(e);
    }
  }
  if (e == cudaSuccess && L > 0) {
    if (LU > 0x7fffffffull) return B2_NOT_SUPPORTED;   // segmented sort item count is int
    if (col0.alloc(LU, st) != cudaSuccess || col1.alloc(LU, st) != cudaSuccess || val0.alloc(LU, st) != cudaSuccess ||
        val1.alloc(LU, st) != cudaSuccess)
      return B2_OUT_OF_MEMORY;
    k_expand<T><<<grid_rows(L), 256, 0, st>>>(L, wrows, N, arp, A->colind, (const T*)A->values, brp, B->colind,
                                              (const T*)B->values, loff.p, col0.p, val0.p, status);
    e = cudaGetLastError();
    size_t tbs = 0;
    if (e == cudaSuccess)
      e = cub::DeviceSegmentedSort::StableSortPairs(nullptr, tbs, col0.p, col1.p, val0.p, val1.p, (int)LU, (int)L,
                                                    loff.p, loff.p + 1, st);
    if (e == cudaSuccess) e = tmp3.alloc(tbs, st);
    if (e == cudaSuccess)
      e = cub::DeviceSegmentedSort::StableSortPairs(tmp3.p, tbs, col0.p, col1.p, val0.p, val1.p, (int)LU, (int)L,
                                                    loff.p, loff.p + 1, st);
    if (e == cudaSuccess) {
      k_compress<T><<<grid_rows(L), 256, 0, st>>>(L, wrows, loff.p, col1.p, val1.p, off.p, tcol.p, tval.p, cnt.p);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(cnt.p + M, 0, 8, st);
  size_t tb4 = 0;
  DBuf<unsigned char> tmp4;
  if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(nullptr, tb4, cnt.p, crp.p, M + 1, st);
  if (e == cudaSuccess) e = tmp4.alloc(tb4, st);
  if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp4.p, tb4, cnt.p, crp.p, M + 1, st);
  int64_t nnz = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&nnz, crp.p + M, 8, cudaMemcpyDeviceToHost, st);
  uint32_t hs = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&hs, status, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return from_cuda(e);
  if (hs == kSpBadIndex) return B2_INVALID_INDEX;
  if (hs == kSpBadRowptr) return B2_INVALID_ROWPTR;
  plan.nnz = nnz;
  plan.crp = crp.release();
  plan.off = off.release();
  plan.tcol = tcol.release();
  plan.tval = tval.release();
  return B2_SUCCESS;
}

// Scratch slots -> caller-visible outputs (stream-ordered).
template <typename T>
cudaError_t fill(const SpPlan& plan, int64_t* crp, int32_t* cci, T* cv, cudaStream_t st) {
  cudaError_t e = cudaMemcpyAsync(crp, plan.crp, (size_t)(plan.M + 1) * sizeof(int64_t), cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess && plan.nnz > 0) {
    k_compact<T><<<grid_rows(plan.M), 256, 0, st>>>(plan.M, plan.off, plan.crp, plan.tcol, (const T*)plan.tval,
                                                    cci, cv);
    e = cudaGetLastError();
  }
  return e;
}

// The reference's one-call form: outputs cudaMalloc'd here, freed by the caller.
template <typename T>
b2_status spgemm(const b2_csr* A, const b2_csr* B, int64_t** dC_rowptr, int32_t** dC_colind, T** dC_values,
                 int64_t* hC_nnz, cudaStream_t st) {
  if (!dC_rowptr || !dC_colind || !dC_values || !hC_nnz) return B2_INVALID_ARGUMENT;
  *dC_rowptr = nullptr;
  *dC_colind = nullptr;
  *dC_values = nullptr;
  *hC_nnz = 0;
  SpPlan plan;
  b2_status s = compute<T>(A, B, st, plan);
  if (s != B2_SUCCESS) {
    plan.release();
    return s;
  }
  int64_t* crp = nullptr;
  int32_t* cci = nullptr;
  T* cv = nullptr;
  cudaError_t e = cudaMalloc((void**)&crp, (size_t)(plan.M + 1) * sizeof(int64_t));
  if (e == cudaSuccess && plan.nnz > 0) e = cudaMalloc((void**)&cci, (size_t)plan.nnz * sizeof(int32_t));
  if (e == cudaSuccess && plan.nnz > 0) e = cudaMalloc((void**)&cv, (size_t)plan.nnz * sizeof(T));
  if (e == cudaSuccess) e = fill<T>(plan, crp, cci, cv, st);
  plan.release();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaFree(crp);
    cudaFree(cci);
    cudaFree(cv);
    return e == cudaErrorMemoryAllocation ? B2_OUT_OF_MEMORY : from_cuda(e);
  }
  *dC_rowptr = crp;
  *dC_colind = cci;
  *dC_values = cv;
  *hC_nnz = plan.nnz;
  return B2_SUCCESS;
}

}  // namespace
}  // namespace b2

extern "C" b2_status b2_release_scratch(void) {
  cudaMemPool_t pool;
  B2_CUDA_TRY(b2::scratch_pool(&pool));
  B2_CUDA_TRY(cudaDeviceSynchronize());   // releases queued on streams are made
  return b2::from_cuda(cudaMemPoolTrimTo(pool, 0));
}

extern "C" b2_status b2_minplus_spgemm_f32(const b2_csr* A, const b2_csr* B, int64_t** dC_rowptr,
                                           int32_t** dC_colind, float** dC_values, int64_t* hC_nnz,
                                           b2_stream stream) {
  if (A && A->weight_type != B2_W_F32) return B2_INVALID_ARGUMENT;
  if (B && B->weight_type != B2_W_F32) return B2_INVALID_ARGUMENT;
  return b2::spgemm<float>(A, B, dC_rowptr, dC_colind, dC_values, hC_nnz, (cudaStream_t)stream);
}

extern "C" b2_status b2_minplus_spgemm_i32(const b2_csr* A, const b2_csr* B, int64_t** dC_rowptr,
                                           int32_t** dC_colind, int32_t** dC_values, int64_t* hC_nnz,
                                           b2_stream stream) {
  return b2::spgemm<int32_t>(A, B, dC_rowptr, dC_colind, dC_values, hC_nnz, (cudaStream_t)stream);
}

extern "C" b2_status b2_minplus_spgemm_plan(const b2_csr* A, const b2_csr* B, b2_stream stream,
                                            b2_spgemm_plan* plan, int64_t* hC_nnz) {
  if (!A || !B || !plan || !hC_nnz) return B2_INVALID_ARGUMENT;
  *plan = nullptr;
  *hC_nnz = 0;
  if (A->weight_type != B->weight_type) return B2_INVALID_ARGUMENT;
  b2::SpPlan* p = new b2::SpPlan();
  p->wt = A->weight_type;
  const b2_status s = A->weight_type == B2_W_F32 ? b2::compute<float>(A, B, (cudaStream_t)stream, *p)
                                                  : b2::compute<int32_t>(A, B, (cudaStream_t)stream, *p);
  if (s != B2_SUCCESS) {
    p->release();
    delete p;
    return s;
  }
  *plan = reinterpret_cast<b2_spgemm_plan>(p);
  *hC_nnz = p->nnz;
  return B2_SUCCESS;
}

extern "C" b2_status b2_minplus_spgemm_fill(b2_spgemm_plan plan, int64_t* dC_rowptr, int32_t* dC_colind,
                                            void* dC_values, b2_stream stream) {
  b2::SpPlan* p = reinterpret_cast<b2::SpPlan*>(plan);
  if (!p || !dC_rowptr || (p->nnz > 0 && (!dC_colind || !dC_values))) return B2_INVALID_ARGUMENT;
  const cudaStream_t st = (cudaStream_t)stream;
  p->st = st;   // scratch is released in the order of this stream
  const cudaError_t e = p->wt == B2_W_F32 ? b2::fill<float>(*p, dC_rowptr, dC_colind, (float*)dC_values, st)
                                          : b2::fill<int32_t>(*p, dC_rowptr, dC_colind, (int32_t*)dC_values, st);
  p->release();
  delete p;
  return b2::from_cuda(e);
}

extern "C" b2_status b2_minplus_spgemm_plan_free(b2_spgemm_plan plan) {
  b2::SpPlan* p = reinterpret_cast<b2::SpPlan*>(plan);
  if (!p) return B2_INVALID_ARGUMENT;
  p->release();
  delete p;
  return B2_SUCCESS;
}
