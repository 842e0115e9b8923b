// t(X) X of more than 128 columns on the 8-bit tensor cores, in exact integer arithmetic.
//
// Every cell is split into seven signed base-256 digits relative to its column's largest magnitude (56 bits with the
// sign: x = 2^e * sum of d_i 2^(-8 i - 7)), the digits are multiplied by tcgen05.mma (kind::i8) with 32-bit sums in tensor memory,
// and the products of the same weight i + j are added up as 64-bit integers: no rounding, no order (the scheme of Ozaki and others for
// integer matrix units). Kept are the products with i + j <= 7. So a cell is off by 2^-56 of its column's 2^e at most, whatever its own
// size, and a row's product by 2^-61.6 of the two columns' 2^e. That is little for an entry whose cells come near their columns' largest
// magnitudes, and all of it for one whose cells are small where the other column is not zero. The guard, which a block's first product
// runs before it (k_split_guard), therefore bounds the error of every entry of the result against the sum of its terms' magnitudes, and
// takes the digits only where all of them stay within SP_LOSS = 2^-50 of it, whatever the order of the rows; else, and where a value
// is not finite, the FP64 tensor core does the sums (k_gemm_tn, 37 TFLOP/s), whose own bound is a rounding of 2^-53 per four rows.
// Measured, error over the sum of the terms' magnitudes, mean square and largest (FP64 products beside it): 200,000 x 250 of lists, runs,
// small dictionaries and normal values 1.2e-17 and 1.1e-16 (1.6e-15 and 4.8e-14), 20,011 x 257 of six kinds 2.0e-17 and 2.7e-16 (1.2e-15
// and 1.6e-14), 8,000 x 250 1.8e-17 and 2.9e-16 (2.8e-16 and 4.1e-15), 4,096 x 500 2.2e-17 and 3.2e-16 (4.0e-16 and 9.1e-15).
//
//  * k_split_maps, k_split_cols (cla_generic.cu), k_split: dense maps, other columns by kind, decompressed rows -> planes [block of 128 columns][16 rows][digit][column][16 bytes], which is at once the layout of
//    the operands in shared memory (K-major, no swizzle: a core matrix is 8 columns x 16 rows), so that a stage is copied as it lies.
//  * k_syrk_i8: a CTA takes one pair of column blocks, half of the weights and a range of rows: bulk copies in a ring of
//    four stages, a warp per sum issues its products, four warps take the sums out of tensor memory every 16,384 rows.
//  * k_syrk_final: the integers to doubles, both triangles.
//  * k_split_guard: the verdict over the guard's sums, which the same kernels form: planes of two digits a cell, "not zero" u and the
//    leading seven bits of the magnitude a, and their four products.
#include "cla_common.cuh"
#include "cla_split.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace cla {

constexpr int SP_STAGES = 4;
constexpr int SP_RING = 224 * 1024;
constexpr int SP_T = 288;                               // four warps that take sums out, one that copies, four that multiply
constexpr int SP_BLOCKS = 16;                           // 2048 columns
constexpr int SP_ITEMS = SP_BLOCKS * (SP_BLOCKS - 1) + 3 * SP_BLOCKS;
constexpr int64_t SP_TOTAL = 4 << 20;                   // rows whose 64-bit sums are safe: five products of 2^14 in units of 2^24 a row, with room
// rows whose sums stay below 2^31: seven products of 2^14 a row and weight
constexpr int SP_ROWS = 16384;
constexpr int SP_PAD = 24;                              // halves: whole stages of every set
// What a CTA multiplies: a set of products d_i d_j whose sums fit tensor memory, four of 128 columns. Two sets for a pair of
// different blocks (weights 0..3 and 4..7), three for a block with itself, where i < j stands for j < i too: those sums D are kept apart
// from the E of i = j.
struct SplitSet {
  int products, digits, steps;  // steps of 32 rows in a stage
  int clocks;                   // measured, of a step: what the CTAs are dealt by
};
__host__ __device__ constexpr SplitSet sp_set(int t) {
  return t == 0 ? SplitSet{10, 4, 2, 770} : t == 1 ? SplitSet{24, 7, 1, 1690} : t == 2 ? SplitSet{4, 3, 4, 380} : t == 3 ? SplitSet{5, 5, 3, 470}
                                                                                                 : t == 4 ? SplitSet{10, 7, 2, 755}
                                                                                                          : SplitSet{4, 2, 3, 400};
}
constexpr int SP_GUARD = 5;  // the guard's set, of any pair of blocks: u u', u a', a u', a a' (its clocks: all items are alike)
// The sum (0..3) that product i, j of set t goes to, -1: not in the set
__host__ __device__ constexpr int sp_sum(int t, int i, int j) {
  const int w = i + j;
  if (t == 0) return w <= 3 ? w : -1;
  if (t == 1) return w >= 4 && w <= 7 ? w - 4 : -1;
  if (t == SP_GUARD) return i < 2 && j < 2 ? 2 * i + j : -1;
  if (i > j) return -1;
  if (t == 2) return w == 0 ? 0 : w == 1 ? 1 : w == 2 ? (i < j ? 2 : 3) : -1;          // E0 D1 D2 E2
  if (t == 3) return w == 3 ? 0 : w == 4 ? (i < j ? 1 : 2) : -1;                       // D3 D4 E4
  return w == 5 ? 0 : w == 6 ? (i < j ? 1 : 2) : w == 7 ? 3 : -1;                       // D5 D6 E6 D7
}
// Whether it is the first of its sum, products in the order of i
__host__ __device__ constexpr bool sp_first(int t, int i, int j) {
  for (int a = 0; a < i; a++)
    for (int b = 0; b < SP_DIG; b++)
      if (sp_sum(t, a, b) == sp_sum(t, i, j)) return false;
  for (int b = 0; b < j; b++)
    if (sp_sum(t, i, b) == sp_sum(t, i, j)) return false;
  return true;
}
// Error of an entry over the sum of its terms' magnitudes, at most. With 2^-50 columns of the usual distributions are taken (bounds
// found: 200,000 x 250 of lists, runs, small dictionaries and normal values 2^-51.3, six kinds of column on 4,096 to 40,001 rows 2^-51,
// exponentially distributed values up to 2^e = 16 times their mean), some blocks whose lists have only a few rows in common are not.
constexpr int SP_LOSS = -50;
// Below these the FP64 products are as fast or nearly (us, FP64 / digits; mixed columns, whose kinds per 32 columns decide how they are decompressed): 200,000 x 130
// 367 / 369, x 140 366 / 379, x 150 375 / 399, x 160 311 / 247, x 170 466 / 430, x 176 455 / 438, 100,000 x 180 234 / 230, 60,000 x 150 132 / 128; 2,500 x 250
// 42 / 42, 5,000 x 250 44 / 44, 9,000 x 250 54 / 48, 12,000 x 180 47 / 47, 5,000 x 800 225 / 108.
constexpr int SP_MIN_COLS = 176, SP_MIN_ROWS = 4096;
constexpr int64_t SP_MIN_CELLS = 2000000;
constexpr int SP_MAPS_COLS = 129;  // where k_split_maps takes the block (200,000 x 130 bytes 319 / 222, 1000 values 359 / 260; 16,000 x 130 47 / 38)
constexpr size_t SP_CHUNK = 192ull << 20;  // bytes of a chunk of rows (200,000 x 250: 280 us in one chunk of 358 MB, 293 in two, 345 in four; 100 MB more cost a first call a millisecond)
constexpr size_t SP_SMEM = (size_t)SP_RING + 1024;

struct SplitPlan {
  bool tried = false, ok = false;  // ok: the guard has let the block pass
  int32_t* expo = nullptr;         // [nCols] e of every column
};

// --------------------------------------------------------------------------------------------------
// A thread per column and 16 rows; rows behind the last one count as zeros. Bound: the two streams (8 bytes in, 7 out).
template <bool GUARD>
__global__ void __launch_bounds__(128) k_split(const double* __restrict__ X, size_t ld, int rows, int n, const int32_t* __restrict__ expo,
                                               int64_t halves, uint8_t* __restrict__ planes, int32_t* __restrict__ refused) {
  const int c = blockIdx.y * SP_COLS + threadIdx.x;
  if (c >= n) return;
  const double scale = split_scale(expo[c]);
  bool bad = false;
  for (int64_t h = blockIdx.x; h < halves; h += gridDim.x) {
    unsigned long long v[16];
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = split_pack<GUARD>(h * 16 + i < rows ? __ldcs(X + (size_t)(h * 16 + i) * ld + c) : 0.0, scale, bad);
    split_store<GUARD>(planes + ((size_t)blockIdx.y * halves + h) * SP_HALF, c, v);
  }
  if (GUARD && bad) *refused = 1;
}

// Dense maps straight to planes: a CTA owns 16 columns, their tables of digits in shared memory (entry k of slot s at k * 16 + s, so that a
// lane stays in its banks), and a range of rows; a lane takes 16 rows of its column.
// Bound: the latency of the maps' loads, a sector a lane, next to the planes written (7 bytes a cell). The self product of 160,000 x 250 of 1000 values
// took 421 us with the rows decompressed and split, 232 with this (256 values: 380 and 211).
constexpr int SM_W = 24;        // (16: 160,000 x 250 of 256 values 211 us instead of 205)
constexpr int SM_VALS = 1600;  // tuples, at most: 200 KB
template <bool GUARD>
__global__ void __launch_bounds__(SM_W * 32, 1) k_split_maps(const DevGroup* __restrict__ groups, const int32_t* __restrict__ colSrc, const double* __restrict__ constV,
                                                             const int32_t* __restrict__ expo, int n, int r0, int r1, int64_t halves,
                                                             uint8_t* __restrict__ planes, int32_t* __restrict__ refused) {
  extern __shared__ unsigned long long smt[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.y * 16 + (lane & 15), up = lane >> 4;
  const bool on = c < n;
  const DevGroup& g = groups[colSrc[2 * (on ? c : 0)]];
  const int nv = g.nVals, mt = g.mapType;
  unsigned long long* T = smt + (lane & 15);
  bool bad = false;
  if (on) {
    const double* dict = g.dict + colSrc[2 * c + 1];
    const double cst = constV ? constV[c] : 0.0, scale = split_scale(expo[c]);
    const int gc = g.gCols;
#pragma unroll 4
    for (int k = warp * 2 + up; k < nv; k += SM_W * 2) T[k * 16] = split_pack<GUARD>(cst + dict[(size_t)k * gc], scale, bad);
  }
  __syncthreads();
  uint8_t* o = planes + (size_t)(c / SP_COLS) * halves * SP_HALF;
  const int64_t h0 = halves * blockIdx.x / gridDim.x, h1 = halves * (blockIdx.x + 1) / gridDim.x;
  const void* map = g.map;
  // the ids of a lane's next 16 rows are under way while it works on these
  uint4 a0 = make_uint4(0, 0, 0, 0), b0 = a0;
  auto load = [&](int64_t h) {
    const int64_t r = r0 + h * 16;
    if (h >= h1 || r + 16 > r1 || !on) return;
    if (mt == CLA_MAP_CHAR) {
      a0 = __ldg((const uint4*)((const uint16_t*)map + r));
      b0 = __ldg((const uint4*)((const uint16_t*)map + r) + 1);
    } else if (mt != CLA_MAP_BIT) a0 = __ldg((const uint4*)((const uint8_t*)map + r));
  };
  load(h0 + warp * 2 + up);
  for (int64_t h = h0 + warp * 2 + up; h < h1; h += SM_W * 2) {
    if (!on) continue;
    const int64_t r = r0 + h * 16;
    const uint32_t w[8] = {a0.x, a0.y, a0.z, a0.w, b0.x, b0.y, b0.z, b0.w};
    load(h + SM_W * 2);
    unsigned long long v[16];
    if (r + 16 <= r1 && mt == CLA_MAP_CHAR) {
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = T[(i & 1 ? w[i >> 1] >> 16 : w[i >> 1] & 0xFFFFu) * 16];
    } else if (r + 16 <= r1 && mt != CLA_MAP_BIT) {
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = T[((w[i >> 2] >> (8 * (i & 3))) & 0xFFu) * 16];
    } else {
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = r + i < r1 ? T[map_get(mt, map, nullptr, r + i) * 16] : 0ull;
    }
    split_store<GUARD>(o + (size_t)h * SP_HALF, c, v);
  }
  if (GUARD && bad) *refused = 1;
}

// --------------------------------------------------------------------------------------------------
struct SyrkArgs {
  const uint8_t* planes;
  int64_t halves;               // of every block: 16 rows each, even
  int nBlocks, lastN;           // columns of the last block, a multiple of 16
  int nItems;
  int16_t cta0[SP_ITEMS + 1];   // first CTA of an item: pairs of blocks row by row of the upper triangle, their sets in order
  long long* sums;              // [pairs of blocks][weights 0..3, weights 4..7][column][row]
  int32_t* err;
};

__device__ __forceinline__ uint32_t sp_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool sp_wait(uint32_t bar, uint32_t parity) {
  uint32_t done = 0;
  for (int it = 0; it < (1 << 22) && !done; it++) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
  }
  return done != 0;
}
// Operand of one digit of a stage: no swizzle, K-major; core matrices 128 bytes apart along the columns, `half` along the rows
__device__ __forceinline__ uint64_t sp_desc(uint32_t addr, uint32_t half) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(half >> 4) << 16 | (uint64_t)(128 >> 4) << 32 | (uint64_t)1 << 46;
}
__device__ __forceinline__ void sp_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b),
               "r"(idesc), "r"((uint32_t)add)
               : "memory");
}
// The products of one stage that go to one sum
template <int T, int SUM, int P = 0>
__device__ __forceinline__ void sp_products(uint32_t sum, uint64_t a, uint64_t b, uint32_t idesc, bool fresh) {
  if constexpr (P < SP_DIG * SP_DIG) {
    constexpr int i = P / SP_DIG, j = P % SP_DIG;
    if constexpr (sp_sum(T, i, j) == SUM) {
      constexpr uint64_t DIG = SP_PLANE >> 4;
      sp_mma(sum, a + i * DIG, b + j * DIG, idesc, !(fresh && sp_first(T, i, j)));
    }
    sp_products<T, SUM, P + 1>(sum, a, b, idesc, fresh);
  }
}
// One lane of the warp, the same each time: the loops around stay uniform
__device__ __forceinline__ bool sp_elect() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r != 0;
}
__device__ __forceinline__ void sp_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Bound: the tensor pipe, 64 clocks a product of 128 x 128 x 32, next to the shared memory it reads its operands from, 8 KB a product, and
// the stages are written to. A set of products is what four sums of 128 columns leave of tensor memory (SplitSet). 200,000 x 250 in one
// launch: 150 us, tensor pipe 71 % active; 485 us for the FP64 products. On the way (one launch, some with fewer products): 338 with
// stages of 32 rows, whose waits cost sets of few products more than their products; 328 with the CTAs of an item in row ranges of
// their own, which read the planes from memory three times.
// GUARD: an item per pair, the guard's set.
template <bool GUARD>
__global__ void __launch_bounds__(SP_T, 1) k_syrk_i8(const __grid_constant__ SyrkArgs A) {
  extern __shared__ __align__(1024) unsigned char spsm[];
  __shared__ __align__(8) uint64_t full[SP_STAGES], empty[SP_STAGES], sumFull, sumEmpty;
  __shared__ uint32_t tmemAt;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int item = 0;
  for (int lo = 0, hi = A.nItems; lo < hi;) {  // the last item that starts at or before this CTA
    const int mid = (lo + hi) / 2;
    if (A.cta0[mid] <= (int)blockIdx.x) item = mid, lo = mid + 1;
    else hi = mid;
  }
  int I = 0, J = 0, pair = 0, set = 0;
  for (int it = 0; it + (GUARD ? 1 : I == J ? 3 : 2) <= item; pair++) {
    it += GUARD ? 1 : I == J ? 3 : 2;
    set = it;
    if (++J == A.nBlocks) J = ++I;
  }
  set = GUARD ? SP_GUARD : item - set + (I == J ? 2 : 0);
  const int N = J == A.nBlocks - 1 ? A.lastN : SP_COLS;
  const int part = blockIdx.x - A.cta0[item], parts = A.cta0[item + 1] - A.cta0[item];
  const int digits = sp_set(set).digits, nSums = set == 3 ? 3 : 4;
  const uint32_t smem = (sp_smem(spsm) + 1023u) & ~1023u;
  // A stage: the item's digits of 16 rows and of the next 16, so many times, of the first block and then of the second. The CTAs of an
  // item take stages in turn, so that all items go down the rows together and the planes come from memory once.
  const int R = sp_set(set).steps, nStages = (int)(A.halves / (2 * R)), mine = part < nStages ? (nStages - part + parts - 1) / parts : 0;
  const uint32_t half = (uint32_t)digits * SP_PLANE, block = half * 2 * R, step = block * (I == J ? 1 : 2);
  const int stages = min(SP_STAGES, SP_RING / (int)step);
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(sp_smem(&tmemAt)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < SP_STAGES; i++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sp_smem(full + i)));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sp_smem(empty + i)), "r"(nSums));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sp_smem(&sumFull)), "r"(nSums));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 128;" ::"r"(sp_smem(&sumEmpty)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmemAt;
  const int PIECE = SP_ROWS / 32 / R, pieces = (mine + PIECE - 1) / PIECE;  // stages between two times the sums are taken out
  bool ok = true;
  if (warp == 4) {
    const uint8_t* a = A.planes + (size_t)I * A.halves * SP_HALF;
    const uint8_t* b = A.planes + (size_t)J * A.halves * SP_HALF;
    int s = 0;
    uint32_t ph = 1;
    for (int n = 0; n < mine; n++) {
      ok = sp_wait(sp_smem(empty + s), ph);
      if (!__all_sync(0xffffffffu, ok)) break;
      if (sp_elect()) {
        const uint32_t bar = sp_smem(full + s), dst = smem + (uint32_t)s * step;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(step) : "memory");
        const size_t at = (size_t)(part + (int64_t)n * parts) * (2 * R) * SP_HALF;
        for (int h = 0; h < 2 * R; h++) {
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst + h * half),
                       "l"(a + at + (size_t)h * SP_HALF), "r"(half), "r"(bar)
                       : "memory");
          if (I != J)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst + block + h * half),
                         "l"(b + at + (size_t)h * SP_HALF), "r"(half), "r"(bar)
                         : "memory");
        }
      }
      __syncwarp();
      if (++s == stages) s = 0, ph ^= 1;
    }
  } else if (warp >= 5) {
    // A warp per sum: what a stage costs beside its products (waits, commit, operands to uniform registers: 400 clocks against 64 a product) it
    // costs one warp while the others' products run.
    const uint32_t sum = tmem + (warp - 5) * SP_COLS;
    // 32-bit sums of signed bytes, both operands K-major, N x 128
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(SP_COLS >> 4) << 24);
    int s = 0, done = 0, at = 0;
    uint32_t ph = 0;
    for (int n = 0; n < (warp - 5 < nSums ? mine : 0); n++) {
      ok = true;
      if (at == 0 && n > 0) {  // the sums have been taken out
        ok = sp_wait(sp_smem(&sumEmpty), (uint32_t)(done - 1) & 1u);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      ok = ok && sp_wait(sp_smem(full + s), ph);
      if (!__all_sync(0xffffffffu, ok)) break;
      const uint32_t base = smem + (uint32_t)s * step;
      uint64_t a = sp_desc(base, half), b = sp_desc(I == J ? base : base + block, half);
      const bool out = at == PIECE - 1 || n + 1 == mine;
      if (sp_elect()) {
        for (int r = 0; r < R; r++, a += half >> 3, b += half >> 3)
#define SP_CASE(T, SUM) case T * 4 + SUM: sp_products<T, SUM>(sum, a, b, idesc, at == 0 && r == 0); break;
        if (GUARD) switch (set * 4 + warp - 5) { SP_CASE(5, 0) SP_CASE(5, 1) SP_CASE(5, 2) SP_CASE(5, 3) }
        else switch (set * 4 + warp - 5) {
          SP_CASE(0, 0) SP_CASE(0, 1) SP_CASE(0, 2) SP_CASE(0, 3) SP_CASE(1, 0) SP_CASE(1, 1) SP_CASE(1, 2) SP_CASE(1, 3)
          SP_CASE(2, 0) SP_CASE(2, 1) SP_CASE(2, 2) SP_CASE(2, 3) SP_CASE(3, 0) SP_CASE(3, 1) SP_CASE(3, 2)
          SP_CASE(4, 0) SP_CASE(4, 1) SP_CASE(4, 2) SP_CASE(4, 3)
        }
#undef SP_CASE
        sp_commit(sp_smem(empty + s));
        if (out) sp_commit(sp_smem(&sumFull));
      }
      __syncwarp();
      at = out ? 0 : at + 1;
      done += out;
      if (++s == stages) s = 0, ph ^= 1;
    }
  } else {
    long long* hi = A.sums + (size_t)pair * 2 * SP_COLS * SP_COLS + warp * 32 + lane;
    long long* lo = hi + SP_COLS * SP_COLS;
    const uint32_t t0 = tmem + ((uint32_t)warp << 21);
    for (int p = 0; p < pieces && ok; p++) {
      ok = sp_wait(sp_smem(&sumFull), (uint32_t)p & 1u);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int c = 0; c < N; c += 8) {
        int32_t v[4][8];
#pragma unroll
        for (int w = 0; w < 4; w++)
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                       : "=r"(v[w][0]), "=r"(v[w][1]), "=r"(v[w][2]), "=r"(v[w][3]), "=r"(v[w][4]), "=r"(v[w][5]), "=r"(v[w][6]), "=r"(v[w][7])
                       : "r"(t0 + min(w, nSums - 1) * SP_COLS + c)
                       : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int w = 0; w < 4; w++)  // (nothing reads the registers before the wait)
          asm volatile("" : "+r"(v[w][0]), "+r"(v[w][1]), "+r"(v[w][2]), "+r"(v[w][3]), "+r"(v[w][4]), "+r"(v[w][5]), "+r"(v[w][6]), "+r"(v[w][7]));
#pragma unroll
        for (int i = 0; i < 8; i++) {
          // in units of weight 3 and of weight 7; of a block with itself 2 D + E, whose mean with its mirror image is D + D' + E
          const long long x = v[0][i], y = v[1][i], z = v[2][i], u = v[3][i];
          unsigned long long* h = (unsigned long long*)(hi + (size_t)(c + i) * SP_COLS);
          unsigned long long* l = (unsigned long long*)(lo + (size_t)(c + i) * SP_COLS);
          if (GUARD) {  // a a', and what the error is bounded by (k_split_guard)
            atomicAdd(h, (unsigned long long)u);
            atomicAdd(l, (unsigned long long)(y + z + 5 * x));
          } else if (set < 2) atomicAdd(set == 0 ? h : l, (unsigned long long)(((x * 256 + y) * 256 + z) * 256 + u));
          else if (set == 2) atomicAdd(h, (unsigned long long)(((x * 256 + 2 * y) * 256 + 2 * z + u) * 256));
          else if (set == 3) {
            atomicAdd(h, (unsigned long long)(2 * x));
            atomicAdd(l, (unsigned long long)((2 * y + z) * (1 << 24)));
          } else atomicAdd(l, (unsigned long long)((2 * x * 256 + 2 * y + z) * 256 + 2 * u));
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sp_smem(&sumEmpty)) : "memory");
    }
  }
  if (!ok) atomicExch(A.err, 106);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  __syncwarp();
  if (warp == 5) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

// Cells of the upper triangle's blocks from their two sums, to both triangles. grid: (pairs of blocks, rows of a block)
__global__ void __launch_bounds__(SP_COLS) k_syrk_final(const long long* __restrict__ sums, int nBlocks, int n, const int32_t* __restrict__ expo,
                                                        double* __restrict__ out, int add, const int32_t* __restrict__ err) {
  int I = 0, first = 0;
  while (first + nBlocks - I <= (int)blockIdx.x) first += nBlocks - I++;
  const int J = I + blockIdx.x - first, r = I * SP_COLS + threadIdx.x, c = J * SP_COLS + blockIdx.y;
  if (r >= n || c >= n) return;
  const long long* p = sums + (size_t)blockIdx.x * 2 * SP_COLS * SP_COLS + blockIdx.y * SP_COLS + threadIdx.x;
  long long hi = p[0], lo = p[SP_COLS * SP_COLS];
  if (I == J) {  // the mean with the mirror image
    const long long* q = sums + (size_t)blockIdx.x * 2 * SP_COLS * SP_COLS + threadIdx.x * SP_COLS + blockIdx.y;
    hi = hi / 2 + q[0] / 2 + (hi % 2 + q[0] % 2) / 2;
    lo = lo / 2 + q[SP_COLS * SP_COLS] / 2 + (lo % 2 + q[SP_COLS * SP_COLS] % 2) / 2;
  }
  // in units of weights 3 and 7: 2^72 and 2^40, times 2^(e + e' - 110)
  const double h = (double)hi, rest = (double)(hi - (long long)h);
  double x = scalbn(h + fma((double)lo, 0x1p-32, rest), expo[r] + expo[c] - 38);
  if (*err) x = __longlong_as_double(0x7ff8000000000000ll);  // (a kernel gave up: visible in the result as well)
  if (I == J && c < r) return;  // (written from the other side)
  if (add) x += out[(size_t)r * n + c];
  out[(size_t)r * n + c] = x;
  out[(size_t)c * n + r] = x;
}

// Whether an entry of the result could be off by more than 2^SP_LOSS of the sum of its terms' magnitudes. In units of 2^(e + e') a row's
// product is off by 2^-56 |y| + 2^-56 |x| (the cells' last digits, where the other cell is not zero) and 2^-61.6 (the products left out) at
// most. With |x| < (a + 1) 2^-7 that is 2^-63 (u a' + a u' + 5 u u'); the magnitudes add up to 2^-14 a a' at least. grid: (pairs of blocks, rows
// of a block)
__global__ void __launch_bounds__(SP_COLS) k_split_guard(const long long* __restrict__ sums, int nBlocks, int n, const int32_t* __restrict__ err,
                                                         int32_t* __restrict__ refused) {
  int I = 0, first = 0;
  while (first + nBlocks - I <= (int)blockIdx.x) first += nBlocks - I++;
  const int J = I + blockIdx.x - first, r = I * SP_COLS + threadIdx.x, c = J * SP_COLS + blockIdx.y;
  if (r >= n || c >= n) return;
  const long long* p = sums + (size_t)blockIdx.x * 2 * SP_COLS * SP_COLS + blockIdx.y * SP_COLS + threadIdx.x;
  const long long magnitudes = p[0], lost = p[SP_COLS * SP_COLS];
  if ((lost << (-49 - SP_LOSS)) > magnitudes || *err) *refused = 1;
}

// --------------------------------------------------------------------------------------------------
static int blocks_of(const Matrix* m) { return (m->nCols + SP_COLS - 1) / SP_COLS; }
// Rows of a chunk, in even parts of about SP_CHUNK bytes, a multiple of SKIP_ROWS; dense: it is decompressed first
static int64_t split_chunk(const Matrix* m, bool dense) {
  const double row = (dense ? ((m->nCols + 1) & ~1) * 8.0 : 0.0) + (double)blocks_of(m) * SP_COLS * SP_DIG;
  const int64_t parts = std::max<int64_t>(1, (int64_t)(m->nRows * row / SP_CHUNK + 0.5));
  return std::max<int64_t>(SKIP_ROWS, ((m->nRows + parts - 1) / parts + SKIP_ROWS - 1) / SKIP_ROWS * SKIP_ROWS);
}

// Every column in a dense map of bits, bytes or 16 bits whose table fits: k_split_maps; the longest table, 0: no
static int split_maps_vals(const Matrix* m) {
  if (!m->colSrcValid || m->multiCover) return 0;
  int64_t covered = 0;
  int vals = 0;
  for (auto& g : m->groups) {
    if (g.type != GT_DDC || g.nVals > SM_VALS) return 0;
    if (g.mapType != CLA_MAP_BIT && g.mapType != CLA_MAP_BYTE && g.mapType != CLA_MAP_UBYTE && g.mapType != CLA_MAP_CHAR) return 0;
    covered += g.gCols;
    vals = std::max(vals, g.nVals);
  }
  return covered == m->nCols ? vals : 0;
}
static bool split_covers(const Matrix* m, bool maps) {
  const int64_t cells = (int64_t)m->nRows * m->nCols;
  return m->nCols >= (maps ? SP_MAPS_COLS : SP_MIN_COLS) && m->nCols <= SP_BLOCKS * SP_COLS && m->nRows >= SP_MIN_ROWS && cells >= SP_MIN_CELLS && m->colSrcValid && !m->overlapping;
}

// How the rows get to planes, and what of scratch2 that and the sums take
struct SplitShape {
  int vals;          // k_split_maps, its longest table; 0: not
  bool cols, dense;  // k_split_cols; k_split of decompressed rows
  int64_t chunk;
  size_t ld, denseBytes, planeBytes, sumBytes;
};
static SplitShape split_shape(Matrix* m, int vals, cudaStream_t s) {
  SplitShape S{};
  const int nb = blocks_of(m), pairs = nb * (nb + 1) / 2;
  S.vals = vals;
  S.cols = !vals && split_cols_covers(m, s);
  S.dense = !vals && !S.cols;
  S.chunk = split_chunk(m, S.dense);
  S.ld = (size_t)((m->nCols + 1) & ~1);
  S.denseBytes = S.dense ? (size_t)S.chunk * S.ld * 8 : 0;
  S.planeBytes = (size_t)nb * (S.chunk / 16 + SP_PAD) * SP_HALF;
  S.sumBytes = (size_t)pairs * 2 * SP_COLS * SP_COLS * 8;
  return S;
}
// All rows through planes and products. refused: the guard's planes, sums and verdict (set, or left), dOut null; else the product.
static int64_t split_run(Matrix* m, const SplitShape& S, const int32_t* expo, double* dOut, int32_t* refused, cudaStream_t s) {
  const int n = m->nCols, nb = blocks_of(m), pairs = nb * (nb + 1) / 2;
  const bool guard = refused != nullptr;
  int64_t rc;
  if ((rc = ensure_scratch2(m, S.denseBytes + S.planeBytes + S.sumBytes)) < 0) return rc;
  double* X = (double*)m->scratch2;
  uint8_t* planes = (uint8_t*)m->scratch2 + S.denseBytes;
  long long* sums = (long long*)(planes + S.planeBytes);
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, SP_SMEM, k_syrk_i8<false>, k_syrk_i8<true>); e < 0) return e;
  static OncePerDevice onceMaps;
  if (const int64_t e = allow_smem(onceMaps, m->device, (size_t)SM_VALS * 128, k_split_maps<false>, k_split_maps<true>); e < 0) return e;
  SyrkArgs A{};
  A.planes = planes;
  A.nBlocks = nb;
  A.lastN = (n - (nb - 1) * SP_COLS + 15) / 16 * 16;
  A.nItems = guard ? pairs : pairs * 2 + nb;
  A.sums = sums;
  A.err = m->dErr;
  // CTAs by the time of an item
  {
    double total = 0.0, at = 0.0;
    auto each = [&](auto&& f) {
      int it = 0;
      for (int I = 0; I < nb; I++)
        for (int J = I; J < nb; J++)
          for (int t = guard ? SP_GUARD : I == J ? 2 : 0; t < (guard ? SP_GUARD + 1 : I == J ? 5 : 2); t++, it++) {
            const SplitSet set = sp_set(t);
            f(it, J == nb - 1 ? std::max(set.clocks * A.lastN / (double)SP_COLS, set.clocks * 0.6) : set.clocks);
          }
    };
    each([&](int, double c) { total += c; });
    const int ctas = std::max(m->smCount, A.nItems);
    each([&](int it, double c) {
      const int want = (int)(at / total * ctas + 0.5);
      A.cta0[it] = (int16_t)std::min(std::max(want, it == 0 ? 0 : A.cta0[it - 1] + 1), ctas - (A.nItems - it));
      at += c;
    });
    A.cta0[A.nItems] = (int16_t)ctas;
  }
  int64_t summed = 0;  // rows in the 64-bit sums
  bool add = false;
  for (int64_t r0 = 0; r0 < m->nRows; r0 += S.chunk) {
    const int r1 = (int)std::min<int64_t>(m->nRows, r0 + S.chunk), rows = r1 - (int)r0;
    if (summed == 0) CLA_CUDA(cudaMemsetAsync(sums, 0, S.sumBytes, s));
    A.halves = ((int64_t)rows + 16 * SP_PAD - 1) / (16 * SP_PAD) * SP_PAD;
    if (S.vals) {
      const dim3 grid((unsigned)std::max<int64_t>(1, std::min<int64_t>(A.halves / (SM_W * 2) + 1, m->smCount / ((n + 15) / 16))), (n + 15) / 16);
      const double* constV = m->hasConst ? m->dConstV : nullptr;
      const size_t smem = (size_t)S.vals * 128;
      if (guard) k_split_maps<true><<<grid, SM_W * 32, smem, s>>>(m->dGroups, m->dColSrc, constV, expo, n, (int)r0, r1, A.halves, planes, refused);
      else k_split_maps<false><<<grid, SM_W * 32, smem, s>>>(m->dGroups, m->dColSrc, constV, expo, n, (int)r0, r1, A.halves, planes, nullptr);
      m->stats.kernel_launches++;
    } else if (S.cols) {
      if ((rc = launch_split_cols(m, (int)r0, r1, expo, A.halves, planes, refused, s)) < 0) return rc;
    } else {
      if ((rc = launch_decompress_range(m, (int)r0, r1, X, s, S.ld)) < 0) return rc;
      const dim3 grid((unsigned)std::min<int64_t>(A.halves, 16 * m->smCount / nb), nb);
      if (guard) k_split<true><<<grid, SP_COLS, 0, s>>>(X, S.ld, rows, n, expo, A.halves, planes, refused);
      else k_split<false><<<grid, SP_COLS, 0, s>>>(X, S.ld, rows, n, expo, A.halves, planes, nullptr);
      m->stats.kernel_launches++;
    }
    if (r0 == 0 && !guard) prof_begin(m, s);
    if (guard) k_syrk_i8<true><<<A.cta0[A.nItems], SP_T, SP_SMEM, s>>>(A);
    else k_syrk_i8<false><<<A.cta0[A.nItems], SP_T, SP_SMEM, s>>>(A);
    if (r0 == 0 && !guard) prof_end(m, s);
    m->stats.kernel_launches++;
    summed += rows;
    if (guard) continue;  // (its sums are safe for any number of rows: below 2^14 a row)
    if (r1 == m->nRows || summed + S.chunk > SP_TOTAL) {
      k_syrk_final<<<dim3(pairs, SP_COLS), SP_COLS, 0, s>>>(sums, nb, n, expo, dOut, add ? 1 : 0, m->dErr);
      m->stats.kernel_launches++;
      summed = 0;
      add = true;
    }
  }
  if (guard) {
    k_split_guard<<<dim3(pairs, SP_COLS), SP_COLS, 0, s>>>(sums, nb, n, m->dErr, refused);
    m->stats.kernel_launches++;
  }
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

// The columns' exponents, from the extrema (a bound on the cells is enough), and the guard's verdict, which the host waits for: once per
// block, in its first product (200,000 x 250 mixed: that product 639 us, the others 300).
static int64_t ensure_split(Matrix* m, const SplitShape& S, cudaStream_t s) {
  SplitPlan& P = *m->split;
  const int n = m->nCols;
  std::vector<double> lo, hi;
  int64_t rc;
  P.tried = true;  // (whatever comes: not again)
  if ((rc = col_minmax(m, lo, hi, s)) < 0) return rc;
  std::vector<int32_t> e(n + 1, 0);
  for (int c = 0; c < n; c++) {
    const double M = std::max(std::fabs(lo[c]), std::fabs(hi[c]));
    if (M == 0.0) continue;
    if (!(M < 1e140 && M > 1e-140)) return CLA_OK;  // the scale or the sums would leave the range of doubles
    int x;
    if (std::frexp(M, &x) > 0.99) x++;  // the leading digit stays within a byte when the others carry
    e[c] = x;
  }
  void* p = nullptr;
  if (plan_alloc(m, &p, ((size_t)n + 1) * 4) < 0) return CLA_OK;
  P.expo = (int32_t*)p;
  int32_t* refused = P.expo + n;
  CLA_CUDA(cudaMemcpyAsync(p, e.data(), ((size_t)n + 1) * 4, cudaMemcpyHostToDevice, s));
  if ((rc = split_run(m, S, P.expo, nullptr, refused, s)) < 0) return rc;
  int32_t no = 1;
  CLA_CUDA(cudaMemcpyAsync(&no, refused, 4, cudaMemcpyDeviceToHost, s));
  CLA_CUDA(cudaStreamSynchronize(s));
  P.ok = no == 0;
  return CLA_OK;
}

int64_t split_tsmm(Matrix* m, double* dOut, cudaStream_t s) {
  const int vals = split_maps_vals(m);
  if (!split_covers(m, vals > 0)) return 0;
  if (!m->split) m->split = new SplitPlan();
  if (m->split->tried && !m->split->ok) return 0;
  if (!m->split->tried) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
      cudaGetLastError();
      return 0;  // (a call that is being captured runs nothing yet: no plan from it)
    }
  }
  const SplitShape S = split_shape(m, vals, s);
  int64_t rc = m->split->tried ? CLA_OK : ensure_split(m, S, s);
  if (rc == CLA_OK && !m->split->ok) return 0;
  if (rc == CLA_OK) rc = split_run(m, S, m->split->expo, dOut, nullptr, s);
  if (rc != CLA_ERR_NOMEM) return rc < 0 ? rc : 1;
  // Planes and sums can take more scratch than the FP64 products' chunk (100,000 x 130: 188 MiB against 115): no room, no digits from now on
  m->split->ok = false;
  return 0;
}

void split_plan_free(Matrix* m) {
  delete m->split;
  m->split = nullptr;
}

}  // namespace cla
