// t(X) %*% X on a compressed matrix (CLALibTSMM.leftMultByTransposeSelf, lib/CLALibTSMM.java:59-94).
//
// The reference multiplies dictionaries when there are few groups and otherwise decompresses the
// whole matrix and runs a dense self product (:73-77). Here the second strategy is used for all
// inputs, but blocked so the dense form never exists in full: a chunk of rows is decompressed into scratch, an FP64
// tensor-core SYRK adds chunk^T * chunk into the upper triangle of the result, and the next chunk reuses the scratch.
// Constant columns are part of the decompressed chunk, so no correction layer is needed.
#include "cla_common.cuh"
#include <algorithm>
#include <cstdlib>
#include <type_traits>

namespace cla {

__device__ __forceinline__ void dmma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// m16n8k8: eight times the flops of m8n8k4 per instruction and, per flop, half the B-fragment bytes (a 16-row tile
// reuses each B value for twice the rows). Fragments (PTX ISA, mma.m16n8k8 .f64): a0 (g, t), a1 (g + 8, t),
// a2 (g, t + 4), a3 (g + 8, t + 4); b0 (k = t, n = g), b1 (k = t + 4, n = g); c0 (g, 2t), c1 (g, 2t + 1),
// c2 (g + 8, 2t), c3 (g + 8, 2t + 1), with g = lane >> 2, t = lane & 3.
__device__ __forceinline__ void dmma1688(double (&c)[4], double a0, double a1, double a2, double a3, double b0, double b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// Loads pinned where they are written: volatile asm is not moved across the (volatile) DMMAs, so a load issued
// before a block of DMMAs stays in flight during them instead of being sunk to its first use behind them.
__device__ __forceinline__ double ld_f64_here(const double* p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ld_u8_here(const uint8_t* p) {
  uint32_t v;
  asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ld_u16_here(const uint16_t* p) {
  uint32_t v;
  asm volatile("ld.global.nc.u16 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// C [aCols x bCols] += A^T B for row-major chunks A [rows x lda], B [rows x ldb] of the same rows, on 128 x 128 blocks of C:
// a CTA owns one block (or, on the diagonal of a self product, its upper triangle of 32 x 32 tiles) over a range of rows,
// a warp one 32 x 32 tile in registers (eight m16n8k8 per eight rows from 16 fragment loads). 16-row stages arrive row by
// row by TMA bulk copies in a ring of six; full / empty mbarriers let the warps drift apart, so
// that one's fragment loads hide behind the others' products. Rows of a stage are 132 doubles apart (4 mod 16:
// conflict-free fragment loads). The blocks get CTAs in proportion to their tiles.
// Bound: the FP64 tensor pipe, 1024 clocks per tile and stage on a scheduler. 98,304 rows x 250 columns: 308 us with the
// copies made by warp 0 between its products (64 x 64 blocks of m8n8k4 with the stage loaded through registers: 316 at 45 %
// of the pipe and atomics four times as often; cp.async by all threads and a barrier per stage: 318); with warps for the
// copies, 100,001 rows: 129 columns 508 -> 224 us, 200: 283 -> 230, 250: 350 -> 313 (every warp copying its row of each
// stage: 319, 226, 326; one warp for all copies and 96 registers for the others: 352, 232, 317).
constexpr int GT_KT = 16;
constexpr int GT_BLK = 128;
constexpr int GT_LD = GT_BLK + 4;
constexpr int GT_WARPS = 16;
constexpr int GT_COPY = 4;  // warps that make the copies: a warpgroup, which hands its registers to the others
constexpr int GT_T = (GT_WARPS + GT_COPY) * 32;
constexpr int GT_STAGES = 6;
constexpr int GT_STAGE = 2 * GT_KT * GT_LD;  // doubles
constexpr size_t GT_SMEM = (size_t)GT_STAGES * GT_STAGE * sizeof(double) + 2 * GT_STAGES * sizeof(uint64_t);
constexpr int GT_PAIRS = 64;  // blocks per launch
struct GemmBlocks {
  int n;
  int cta0[GT_PAIRS + 1];   // CTAs [cta0[p], cta0[p + 1]) split the rows of block p
  int16_t bi[GT_PAIRS], bj[GT_PAIRS];
};
__device__ __forceinline__ bool gt_wait(uint32_t bar, uint32_t parity) {
  uint32_t done = 0;
  for (int it = 0; it < (1 << 20) && !done; it++)
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
  return done != 0;
}
// lda, ldb: even, rows 16-byte aligned; the rows up to the next multiple of GT_KT behind `rows` are zero.
template <bool SYRK>
__global__ void __launch_bounds__(GT_T, 1)
k_gemm_tn(const double* __restrict__ A, int aCols, int lda, const double* __restrict__ B, int bCols, int ldb, int rows,
          double* __restrict__ C, const __grid_constant__ GemmBlocks G, int32_t* err) {
  extern __shared__ __align__(128) double gts[];  // [GT_STAGES][A | B][GT_KT][GT_LD], full and empty barriers
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  int p = 0;
  while (p + 1 < G.n && (int)blockIdx.x >= G.cta0[p + 1]) p++;
  const int i0 = G.bi[p] * GT_BLK, j0 = G.bj[p] * GT_BLK;
  const bool diag = SYRK && i0 == j0;
  const int nCta = G.cta0[p + 1] - G.cta0[p], c = blockIdx.x - G.cta0[p];
  const int nSt = (rows + GT_KT - 1) / GT_KT;
  const int s0 = (int)((int64_t)nSt * c / nCta), s1 = (int)((int64_t)nSt * (c + 1) / nCta);
  // The block's tiles are dealt to the warps in turn, so that they spread over the SM's four schedulers (by position in
  // the block, the triangle's tiles fell 1 : 2 : 3 : 4 on them and cost as much as a whole block); with eight tiles or
  // fewer two warps share a tile, one for each eight rows of a stage. Tiles on the diagonal do without the products of
  // their lower left quarter and go to warps 0, 1, 4, 5: a triangle's ten tiles load the schedulers 2.5 : 2.5 : 2 : 2.
  const int ti = (min(GT_BLK, aCols - i0) + 31) / 32, tj = (min(GT_BLK, bCols - j0) + 31) / 32;
  const int nT = diag ? ti * (ti + 1) / 2 : ti * tj, split = nT <= GT_WARPS / 2 ? 2 : 1;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(gts);
  const uint32_t full = base + (uint32_t)(GT_STAGES * GT_STAGE * 8), empty = full + GT_STAGES * 8;
  if (tid == 0) {
    for (int i = 0; i < GT_STAGES; i++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + 8 * i));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty + 8 * i), "r"(nT * split));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  // The copies of a stage, 16 rows of A and of B, by four warps of their own that run ahead (a warp takes about as long
  // for 32 copies as for a tile's products). Registers: 640 threads start with 96; 128 x 24 + 512 x 112 of them remain.
  if (warp >= GT_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
    const int row = (warp - GT_WARPS) * (GT_KT / GT_COPY) + (lane & 3);
    const bool isB = lane >= GT_KT / GT_COPY;
    const uint32_t wA = (uint32_t)min(GT_BLK, lda - i0) * 8u, wB = diag ? 0u : (uint32_t)min(GT_BLK, ldb - j0) * 8u;
    const uint32_t bytes = lane >= 2 * (GT_KT / GT_COPY) ? 0u : isB ? wB : wA;
    const size_t ld = isB ? ldb : lda;
    const double* src = (isB ? B + j0 : A + i0) + ((size_t)s0 * GT_KT + row) * ld;
    const uint32_t dst = base + (uint32_t)(row + (isB ? GT_KT : 0)) * GT_LD * 8u;
    for (int k = 0; k < s1 - s0; k++, src += GT_KT * ld) {
      const int b = k % GT_STAGES;
      if (k >= GT_STAGES && !gt_wait(empty + 8 * b, (uint32_t)(k / GT_STAGES - 1) & 1u)) {
        if (lane == 0) atomicExch(err, 111);
        return;
      }
      if (warp == GT_WARPS && lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + 8 * b), "r"((wA + wB) * GT_KT) : "memory");
      if (bytes)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         dst + (uint32_t)(b * GT_STAGE) * 8u),
                     "l"(src), "r"(bytes), "r"(full + 8 * b)
                     : "memory");
    }
    return;
  }
  asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
  if (warp >= nT * split) return;
  const int tile = warp % nT;
  const int kBeg = split == 2 ? warp / nT * 8 : 0, kEnd = split == 2 ? kBeg + 8 : GT_KT;
  int wi, wj;
  if (!diag)
    wi = tile / tj, wj = tile - wi * tj;
  else if (tile < 8 && !(tile & 2) && (tile & 1) + (tile >> 2) * 2 < ti)
    wi = wj = (tile & 1) + (tile >> 2) * 2;
  else {
    int rest = tile - min(ti, min(tile, 2) + max(0, min(tile - 4, 2)));  // of the tiles above the diagonal
    for (wi = 0; rest >= ti - 1 - wi; wi++) rest -= ti - 1 - wi;
    wj = wi + 1 + rest;
  }
  double acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int u = 0; u < 4; u++) acc[i][j][u] = 0.0;
  auto run = [&](auto onDiagonal) {  // (a product skipped by a predicate would still take its turn in the tensor pipe)
    constexpr int J1 = decltype(onDiagonal)::value ? 2 : 0;
    for (int st = s0; st < s1; st++) {
      const int n = st - s0, b = n % GT_STAGES;
      if (!gt_wait(full + 8 * b, (uint32_t)(n / GT_STAGES) & 1u)) {
        if (lane == 0) atomicExch(err, 112);
        return false;
      }
      const double* sA = gts + (size_t)b * GT_STAGE + wi * 32 + g;
      const double* sB = gts + (size_t)b * GT_STAGE + (diag ? 0 : GT_KT * GT_LD) + wj * 32 + g;
#pragma unroll 1
      for (int k = kBeg; k < kEnd; k += 8) {
        double a[2][4], bb[4][2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const double* x = sA + (k + t) * GT_LD + i * 16;
          a[i][0] = x[0];
          a[i][1] = x[8];
          a[i][2] = x[4 * GT_LD];
          a[i][3] = x[4 * GT_LD + 8];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
          bb[j][0] = sB[(k + t) * GT_LD + j * 8];
          bb[j][1] = sB[(k + 4 + t) * GT_LD + j * 8];
        }
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int j = i * J1; j < 4; j++) dmma1688(acc[i][j], a[i][0], a[i][1], a[i][2], a[i][3], bb[j][0], bb[j][1]);
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + 8 * b) : "memory");
    }
    return true;
  };
  if (!((SYRK && diag && wi == wj) ? run(std::true_type{}) : run(std::false_type{}))) return;
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int gi = i0 + wi * 32 + i * 16 + g + 8 * (u >> 1), gj = j0 + wj * 32 + j * 8 + 2 * t + (u & 1);
        if (gi < aCols && gj < bCols && (!SYRK || gi <= gj) && acc[i][j][u] != 0.0) atomicAdd(&C[(size_t)gi * bCols + gj], acc[i][j][u]);
      }
}

template <bool SYRK>
static int64_t launch_gemm_tn(Matrix* m, const double* A, int aCols, int lda, const double* B, int bCols, int ldb, int rows, double* C,
                              cudaStream_t s) {
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, GT_SMEM, k_gemm_tn<SYRK>); e < 0) return e;
  const int nA = (aCols + GT_BLK - 1) / GT_BLK, nB = (bCols + GT_BLK - 1) / GT_BLK, nSt = (rows + GT_KT - 1) / GT_KT;
  auto tiles = [](int cols, int b) { return (std::min(GT_BLK, cols - b * GT_BLK) + 31) / 32; };
  int bi = 0, bj = 0;
  while (bi < nA) {  // up to GT_PAIRS blocks per launch
    GemmBlocks G;
    G.n = 0;
    double w[GT_PAIRS], sum = 0.0;
    while (bi < nA && G.n < GT_PAIRS) {
      G.bi[G.n] = (int16_t)bi;
      G.bj[G.n] = (int16_t)bj;
      const int ti = tiles(aCols, bi), tj = tiles(bCols, bj);
      const int nT = (SYRK && bi == bj) ? ti * (ti + 1) / 2 : ti * tj;
      // Tiles of the busiest scheduler, at least one: a stage of a narrow block takes its latency (100,001 rows x 129
      // columns: 225 us without that floor, 188 with half a tile, 175 with one).
      constexpr double DIAG[5] = {0.0, 1.0, 1.0, 1.375, 2.5};
      sum += w[G.n++] = (SYRK && bi == bj) ? DIAG[ti] : nT <= 8 ? std::max(1.0, (nT + 1) / 2 * 0.5) : (nT + 3) / 4;
      if (++bj == nB) {
        bi++;
        bj = SYRK ? bi : 0;
      }
    }
    int at = 0;
    double cum = 0.0;
    for (int p = 0; p < G.n; p++) {
      G.cta0[p] = at;
      cum += w[p];
      const int want = std::max(at + 1, (int)(cum / sum * m->smCount + 0.5));
      at += std::max(1, std::min(want - at, (nSt + 1) / 2));  // at least two stages each
    }
    G.cta0[G.n] = at;
    k_gemm_tn<SYRK><<<at, GT_T, GT_SMEM, s>>>(A, aCols, lda, B, bCols, ldb, rows, C, G, m->dErr);
    m->stats.kernel_launches++;
  }
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

// Rows [r0, r1) decompressed into X as k_gemm_tn wants them: ld even, zeros up to a whole stage.
static int64_t decompress_chunk(Matrix* m, int r0, int r1, double* X, int ld, cudaStream_t s) {
  const int rows = r1 - r0, pad = (rows + GT_KT - 1) / GT_KT * GT_KT - rows;
  if (pad) CLA_CUDA(cudaMemsetAsync(X + (size_t)rows * ld, 0, (size_t)pad * ld * sizeof(double), s));
  return launch_decompress_range(m, r0, r1, X, s, (size_t)ld);
}

// Rows of a decompressed chunk, about 192 MB in even parts: enough that the partial sums every CTA adds to the result at its
// end do not count (200,000 x 250 mixed: 616 us with 192 MB and a third chunk for the last 3,392 rows, 600 with 512 MB),
// little enough that the first call's allocation does not (512 MB: 0.9 ms more there).
static int64_t chunk_rows(int64_t nRows, int64_t cols) {
  const int64_t parts = std::max<int64_t>(1, (nRows * cols * 8 + (96ll << 20)) / (192ll << 20));
  return std::max<int64_t>(SKIP_ROWS, ((nRows + parts - 1) / parts + SKIP_ROWS - 1) / SKIP_ROWS * SKIP_ROWS);
}

// --------------------------------------------------------------------------------------------------
// Up to 128 columns: one CTA holds the whole upper triangle of the result as 16x8 DMMA tiles, so nothing of the
// product is computed twice and only the triangle's tiles are computed at all. Rows are split across CTAs; each
// adds its partial triangle to the result with atomics at the end.
// FUSED: the 32-row stage is decoded straight from the maps and dictionaries (dense-map and uncompressed groups
// only), so the dense form of X never exists, not even in L2. Otherwise the stage is read from a decompressed chunk.
// --------------------------------------------------------------------------------------------------
constexpr int TT_KT = 32;             // rows per stage

// What the staging loop needs to know about one matrix column, kept in shared memory.
struct TsmmCol {
  const void* map;     // null: no dense-map / uncompressed group holds the column
  const void* mapHi;
  const double* src;   // dictionary (or the dense block) already offset to the column inside the group
  double cst;          // constant part of the column
  int32_t mapType;     // -1: uncompressed (src is the dense block + j)
  int32_t gCols;
};

// --------------------------------------------------------------------------------------------------
// 16 warps in one CTA per SM. The triangle's tiles are dealt to the warps as contiguous runs of the row-major tile
// order (TPW tiles each, so a warp's A fragment changes at most a few times), which keeps the accumulators at
// 2 * TPW registers per thread and leaves room for a two-deep register pipeline of the decode: while the DMMAs of stage s run, the dictionary gathers of stage s+2 and the map loads
// of stage s+3 are in flight; their values go to one of four shared-memory stage buffers an iteration later.
// (An earlier 8-warp version, whose decode had to finish, values in shared memory, before its DMMAs started,
// stalled 7.6 cycles per issue on those gathers; this one 0.5.)
// --------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

constexpr int T16_WARPS = 16;
constexpr int T16_THREADS = T16_WARPS * 32;
constexpr int T16_MAXC = 8;   // columns decoded per warp and stage at 128 columns

// SIMPLE (with MT = byte or char): every column is held by a dense-map group of that width, so a column needs two
// pointers (map, dictionary) instead of the full record, whose reads were 40 % of the kernel's shared-memory load
// instructions. SIMPLE = 1: single-column groups and no constant part; SIMPLE = 2: also the group width (co-coded
// columns) and the constant part of the column.
// The MMAs of one 32-row stage on 16 x 8 tiles for a warp that owns N of its TPW tile slots. N is a template
// parameter, not a predicate on each MMA: a predicated-off MMA still takes its turn in the tensor pipe.
// The fragments of k-step ks + 8 are loaded before the MMAs of k-step ks are issued.
template <int N, int TPW, int LD>
__device__ __forceinline__ void tsmm_stage_1688(const double* __restrict__ Xt, const int (&offA)[TPW], const int (&offB)[TPW],
                                                uint32_t aMask, double (&c)[TPW][4]) {
  double2 bC[N], aC0 = *(const double2*)&Xt[offA[0]], aC1 = *(const double2*)&Xt[offA[0] + 8 * LD];
#pragma unroll
  for (int sl = 0; sl < N; sl++) bC[sl] = *(const double2*)&Xt[offB[sl]];
#pragma unroll
  for (int ks = 0; ks < 32; ks += 8) {
    double2 bN[N], aN0 = make_double2(0.0, 0.0), aN1 = make_double2(0.0, 0.0);
    if (ks + 8 < 32) {
      aN0 = *(const double2*)&Xt[offA[0] + ks + 8];
      aN1 = *(const double2*)&Xt[offA[0] + 8 * LD + ks + 8];
#pragma unroll
      for (int sl = 0; sl < N; sl++) bN[sl] = *(const double2*)&Xt[offB[sl] + ks + 8];
    }
    double2 a0 = aC0, a1 = aC1;
#pragma unroll
    for (int sl = 0; sl < N; sl++) {
      if (sl > 0 && ((aMask >> sl) & 1u)) {
        a0 = *(const double2*)&Xt[offA[sl] + ks];
        a1 = *(const double2*)&Xt[offA[sl] + 8 * LD + ks];
      }
      dmma1688(c[sl], a0.x, a1.x, a0.y, a1.y, bC[sl].x, bC[sl].y);
    }
    if (ks + 8 < 32) {
      aC0 = aN0;
      aC1 = aN1;
#pragma unroll
      for (int sl = 0; sl < N; sl++) bC[sl] = bN[sl];
    }
  }
}

// The triangle is cut into 16 x 8 tiles for m16n8k8 (8 x 8 tiles on m8n8k4 needed twice the B-fragment bytes per
// flop and four times the instructions; measured 10.6 -> 10.3 ms on 20M x 100). The stage keeps its rows (the k dimension) in the
// order 0, 4, 1, 5, 2, 6, 3, 7 within every group of eight, so that the two k values a lane needs of an A or B
// fragment are adjacent: one 128-bit load per fragment half; its stride TT_LDB = 8 mod 16 makes those loads
// conflict free (a quarter-warp reads 64 contiguous bytes of two columns).
constexpr int TT_LDB = TT_KT + 8;
template <bool FUSED, int MT, int TPW, int SIMPLE>
__global__ void __launch_bounds__(T16_THREADS, 1)
k_tsmm_tri16(const DevGroup* __restrict__ groups, const int32_t* __restrict__ colSrc, const double* __restrict__ constV,
             const double* __restrict__ X, int rowBegin, int rowEnd, int nCols, double* __restrict__ C, int32_t* err) {
  extern __shared__ __align__(16) double XtAll[];  // four stages of [nColsPad][TT_LDB], the column records, four mbarriers
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int LD = TT_LDB;
  constexpr int CW = 4;                             // accumulator doubles per tile slot
  const int NT = (nCols + 7) >> 3;                  // 8-column tiles
  const int NI = (nCols + 15) >> 4;                 // tile rows (16 matrix columns each)
  const int nColsPad = NI * 16;                     // columns of the stage (zero beyond nCols)
  const int stageDoubles = nColsPad * LD;
  TsmmCol* cols = (TsmmCol*)(XtAll + 4 * stageDoubles);
  uint64_t* bars = (uint64_t*)(cols + nColsPad);
  if (tid == 0) {
    for (int b = 0; b < 4; b++) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&bars[b])), "r"(T16_THREADS));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (FUSED) {
    for (int cc = tid; cc < nColsPad; cc += T16_THREADS) {
      TsmmCol d;
      d.map = nullptr;
      d.mapHi = nullptr;
      d.src = nullptr;
      d.cst = (constV && cc < nCols) ? constV[cc] : 0.0;
      d.mapType = 0;
      d.gCols = 1;
      if (cc < nCols && colSrc[2 * cc] >= 0) {
        const DevGroup& g = groups[colSrc[2 * cc]];
        const int j = colSrc[2 * cc + 1];
        d.gCols = g.gCols;
        if (g.type == GT_UNC) {
          d.mapType = -1;
          d.src = g.dense + j;
          d.map = g.dense;  // non-null marker
        } else {
          d.mapType = g.mapType;
          d.map = g.mapType == CLA_MAP_ZERO ? (const void*)g.dict : g.map;
          d.mapHi = g.mapHi;
          d.src = g.dict + j;
        }
      }
      cols[cc] = d;
    }
    __syncthreads();
  }
  // SIMPLE: the two pointers per column, packed behind the mbarriers
  const void** mapArr = (const void**)(bars + 4);
  const double** srcArr = (const double**)(mapArr + nColsPad);
  double* cstArr = (double*)(srcArr + nColsPad);
  int* gcArr = (int*)(cstArr + nColsPad);
  if (SIMPLE) {
    for (int cc = tid; cc < nColsPad; cc += T16_THREADS) {
      mapArr[cc] = cols[cc].map;
      srcArr[cc] = cols[cc].src;
      cstArr[cc] = cols[cc].cst;
      gcArr[cc] = cols[cc].gCols;
    }
    __syncthreads();
  }
  // this warp's tiles: [t0, t1) of the row-major order of the upper triangle
  // tile row I holds the tiles (I, J) with J >= firstJ(I): every 8-column tile that reaches the diagonal or lies above it
  auto rowLen = [&](int I) { return NT - 2 * I; };
  auto firstJ = [&](int I) { return 2 * I; };
  const int nTiles = NI * NT - NI * (NI - 1);
  const int t0 = nTiles * warp / T16_WARPS, t1 = nTiles * (warp + 1) / T16_WARPS;
  const int am = lane >> 2, ak = lane & 3;
  // Fragment offsets of each of the TPW tile slots. A slot the warp does not own points at tile (0, 0) and its
  // accumulator is never written out: the inner loop then needs no test per slot. aMask bit sl: slot sl starts
  // a new tile row, i.e. needs a fresh A fragment (bit 0 always).
  int offA[TPW], offB[TPW];
  uint32_t aMask = 1;
  {
    int I = 0, base = 0;  // base = linear index of the first tile of row I
    while (I < NI && base + rowLen(I) <= t0) {
      base += rowLen(I);
      I++;
    }
    int J = firstJ(I) + (t0 - base);
#pragma unroll
    for (int sl = 0; sl < TPW; sl++) {
      if (t0 + sl < t1) {
        offA[sl] = (I * 16 + am) * LD + 2 * ak;
        offB[sl] = (J * 8 + am) * LD + 2 * ak;
        if (J == firstJ(I)) aMask |= 1u << sl;
        if (++J == NT) {
          I++;
          J = firstJ(I);
        }
      } else {
        offA[sl] = offB[sl] = am * LD + 2 * ak;
        aMask |= 1u << sl;
      }
    }
  }
  const int nMine = t1 - t0;
  double c[TPW][CW];
#pragma unroll
  for (int i = 0; i < TPW; i++)
#pragma unroll
    for (int u = 0; u < CW; u++) c[i][u] = 0.0;

  const int64_t nStages = ((int64_t)(rowEnd - rowBegin) + TT_KT - 1) / TT_KT;
  const int64_t sa = nStages * blockIdx.x / gridDim.x, sb = nStages * (blockIdx.x + 1) / gridDim.x;
  if (sa >= sb) return;

  // ---- decode pipeline: column warp + 16 * b of the stage, lanes along the 32 rows ----
  uint32_t ids[T16_MAXC];  // dictionary ids of the stage two ahead
  double vals[T16_MAXC];   // values of the stage one ahead
  auto load_ids = [&](int64_t st) {
    if (!FUSED) return;
    const int row = rowBegin + (int)st * TT_KT + lane;
    const bool inRange = row < rowEnd;
#pragma unroll
    for (int b = 0; b < T16_MAXC; b++) {
      const int cc = warp + T16_WARPS * b;
      ids[b] = 0;
      if (SIMPLE) {
        if (cc < nCols && inRange)
          ids[b] = MT == CLA_MAP_BYTE ? ld_u8_here((const uint8_t*)mapArr[cc] + row) : ld_u16_here((const uint16_t*)mapArr[cc] + row);
      } else if (cc < nColsPad && inRange) {
        const TsmmCol& d = cols[cc];
        if (d.map && d.mapType >= 0) {
          // the raw id only: any arithmetic on it here would wait for the load
          if (MT == CLA_MAP_BYTE) ids[b] = ld_u8_here((const uint8_t*)d.map + row);
          else if (MT == CLA_MAP_CHAR) ids[b] = ld_u16_here((const uint16_t*)d.map + row);
          else ids[b] = (uint32_t)map_get(d.mapType, d.map, d.mapHi, row);
        }
      }
    }
  };
  auto gather = [&](int64_t st) {  // issues the loads of a stage's values (uses ids for dense-map columns)
    const int row = rowBegin + (int)st * TT_KT + lane;
    const bool inRange = row < rowEnd;
#pragma unroll
    for (int b = 0; b < T16_MAXC; b++) {
      const int cc = warp + T16_WARPS * b;
      vals[b] = 0.0;
      if (SIMPLE) {
        if (cc < nCols && inRange) vals[b] = ld_f64_here(srcArr[cc] + (SIMPLE == 2 ? (size_t)ids[b] * gcArr[cc] : (size_t)ids[b]));
      } else if (cc < nColsPad && inRange) {
        // volatile asm keeps the load where it is written, ahead of the (volatile) DMMAs: left to itself the
        // compiler sinks it to its use behind them and the pipeline is gone
        if (FUSED) {
          const TsmmCol& d = cols[cc];
          if (d.map) vals[b] = ld_f64_here(d.src + (d.mapType < 0 ? (size_t)row : (size_t)ids[b]) * d.gCols);
        } else if (cc < nCols)
          vals[b] = ld_f64_here(X + (size_t)(row - rowBegin) * nCols + cc);
      }
    }
  };
  auto store = [&](int64_t st, double* Xt) {  // adds the constant part of the column (rows inside the matrix only)
    const bool inRange = rowBegin + (int)st * TT_KT + lane < rowEnd;
#pragma unroll
    for (int b = 0; b < T16_MAXC; b++) {
      const int cc = warp + T16_WARPS * b;
      if (cc < nColsPad)
        Xt[cc * LD + ((lane & ~7) | ((lane & 3) << 1) | ((lane >> 2) & 1))] =
            vals[b] + ((FUSED && inRange && SIMPLE != 1) ? (SIMPLE == 2 ? cstArr[cc] : cols[cc].cst) : 0.0);
    }
  };
  // Four stage buffers, each with an mbarrier that counts the 512 threads' "my part of this stage is stored". A warp
  // stores its part of stage s + 1 and signals, issues the loads of the stages behind it, and only then waits for
  // stage s -- which every warp finished storing a whole iteration earlier -- so the warps drift up to a stage apart
  // and their DMMA phases no longer coincide (with one __syncthreads per stage they did: the tensor pipe was 47 %
  // busy yet throttling). Buffer (s + 1) % 4 was last read by the DMMAs of stage s - 3; a warp that is about to
  // store stage s + 1 has seen stage s - 1 complete, i.e. every warp had stored it, which each did after its
  // DMMAs of stage s - 3: no barrier is needed before the store.
  auto bar_addr = [&](int b) { return smem_addr(&bars[b]); };
  auto signal = [&](int b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_addr(b)) : "memory"); };
  auto wait_for = [&](int b, uint32_t parity) -> bool {  // bounded: gives up after 2^20 polls and reports it
    uint32_t done = 0;
    for (int it = 0; it < (1 << 20) && !done; it++)
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(done)
                   : "r"(bar_addr(b)), "r"(parity)
                   : "memory");
    return done != 0;
  };
  load_ids(sa);
  gather(sa);
  store(sa, XtAll);
  signal(0);
  if (sa + 1 < sb) {
    load_ids(sa + 1);
    gather(sa + 1);
  }
  if (sa + 2 < sb) load_ids(sa + 2);
  for (int64_t st = sa; st < sb; st++) {
    const int it = (int)(st - sa);
    if (st + 1 < sb) {  // vals holds stage st + 1 (gathered one iteration ago)
      store(st + 1, XtAll + ((it + 1) & 3) * stageDoubles);
      signal((it + 1) & 3);
    }
    if (st + 2 < sb) gather(st + 2);    // addresses from ids (loaded one iteration ago)
    if (st + 3 < sb) load_ids(st + 3);  // then the registers take the ids of the stage after that
    if (!wait_for(it & 3, (uint32_t)(it >> 2) & 1u)) {
      if (lane == 0) atomicExch(err, 7);  // stage never completed: give up, the host reports the self-check
      return;
    }
    const double* Xt = XtAll + (it & 3) * stageDoubles;
    // k-step outermost, tile slots innermost: consecutive DMMAs go to different accumulators, so none waits for
    // the one before it; no branch in the loop body (the A reload is a predicated load)
    // (the fragments of k-step ks + 4 are loaded into registers before the DMMAs of k-step ks are issued, so the
    // shared-memory latency is covered by the warp's own DMMAs rather than by the three other warps of its scheduler)
    {
      static_assert(TT_KT == 32, "tsmm_stage_1688 walks 32 rows");
      if (nMine == TPW) tsmm_stage_1688<TPW, TPW, LD>(Xt, offA, offB, aMask, c);
      else if (nMine == TPW - 1) tsmm_stage_1688<(TPW > 1 ? TPW - 1 : 1), TPW, LD>(Xt, offA, offB, aMask, c);
      else if (nMine == TPW - 2) tsmm_stage_1688<(TPW > 2 ? TPW - 2 : 1), TPW, LD>(Xt, offA, offB, aMask, c);
      else if (nMine > 0) tsmm_stage_1688<1, TPW, LD>(Xt, offA, offB, aMask, c);
    }
  }
  // ---- add the partial tiles ----
  {
    int I = 0, base = 0;
    while (I < NI && base + rowLen(I) <= t0) {
      base += rowLen(I);
      I++;
    }
    int J = firstJ(I) + (t0 - base);
#pragma unroll
    for (int sl = 0; sl < TPW; sl++) {
      if (t0 + sl < t1) {
#pragma unroll
        for (int u = 0; u < CW; u++) {
          const int gi = I * 16 + (lane >> 2) + 8 * (u >> 1);
          const int gj = J * 8 + (lane & 3) * 2 + (u & 1);
          if (gi < nCols && gj < nCols && gi <= gj && c[sl][u] != 0.0) atomicAdd(&C[(size_t)gi * nCols + gj], c[sl][u]);
        }
        if (++J == NT) {
          I++;
          J = firstJ(I);
        }
      }
    }
  }
}

// LibMatrixMult.copyUpperToLowerTriangle (runtime/matrix/data/LibMatrixMult.java:4769-4799)
__global__ void k_mirror(double* __restrict__ C, int n) {
  const int64_t total = (int64_t)n * n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / n), j = (int)(e - (int64_t)i * n);
    if (j < i) C[e] = C[(size_t)j * n + i];
  }
}

// --------------------------------------------------------------------------------------------------
// FP64 peak probes: the denominators for the tensor-pipe and FMA-pipe fractions quoted for the kernels above.
// --------------------------------------------------------------------------------------------------
__global__ void k_peak_dmma(int iters, double* sink) {
  double c[8][2];
#pragma unroll
  for (int i = 0; i < 8; i++) c[i][0] = c[i][1] = 0.0;
  const double a = 1.0 + threadIdx.x * 1e-9, b = 1.0 - threadIdx.x * 1e-9;
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int i = 0; i < 8; i++) dmma884(c[i][0], c[i][1], a, b);
  }
  double s = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) s += c[i][0] + c[i][1];
  if (s == 12345.678) sink[0] = s;  // keeps the loop alive
}
__global__ void k_peak_dfma(int iters, double* sink) {
  double c[16];
#pragma unroll
  for (int i = 0; i < 16; i++) c[i] = threadIdx.x * 1e-3 + i;
  const double a = 1.0000001, b = 1e-9;
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int i = 0; i < 16; i++) c[i] = fma(c[i], a, b);
  }
  double s = 0;
#pragma unroll
  for (int i = 0; i < 16; i++) s += c[i];
  if (s == 12345.678) sink[0] = s;
}

// TFLOP/s of back-to-back DMMA m8n8k4 (512 flop per warp instruction) and of FP64 FMA, on `device`.
int64_t measure_fp64_peaks(int device, double* dmmaTflops, double* dfmaTflops) {
  CLA_CUDA(cudaSetDevice(device));
  cudaDeviceProp prop;
  CLA_CUDA(cudaGetDeviceProperties(&prop, device));
  double* sink = nullptr;
  CLA_CUDA(cudaMalloc(&sink, 8));
  cudaEvent_t e0, e1;
  CLA_CUDA(cudaEventCreate(&e0));
  CLA_CUDA(cudaEventCreate(&e1));
  const int blocks = prop.multiProcessorCount * 4, threads = 256, iters = 20000;
  float ms = 0;
  for (int pass = 0; pass < 2; pass++) {  // first pass warms up
    CLA_CUDA(cudaEventRecord(e0));
    k_peak_dmma<<<blocks, threads>>>(iters, sink);
    CLA_CUDA(cudaEventRecord(e1));
    CLA_CUDA(cudaEventSynchronize(e1));
    CLA_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  }
  *dmmaTflops = (double)blocks * (threads / 32) * iters * 8.0 * 512.0 / (ms * 1e-3) / 1e12;
  for (int pass = 0; pass < 2; pass++) {
    CLA_CUDA(cudaEventRecord(e0));
    k_peak_dfma<<<blocks, threads>>>(iters, sink);
    CLA_CUDA(cudaEventRecord(e1));
    CLA_CUDA(cudaEventSynchronize(e1));
    CLA_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  }
  *dfmaTflops = (double)blocks * threads * iters * 16.0 * 2.0 / (ms * 1e-3) / 1e12;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(sink);
  return CLA_OK;
}

// The 16-warp kernel is instantiated for the map widths the decode specialises on and for 2, 4 and 5 slots of 16 x 8 tiles
// per warp (up to 80, 120 and 128 columns), decoded on the fly or read from a decompressed chunk.
template <int TPW>
static void tri16_go(bool fused, int mt, int simple, int grid, size_t smem, cudaStream_t s, const DevGroup* groups,
                     const int32_t* colSrc, const double* constV, const double* X, int rows, int n, double* dOut, int32_t* err) {
#define TRI16(F, M, S) k_tsmm_tri16<F, M, TPW, S><<<grid, T16_THREADS, smem, s>>>(groups, colSrc, constV, X, 0, rows, n, dOut, err)
  if (!fused) TRI16(false, -2, 0);
  else if (mt == CLA_MAP_BYTE && simple == 1) TRI16(true, CLA_MAP_BYTE, 1);
  else if (mt == CLA_MAP_BYTE && simple == 2) TRI16(true, CLA_MAP_BYTE, 2);
  else if (mt == CLA_MAP_CHAR && simple == 1) TRI16(true, CLA_MAP_CHAR, 1);
  else if (mt == CLA_MAP_CHAR && simple == 2) TRI16(true, CLA_MAP_CHAR, 2);
  else if (mt == CLA_MAP_BYTE) TRI16(true, CLA_MAP_BYTE, 0);
  else if (mt == CLA_MAP_CHAR) TRI16(true, CLA_MAP_CHAR, 0);
  else TRI16(true, -2, 0);
#undef TRI16
}
static void launch_tri16(bool fused, int mt, int simple, int n, int grid, size_t smem, cudaStream_t s, const DevGroup* groups,
                         const int32_t* colSrc, const double* constV, const double* X, int rows, double* dOut, int32_t* err) {
  const int NT = (n + 7) / 8, NI = (n + 15) / 16, perWarp = (NI * NT - NI * (NI - 1) + T16_WARPS - 1) / T16_WARPS;
  if (perWarp <= 2) tri16_go<2>(fused, mt, simple, grid, smem, s, groups, colSrc, constV, X, rows, n, dOut, err);
  else if (perWarp <= 4) tri16_go<4>(fused, mt, simple, grid, smem, s, groups, colSrc, constV, X, rows, n, dOut, err);
  else tri16_go<5>(fused, mt, simple, grid, smem, s, groups, colSrc, constV, X, rows, n, dOut, err);
}
template <int TPW>
static int64_t tri16_set_smem_t(int bytes) {
#define TRI16_ATTR(F, M, S) \
  CLA_CUDA(cudaFuncSetAttribute(k_tsmm_tri16<F, M, TPW, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes))
  TRI16_ATTR(true, -2, 0);
  TRI16_ATTR(true, CLA_MAP_BYTE, 0);
  TRI16_ATTR(true, CLA_MAP_CHAR, 0);
  TRI16_ATTR(true, CLA_MAP_BYTE, 1);
  TRI16_ATTR(true, CLA_MAP_CHAR, 1);
  TRI16_ATTR(true, CLA_MAP_BYTE, 2);
  TRI16_ATTR(true, CLA_MAP_CHAR, 2);
  TRI16_ATTR(false, -2, 0);
#undef TRI16_ATTR
  return CLA_OK;
}
static int64_t tri16_set_smem(int bytes) {
  int64_t rc;
  if ((rc = tri16_set_smem_t<2>(bytes)) < 0) return rc;
  if ((rc = tri16_set_smem_t<4>(bytes)) < 0) return rc;
  return tri16_set_smem_t<5>(bytes);
}

int64_t launch_tsmm(Matrix* m, double* dOut, cudaStream_t s) {
  const int n = m->nCols;
  if (n == 0) return CLA_OK;
  if (m->nRows > 0 && pairs_eligible(m, m, true)) {  // few co-coded groups: on the dictionaries
    const int64_t rc = launch_pairs(m, m, true, dOut, s);
    if (rc < 0) return rc;
    // overlapping groups add to a cell from several pairs, in no fixed order: copy the upper triangle down
    k_mirror<<<std::max(1, std::min(1024, (int)(((int64_t)n * n + 255) / 256))), 256, 0, s>>>(dOut, n);
    m->stats.kernel_launches++;
    CLA_CUDA(cudaGetLastError());
    return CLA_OK;
  }
  int64_t rc;
  if ((rc = split_tsmm(m, dOut, s)) != 0) return rc < 0 ? rc : CLA_OK;
  CLA_CUDA(cudaMemsetAsync(dOut, 0, sizeof(double) * (size_t)n * n, s));
  if (m->nRows == 0) return CLA_OK;
  const bool tri = n <= 128;
  bool denseOnly = m->colSrcValid;
  for (auto& g : m->groups) denseOnly &= (g.type == GT_DDC || g.type == GT_UNC);
  const size_t tri16Smem = (size_t)((n + 15) / 16 * 16) * (4 * TT_LDB * sizeof(double) + sizeof(TsmmCol) + 28) + 4 * sizeof(uint64_t);
  static OncePerDevice once;
  if ((rc = once(m->device, [&] { return tri16_set_smem(128 * (4 * TT_LDB * 8 + (int)sizeof(TsmmCol) + 28) + 32); })) < 0) return rc;
  if (tri && denseOnly) {  // one launch over all rows, decoding as it goes
    const int64_t nStages = ((int64_t)m->nRows + TT_KT - 1) / TT_KT;
    // one map width for every column (and every column held by a dense-map group): the specialised decode
    int mt = -1;
    for (auto& g : m->groups) {
      const int w = (g.type != GT_DDC) ? -2
                    : (g.mapType == CLA_MAP_UBYTE || g.mapType == CLA_MAP_BYTE) ? CLA_MAP_BYTE
                    : (g.mapType == CLA_MAP_CHAR ? CLA_MAP_CHAR : -2);
      mt = (mt == -1 || mt == w) ? w : -2;
    }
    // the compact records: every column in exactly one dense-map group of that width (1: single-column groups
    // and no constant part; 2: any group width, constants allowed)
    int simple = 0;
    if (mt == CLA_MAP_BYTE || mt == CLA_MAP_CHAR) {
      int covered = 0;
      bool single = true;
      for (auto& g : m->groups) {
        covered += g.gCols;
        single &= g.gCols == 1;
      }
      if (covered == n) simple = (single && !m->hasConst) ? 1 : 2;  // colSrcValid: no column is counted twice
    }
    prof_begin(m, s);
    launch_tri16(true, mt, simple, n, (int)std::min<int64_t>(m->smCount, nStages), tri16Smem, s, m->dGroups, m->dColSrc,
                 m->hasConst ? m->dConstV : nullptr, nullptr, m->nRows, dOut, m->dErr);
    prof_end(m, s);
    m->stats.kernel_launches++;
  } else {
    const int64_t chunk = chunk_rows(m->nRows, n);
    const int ld = tri ? n : (n + 1) & ~1;
    if ((rc = ensure_scratch2(m, (size_t)chunk * ld * sizeof(double))) < 0) return rc;
    double* X = (double*)m->scratch2;
    for (int64_t r0 = 0; r0 < m->nRows; r0 += chunk) {
      const int r1 = (int)std::min<int64_t>(m->nRows, r0 + chunk);
      const int rows = r1 - (int)r0;
      if ((rc = tri ? launch_decompress_range(m, (int)r0, r1, X, s) : decompress_chunk(m, (int)r0, r1, X, ld, s)) < 0) return rc;
      if (tri) {
        const int64_t nStages = ((int64_t)rows + TT_KT - 1) / TT_KT;
        launch_tri16(false, -2, 0, n, (int)std::min<int64_t>(m->smCount, nStages), tri16Smem, s, nullptr, nullptr, nullptr,
                     X, rows, dOut, m->dErr);
        m->stats.kernel_launches++;
      } else if ((rc = launch_gemm_tn<true>(m, X, n, ld, X, n, ld, rows, dOut, s)) < 0)
        return rc;
    }
  }
  k_mirror<<<std::max(1, std::min(1024, (int)(((int64_t)n * n + 255) / 256))), 256, 0, s>>>(dOut, n);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

// t(L) %*% R for two compressed matrices over the same rows (CLALibLeftMultBy.leftMultByMatrixTransposed on two
// compressed blocks, lib/CLALibLeftMultBy.java:100-112,170-284). Both sides are decompressed one L2-sized row
// chunk at a time (constants included, so no rank-1 corrections are needed) and the chunks are multiplied on
// the FP64 tensor cores; the dense forms never reach HBM-sized buffers.
int64_t launch_tmm(Matrix* L, Matrix* R, double* dOut, cudaStream_t s) {
  const int a = L->nCols, b = R->nCols;
  if ((int64_t)a * b == 0) return CLA_OK;
  if (L->nRows > 0 && pairs_eligible(L, R, false)) return launch_pairs(L, R, false, dOut, s);  // pair pre-aggregation
  CLA_CUDA(cudaMemsetAsync(dOut, 0, sizeof(double) * (size_t)a * b, s));
  if (L->nRows == 0) return CLA_OK;
  int64_t rc;
  const int64_t chunk = chunk_rows(L->nRows, a + b);
  const int la = (a + 1) & ~1, lb = (b + 1) & ~1;
  if ((rc = ensure_scratch2(L, (size_t)chunk * la * sizeof(double))) < 0) return rc;
  if ((rc = ensure_scratch2(R, (size_t)chunk * lb * sizeof(double))) < 0) return rc;
  double* XL = (double*)L->scratch2;
  double* XR = (double*)R->scratch2;
  for (int64_t r0 = 0; r0 < L->nRows; r0 += chunk) {
    const int r1 = (int)std::min<int64_t>(L->nRows, r0 + chunk);
    if ((rc = decompress_chunk(L, (int)r0, r1, XL, la, s)) < 0) return rc;
    if ((rc = decompress_chunk(R, (int)r0, r1, XR, lb, s)) < 0) return rc;
    const int rows = r1 - (int)r0;
    if (r0 == 0) prof_begin(L, s);
    if ((rc = launch_gemm_tn<false>(L, XL, a, la, XR, b, lb, rows, dOut, s)) < 0) return rc;
    if (r0 == 0) prof_end(L, s);
  }
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

}  // namespace cla
