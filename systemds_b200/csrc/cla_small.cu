// Products on short blocks (fewer than SMALL_ROWS rows: the blocks of a blocked matrix, mini-batches, the tail shard
// of a row-partitioned matrix). Such a product touches a few hundred kilobytes, so its time is launches, dependent
// memory round trips and idle SMs; one kernel per product, no tables prepared beforehand, every group type.
//
//  * k_small_rmm: X %*% V. A CTA owns 32 rows (lane = row) and up to KT result columns; its warps share the
//    groups and their partial sums are added in a fixed order. Cells are dictionary value x V directly: with a few
//    dozen rows per CTA a table D * V would cost more to build than it saves.
//  * k_small_lmm: Yt %*% X. Four warps own one matrix column (and QT left rows) over all rows and write the result
//    cell; nothing is accumulated across CTAs, so there is nothing to clear, no atomics and one fixed order.
//
// Measured on 1000 rows x 100 byte-map columns, host arrays in and out: X %*% v 199 us before (a dictionary kernel, one
// CTA of the general row kernel, a count kernel, five pageable copies, three synchronisations).
#include "cla_common.cuh"
#include <algorithm>
#include <cstring>

namespace cla {

constexpr int SMALL_ROWS = 4096;
constexpr int SR_T = 256;
// Warps of a k_small_rmm CTA: what a warp waits for is a chain of three dependent reads (column record, id, value) per
// batch of four columns, so for one result column 32 warps share the columns (measured with 8: four batches per warp);
// with several result columns the partial sums would not fit.
template <int KT> struct SmallRmm { static constexpr int WARPS = KT == 1 ? 32 : 16; };
constexpr int SR_VMAX = 6144;  // doubles of V kept in shared memory

// The end of a small host-buffer call: every CTA has stored its part of the result (to pinned host memory); the last
// one to arrive publishes the non-zero count and raises the flag the host polls. Called by all threads of the CTA.
__device__ __forceinline__ void finish_cta(const Finish& fin, unsigned nonZeros) {
  if (!fin.box) return;
  __shared__ unsigned cnt;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  for (int d = 16; d; d >>= 1) nonZeros += __shfl_down_sync(0xffffffffu, nonZeros, d);
  if ((threadIdx.x & 31) == 0 && nonZeros) atomicAdd(&cnt, nonZeros);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    const unsigned long long mine = cnt;
    if (mine) atomicAdd(fin.nnz, mine);
    __threadfence();
    const unsigned total = gridDim.x * gridDim.y;
    if (atomicAdd(fin.ticket, 1u) + 1 == total) {
      __threadfence();
      const unsigned long long nnz = atomicExch(fin.nnz, 0ull);
      const unsigned err = (unsigned)atomicExch(fin.err, 0);
      *fin.ticket = 0;
      asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(fin.box), "r"(fin.seq), "r"(err), "r"((unsigned)nnz),
                   "r"((unsigned)(nnz >> 32))
                   : "memory");
    }
  }
}

// V handed over by value in the launch itself (host-buffer calls with a short right operand): the kernel would
// otherwise wait for a read across the bus, or for a copy, before its first multiplication.
template <int N> struct VArg { double v[N]; };
template <> struct VArg<0> {};

template <int KT, int NV>
__global__ void __launch_bounds__(SmallRmm<KT>::WARPS * 32)
k_small_rmm(const ColRef* __restrict__ dense, int nDense, const DevGroup* __restrict__ groups, const SparseVal* __restrict__ sv,
            const int32_t* __restrict__ svOff, const uint32_t* __restrict__ rowPtr, const uint32_t* __restrict__ rowItems,
            const uint32_t* __restrict__ fullPtr, const uint32_t* __restrict__ fullItems, const uint32_t* __restrict__ partPtr,
            const uint2* __restrict__ partItems, int nRows, const double* __restrict__ V, int nCols, int vCols,
            const double* __restrict__ constV, const double* __restrict__ rowScale, double* __restrict__ out, int vShared,
            const Finish fin, const __grid_constant__ VArg<NV> varg) {
  constexpr int WARPS = SmallRmm<KT>::WARPS, THREADS = WARPS * 32;
  extern __shared__ __align__(16) double srsm[];  // [WARPS][KT][33] partial sums, then V [nCols][KT]
  double* part = srsm;
  double* Vs = srsm + WARPS * KT * 33;
  __shared__ double cpart[WARPS][KT];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j0 = blockIdx.y * KT, kc = min(KT, vCols - j0);
  const int r0 = blockIdx.x * 32, r = min(r0 + lane, nRows - 1);
  if (vShared) {
    for (int e = tid; e < nCols * KT; e += THREADS) {
      const int c = e / KT, j = e - c * KT;
      double x = 0.0;
      if constexpr (NV > 0) { if (j < kc) x = varg.v[c * vCols + j0 + j]; }
      else { if (j < kc) x = V[(size_t)c * vCols + j0 + j]; }
      Vs[e] = x;
    }
    __syncthreads();
  }
  auto vat = [&](int c, int j) -> double {
    if (vShared) return Vs[c * KT + j];
    return j < kc ? V[(size_t)c * vCols + j0 + j] : 0.0;
  };
  double acc[KT];
#pragma unroll
  for (int j = 0; j < KT; j++) acc[j] = 0.0;
  // dense-map and uncompressed columns, four in flight
  for (int d0 = warp; d0 < nDense; d0 += 4 * WARPS) {
    double x[4];
    int col[4];
    int64_t at[4];
    const double* src[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int d = d0 + u * WARPS;
      at[u] = 0;
      col[u] = -1;
      if (d < nDense) {
        const ColRef c = dense[d];
        col[u] = c.col;
        src[u] = c.src;
        const int64_t id = c.kind == GT_UNC ? r : map_get(c.mapType, c.map, c.mapHi, r);
        at[u] = id * c.stride;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) x[u] = col[u] >= 0 ? src[u][at[u]] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (col[u] >= 0)
#pragma unroll
        for (int j = 0; j < KT; j++) acc[j] = fma(x[u], vat(col[u], j), acc[j]);
  }
  // a listed tuple (or run) of table row p
  auto add_sparse = [&](uint32_t p) {
    const SparseVal s = sv[p];
    if (s.col >= 0) {
#pragma unroll
      for (int j = 0; j < KT; j++) acc[j] = fma(s.val, vat(s.col, j), acc[j]);
    } else {
      const DevGroup& g = groups[s.group];
      const double* d = g.dict + (size_t)(p - (uint32_t)svOff[s.group]) * g.gCols;
      for (int h = 0; h < g.gCols; h++) {
        const double x = d[h];
        const int c = g.cols[h];
#pragma unroll
        for (int j = 0; j < KT; j++) acc[j] = fma(x, vat(c, j), acc[j]);
      }
    }
  };
  if (rowPtr) {
    const uint32_t p0 = rowPtr[r], p1 = rowPtr[r + 1];
    for (uint32_t p = p0 + warp; p < p1; p += WARPS) add_sparse(rowItems[p]);
  }
  if (fullPtr) {
    const int w = r0 / WIN_ROWS, rw = r - w * WIN_ROWS;  // 32 rows lie inside one window
    for (uint32_t p = fullPtr[w] + warp; p < fullPtr[w + 1]; p += WARPS) add_sparse(fullItems[p]);
    for (uint32_t p = partPtr[w] + warp; p < partPtr[w + 1]; p += WARPS) {
      const uint2 it = partItems[p];
      if (rw >= (int)(it.y & 0xFF) && rw < (int)(it.y >> 8)) add_sparse(it.x);
    }
  }
  double c0[KT];
#pragma unroll
  for (int j = 0; j < KT; j++) c0[j] = 0.0;
  if (constV) {
    for (int c = tid; c < nCols; c += THREADS) {
      const double x = constV[c];
      if (x != 0.0)
#pragma unroll
        for (int j = 0; j < KT; j++) c0[j] = fma(x, vat(c, j), c0[j]);
    }
#pragma unroll
    for (int j = 0; j < KT; j++) {
      for (int d = 16; d; d >>= 1) c0[j] += __shfl_xor_sync(0xffffffffu, c0[j], d);
      if (lane == 0) cpart[warp][j] = c0[j];
    }
  }
#pragma unroll
  for (int j = 0; j < KT; j++) part[(warp * KT + j) * 33 + lane] = acc[j];
  __syncthreads();
  unsigned nz = 0;
  for (int e = warp; e < 32 * KT; e += WARPS) {  // a warp per output cell, lanes over the partial sums
    const int rr = e / KT, j = e - rr * KT;
    double s = lane < WARPS ? part[(lane * KT + j) * 33 + rr] : 0.0;
    if (constV && lane < WARPS) s += cpart[lane][j];
    for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (lane == 0 && r0 + rr < nRows && j < kc) {
      if (rowScale) s *= rowScale[r0 + rr];
      out[(size_t)(r0 + rr) * vCols + j0 + j] = s;
      nz += s != 0.0;
    }
  }
  finish_cta(fin, nz);
}

constexpr int SL_WARPS = SR_T / 32, SL_WPC = 4;  // warps per CTA, per column
template <int QT>
__global__ void __launch_bounds__(SR_T)
k_small_lmm(const ColRef* __restrict__ refs, const int32_t* __restrict__ refPtr, const DevGroup* __restrict__ groups, int nRows,
            int nCols, const double* __restrict__ Yt, int q, const double* __restrict__ constV, double* __restrict__ out,
            const Finish fin) {
  __shared__ double part[SL_WARPS][QT], ysum[SL_WARPS][QT];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = blockIdx.x * (SL_WARPS / SL_WPC) + warp / SL_WPC, wq = warp % SL_WPC;
  const int q0 = blockIdx.y * QT, qc = min(QT, q - q0);
  const double* y[QT];
#pragma unroll
  for (int i = 0; i < QT; i++) y[i] = Yt + (size_t)(q0 + min(i, qc - 1)) * nRows;
  double acc[QT];
#pragma unroll
  for (int i = 0; i < QT; i++) acc[i] = 0.0;
  if (c < nCols)
    for (int k = refPtr[c]; k < refPtr[c + 1]; k++) {
      const ColRef cr = refs[k];
      if (cr.kind == GT_DDC || cr.kind == GT_UNC) {
        const bool bytes = cr.mapType == CLA_MAP_UBYTE || cr.mapType == CLA_MAP_BYTE;
        for (int r = (wq * 32 + lane) * 4; r < nRows; r += SL_WPC * 128) {  // four consecutive rows per lane
          double x[4];
          int64_t at[4];
          if (cr.kind == GT_DDC && bytes && r + 4 <= nRows) {
            const uint32_t w = *(const uint32_t*)((const uint8_t*)cr.map + r);
#pragma unroll
            for (int u = 0; u < 4; u++) at[u] = (w >> (8 * u)) & 0xFF;
          } else {
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const int rr = min(r + u, nRows - 1);
              at[u] = cr.kind == GT_UNC ? rr : map_get(cr.mapType, cr.map, cr.mapHi, rr);
            }
          }
#pragma unroll
          for (int u = 0; u < 4; u++) x[u] = r + u < nRows ? cr.src[at[u] * cr.stride] : 0.0;
#pragma unroll
          for (int u = 0; u < 4; u++)
#pragma unroll
            for (int i = 0; i < QT; i++) acc[i] = fma(x[u], y[i][min(r + u, nRows - 1)], acc[i]);
        }
      } else if (cr.kind == GT_SDC) {
        const DevGroup& g = groups[cr.group];
        for (int b = wq * SKIP_ROWS; b < nRows; b += SL_WPC * SKIP_ROWS)
          sdc_walk_block(g, b, min(nRows, b + SKIP_ROWS), [&](int row, int e) {
            const double x = cr.src[(size_t)(g.single ? 0 : map_get(cr.mapType, cr.map, cr.mapHi, e)) * cr.stride];
#pragma unroll
            for (int i = 0; i < QT; i++) acc[i] = fma(x, y[i][row], acc[i]);
          });
        __syncwarp();
      } else {  // RLE: the left values of a run are summed, then multiplied once per lane
        const DevGroup& g = groups[cr.group];
        for (int64_t ri = wq; ri < g.nRuns; ri += SL_WPC) {
          const RleRun run = g.runs[ri];
          const double x = cr.src[(size_t)run.k * cr.stride];
          double s[QT];
#pragma unroll
          for (int i = 0; i < QT; i++) s[i] = 0.0;
          for (int r = run.start + lane; r < run.start + (int)run.len; r += 32)
#pragma unroll
            for (int i = 0; i < QT; i++) s[i] += y[i][r];
#pragma unroll
          for (int i = 0; i < QT; i++) acc[i] = fma(x, s[i], acc[i]);
        }
      }
    }
  double ys[QT];
#pragma unroll
  for (int i = 0; i < QT; i++) ys[i] = 0.0;
  if (constV && c < nCols && constV[c] != 0.0)
    for (int r = wq * 32 + lane; r < nRows; r += SL_WPC * 32)
#pragma unroll
      for (int i = 0; i < QT; i++) ys[i] += y[i][r];
#pragma unroll
  for (int i = 0; i < QT; i++) {
    for (int d = 16; d; d >>= 1) {
      acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], d);
      if (constV) ys[i] += __shfl_xor_sync(0xffffffffu, ys[i], d);
    }
    if (lane == 0) {
      part[warp][i] = acc[i];
      ysum[warp][i] = ys[i];
    }
  }
  __syncthreads();
  unsigned nz = 0;
  if (c < nCols && wq == 0 && lane < qc) {
    double s = 0.0, t = 0.0;
#pragma unroll
    for (int w = 0; w < SL_WPC; w++) {
      s += part[warp + w][lane];
      t += ysum[warp + w][lane];
    }
    if (constV) s = fma(t, constV[c], s);
    out[(size_t)(q0 + lane) * nCols + c] = s;
    nz = s != 0.0;
  }
  finish_cta(fin, nz);
}

// Result of a small host-buffer call whose kernels left it in device memory: copied to the pinned mailbox, counted.
__global__ void __launch_bounds__(SR_T) k_finish(const double* __restrict__ d, int n, double* __restrict__ out, const Finish fin) {
  unsigned nz = 0;
  for (int i = blockIdx.x * SR_T + threadIdx.x; i < n; i += gridDim.x * SR_T) {
    const double x = d[i];
    out[i] = x;
    nz += x != 0.0;
  }
  finish_cta(fin, nz);
}
int64_t launch_finish(Matrix* m, const double* d, int n, double* out, cudaStream_t s, const Finish& fin) {
  k_finish<<<std::max(1, std::min(64, (n + 4 * SR_T - 1) / (4 * SR_T))), SR_T, 0, s>>>(d, n, out, fin);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

bool small_block(const Matrix* m) { return m->nRows > 0 && m->nRows < SMALL_ROWS && m->nCols > 0; }

// hostV: V in host memory as well (null: not); dV may then be host memory the device can read
int64_t small_rmm(Matrix* m, const double* dV, int vCols, double* dOut, const double* dW, cudaStream_t s, const Finish& fin,
                  const double* hostV) {
  if (!small_block(m) || vCols <= 0) return 0;
  int64_t rc;
  if ((rc = ensure_col_plan(m)) < 0 || (rc = ensure_row_lists(m, s)) < 0) return rc;
  const RowLists& L = m->rows;
  if (!m->cols.ok || !L.ok) return 0;
  const int KT = vCols == 1 ? 1 : (vCols <= 4 ? 4 : 8);
  const bool vShared = (int64_t)m->nCols * KT <= SR_VMAX;
  const int warps = KT == 1 ? SmallRmm<1>::WARPS : SmallRmm<8>::WARPS;
  const size_t smem = ((size_t)warps * KT * 33 + (vShared ? (size_t)m->nCols * KT : 0)) * sizeof(double);
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, (16 * 8 * 33 + SR_VMAX) * sizeof(double), k_small_rmm<1, 0>,
                                         k_small_rmm<4, 0>, k_small_rmm<8, 0>);
      e < 0)
    return e;
  const dim3 grid((m->nRows + 31) / 32, (vCols + KT - 1) / KT);
  prof_begin(m, s);
#define SMALL_RMM(K, N, ARG)                                                                                                   \
  k_small_rmm<K, N><<<grid, warps * 32, smem, s>>>(m->cols.dense, m->cols.nDense, m->dGroups, L.sv, L.svOff,                   \
                                                   L.nSdc ? L.rowPtr : nullptr, L.rowItems, L.nRle ? L.fullPtr : nullptr,      \
                                                   L.fullItems, L.partPtr, L.partItems, m->nRows, dV, m->nCols, vCols,         \
                                                   m->hasConst ? m->dConstV : nullptr, dW, dOut, vShared ? 1 : 0, fin, ARG)
  const size_t nV = (size_t)m->nCols * vCols;
  if (hostV && KT == 1 && nV <= 128) {
    VArg<128> a;
    memcpy(a.v, hostV, nV * sizeof(double));
    SMALL_RMM(1, 128, a);
  } else if (hostV && KT == 1 && nV <= 448) {
    VArg<448> a;
    memcpy(a.v, hostV, nV * sizeof(double));
    SMALL_RMM(1, 448, a);
  } else if (KT == 1)
    SMALL_RMM(1, 0, VArg<0>());
  else if (KT == 4)
    SMALL_RMM(4, 0, VArg<0>());
  else
    SMALL_RMM(8, 0, VArg<0>());
#undef SMALL_RMM
  prof_end(m, s);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  return 1;
}

int64_t small_lmm(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s, const Finish& fin) {
  if (!small_block(m) || q <= 0) return 0;
  int64_t rc;
  if ((rc = ensure_col_plan(m)) < 0) return rc;
  if (!m->cols.ok) return 0;
  const int QT = q == 1 ? 1 : 4;
  const dim3 grid((m->nCols + SL_WARPS / SL_WPC - 1) / (SL_WARPS / SL_WPC), (q + QT - 1) / QT);
  auto kern = QT == 1 ? k_small_lmm<1> : k_small_lmm<4>;
  prof_begin(m, s);
  kern<<<grid, SR_T, 0, s>>>(m->cols.refs, m->cols.refPtr, m->dGroups, m->nRows, m->nCols, dYt, q, m->hasConst ? m->dConstV : nullptr,
                             dOut, fin);
  prof_end(m, s);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  return 1;
}

}  // namespace cla
