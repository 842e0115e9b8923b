// Vector products over the groups the column-per-lane kernels do not take: SDC, RLE, uncompressed and wide dense maps.
//
//  * k_rest_rmm: X v. A warp owns 32 consecutive rows (lane = row) and needs no other warp: listed SDC tuples and RLE
//    pieces come from the row lists (cla_rows.cu) and their table P = D v in shared memory, uncompressed columns from the
//    FP64 tensor core (eight rows x four columns per product, v in one column of B: the dense block streams through with
//    no shuffle reduction), remaining dense-map columns by gathers. Nothing is staged and no barrier is passed, so the
//    dense block's loads of one warp hide the list walks of the others. Bound: the bytes of the dense block; on
//    1M x 500 mixed (400 MB dense) the kernel this replaces, a CTA per 1024 rows with its phases one after the other
//    and a thread per 8-row step on the lists, took 222 us.
//  * k_rest_lmm: Yt X for up to QT left rows. CTAs [0, nA) walk the SDC / RLE / dense-map columns over 1024-row blocks whose
//    left values are in shared memory: a warp owns a fixed set of columns, multiplies left value and dictionary value
//    directly (no histogram, no atomics) and keeps the column's sums in shared memory. CTAs [nA, ...) take 64 columns of
//    an uncompressed group each on the tensor core (A = left rows, B = the block). Before: per-tuple sums by
//    shared-memory FP64 atomics, every RLE group reading all of y; 346 + 246 us on 500k x 250 with eight left rows.
#include "cla_common.cuh"
#include <algorithm>
#include <cstring>

namespace cla {

__device__ __forceinline__ void dmma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// --------------------------------------------------------------------------------------------------
// X v
// --------------------------------------------------------------------------------------------------
constexpr int RR_WARPS = 8;
constexpr int RR_T = RR_WARPS * 32;
constexpr int RR_PMAX = 8192;  // sparse table rows kept in shared memory (64 KB)

__device__ __forceinline__ double sparse_term(const SparseVal& s, uint32_t p, const DevGroup* __restrict__ groups,
                                              const int32_t* __restrict__ svOff, const double* __restrict__ v) {
  if (s.col >= 0) return s.val * v[s.col];
  const DevGroup& g = groups[s.group];
  const double* d = g.dict + (size_t)(p - (uint32_t)svOff[s.group]) * g.gCols;
  double x = 0.0;
  for (int h = 0; h < g.gCols; h++) x += d[h] * v[g.cols[h]];
  return x;
}
__global__ void k_rest_terms(const SparseVal* __restrict__ sv, int nSv, const DevGroup* __restrict__ groups,
                             const int32_t* __restrict__ svOff, const double* __restrict__ v, double* __restrict__ P) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nSv; p += gridDim.x * blockDim.x) P[p] = sparse_term(sv[p], p, groups, svOff, v);
}

struct UncGroup {
  const double* dense;
  const int32_t* cols;
  int32_t gCols, pad;
};
constexpr int RR_UNC = 8;  // uncompressed groups per launch
struct RestRmmArgs {
  const SparseVal* sv;
  const int32_t* svOff;
  const DevGroup* groups;
  const double* P;          // null: the CTA builds the table in shared memory
  int nSv, nRows, nDense, nUnc, nCols, addTo;
  const uint32_t *rowPtr, *rowItems, *fullPtr, *fullItems, *partPtr;
  const uint2* partItems;
  const ColRef* dense;
  UncGroup unc[RR_UNC];
  const double* v;
  const double* constV;
  const double* rowScale;
  double* out;
};

__global__ void __launch_bounds__(RR_T, 4) k_rest_rmm(const __grid_constant__ RestRmmArgs A) {
  extern __shared__ __align__(16) double ps[];
  __shared__ double cred[RR_WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* P = A.P;
  if (!P && A.nSv) {
    for (int p = tid; p < A.nSv; p += RR_T) ps[p] = sparse_term(A.sv[p], p, A.groups, A.svOff, A.v);
    P = ps;
  }
  double c0 = 0.0;
  if (A.constV) {
    for (int c = tid; c < A.nCols; c += RR_T) c0 = fma(A.constV[c], A.v[c], c0);
    for (int d = 16; d; d >>= 1) c0 += __shfl_xor_sync(0xffffffffu, c0, d);
    if (lane == 0) cred[warp] = c0;
  }
  __syncthreads();
  if (A.constV) {
    c0 = 0.0;
    for (int w = 0; w < RR_WARPS; w++) c0 += cred[w];
  }
  const int g = lane >> 2, t = lane & 3;
  const int nSteps = (A.nRows + 31) / 32;
  for (int st = blockIdx.x * RR_WARPS + warp; st < nSteps; st += gridDim.x * RR_WARPS) {
    const int r0 = st * 32, r = min(r0 + lane, A.nRows - 1);
    double acc = 0.0;
    uint32_t p0 = 0, p1 = 0;
    if (A.rowPtr) {
      p0 = A.rowPtr[r];
      p1 = A.rowPtr[r + 1];
    }
    // uncompressed: rows 8 j + g of the step, columns c + t
    for (int i = 0; i < A.nUnc; i++) {
      const UncGroup& U = A.unc[i];
      const int gc = U.gCols;
#pragma unroll 1
      for (int j = 0; j < 4; j++) {
        const int row = min(r0 + 8 * j + g, A.nRows - 1);
        const double* x = U.dense + (size_t)row * gc + t;
        double s0 = 0.0, s1 = 0.0;
        int c = 0;
        for (; c + 32 <= gc; c += 32) {
          double xv[8];
#pragma unroll
          for (int u = 0; u < 8; u++) xv[u] = __ldcs(x + c + 4 * u);
#pragma unroll
          for (int u = 0; u < 8; u++) {
            const double b = g == 0 ? A.v[U.cols[c + 4 * u + t]] : 0.0;
            dmma884(s0, s1, xv[u], b);
          }
        }
        {
          double xv[8];
#pragma unroll
          for (int u = 0; u < 8; u++) xv[u] = c + 4 * u + t < gc ? __ldcs(x + c + 4 * u) : 0.0;
#pragma unroll
          for (int u = 0; u < 8; u++)
            if (c + 4 * u < gc) {
              const double b = (g == 0 && c + 4 * u + t < gc) ? A.v[U.cols[c + 4 * u + t]] : 0.0;
              dmma884(s0, s1, xv[u], b);
            }
        }
        // lane 4 g' holds row g' of the eight: hand it to the lane of that row
        const double mine = __shfl_sync(0xffffffffu, s0, 4 * (lane & 7));
        if ((lane >> 3) == j) acc += mine;
      }
    }
    // remaining dense-map columns
    for (int d0 = 0; d0 < A.nDense; d0 += 4) {
      double x[4];
      int64_t at[4];
      const double* src[4];
      int col[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        col[u] = -1;
        if (d0 + u < A.nDense) {
          const ColRef& cr = A.dense[d0 + u];
          col[u] = cr.col;
          src[u] = cr.src;
          at[u] = (int64_t)map_get(cr.mapType, cr.map, cr.mapHi, r) * cr.stride;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++) x[u] = col[u] >= 0 ? src[u][at[u]] : 0.0;
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (col[u] >= 0) acc = fma(x[u], A.v[col[u]], acc);
    }
    // listed tuples of this lane's row
    for (uint32_t p = p0; p < p1; p++) acc += P[A.rowItems[p]];
    if (A.fullPtr) {
      const int w = r0 / WIN_ROWS, rw = r0 + lane - w * WIN_ROWS;
      double full = 0.0;  // runs over the whole window: lanes share the sum
      for (uint32_t p = A.fullPtr[w] + lane; p < A.fullPtr[w + 1]; p += 32) full += P[A.fullItems[p]];
      for (int d = 16; d; d >>= 1) full += __shfl_xor_sync(0xffffffffu, full, d);
      acc += full;
      for (uint32_t p = A.partPtr[w]; p < A.partPtr[w + 1]; p++) {
        const uint2 it = A.partItems[p];
        const double x = P[it.x];
        if (rw >= (int)(it.y & 0xFF) && rw < (int)(it.y >> 8)) acc += x;
      }
    }
    if (r0 + lane < A.nRows) {
      double x = acc + (A.addTo ? A.out[r] : c0);
      if (A.rowScale) x *= A.rowScale[r];
      A.out[r] = x;
    }
  }
}

// --------------------------------------------------------------------------------------------------
// Yt X
// --------------------------------------------------------------------------------------------------
constexpr int RL_WARPS = 8;     // two CTAs per SM
constexpr int RL_T = RL_WARPS * 32;
constexpr int RL_TASKS = 320;   // columns per CTA of the first kind
constexpr int RL_UC = 64;       // columns per CTA of the second
constexpr int RL_WIN = SKIP_ROWS / WIN_ROWS;
struct RestLmmArgs {
  const RestTask* tasks;
  int nTasks, nChunks;       // chunks of RL_TASKS columns
  int ctaTasks;              // CTAs per chunk
  const double* dense;       // uncompressed group (null: none), its width, chunks of RL_UC columns, CTAs per chunk
  const int32_t* uncCols;
  int gCols, nUncChunks, ctaUnc;
  int nRows, q, nCols;
  const double* Yt;
  double* partT;             // [nChunks][ctaTasks][RL_TASKS][QT]
  double* partU;             // [nUncChunks][ctaUnc][RL_UC][QT]
  double* out;
};

template <int QT>
__device__ __forceinline__ void rest_lmm_tasks(const RestLmmArgs& A, int chunk, int cta, unsigned char* sm) {
  double* ys = (double*)sm;                         // [QT][SKIP_ROWS]
  double* ws = ys + QT * SKIP_ROWS;                 // [QT][RL_WIN]: sums of 64 rows
  double* sums = ws + QT * RL_WIN;                  // [RL_TASKS][QT]
  RestTask* T = (RestTask*)(sums + RL_TASKS * QT);  // [RL_TASKS]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = chunk * RL_TASKS, nt = min(RL_TASKS, A.nTasks - t0);
  for (int i = tid; i < nt; i += RL_T) T[i] = A.tasks[t0 + i];
  for (int i = tid; i < nt * QT; i += RL_T) sums[i] = 0.0;
  const int nBlocks = (A.nRows + SKIP_ROWS - 1) / SKIP_ROWS;
  const int b0 = (int)((int64_t)nBlocks * cta / A.ctaTasks), b1 = (int)((int64_t)nBlocks * (cta + 1) / A.ctaTasks);
  for (int b = b0; b < b1; b++) {
    const int r0 = b * SKIP_ROWS, nr = min(SKIP_ROWS, A.nRows - r0);
    __syncthreads();  // the previous block's readers are done (and T, sums are in place)
    for (int e = tid; e < QT * SKIP_ROWS; e += RL_T) {
      const int i = e / SKIP_ROWS, r = e - i * SKIP_ROWS;
      ys[e] = (i < A.q && r < nr) ? A.Yt[(size_t)i * A.nRows + r0 + r] : 0.0;
    }
    __syncthreads();
    for (int e = warp; e < QT * RL_WIN; e += RL_WARPS) {  // a warp per window and left row
      const double* y = ys + (e / RL_WIN) * SKIP_ROWS + (e % RL_WIN) * WIN_ROWS;
      double s = y[lane] + y[lane + 32];
      for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      if (lane == 0) ws[e] = s;
    }
    __syncthreads();
    for (int i0 = warp; i0 < nt; i0 += 32 * RL_WARPS) {
      // this warp's next 32 columns: lane l looks up where column i0 + RL_WARPS l starts in the block
      const int ti = i0 + lane * RL_WARPS;
      int64_t e0 = 0, e1 = 0;
      if (ti < nt) {
        const RestTask& k = T[ti];
        if (k.kind == GT_SDC) {
          const SdcSkip* sk = (const SdcSkip*)k.b;
          e0 = sk[b].elem;
          e1 = b + 1 < nBlocks ? (int64_t)sk[b + 1].elem : k.n;
        } else if (k.kind == GT_RLE) {
          e0 = ((const int32_t*)k.b)[b];
          e1 = k.n;
        }
      }
      const int n = min(32, (nt - i0 + RL_WARPS - 1) / RL_WARPS);
      uint2 next = make_uint2(0, 0);
      auto fetch = [&](int j) {  // the first 32 items of column j of the 32
        const int64_t a = __shfl_sync(0xffffffffu, e0, j & 31), z = __shfl_sync(0xffffffffu, e1, j & 31);
        uint2 v = make_uint2(0xFFFFFFFFu, 0);
        if (j < n) {
          const RestTask& k = T[i0 + j * RL_WARPS];
          if (a + lane < z) {
            if (k.kind == GT_SDC) v.x = ((const uint32_t*)k.a)[a + lane];
            else if (k.kind == GT_RLE) v = ((const uint2*)k.a)[a + lane];
          }
        }
        return v;
      };
      next = fetch(0);
      for (int j = 0; j < n; j++) {
        const uint2 item = next;
        next = fetch(j + 1);
        const int task = i0 + j * RL_WARPS;
        const RestTask& k = T[task];
        const int64_t a = __shfl_sync(0xffffffffu, e0, j), z = __shfl_sync(0xffffffffu, e1, j);
        double acc[QT];
#pragma unroll
        for (int i = 0; i < QT; i++) acc[i] = 0.0;
        if (k.kind == GT_SDC) {
          auto one = [&](uint32_t it) {
            const double x = k.src[(size_t)(it >> 10) * k.stride];
            const double* y = ys + (it & 1023u);
#pragma unroll
            for (int i = 0; i < QT; i++) acc[i] = fma(x, y[i * SKIP_ROWS], acc[i]);
          };
          if (a + lane < z) one(item.x);
          for (int64_t e = a + 32 + lane; e < z; e += 32) one(((const uint32_t*)k.a)[e]);
        } else if (k.kind == GT_RLE) {
          for (int64_t e = a;; e += 32) {
            uint2 it = item;
            if (e > a) it = e + lane < z ? ((const uint2*)k.a)[e + lane] : make_uint2(0xFFFFFFFFu, 0);
            const bool in = e + lane < z && (int)it.x < r0 + nr;  // the runs of a group are sorted by row
            const unsigned mask = __ballot_sync(0xffffffffu, in);
            for (unsigned left = mask; left; left &= left - 1) {
              const int l = __ffs(left) - 1;
              const int start = (int)__shfl_sync(0xffffffffu, it.x, l) - r0;
              const uint32_t lk = __shfl_sync(0xffffffffu, it.y, l);
              const int ra = max(start, 0), rb = min(start + (int)(lk & 0xFFFF), nr);
              if (ra >= rb) continue;
              const double x = k.src[(size_t)(lk >> 16) * k.stride];
              const int wa = (ra + WIN_ROWS - 1) / WIN_ROWS, wb = rb / WIN_ROWS;  // whole windows [wa, wb)
              double s[QT];
#pragma unroll
              for (int i = 0; i < QT; i++) s[i] = 0.0;
              if (wa < wb) {
                if (lane >= wa && lane < wb)
#pragma unroll
                  for (int i = 0; i < QT; i++) s[i] += ws[i * RL_WIN + lane];
                for (int r = ra + lane; r < wa * WIN_ROWS; r += 32)
#pragma unroll
                  for (int i = 0; i < QT; i++) s[i] += ys[i * SKIP_ROWS + r];
                for (int r = wb * WIN_ROWS + lane; r < rb; r += 32)
#pragma unroll
                  for (int i = 0; i < QT; i++) s[i] += ys[i * SKIP_ROWS + r];
              } else
                for (int r = ra + lane; r < rb; r += 32)
#pragma unroll
                  for (int i = 0; i < QT; i++) s[i] += ys[i * SKIP_ROWS + r];
#pragma unroll
              for (int i = 0; i < QT; i++) acc[i] = fma(x, s[i], acc[i]);
            }
            if (mask != 0xffffffffu) break;
          }
        } else {  // dense map, lanes along the rows
          for (int rr = lane; rr < nr; rr += 256) {
            int64_t at[8];
            double x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) at[u] = rr + 32 * u < nr ? (int64_t)map_get(k.mapType, k.a, k.b, r0 + rr + 32 * u) * k.stride : 0;
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = rr + 32 * u < nr ? k.src[at[u]] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; u++)
              if (rr + 32 * u < nr)
#pragma unroll
                for (int i = 0; i < QT; i++) acc[i] = fma(x[u], ys[i * SKIP_ROWS + rr + 32 * u], acc[i]);
          }
        }
        // lane i ends with the sum of left row i (reduce-scatter while there are several)
        if constexpr (QT == 1) {
          for (int d = 16; d; d >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], d);
          if (lane == 0) sums[task] += acc[0];
        } else {
#pragma unroll
          for (int d = QT / 2; d; d >>= 1) {
            const bool up = (lane & d) != 0;
#pragma unroll
            for (int i = 0; i < d; i++) {
              const double recv = __shfl_xor_sync(0xffffffffu, up ? acc[i] : acc[i + d], d);
              acc[i] = (up ? acc[i + d] : acc[i]) + recv;
            }
          }
          for (int d = 16; d >= QT; d >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], d);
          if (lane < QT) sums[task * QT + lane] += acc[0];
        }
      }
    }
  }
  __syncthreads();
  double* o = A.partT + ((size_t)chunk * A.ctaTasks + cta) * RL_TASKS * QT;
  for (int i = tid; i < nt * QT; i += RL_T) o[i] = sums[i];
}

// 64 columns of the uncompressed group: per product four rows x eight columns of the block and four left values of each
// left row; a warp takes every RL_WARPS-th group of 16 rows of the CTA's range.
template <int QT>
__device__ __forceinline__ void rest_lmm_unc(const RestLmmArgs& A, int chunk, int cta, unsigned char* sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int c0 = chunk * RL_UC, nc = min(RL_UC, A.gCols - c0), gc = A.gCols;
  const int nG = (A.nRows + 15) / 16;
  const int g0 = (int)((int64_t)nG * cta / A.ctaUnc), g1 = (int)((int64_t)nG * (cta + 1) / A.ctaUnc);
  double c[8][2];
#pragma unroll
  for (int i = 0; i < 8; i++) c[i][0] = c[i][1] = 0.0;
  const bool live = g < A.q;
  const double* yr = A.Yt + (size_t)(live ? g : 0) * A.nRows;
  for (int gi = g0 + warp; gi < g1; gi += RL_WARPS) {
    double x[4][8], y[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int row = gi * 16 + u * 4 + t;
      const bool in = row < A.nRows;
      y[u] = (live && in) ? yr[row] : 0.0;
      const double* d = A.dense + (size_t)row * gc + c0 + g;
#pragma unroll
      for (int i = 0; i < 8; i++) x[u][i] = (in && i * 8 + g < nc) ? __ldcs(d + i * 8) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int i = 0; i < 8; i++)
        if (i * 8 < nc) dmma884(c[i][0], c[i][1], y[u], x[u][i]);
  }
  // C: left row g, columns i * 8 + 2 t + {0, 1}; the warps' sums through shared memory
  double* red = (double*)sm;  // [RL_WARPS][RL_UC][QT]
  if (g < QT)
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int u = 0; u < 2; u++) red[(warp * RL_UC + i * 8 + 2 * t + u) * QT + g] = c[i][u];
  __syncthreads();
  double* o = A.partU + ((size_t)chunk * A.ctaUnc + cta) * RL_UC * QT;
  for (int e = tid; e < RL_UC * QT; e += RL_T) {
    double s = 0.0;
    for (int w = 0; w < RL_WARPS; w++) s += red[w * RL_UC * QT + e];
    o[e] = s;
  }
}

template <int QT>
__global__ void __launch_bounds__(RL_T, 2) k_rest_lmm(const __grid_constant__ RestLmmArgs A) {
  extern __shared__ __align__(16) unsigned char rlsm[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int nA = A.nChunks * A.ctaTasks;
  // the two kinds are interleaved so that both are resident from the start
  int b = blockIdx.x;
  if (b < nA) rest_lmm_tasks<QT>(A, b / A.ctaTasks, b % A.ctaTasks, rlsm);
  else {
    b -= nA;
    rest_lmm_unc<QT>(A, b / A.ctaUnc, b % A.ctaUnc, rlsm);
  }
}

// out += the CTAs' partial sums: 32 outputs per CTA, eight threads each, a fixed order
template <int QT>
__global__ void __launch_bounds__(256) k_rest_lmm_final(const __grid_constant__ RestLmmArgs A) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ double red[8][33];
  const int x = threadIdx.x & 31, sub = threadIdx.x >> 5;
  const int nT = A.nTasks * QT, nU = A.gCols * QT;
  const int e = blockIdx.x * 32 + x;
  double s = 0.0;
  int col = -1, i = 0;
  if (e < nT) {
    const int task = e / QT, chunk = task / RL_TASKS;
    i = e - task * QT;
    col = A.tasks[task].col;
    const double* p = A.partT + (size_t)chunk * A.ctaTasks * RL_TASKS * QT + (task - chunk * RL_TASKS) * QT + i;
#pragma unroll 4
    for (int k = sub; k < A.ctaTasks; k += 8) s += __ldcg(p + (size_t)k * RL_TASKS * QT);
  } else if (e < nT + nU) {
    const int c = (e - nT) / QT, chunk = c / RL_UC;
    i = (e - nT) - c * QT;
    col = A.uncCols[c];
    const double* p = A.partU + (size_t)chunk * A.ctaUnc * RL_UC * QT + (c - chunk * RL_UC) * QT + i;
#pragma unroll 4
    for (int k = sub; k < A.ctaUnc; k += 8) s += __ldcg(p + (size_t)k * RL_UC * QT);
  }
  red[sub][x] = s;
  __syncthreads();
  if (sub == 0 && col >= 0 && i < A.q) {
    for (int k = 1; k < 8; k++) s += red[k][x];
    atomicAdd(&A.out[(size_t)i * A.nCols + col], s);  // (a column may be held by several groups)
  }
}

// --------------------------------------------------------------------------------------------------
// plan and launchers
// --------------------------------------------------------------------------------------------------
static int64_t ensure_rest(Matrix* m, cudaStream_t s) {
  RestPlan& R = m->rest;
  if (R.tried) return CLA_OK;
  R.tried = true;
  int64_t rc;
  if ((rc = ensure_row_lists(m, s)) < 0) return rc;
  if (!m->rows.ok) return CLA_OK;
  std::vector<RestTask> sdc, rle, ddc;
  std::vector<ColRef> dense;
  for (size_t hi = 0; hi < m->hg.size(); hi++) {
    const int gi = m->regToDev[hi];
    if (gi < 0) continue;
    const DevGroup& g = m->groups[gi];
    if (g.type == GT_UNC) R.unc.push_back(gi);
    if (g.type == GT_UNC || g.inFast) continue;
    for (int j = 0; j < g.gCols; j++) {
      RestTask t{};
      t.src = g.dict + j;
      t.kind = g.type;
      t.mapType = g.mapType;
      t.stride = g.gCols;
      t.col = m->hg[hi].cols[j];
      if (g.type == GT_SDC) {
        if (g.nOff == 0) continue;
        t.a = m->rows.sdcItems + m->rows.sdcBase[gi];
        t.b = g.skip;
        t.n = g.nOff;
        sdc.push_back(t);
      } else if (g.type == GT_RLE) {
        if (g.nRuns == 0) continue;
        t.a = g.runs;
        t.b = g.runSkip;
        t.n = g.nRuns;
        rle.push_back(t);
      } else {
        t.a = g.map;
        t.b = g.mapHi;
        ddc.push_back(t);
        dense.push_back(ColRef{g.map, g.mapHi, g.dict + j, GT_DDC, g.mapType, g.gCols, t.col, gi, 0});
      }
    }
  }
  std::vector<RestTask> all(sdc);
  all.insert(all.end(), rle.begin(), rle.end());
  all.insert(all.end(), ddc.begin(), ddc.end());
  R.nTasks = (int)all.size();
  R.nDense = (int)dense.size();
  R.nUnc = (int)R.unc.size();
  const size_t bt = (all.size() * sizeof(RestTask) + 255) & ~(size_t)255, bd = dense.size() * sizeof(ColRef);
  std::vector<char> blob(bt + bd);
  if (!all.empty()) memcpy(blob.data(), all.data(), all.size() * sizeof(RestTask));
  if (bd) memcpy(blob.data() + bt, dense.data(), bd);
  if (!blob.empty()) {
    void* d = nullptr;
    if ((rc = plan_alloc(m, &d, blob.size())) < 0) return rc;
    CLA_CUDA(cudaMemcpy(d, blob.data(), blob.size(), cudaMemcpyHostToDevice));
    R.tasks = (RestTask*)d;
    R.dense = (ColRef*)((char*)d + bt);
  }
  R.ok = true;
  return CLA_OK;
}

// addTo: dOut holds the specialised kernels' part (constants included)
int64_t rest_rmm(Matrix* m, const double* dV, double* dOut, const double* dW, cudaStream_t s, bool addTo) {
  int64_t rc;
  if ((rc = ensure_rest(m, s)) < 0) return rc;
  const RestPlan& R = m->rest;
  const RowLists& L = m->rows;
  if (!R.ok) return 0;
  RestRmmArgs A{};
  A.sv = L.sv;
  A.svOff = L.svOff;
  A.groups = m->dGroups;
  A.nSv = (L.nSdc || L.nRle) ? (int)L.nSv : 0;
  A.nRows = m->nRows;
  A.nCols = m->nCols;
  A.nDense = R.nDense;
  A.dense = R.dense;
  A.rowPtr = L.nSdc ? L.rowPtr : nullptr;
  A.rowItems = L.rowItems;
  A.fullPtr = L.nRle ? L.fullPtr : nullptr;
  A.fullItems = L.fullItems;
  A.partPtr = L.partPtr;
  A.partItems = L.partItems;
  A.v = dV;
  A.out = dOut;
  size_t smem = 0;
  if (A.nSv > RR_PMAX) {
    if ((rc = ensure_scratch(m, (size_t)A.nSv * sizeof(double))) < 0) return rc;
    k_rest_terms<<<std::min(1024, (A.nSv + 255) / 256), 256, 0, s>>>(L.sv, A.nSv, m->dGroups, L.svOff, dV, (double*)m->scratch);
    m->stats.kernel_launches++;
    A.P = (const double*)m->scratch;
  } else
    smem = (size_t)A.nSv * sizeof(double);
  static bool attrSet[64] = {};  // per device
  if (!attrSet[m->device & 63]) {
    CLA_CUDA(cudaFuncSetAttribute(k_rest_rmm, cudaFuncAttributeMaxDynamicSharedMemorySize, RR_PMAX * (int)sizeof(double)));
    attrSet[m->device & 63] = true;
  }
  const int perSm = smem <= 50 * 1024 ? 4 : 3;
  const int grid = std::max(1, std::min((m->nRows + RR_T - 1) / RR_T, perSm * m->smCount));
  int u0 = 0;
  prof_begin(m, s);
  do {  // uncompressed groups RR_UNC at a time; the first launch adds everything else
    A.nUnc = std::min(RR_UNC, R.nUnc - u0);
    for (int i = 0; i < A.nUnc; i++) {
      const DevGroup& g = m->groups[R.unc[u0 + i]];
      A.unc[i] = UncGroup{g.dense, g.cols, g.gCols, 0};
    }
    u0 += A.nUnc;
    A.addTo = addTo ? 1 : 0;
    A.constV = (!addTo && m->hasConst) ? m->dConstV : nullptr;
    A.rowScale = u0 >= R.nUnc ? dW : nullptr;
    k_rest_rmm<<<grid, RR_T, smem, s>>>(A);
    m->stats.kernel_launches++;
    A.nSv = A.nDense = 0;
    A.rowPtr = A.fullPtr = nullptr;
    addTo = true;
  } while (u0 < R.nUnc);
  prof_end(m, s);
  CLA_CUDA(cudaGetLastError());
  return 1;
}

template <int QT>
static int64_t rest_lmm_go(Matrix* m, RestLmmArgs& A, int grid, size_t smem, cudaStream_t s) {
  static bool attrSet[64] = {};  // per device
  if (!attrSet[m->device & 63]) {
    CLA_CUDA(cudaFuncSetAttribute(k_rest_lmm<QT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024));
    attrSet[m->device & 63] = true;
  }
  k_rest_lmm<QT><<<grid, RL_T, smem, s>>>(A);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::max(1, (int)(((int64_t)A.nTasks * QT + (int64_t)A.gCols * QT + 31) / 32)));
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CLA_CUDA(cudaLaunchKernelEx(&cfg, k_rest_lmm_final<QT>, A));
  m->stats.kernel_launches += 2;
  return CLA_OK;
}

// Adds the remaining groups' part of Yt X to dOut (which holds the specialised kernels' part, or zeros and constants).
int64_t rest_lmm(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s) {
  int64_t rc;
  if ((rc = ensure_rest(m, s)) < 0) return rc;
  const RestPlan& R = m->rest;
  if (!R.ok) return 0;
  for (int q0 = 0; q0 < q;) {
    const int left = q - q0, QT = left >= 5 ? 8 : (left >= 2 ? 4 : 1), qc = std::min(QT, left);
    for (int u = 0; u == 0 || u < R.nUnc; u++) {  // one uncompressed group per launch; the first takes the other groups too
      RestLmmArgs A{};
      A.tasks = R.tasks;
      A.nTasks = u == 0 ? R.nTasks : 0;
      if (u < R.nUnc) {
        const DevGroup& g = m->groups[R.unc[u]];
        A.dense = g.dense;
        A.uncCols = g.cols;
        A.gCols = g.gCols;
      }
      if (A.nTasks == 0 && A.gCols == 0) break;
      A.nChunks = (A.nTasks + RL_TASKS - 1) / RL_TASKS;
      A.nUncChunks = (A.gCols + RL_UC - 1) / RL_UC;
      A.nRows = m->nRows;
      A.q = qc;
      A.nCols = m->nCols;
      A.Yt = dYt + (size_t)q0 * m->nRows;
      A.out = dOut + (size_t)q0 * m->nCols;
      const size_t smT = A.nTasks ? ((size_t)QT * (SKIP_ROWS + RL_WIN) + (size_t)RL_TASKS * QT) * 8 + RL_TASKS * sizeof(RestTask) : 0;
      const size_t smU = A.gCols ? (size_t)RL_WARPS * RL_UC * QT * 8 : 0;
      const size_t smem = std::max(smT, smU);
      const int slots = 2 * m->smCount;
      // CTAs of the two kinds: the block's bytes against the list walks, about 1 us of an SM per 350 columns and block
      const int nBlocks = (m->nRows + SKIP_ROWS - 1) / SKIP_ROWS;
      const double wT = A.nTasks * 1.0, wU = A.gCols * 2.5;
      int nT = A.nTasks ? (A.gCols ? std::max(1, (int)(slots * wT / (wT + wU))) : slots) : 0;
      A.ctaTasks = A.nTasks ? std::max(1, std::min(nBlocks, nT / A.nChunks)) : 0;
      const int nU = std::max(1, slots - A.ctaTasks * A.nChunks);
      A.ctaUnc = A.gCols ? std::max(1, std::min((m->nRows + 255) / 256, nU / A.nUncChunks)) : 0;
      const size_t bT = (size_t)A.nChunks * A.ctaTasks * RL_TASKS * QT * 8, bU = (size_t)A.nUncChunks * A.ctaUnc * RL_UC * QT * 8;
      if ((rc = ensure_scratch(m, bT + bU + 256)) < 0) return rc;
      A.partT = (double*)m->scratch;
      A.partU = (double*)((char*)m->scratch + bT);
      const int grid = A.nChunks * A.ctaTasks + A.nUncChunks * A.ctaUnc;
      if (u == 0) prof_begin(m, s);
      rc = QT == 8 ? rest_lmm_go<8>(m, A, grid, smem, s) : (QT == 4 ? rest_lmm_go<4>(m, A, grid, smem, s) : rest_lmm_go<1>(m, A, grid, smem, s));
      if (rc < 0) return rc;
      if (u == 0) prof_end(m, s);
    }
    q0 += qc;
  }
  CLA_CUDA(cudaGetLastError());
  return 1;
}

}  // namespace cla
