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
  int32_t gCols, at;  // at: its first column among the launch's
};
constexpr int RR_UNC = 8;       // uncompressed groups per launch
constexpr int RR_UCOLS = 1024;  // their columns (their part of v in shared memory); a wider group goes by itself, v unstaged
struct RestRmmArgs {
  const SparseVal* sv;
  const int32_t* svOff;
  const DevGroup* groups;
  const double* P;          // null: the CTA builds the table in shared memory
  int nSv, nRows, nDense, nUnc, nCols, addTo;
  int nUncCols;             // 0: v of the uncompressed columns is not staged
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
  double* uv = ps + (A.P ? 0 : A.nSv);
  for (int i = 0; i < A.nUnc && A.nUncCols; i++)
    for (int c = tid; c < A.unc[i].gCols; c += RR_T) uv[A.unc[i].at + c] = A.v[A.unc[i].cols[c]];
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
      const double* vs = uv + U.at;
      auto v_at = [&](int c) { return g == 0 ? (A.nUncCols ? vs[c] : A.v[U.cols[c]]) : 0.0; };
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
          for (int u = 0; u < 8; u++) dmma884(s0, s1, xv[u], v_at(c + 4 * u + t));
        }
        {
          double xv[8];
#pragma unroll
          for (int u = 0; u < 8; u++) xv[u] = c + 4 * u + t < gc ? __ldcs(x + c + 4 * u) : 0.0;
#pragma unroll
          for (int u = 0; u < 8; u++)
            if (c + 4 * u < gc) {
              dmma884(s0, s1, xv[u], c + 4 * u + t < gc ? v_at(c + 4 * u + t) : 0.0);
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
    for (; p0 + 4 <= p1; p0 += 4) {
      uint32_t it[4];
#pragma unroll
      for (int u = 0; u < 4; u++) it[u] = A.rowItems[p0 + u];
#pragma unroll
      for (int u = 0; u < 4; u++) acc += P[it[u]];
    }
    {
      uint32_t it[3];
#pragma unroll
      for (int u = 0; u < 3; u++) it[u] = p0 + u < p1 ? A.rowItems[p0 + u] : 0u;
#pragma unroll
      for (int u = 0; u < 3; u++)
        if (p0 + u < p1) acc += P[it[u]];
    }
    if (A.fullPtr) {
      const int w = r0 / WIN_ROWS, rw = r0 + lane - w * WIN_ROWS;
      double full = 0.0;  // runs over the whole window: lanes share the sum
      for (uint32_t p = A.fullPtr[w] + lane; p < A.fullPtr[w + 1]; p += 32) full += P[A.fullItems[p]];
      for (int d = 16; d; d >>= 1) full += __shfl_xor_sync(0xffffffffu, full, d);
      acc += full;
      const uint32_t q1 = A.partPtr[w + 1];
      for (uint32_t p = A.partPtr[w]; p < q1; p += 4) {
        uint2 it[4];
#pragma unroll
        for (int u = 0; u < 4; u++) it[u] = p + u < q1 ? A.partItems[p + u] : make_uint2(0, 0);  // no rows
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const double x = P[it[u].x];
          if (rw >= (int)(it[u].y & 0xFF) && rw < (int)(it[u].y >> 8)) acc += x;
        }
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
constexpr int RL_WARPS = 8;     // two CTAs per SM (three or four, of 80 or 64 registers: 5 to 35 % slower)
constexpr int RL_T = RL_WARPS * 32;
constexpr int RL_TASKS = 320;   // columns per CTA of the first kind, at most
constexpr int RL_UC = 64;       // columns per CTA of the second
constexpr int RL_WIN = SKIP_ROWS / WIN_ROWS;
struct RestLmmArgs {
  const RestTask* tasks;
  int nTasks, nChunks, per;  // chunks of per columns; the first nSparse are SDC / RLE columns
  int nSparse;
  int ctaTasks;              // CTAs per chunk
  const double* dense;       // uncompressed group (null: none), its width, chunks of RL_UC columns, CTAs per chunk
  const int32_t* uncCols;
  int gCols, nUncChunks, ctaUnc;
  int nRows, q, nCols;
  const double* Yt;
  double* partT;             // [nChunks][ctaTasks][per][QT]
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
  const int t0 = chunk * A.per, nt = min(A.per, A.nTasks - t0), nSparse = max(0, min(nt, A.nSparse - t0));
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
    // SDC and RLE columns: eight lanes each, four columns of a warp at a time (a column has a few dozen items per block,
    // and with eight lanes the walks of four columns and one reduction of three steps serve what took four)
    const int l8 = lane & 7, grp = lane >> 3;
    const unsigned gmask = 0xFFu << (grp * 8);
    for (int i0 = warp * 4; i0 < nSparse; i0 += RL_WARPS * 4) {
      const int task = i0 + grp;
      double acc[QT];
#pragma unroll
      for (int i = 0; i < QT; i++) acc[i] = 0.0;
      if (task < nSparse) {
        const RestTask& k = T[task];
        if (k.kind == GT_SDC) {
          const SdcSkip* sk = (const SdcSkip*)k.b;
          const int64_t e1 = b + 1 < nBlocks ? (int64_t)sk[b + 1].elem : k.n;
          const uint32_t* items = (const uint32_t*)k.a;
          for (int64_t e = (int64_t)sk[b].elem + l8; e < e1; e += 32) {
            uint32_t it[4];
            double x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) it[u] = e + 8 * u < e1 ? items[e + 8 * u] : 0u;
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = k.src[(size_t)(it[u] >> 10) * k.stride];
#pragma unroll
            for (int u = 0; u < 4; u++)
              if (e + 8 * u < e1) {
                const double* y = ys + (it[u] & 1023u);
#pragma unroll
                for (int i = 0; i < QT; i++) acc[i] = fma(x[u], y[i * SKIP_ROWS], acc[i]);
              }
          }
        } else {
          const RleRun* runs = (const RleRun*)k.a;
          for (int64_t e = ((const int32_t*)k.b)[b]; e < k.n; e++) {
            const RleRun run = runs[e];
            if (run.start >= r0 + nr) break;  // the runs of a group are sorted by row
            const int ra = max(run.start - r0, 0), rb = min(run.start - r0 + (int)run.len, nr);
            if (ra >= rb) continue;
            const double x = k.src[(size_t)run.k * k.stride];
            const int wa = (ra + WIN_ROWS - 1) / WIN_ROWS, wb = rb / WIN_ROWS;  // whole windows [wa, wb)
            double s[QT];
#pragma unroll
            for (int i = 0; i < QT; i++) s[i] = 0.0;
            const int h = wa < wb ? wa * WIN_ROWS : rb;  // rows [ra, h) and, behind the windows, [wb * 64, rb)
            for (int r = ra + l8; r < h; r += 8)
#pragma unroll
              for (int i = 0; i < QT; i++) s[i] += ys[i * SKIP_ROWS + r];
            if (wa < wb) {
              for (int w = wa + l8; w < wb; w += 8)
#pragma unroll
                for (int i = 0; i < QT; i++) s[i] += ws[i * RL_WIN + w];
              for (int r = wb * WIN_ROWS + l8; r < rb; r += 8)
#pragma unroll
                for (int i = 0; i < QT; i++) s[i] += ys[i * SKIP_ROWS + r];
            }
#pragma unroll
            for (int i = 0; i < QT; i++) acc[i] = fma(x, s[i], acc[i]);
          }
        }
      }
      __syncwarp();
      // lane i of the eight ends with the sum of left row i (reduce-scatter while there are several)
#pragma unroll
      for (int d = QT / 2; d; d >>= 1) {
        const bool up = (lane & d) != 0;
#pragma unroll
        for (int i = 0; i < d; i++) {
          const double recv = __shfl_xor_sync(gmask, up ? acc[i] : acc[i + d], d);
          acc[i] = (up ? acc[i + d] : acc[i]) + recv;
        }
      }
      for (int d = 4; d >= QT; d >>= 1) acc[0] += __shfl_xor_sync(gmask, acc[0], d);
      if (task < nSparse && l8 < QT) sums[task * QT + l8] += acc[0];
    }
    for (int task = nSparse + warp; task < nt; task += RL_WARPS) {  // dense map, lanes along the rows
      const RestTask& k = T[task];
      double acc[QT];
#pragma unroll
      for (int i = 0; i < QT; i++) acc[i] = 0.0;
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
  __syncthreads();
  double* o = A.partT + ((size_t)chunk * A.ctaTasks + cta) * A.per * QT;
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
  // (the launcher aims at no more CTAs than are resident at once, so that the second kind does not wait for the first)
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
    const int task = e / QT, chunk = task / A.per;
    i = e - task * QT;
    col = A.tasks[task].col;
    const double* p = A.partT + (size_t)chunk * A.ctaTasks * A.per * QT + (task - chunk * A.per) * QT + i;
#pragma unroll 4
    for (int k = sub; k < A.ctaTasks; k += 8) s += __ldcg(p + (size_t)k * A.per * QT);
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
// Yt X over 16-bit maps from TL_ROWS rows on: a CTA keeps the tables of up to sixteen columns in shared memory and walks a
// range of rows, a warp (or several, where long tables leave fewer columns) per column, lanes along the rows.
// Bound: the L1 / shared data pipe. Per 32 cells two 128-byte accesses for the left values, one for the ids and about six for
// random 8-byte reads of the table; from global memory, as the blockwise kernel reads them, each such read goes to its own
// line. 1,000,003 rows x 300 columns of 500 tuples, one left row: 2393 -> 360 us; 27,362 x 391, eight: 511 -> 59.
// --------------------------------------------------------------------------------------------------
constexpr int TL_WARPS = 16;
constexpr int TL_SMEM = 200 * 1024;
constexpr int TL_VALS = TL_SMEM / 8 / 4;  // tuples of a table, at most: four columns per CTA
constexpr int TL_ROWS = 16384;            // fewer rows: filling the tables is most of the time
struct TableLmmArgs {
  const RestTask* tasks;
  int n, vals, C, parts;  // columns, longest table, columns per CTA, row ranges
  int nRows, q, nCols;
  const double* Yt;
  double* part;  // [parts][n][QT]
  double* out;
};
// X v over the same columns, where the rows of an SM outnumber half the longest table (every SM fills every table: 65,537 rows
// x 300 columns of 2,000 tuples took 654 us) and from TL_XROWS rows on: a CTA owns a range of rows, lane = row, and takes the columns in turns,
// the tables D v of up to sixteen in shared memory; a row's sum waits in the result between the turns. Per 32 cells one
// 128-byte access for the ids and about six for the lookups. 1,000,003 x 300 columns of 500 tuples: 1618 -> 480 us.
constexpr int TL_XROWS = 65536;  // 443 rows per SM, a step of nearly every warp
struct TableRmmArgs {
  const RestTask* tasks;
  int n, vals, C, nRows, nCols, addTo;
  const double *v, *constV, *rowScale;
  double* out;
};
__global__ void __launch_bounds__(TL_WARPS * 32, 1) k_table_rmm(const __grid_constant__ TableRmmArgs A) {
  extern __shared__ __align__(16) double tlsm[];  // [C][vals]
  __shared__ const uint16_t* maps[TL_WARPS];
  __shared__ double cred[TL_WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, W = TL_WARPS / A.C;
  const int nSteps = (A.nRows + 31) / 32;
  const int s0 = (int)((int64_t)nSteps * blockIdx.x / gridDim.x), s1 = (int)((int64_t)nSteps * (blockIdx.x + 1) / gridDim.x);
  double c0 = 0.0;
  if (A.constV) {
    for (int c = tid; c < A.nCols; c += TL_WARPS * 32) c0 = fma(A.constV[c], A.v[c], c0);
    for (int d = 16; d; d >>= 1) c0 += __shfl_xor_sync(0xffffffffu, c0, d);
    if (lane == 0) cred[warp] = c0;
    __syncthreads();
    c0 = 0.0;
    for (int w = 0; w < TL_WARPS; w++) c0 += cred[w];
  }
  for (int k0 = 0; k0 < A.n; k0 += A.C) {
    const int nt = min(A.C, A.n - k0), k = warp / W;
    __syncthreads();  // the previous tables' readers are done
    if (k < nt) {
      const RestTask& T = A.tasks[k0 + k];
      const double x = A.v[T.col];
      if (lane == 0) maps[k] = (const uint16_t*)T.a;
      const int n = (int)T.n, stride = T.stride;
      const double* src = T.src;
#pragma unroll 8
      for (int i = (warp - k * W) * 32 + lane; i < n; i += W * 32) tlsm[k * A.vals + i] = src[(size_t)i * stride] * x;
    }
    __syncthreads();
    const bool last = k0 + A.C >= A.n;
    for (int st = s0 + warp; st < s1; st += TL_WARPS) {
      const int r = min(st * 32 + lane, A.nRows - 1);
      double acc = (k0 || A.addTo) ? A.out[r] : c0;
      int c = 0;
      for (; c + 8 <= nt; c += 8) {
        uint32_t id[8];
#pragma unroll
        for (int u = 0; u < 8; u++) id[u] = __ldg(maps[c + u] + r);
#pragma unroll
        for (int u = 0; u < 8; u++) acc += tlsm[(c + u) * A.vals + id[u]];
      }
      for (; c < nt; c++) acc += tlsm[c * A.vals + __ldg(maps[c] + r)];
      if (last && A.rowScale) acc *= A.rowScale[r];
      if (st * 32 + lane < A.nRows) A.out[r] = acc;
    }
  }
}

template <int QT>
__global__ void __launch_bounds__(TL_WARPS * 32, 1) k_table_lmm(const __grid_constant__ TableLmmArgs A) {
  extern __shared__ __align__(16) double tlsm[];  // [C][vals]
  __shared__ double red[TL_WARPS][QT];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = blockIdx.x / A.parts, p = blockIdx.x - chunk * A.parts;
  const int t0 = chunk * A.C, nt = min(A.C, A.n - t0), W = TL_WARPS / A.C, c = warp / W, sub = warp - c * W;
  for (int k = 0; k < nt; k++) {
    const RestTask& T = A.tasks[t0 + k];
    for (int v = tid; v < (int)T.n; v += TL_WARPS * 32) tlsm[k * A.vals + v] = T.src[(size_t)v * T.stride];
  }
  __syncthreads();
  double acc[QT];
#pragma unroll
  for (int i = 0; i < QT; i++) acc[i] = 0.0;
  if (c < nt) {
    const uint16_t* map = (const uint16_t*)A.tasks[t0 + c].a;
    const double* tab = tlsm + c * A.vals;
    const int r0 = (int)((int64_t)A.nRows * p / A.parts), r1 = (int)((int64_t)A.nRows * (p + 1) / A.parts);
    constexpr int U = QT == 1 ? 8 : 4;
    const double* y[QT];
#pragma unroll
    for (int i = 0; i < QT; i++) y[i] = A.Yt + (size_t)min(i, A.q - 1) * A.nRows;
    int r = r0 + sub * 32 * U + lane;
    for (; r - lane + 32 * U <= r1; r += W * 32 * U) {
      uint32_t id[U];
      double l[U][QT];
#pragma unroll
      for (int u = 0; u < U; u++) {
        id[u] = __ldg(map + r + 32 * u);
#pragma unroll
        for (int i = 0; i < QT; i++) l[u][i] = __ldg(y[i] + r + 32 * u);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const double x = tab[id[u]];
#pragma unroll
        for (int i = 0; i < QT; i++) acc[i] = fma(x, l[u][i], acc[i]);
      }
    }
    for (int u = 0; u < U; u++, r += 32)  // the range's last rows (one warp of the column has some)
      if (r < r1) {
        const double x = tab[__ldg(map + r)];
#pragma unroll
        for (int i = 0; i < QT; i++) acc[i] = fma(x, __ldg(y[i] + r), acc[i]);
      }
  }
#pragma unroll
  for (int i = 0; i < QT; i++) {
    for (int d = 16; d; d >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], d);
    if (lane == 0) red[warp][i] = acc[i];
  }
  __syncthreads();
  if (c < nt && sub == 0 && lane < QT) {
    double s = 0.0;
    for (int k = 0; k < W; k++) s += red[warp + k][lane];
    A.part[((size_t)p * A.n + t0 + c) * QT + lane] = s;
  }
}
template <int QT>
__global__ void __launch_bounds__(256) k_table_lmm_final(const __grid_constant__ TableLmmArgs A) {
  const int lane = threadIdx.x & 31, e = blockIdx.x * 8 + (threadIdx.x >> 5);  // a warp per sum
  if (e >= A.n * QT) return;
  double s = 0.0;
  for (int p = lane; p < A.parts; p += 32) s += A.part[(size_t)p * A.n * QT + e];
  for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  const int task = e / QT, i = e - task * QT;
  if (lane == 0 && i < A.q) atomicAdd(&A.out[(size_t)i * A.nCols + A.tasks[task].col], s);  // (several groups may hold a column)
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
  std::vector<RestTask> sdc, rle, ddc, table;
  std::vector<ColRef> dense, denseTable;
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
        t.a = m->sdcItems + g.listAt;
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
        t.n = g.nVals;
        const bool tab = g.mapType == CLA_MAP_CHAR && g.nVals <= TL_VALS;
        (tab ? table : ddc).push_back(t);
        if (tab) R.tableVals = std::max(R.tableVals, g.nVals);
        (tab ? denseTable : dense).push_back(ColRef{g.map, g.mapHi, g.dict + j, GT_DDC, g.mapType, g.gCols, t.col, gi, 0});
      }
    }
  }
  std::vector<RestTask> all(sdc);
  all.insert(all.end(), rle.begin(), rle.end());
  all.insert(all.end(), ddc.begin(), ddc.end());
  all.insert(all.end(), table.begin(), table.end());
  R.nTable = (int)table.size();
  dense.insert(dense.end(), denseTable.begin(), denseTable.end());
  R.nTasks = (int)all.size();
  R.nDense = (int)dense.size();
  R.nUnc = (int)R.unc.size();
  const size_t bt = (all.size() * sizeof(RestTask) + 255) & ~(size_t)255, bd = dense.size() * sizeof(ColRef);
  std::vector<char> blob(bt + bd);
  if (!all.empty()) memcpy(blob.data(), all.data(), all.size() * sizeof(RestTask));
  if (bd) memcpy(blob.data() + bt, dense.data(), bd);
  if (!blob.empty()) {
    void* d = nullptr;
    if (plan_alloc(m, &d, blob.size()) < 0) return CLA_OK;  // (R.ok stays false: the general kernels)
    CLA_CUDA(cudaMemcpy(d, blob.data(), blob.size(), cudaMemcpyHostToDevice));
    R.tasks = (RestTask*)d;
    R.dense = (ColRef*)((char*)d + bt);
  }
  R.ok = true;
  return CLA_OK;
}

static int64_t table_rmm(Matrix* m, const double* dV, double* dOut, const double* dW, cudaStream_t s, bool addTo) {
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, TL_SMEM, k_table_rmm); e < 0) return e;
  const RestPlan& R = m->rest;
  TableRmmArgs A{};
  A.tasks = R.tasks + (R.nTasks - R.nTable);
  A.n = R.nTable;
  A.vals = R.tableVals;
  for (A.C = TL_WARPS; A.C * A.vals * 8 > TL_SMEM; A.C /= 2) {
  }
  A.nRows = m->nRows;
  A.nCols = m->nCols;
  A.addTo = addTo ? 1 : 0;
  A.v = dV;
  A.constV = (!addTo && m->hasConst) ? m->dConstV : nullptr;
  A.rowScale = dW;
  A.out = dOut;
  k_table_rmm<<<m->smCount, TL_WARPS * 32, (size_t)A.C * A.vals * 8, s>>>(A);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

// addTo: dOut holds the specialised kernels' part (constants included)
int64_t rest_rmm(Matrix* m, const double* dV, double* dOut, const double* dW, cudaStream_t s, bool addTo) {
  int64_t rc;
  if ((rc = ensure_rest(m, s)) < 0) return rc;
  const RestPlan& R = m->rest;
  const RowLists& L = m->rows;
  if (!R.ok) return 0;
  const bool table = R.nTable > 0 && m->nRows >= TL_XROWS && (int64_t)m->nRows * 2 >= (int64_t)m->smCount * R.tableVals;
  if (table) {
    const bool all = R.nDense == R.nTable && R.nUnc == 0 && !L.nSdc && !L.nRle;
    if (all) prof_begin(m, s);
    if ((rc = table_rmm(m, dV, dOut, all ? dW : nullptr, s, addTo)) < 0) return rc;
    if (all) prof_end(m, s);
    if (all) return 1;
    addTo = true;
  }
  RestRmmArgs A{};
  A.sv = L.sv;
  A.svOff = L.svOff;
  A.groups = m->dGroups;
  A.nSv = (L.nSdc || L.nRle) ? (int)L.nSv : 0;
  A.nRows = m->nRows;
  A.nCols = m->nCols;
  A.nDense = R.nDense - (table ? R.nTable : 0);
  A.dense = R.dense;
  A.rowPtr = L.nSdc ? L.rowPtr : nullptr;
  A.rowItems = L.rowItems;
  A.fullPtr = L.nRle ? L.fullPtr : nullptr;
  A.fullItems = L.fullItems;
  A.partPtr = L.partPtr;
  A.partItems = L.partItems;
  A.v = dV;
  A.out = dOut;
  if (A.nSv > RR_PMAX) {
    if ((rc = ensure_scratch(m, (size_t)A.nSv * sizeof(double))) < 0) return rc;
    k_rest_terms<<<std::min(1024, (A.nSv + 255) / 256), 256, 0, s>>>(L.sv, A.nSv, m->dGroups, L.svOff, dV, (double*)m->scratch);
    m->stats.kernel_launches++;
    A.P = (const double*)m->scratch;
  }
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, (RR_PMAX + RR_UCOLS) * sizeof(double), k_rest_rmm); e < 0) return e;
  int u0 = 0;
  prof_begin(m, s);
  do {  // uncompressed groups up to RR_UNC and RR_UCOLS columns at a time; the first launch adds everything else
    A.nUnc = A.nUncCols = 0;
    while (u0 < R.nUnc && A.nUnc < RR_UNC) {
      const DevGroup& g = m->groups[R.unc[u0]];
      if (A.nUnc > 0 && A.nUncCols + g.gCols > RR_UCOLS) break;
      A.unc[A.nUnc++] = UncGroup{g.dense, g.cols, g.gCols, A.nUncCols};
      A.nUncCols += g.gCols;
      u0++;
    }
    if (A.nUncCols > RR_UCOLS) A.nUncCols = 0;
    const size_t smem = ((A.P ? 0 : A.nSv) + (size_t)A.nUncCols) * sizeof(double);
    const int perSm = smem <= 50 * 1024 ? 4 : 3;
    const int grid = std::max(1, std::min((m->nRows + RR_T - 1) / RR_T, perSm * m->smCount));
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
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, 112 * 1024, k_rest_lmm<QT>); e < 0) return e;
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

template <int QT>
static int64_t table_lmm_go(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s) {
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, TL_SMEM, k_table_lmm<QT>); e < 0) return e;
  const RestPlan& R = m->rest;
  TableLmmArgs A{};
  A.tasks = R.tasks + (R.nTasks - R.nTable);
  A.n = R.nTable;
  A.vals = R.tableVals;
  for (A.C = TL_WARPS; A.C * A.vals * 8 > TL_SMEM; A.C /= 2) {
  }
  A.nRows = m->nRows;
  A.q = q;
  A.nCols = m->nCols;
  const int chunks = (A.n + A.C - 1) / A.C;
  A.parts = std::max(1, m->smCount / chunks);
  A.Yt = dYt;
  A.out = dOut;
  int64_t rc;
  if ((rc = ensure_scratch(m, (size_t)A.parts * A.n * QT * 8 + 256)) < 0) return rc;
  A.part = (double*)m->scratch;
  k_table_lmm<QT><<<chunks * A.parts, TL_WARPS * 32, (size_t)A.C * A.vals * 8, s>>>(A);
  k_table_lmm_final<QT><<<(A.n * QT + 7) / 8, 256, 0, s>>>(A);
  m->stats.kernel_launches += 2;
  return CLA_OK;
}

// Adds the remaining groups' part of Yt X to dOut (which holds the specialised kernels' part, or zeros and constants).
int64_t rest_lmm(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s) {
  int64_t rc;
  if ((rc = ensure_rest(m, s)) < 0) return rc;
  const RestPlan& R = m->rest;
  if (!R.ok) return 0;
  const bool table = R.nTable > 0 && m->nRows >= TL_ROWS;
  const int nTasks = R.nTasks - (table ? R.nTable : 0);
  for (int q0 = 0; q0 < q;) {
    const int left = q - q0, QT = left >= 5 ? 8 : (left >= 2 ? 4 : 1), qc = std::min(QT, left);
    if (table) {
      const double* y = dYt + (size_t)q0 * m->nRows;
      double* o = dOut + (size_t)q0 * m->nCols;
      if (nTasks == 0 && R.nUnc == 0) prof_begin(m, s);
      rc = QT == 8 ? table_lmm_go<8>(m, y, qc, o, s) : (QT == 4 ? table_lmm_go<4>(m, y, qc, o, s) : table_lmm_go<1>(m, y, qc, o, s));
      if (rc < 0) return rc;
      if (nTasks == 0 && R.nUnc == 0) prof_end(m, s);
    }
    for (int u = 0; u == 0 || u < R.nUnc; u++) {  // one uncompressed group per launch; the first takes the other groups too
      RestLmmArgs A{};
      A.tasks = R.tasks;
      A.nTasks = u == 0 ? nTasks : 0;
      A.nSparse = R.nTasks - R.nDense;
      if (u < R.nUnc) {
        const DevGroup& g = m->groups[R.unc[u]];
        A.dense = g.dense;
        A.uncCols = g.cols;
        A.gCols = g.gCols;
      }
      if (A.nTasks == 0 && A.gCols == 0) break;
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
      const double wT = A.nTasks * 1.0, wU = A.gCols * 4.0;
      int nT = A.nTasks ? (A.gCols ? std::max(1, (int)(slots * wT / (wT + wU))) : slots) : 0;
      // Few blocks: fewer columns per CTA until the CTAs fill the SMs, one per warp at least (320 always: 6,126 rows x 101
      // columns of 16-bit maps took 140 us on 6 CTAs, 18 now).
      const int64_t even = nT ? ((int64_t)A.nTasks * nBlocks + nT - 1) / nT : 0;
      A.per = (int)std::max<int64_t>(RL_WARPS, std::min<int64_t>(RL_TASKS, (even + RL_WARPS - 1) / RL_WARPS * RL_WARPS));
      A.nChunks = (A.nTasks + A.per - 1) / A.per;
      A.ctaTasks = A.nTasks ? std::max(1, std::min(nBlocks, nT / A.nChunks)) : 0;
      const int nU = std::max(1, slots - A.ctaTasks * A.nChunks);
      A.ctaUnc = A.gCols ? std::max(1, std::min((m->nRows + 255) / 256, nU / A.nUncChunks)) : 0;
      const size_t bT = (size_t)A.nChunks * A.ctaTasks * A.per * QT * 8, bU = (size_t)A.nUncChunks * A.ctaUnc * RL_UC * QT * 8;
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
