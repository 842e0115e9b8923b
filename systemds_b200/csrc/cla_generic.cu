// Decompress, X %*% V kept compressed, and the general product kernels: every group type, any number of left rows,
// overlapping groups, from the registered arrays alone. The products come here where the kernels of cla_fast.cu,
// cla_rest.cu and cla_small.cu cannot run because their row lists or plans do not exist: 32-bit positions, device memory or
// the handle's plan limit have no room.
//
//   RMM  (CLALibRightMultBy.RMM, lib/CLALibRightMultBy.java:208-258)
//        1. k_dict_times_v : P_g = D_g * V[cols_g, :] for every dictionary group
//                            (ADictBasedColGroup.rightMultByMatrix, colgroup/ADictBasedColGroup.java:246-275)
//        2. k_rmm_vec_general : one right-hand column; a CTA owns a block of output rows and sums
//                            P_g[id_g(r)] over all groups, then adds constV * v (the decompress-and-sum of
//                            lib/CLALibDecompress.java:310-357). More right-hand columns: cla_rmm_dmma.cu.
//   LMM  (CLALibLeftMultBy.LMM, lib/CLALibLeftMultBy.java:286-346)
//        1. k_lmm_preagg   : A_g[i, k] = sum of Yt[i, r] over rows r holding tuple k
//                            (APreAgg.preAggregateDense, colgroup/APreAgg.java:137)
//        2. k_lmm_post     : out[i, cols_g] += A_g[i, :] * D_g  (APreAgg.mmWithDictionary, :312-322)
//        3. k_lmm_unc      : uncompressed groups, direct product (ColGroupUncompressed.java:429-539)
//        4. k_lmm_const    : out += rowSums(Yt) (x) constV  (lib/CLALibLeftMultBy.java:530-629)
#include "cla_common.cuh"
#include "cla_split.cuh"
#include <algorithm>
#include <climits>

namespace cla {

static inline int grid_for(int64_t n, int block, int cap = 148 * 16) {
  int64_t g = (n + block - 1) / block;
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, cap));
}

// --------------------------------------------------------------------------------------------------
// P arena: [totalVals x vCols]
// --------------------------------------------------------------------------------------------------
__global__ void k_dict_times_v(const DevGroup* __restrict__ groups, const double* __restrict__ V, int vCols,
                               double* __restrict__ P, int skipFast) {
  const DevGroup g = groups[blockIdx.x];
  if (g.type == GT_UNC || (skipFast && g.inFast)) return;
  const int64_t n = (int64_t)g.nVals * vCols;
  for (int64_t e = blockIdx.y * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.y * blockDim.x) {
    const int k = (int)(e / vCols), j = (int)(e - (int64_t)k * vCols);
    double s = 0;
    for (int h = 0; h < g.gCols; h++) s += g.dict[(size_t)k * g.gCols + h] * V[(size_t)g.cols[h] * vCols + j];
    P[(g.valOff + k) * vCols + j] = s;
  }
}

// constRow[j] = sum_c constV[c] * V[c, j]
__global__ void k_const_times_v(const double* __restrict__ constV, int nCols, const double* __restrict__ V, int vCols,
                                double* __restrict__ constRow) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= vCols) return;
  double s = 0;
  for (int c = 0; c < nCols; c++) s += constV[c] * V[(size_t)c * vCols + j];
  constRow[j] = s;
}

// --------------------------------------------------------------------------------------------------
// X %*% v (one column) for every group type. A CTA owns one 1024-row block (the granularity of the skip
// indexes) and keeps its 1024 partial sums in shared memory. Every row's sum is formed in a fixed order, so a
// repeated call returns the same bits whatever else runs on the GPU:
//  1. dense-map groups in list order: a thread per row adds P_g[id];
//  2. uncompressed groups in list order: a warp per row, lanes along the dense row, shuffle reduction;
//  3. SDC and RLE groups in list order, eight at a time: warp w writes the values group 8 i + w contributes to the
//     block's rows into its own row of a staging tile (SDC: warp-scan decode of the delta stream from the block's
//     skip entry; RLE: the runs that reach into the block), then the thread that owns a row adds the eight staged
//     values in group order. No atomics: each staging row has one writer, each sum one owner.
//  4. the constant part.
// (The reference sums a row's groups in list order and the constants last, lib/CLALibDecompress.java:427-434;
// here the order is by kind, then list order.)
// --------------------------------------------------------------------------------------------------
constexpr int RV_THREADS = 256;
constexpr int RV_WARPS = RV_THREADS / 32;
constexpr size_t RV_SMEM = (size_t)(RV_WARPS + 1) * SKIP_ROWS * sizeof(double);
__global__ void __launch_bounds__(RV_THREADS)
k_rmm_vec_general(const DevGroup* __restrict__ groups, const int32_t* __restrict__ ddcIdx, int nDdc,
                  const int32_t* __restrict__ uncIdx, int nUnc, const int32_t* __restrict__ sparseIdx, int nSparse, int nRows, const double* __restrict__ P, const double* __restrict__ v,
                  const double* __restrict__ constRow, double* __restrict__ out, int afterFast) {
  extern __shared__ __align__(16) double rvsm[];
  double* acc = rvsm;                  // [SKIP_ROWS]
  double* stage = rvsm + SKIP_ROWS;    // [RV_WARPS][SKIP_ROWS]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.x * SKIP_ROWS, r1 = min(nRows, r0 + SKIP_ROWS);
  for (int i = tid; i < SKIP_ROWS; i += RV_THREADS) acc[i] = 0.0;
  __syncthreads();
  // dense-map groups (list order; after the specialised kernels only those they left): a thread owns rows tid, tid + 256, ...
  for (int i = 0; i < nDdc; i++) {
    const DevGroup& g = groups[ddcIdx[i]];
    const double* Pg = P + g.valOff;
    for (int r = r0 + tid; r < r1; r += RV_THREADS) acc[r - r0] += Pg[map_get(g.mapType, g.map, g.mapHi, r)];
  }
  __syncthreads();
  // uncompressed groups: a warp owns rows warp, warp + 8, ...; lanes along the dense row, two columns each per pass,
  // four rows in flight (their loads are issued before the first of the four shuffle reductions)
  for (int i = 0; i < nUnc; i++) {
    const DevGroup& g = groups[uncIdx[i]];
    const int gc = g.gCols;
    const double* __restrict__ dense = g.dense;
    for (int cb = 0; cb < gc; cb += 64) {
      const int ca = cb + lane, cc = cb + 32 + lane;
      const double va = ca < gc ? v[g.cols[ca]] : 0.0, vb = cc < gc ? v[g.cols[cc]] : 0.0;
      for (int rb = r0 + warp * 4; rb < r1; rb += RV_WARPS * 4) {
        double sum[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int r = rb + q;
          const double* row = dense + (size_t)r * gc;
          const double xa = (r < r1 && ca < gc) ? row[ca] : 0.0, xb = (r < r1 && cc < gc) ? row[cc] : 0.0;
          sum[q] = xa * va + xb * vb;
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
          for (int d = 16; d; d >>= 1) sum[q] += __shfl_down_sync(0xffffffffu, sum[q], d);
        if (lane == 0) {
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (rb + q < r1) acc[rb + q - r0] += sum[q];
        }
      }
    }
  }
  if (nUnc) __syncthreads();
  // SDC / RLE groups, eight per round. From here on thread t owns rows 4 t .. 4 t + 3.
  double a4[4];
  {
    const double2 lo = *(const double2*)&acc[tid * 4], hi = *(const double2*)&acc[tid * 4 + 2];
    a4[0] = lo.x, a4[1] = lo.y, a4[2] = hi.x, a4[3] = hi.y;
  }
  double* mine = stage + warp * SKIP_ROWS;
  for (int s0 = 0; s0 < nSparse; s0 += RV_WARPS) {
    const int si = s0 + warp;
    if (si < nSparse) {
      double2* m2 = (double2*)mine;
      for (int i = lane; i < SKIP_ROWS / 2; i += 32) m2[i] = make_double2(0.0, 0.0);
      __syncwarp();
      const DevGroup& g = groups[sparseIdx[si]];
      const double* Pg = P + g.valOff;
      if (g.type == GT_SDC) {
        sdc_walk_block(g, r0, r1, [&](int row, int e) {
          mine[row - r0] = Pg[g.single ? 0 : map_get(g.mapType, g.map, g.mapHi, e)];
        });
      } else {  // RLE: a run writes its value to each of its rows (colgroup/ColGroupRLE.java:104-141)
        for (int64_t ri = g.runSkip[blockIdx.x]; ri < g.nRuns; ri++) {
          const RleRun run = g.runs[ri];
          if (run.start >= r1) break;
          const int a = max(run.start, r0), b = min(run.start + (int)run.len, r1);
          const double p = Pg[run.k];
          for (int i = a + lane; i < b; i += 32) mine[i - r0] = p;
        }
      }
    }
    __syncthreads();
    const int nw = min(RV_WARPS, nSparse - s0);
    for (int w = 0; w < nw; w++) {
      const double2 lo = *(const double2*)&stage[w * SKIP_ROWS + tid * 4];
      const double2 hi = *(const double2*)&stage[w * SKIP_ROWS + tid * 4 + 2];
      // rows a group does not list hold 0.0 here; adding it changes nothing
      a4[0] += lo.x, a4[1] += lo.y, a4[2] += hi.x, a4[3] += hi.y;
    }
    __syncthreads();
  }
  const double c0 = (constRow != nullptr && !afterFast) ? constRow[0] : 0.0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r = r0 + tid * 4 + i;
    if (r < r1) {
      const double val = a4[i] + c0;
      out[r] = afterFast ? out[r] + val : val;
    }
  }
}

// SDC groups with listed rows and RLE groups with runs, in list order (built once per handle)
int64_t ensure_sparse_list(Matrix* m) {
  if (m->sparseListBuilt) return CLA_OK;
  std::vector<int32_t> sparse, ddc, ddcRest, unc;
  for (int gi = 0; gi < m->nDev; gi++) {
    const DevGroup& g = m->groups[gi];
    if ((g.type == GT_SDC && g.nOff > 0) || (g.type == GT_RLE && g.nRuns > 0)) sparse.push_back(gi);
    if (g.type == GT_DDC) {
      ddc.push_back(gi);
      if (!g.inFast) ddcRest.push_back(gi);
    }
    if (g.type == GT_UNC) unc.push_back(gi);
  }
  auto up = [&](const std::vector<int32_t>& idx, int32_t** d) -> int64_t {
    if (idx.empty()) return CLA_OK;
    void* p = nullptr;
    cudaError_t e = dev_malloc(m, &p, idx.size() * sizeof(int32_t));
    if (e != cudaSuccess) return fail(CLA_ERR_NOMEM, std::string("cudaMalloc group list: ") + cudaGetErrorString(e));
    m->allocs.push_back(p);
    CLA_CUDA(cudaMemcpy(p, idx.data(), idx.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    *d = (int32_t*)p;
    return CLA_OK;
  };
  int64_t rc;
  if ((rc = up(sparse, &m->dSparseIdx)) < 0 || (rc = up(ddc, &m->dDdcIdx)) < 0 || (rc = up(ddcRest, &m->dDdcRestIdx)) < 0 ||
      (rc = up(unc, &m->dUncIdx)) < 0)
    return rc;
  m->nSparse = (int)sparse.size();
  m->nDdc = (int)ddc.size();
  m->nDdcRest = (int)ddcRest.size();
  m->nUnc = (int)unc.size();
  m->sparseListBuilt = true;
  return CLA_OK;
}

int64_t launch_rmm(Matrix* m, const double* dV, const double* dW, double* dOut, cudaStream_t s, bool afterFast) {
  if (m->nRows == 0) return CLA_OK;
  {
    const int64_t rc = rest_rmm(m, dV, dOut, dW, s, afterFast);
    if (rc != 0) return rc < 0 ? rc : CLA_OK;
  }
  if (dW) {  // no row lists: the kernel below does not scale
    const int64_t rc = launch_rmm(m, dV, nullptr, dOut, s, afterFast);
    return rc < 0 ? rc : launch_scale_rows(m, dOut, dW, m->nRows, s);
  }
  if (afterFast) {  // nothing left for this pass if the specialised kernels covered every group
    bool rest = false;
    for (auto& g : m->groups) rest |= !g.inFast;
    if (!rest) return CLA_OK;
  }
  int64_t rc;
  if ((rc = ensure_sparse_list(m)) < 0) return rc;
  const size_t pBytes = (size_t)std::max<int64_t>(m->totalVals, 1) * sizeof(double);
  const size_t cOff = (pBytes + 255) & ~(size_t)255;
  if ((rc = ensure_scratch(m, cOff + sizeof(double))) < 0) return rc;
  double* P = (double*)m->scratch;
  double* constRow = nullptr;
  if (m->nDev > 0) {
    int maxE = 1;
    for (auto& g : m->groups) maxE = std::max<int64_t>(maxE, (int64_t)g.nVals);
    dim3 grid(m->nDev, std::max(1, std::min(64, (maxE + 255) / 256)));
    k_dict_times_v<<<grid, 256, 0, s>>>(m->dGroups, dV, 1, P, afterFast ? 1 : 0);
    m->stats.kernel_launches++;
  }
  if (m->hasConst && !afterFast) {
    constRow = (double*)((char*)m->scratch + cOff);
    k_const_times_v<<<1, 128, 0, s>>>(m->dConstV, m->nCols, dV, 1, constRow);
    m->stats.kernel_launches++;
  }
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, RV_SMEM, k_rmm_vec_general); e < 0) return e;
  const int32_t* ddcIdx = afterFast ? m->dDdcRestIdx : m->dDdcIdx;
  const int nDdc = afterFast ? m->nDdcRest : m->nDdc;
  prof_begin(m, s);
  const unsigned grid = (unsigned)((m->nRows + SKIP_ROWS - 1) / SKIP_ROWS);
  k_rmm_vec_general<<<grid, RV_THREADS, RV_SMEM, s>>>(m->dGroups, ddcIdx, nDdc, m->dUncIdx, m->nUnc, m->dSparseIdx, m->nSparse, m->nRows, P, dV,
                                                     constRow, dOut, afterFast ? 1 : 0);
  prof_end(m, s);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

// --------------------------------------------------------------------------------------------------
// X %*% V kept compressed (CLALibRightMultBy.RMMOverlapping, lib/CLALibRightMultBy.java:157-201): every dictionary
// group of X becomes a group over all vCols result columns that keeps its index structure (the maps, offset
// streams and run lists are shared with X, not copied) and gets the dictionary P_g = D_g * V[cols_g, :]
// (ADictBasedColGroup.rightMultByMatrix, colgroup/ADictBasedColGroup.java:246-275); an uncompressed group becomes the
// uncompressed product of its block (colgroup/ColGroupUncompressed.java, rightMultByMatrix); the constants become
// constV * V (addConstant, :203-206). The result is an overlapping block: its cells are the sums over the groups.
// --------------------------------------------------------------------------------------------------
__global__ void k_unc_times_v(const double* __restrict__ dense, int gCols, const int32_t* __restrict__ cols, int64_t nRows,
                              const double* __restrict__ V, int vCols, double* __restrict__ out) {
  const int64_t n = nRows * vCols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / vCols;
    const int j = (int)(e - r * vCols);
    double s = 0;
    for (int c = 0; c < gCols; c++) s += dense[r * gCols + c] * V[(size_t)cols[c] * vCols + j];
    out[e] = s;
  }
}
__global__ void k_iota_cols(int32_t* p, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = i;
}

int64_t make_overlapping(Matrix* m, Matrix* child, const double* dV, int vCols, cudaStream_t s) {
  auto dalloc = [&](void** p, size_t bytes) -> int64_t {
    *p = nullptr;
    cudaError_t e = dev_malloc(child, p, std::max<size_t>(bytes, 16));
    if (e != cudaSuccess) return fail(CLA_ERR_NOMEM, std::string("cudaMalloc overlapping result: ") + cudaGetErrorString(e));
    child->allocs.push_back(*p);
    child->deviceBytes += (int64_t)bytes;
    return CLA_OK;
  };
  int64_t rc;
  child->nRows = m->nRows;
  child->nCols = vCols;
  child->overlapping = true;
  child->multiCover = true;
  child->colSrcValid = false;
  child->device = m->device;
  if ((rc = init_device_state(child)) < 0) return rc;
  void *P = nullptr, *iota = nullptr, *cst = nullptr;
  if ((rc = dalloc(&P, (size_t)std::max<int64_t>(m->totalVals, 1) * vCols * sizeof(double))) < 0) return rc;
  if ((rc = dalloc(&iota, (size_t)std::max(vCols, 1) * sizeof(int32_t))) < 0) return rc;
  if ((rc = dalloc(&cst, (size_t)std::max(vCols, 1) * sizeof(double))) < 0) return rc;
  if (vCols > 0) k_iota_cols<<<(vCols + 255) / 256, 256, 0, s>>>((int32_t*)iota, vCols);
  if (m->nDev > 0 && vCols > 0) {
    int64_t maxE = 1;
    for (auto& g : m->groups) maxE = std::max<int64_t>(maxE, (int64_t)g.nVals * vCols);
    dim3 grid(m->nDev, (unsigned)std::max<int64_t>(1, std::min<int64_t>(64, (maxE + 255) / 256)));
    k_dict_times_v<<<grid, 256, 0, s>>>(m->dGroups, dV, vCols, (double*)P, 0);
  }
  child->constV.assign(vCols, 0.0);
  if (m->hasConst && vCols > 0) {
    k_const_times_v<<<(vCols + 127) / 128, 128, 0, s>>>(m->dConstV, m->nCols, dV, vCols, (double*)cst);
    CLA_CUDA(cudaMemcpyAsync(child->constV.data(), cst, (size_t)vCols * sizeof(double), cudaMemcpyDeviceToHost, s));
  } else
    CLA_CUDA(cudaMemsetAsync(cst, 0, (size_t)std::max(vCols, 1) * sizeof(double), s));
  child->dConstV = (double*)cst;
  // the groups: same index structures, new dictionaries / dense blocks, every group over all result columns
  child->groups.clear();
  child->hg.clear();
  child->regToDev.clear();
  for (int gi = 0; gi < m->nDev; gi++) {
    DevGroup g = m->groups[gi];
    HostGroup hg;  // the record kept after finalize: type, width, number of tuples
    hg.type = g.origType;
    hg.cols.resize(vCols);
    for (int j = 0; j < vCols; j++) hg.cols[j] = j;
    hg.nVals = g.origType == GT_OLE ? g.nVals - 1 : g.nVals;
    if (g.type == GT_UNC) {
      void* d = nullptr;
      if ((rc = dalloc(&d, (size_t)m->nRows * vCols * sizeof(double))) < 0) return rc;
      if ((int64_t)m->nRows * vCols > 0)
        k_unc_times_v<<<grid_for((int64_t)m->nRows * vCols, 256), 256, 0, s>>>(g.dense, g.gCols, g.cols, m->nRows, dV, vCols, (double*)d);
      g.dense = (const double*)d;
    } else {
      g.dict = g.dictRaw = (const double*)P + (size_t)g.valOff * vCols;
    }
    g.gCols = vCols;
    g.cols = (const int32_t*)iota;
    g.inFast = 0;
    child->regToDev.push_back((int)child->groups.size());
    child->groups.push_back(g);
    child->hg.push_back(std::move(hg));
  }
  child->nDev = (int)child->groups.size();
  child->totalVals = m->totalVals;
  void* dg = nullptr;
  if ((rc = dalloc(&dg, std::max<size_t>(child->groups.size(), 1) * sizeof(DevGroup))) < 0) return rc;
  if (!child->groups.empty())
    CLA_CUDA(cudaMemcpyAsync(dg, child->groups.data(), child->groups.size() * sizeof(DevGroup), cudaMemcpyHostToDevice, s));
  child->dGroups = (DevGroup*)dg;
  void* cs = nullptr;  // column -> group table: unused for overlapping blocks, but allocated like everywhere else
  if ((rc = dalloc(&cs, (size_t)std::max(vCols, 1) * 2 * sizeof(int32_t))) < 0) return rc;
  CLA_CUDA(cudaMemsetAsync(cs, 0xFF, (size_t)std::max(vCols, 1) * 2 * sizeof(int32_t), s));
  child->dColSrc = (int32_t*)cs;
  CLA_CUDA(cudaStreamSynchronize(s));
  CLA_CUDA(cudaGetLastError());
  child->hasConst = false;
  for (double x : child->constV) child->hasConst |= (x != 0.0);
  child->colMin.assign(vCols, 0.0);  // extrema of an overlapping block are taken from decompressed rows
  child->colMax.assign(vCols, 0.0);
  child->indexBytes = (int64_t)std::max<int64_t>(m->totalVals, 1) * vCols * 8;
  child->stats.n_cols = vCols;
  child->stats.n_groups = (int64_t)child->hg.size();
  child->stats.device_bytes = child->deviceBytes;
  child->stats.index_bytes = child->indexBytes;
  child->finalized = true;
  return CLA_OK;
}

// --------------------------------------------------------------------------------------------------
// decompress = RMM with V = I restricted to the group's own columns: out[r, cols_g] += D_g[id_g(r), :]
// One launch per group keeps the reference's "groups in list order" summation
// (lib/CLALibDecompress.java:427-434) without atomics.
// --------------------------------------------------------------------------------------------------
__global__ void k_decomp_init(double* __restrict__ out, size_t ld, const double* __restrict__ constV, int64_t nRows, int nCols) {
  const int64_t n = nRows * nCols;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[(size_t)(i / nCols) * ld + i % nCols] = constV ? constV[i % nCols] : 0.0;
}
// rows [r0, r1); out points at row r0
__global__ void k_decomp_dense(DevGroup g, double* __restrict__ out, int r0, int r1, size_t ld) {
  const int64_t n = (int64_t)(r1 - r0) * g.gCols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / g.gCols;
    const int c = (int)(e - r * g.gCols);
    double v;
    if (g.type == GT_UNC) v = g.dense[(size_t)(r0 + r) * g.gCols + c];
    else v = g.dict[(size_t)map_get(g.mapType, g.map, g.mapHi, r0 + r) * g.gCols + c];
    out[r * ld + g.cols[c]] += v;
  }
}
__global__ void k_decomp_sdc(DevGroup g, double* __restrict__ out, int r0, int r1, size_t ld) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int rb = r0 + warp * SKIP_ROWS;
  if (rb >= r1) return;
  const int re = min(r1, rb + SKIP_ROWS);
  sdc_walk_block(g, rb, re, [&](int row, int e) {
    const int id = g.single ? 0 : map_get(g.mapType, g.map, g.mapHi, e);
    for (int c = 0; c < g.gCols; c++) out[(size_t)(row - r0) * ld + g.cols[c]] += g.dict[(size_t)id * g.gCols + c];
  });
}
__global__ void k_decomp_rle(DevGroup g, double* __restrict__ out, int r0, int r1, size_t ld) {
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nWarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (int64_t ri = g.runSkip[r0 / SKIP_ROWS] + warp; ri < g.nRuns; ri += nWarps) {
    const RleRun r = g.runs[ri];
    if (r.start >= r1) break;
    const int a = max(r.start, r0), b = min(r.start + (int)r.len, r1);
    for (int i = a + lane; i < b; i += 32)
      for (int c = 0; c < g.gCols; c++) out[(size_t)(i - r0) * ld + g.cols[c]] += g.dict[(size_t)r.k * g.gCols + c];
  }
}

// Decompress of a block whose columns each belong to at most one group, every group type, one pass: a CTA owns
// 128 rows x 32 columns and builds them in shared memory, a warp per column (two columns each) with lanes along the
// rows -- a dense-map column reads four consecutive ids per lane (one 128-byte line per warp for byte maps), an SDC
// column fills its constant and then scatters the listed rows (warp-scan decode from the skip entry), an RLE column
// fills its runs -- and then writes the tile out a row per warp instruction, 256 contiguous bytes per row.
// Uncompressed columns skip the tile: adjacent columns are adjacent in memory, so the write-out loop reads them.
// Every output cell is written exactly once; nothing is read back. (Measured alternatives, both slower: a 256 x 8
// tile, whose 64-byte output pieces lie 4 KB apart; persistent CTAs that keep their columns' dictionaries in shared
// memory -- the kernel is bound by the latency of its load -> lookup -> store chain, which many small CTAs hide
// better than few large ones.)
constexpr int DB_COLS = 32;
constexpr int DB_ROWS = 128;
constexpr int DB_LD = DB_ROWS + 1;   // column stride of the tile (odd: the row-wise read of the write-out is conflict free)
// position of tile row r inside its column: the four rows of a lane go to four different 32-row groups, so a warp's
// store of one of them is contiguous
__device__ __forceinline__ int db_pos(int r) { return (r & 3) * 32 + (r >> 2); }
constexpr int DB_WARPS = 16;  // two columns per warp (measured 4 / 8 / 16 / 32 warps on 1M x 500 mixed: 2.54 / 2.11 / 1.87 / 2.07 ms)
__global__ void __launch_bounds__(DB_WARPS * 32)
k_decomp_block(const DevGroup* __restrict__ groups, const int32_t* __restrict__ colSrc, const double* __restrict__ constV,
               double* __restrict__ out, size_t ld, int r0, int r1, int nCols, int exactSdc) {
  extern __shared__ double dtile[];  // [DB_COLS][DB_LD]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rb = r0 + blockIdx.x * DB_ROWS, re = min(r1, rb + DB_ROWS), nr = re - rb;
  const int c0 = blockIdx.y * DB_COLS, nc = min(DB_COLS, nCols - c0);
  __shared__ const double* uncSrc[DB_COLS];  // uncompressed columns: first value of the column (+ constant below)
  __shared__ int uncStride[DB_COLS];
  __shared__ double uncCst[DB_COLS];
  if (tid < DB_COLS) {
    uncSrc[tid] = nullptr;
    if (tid < nc) {
      const int gi = colSrc[2 * (c0 + tid)];
      if (gi >= 0 && groups[gi].type == GT_UNC) {
        uncSrc[tid] = groups[gi].dense + colSrc[2 * (c0 + tid) + 1];
        uncStride[tid] = groups[gi].gCols;
        uncCst[tid] = constV ? constV[c0 + tid] : 0.0;
      }
    }
  }
  for (int cw = warp; cw < nc; cw += DB_WARPS) {
    const int c = c0 + cw;
    const int gi = colSrc[2 * c];
    const double cst = constV ? constV[c] : 0.0;
    double* col = dtile + cw * DB_LD;
    if (gi < 0) {
      for (int rr = lane; rr < nr; rr += 32) col[db_pos(rr)] = cst;
    } else {
      const DevGroup& g = groups[gi];
      const int j = colSrc[2 * c + 1], gc = g.gCols;
      const double* dict = g.dict + j;
      if (g.type == GT_DDC) {
        const int mt = g.mapType;
        // four consecutive rows per lane; all ids are loaded before the first dictionary read that needs one
        int id[4];
        const int rr0 = lane * 4;
        if ((mt == CLA_MAP_UBYTE || mt == CLA_MAP_BYTE) && nr == DB_ROWS) {
          const uint32_t w = __ldg((const uint32_t*)((const uint8_t*)g.map + rb) + lane);  // rb is a multiple of 128
#pragma unroll
          for (int u = 0; u < 4; u++) id[u] = (w >> (8 * u)) & 0xFF;
        } else if (mt == CLA_MAP_CHAR && nr == DB_ROWS) {
          const uint2 w = __ldg((const uint2*)((const uint16_t*)g.map + rb) + lane);  // four 16-bit ids per lane
          id[0] = w.x & 0xFFFF;
          id[1] = w.x >> 16;
          id[2] = w.y & 0xFFFF;
          id[3] = w.y >> 16;
        } else {
#pragma unroll
          for (int u = 0; u < 4; u++) id[u] = rr0 + u < nr ? map_get(mt, g.map, g.mapHi, rb + rr0 + u) : 0;
        }
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = dict[(size_t)id[u] * gc];
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (rr0 + u < nr) col[u * 32 + lane] = cst + v[u];  // = db_pos(rr0 + u)
      } else if (g.type == GT_SDC) {
        for (int rr = lane; rr < nr; rr += 32) col[db_pos(rr)] = cst;
        __syncwarp();
        // exactSdc: the column belongs to this group alone, so its constant is exactly the group's default tuple and
        // a listed row holds the registered value itself (the reference writes d, lib/CLALibDecompress.java:310-357)
        const double* raw = g.dictRaw + j;
        sdc_walk_block(g, rb, re, [&](int row, int e) {
          const int id = g.single ? 0 : map_get(g.mapType, g.map, g.mapHi, e);
          col[db_pos(row - rb)] = exactSdc ? raw[(size_t)id * gc] : cst + dict[(size_t)id * gc];
        });
      } else if (g.type == GT_RLE) {
        for (int rr = lane; rr < nr; rr += 32) col[db_pos(rr)] = cst;
        __syncwarp();
        for (int64_t ri = g.runSkip[rb / SKIP_ROWS]; ri < g.nRuns; ri++) {
          const RleRun run = g.runs[ri];
          if (run.start >= re) break;
          const int a = max(run.start, rb), b = min(run.start + (int)run.len, re);
          const double v = cst + dict[(size_t)run.k * gc];
          for (int i = a + lane; i < b; i += 32) col[db_pos(i - rb)] = v;
        }
      }
    }
  }
  __syncthreads();
  // a row per warp instruction: lane = column of the tile
  if (lane < nc) {
    const double* us = uncSrc[lane];  // this lane's column: read once, not per row
    const size_t ustride = us ? (size_t)uncStride[lane] : 0;
    const double ucst = us ? uncCst[lane] : 0.0;
    const double* tcol = dtile + lane * DB_LD;
    double* o = out + (size_t)(rb - r0) * ld + c0 + lane;
    for (int rr = warp; rr < nr; rr += DB_WARPS)
      o[(size_t)rr * ld] = us ? ucst + us[(size_t)(rb + rr) * ustride] : tcol[db_pos(rr)];
  }
}

// Decompress, column per lane: a warp owns 32 neighbouring columns and DC_ROWS rows and walks down the rows, every lane
// in its own column: 16 ids per load and a table in shared memory (entry k of lane l at k * 32 + l: no bank conflicts) for
// small dense-map groups, the listed rows and their values for an SDC column, the runs for an RLE column, the dense
// block itself for an uncompressed one. The warps of a CTA write whole stretches of a row at the same time. The tile kernel
// above builds every cell in shared memory and reads it back. What is left is the latency of the chains item -> value and run
// -> value, so lists and runs go sixteen rows at a time: a lane puts its next entries into its own sixteen cells of shared memory, as
// many steps as the fullest column of the warp has entries there, and the sixteen stores then follow without a branch. Row by row,
// with a test for an entry and its loads in each, a warp took sixteen divergent steps: 250,001 x 500 mixed 312 us, 284 with cells for lists,
// 287 -> 273 with CTAs of eight warps. Of runs only the starts and ends go to cells, with a bit set for each (291 against 293 us).
// The records and the items of a block are filled on the device in its first call, without a copy (row lists, which hold the
// items too, take 350 us). 250,001 x 500 mixed (1 GB), tile kernel against this one: 495 -> 273 us, 3.7
// TB/s written.
struct DecCol {
  const double* dict;  // dictionary (or dense block) + position in the group
  const void* a;       // byte / bit map; SDC items; RLE runs
  const void* b;       // SDC skip entries; RLE first run of every block
  int64_t n;           // SDC listed rows; RLE runs
  double cst;          // column constant
  int32_t kind;        // DC_*
  int32_t stride, tbl, nVals;
  int32_t mapType, pad;
};
enum { DC_CONST = 0, DC_BYTES = 1, DC_BITS = 2, DC_MAP = 3, DC_SDC = 4, DC_RLE = 5, DC_UNC = 6 };
__host__ __device__ inline int dc_kind(const DevGroup& g) {
  if (g.type == GT_UNC) return DC_UNC;
  if (g.type == GT_SDC) return g.nOff > 0 ? DC_SDC : DC_CONST;
  if (g.type == GT_RLE) return g.nRuns > 0 ? DC_RLE : DC_CONST;
  if (g.nVals > 256) return DC_MAP;
  return g.mapType == CLA_MAP_UBYTE || g.mapType == CLA_MAP_BYTE ? DC_BYTES : (g.mapType == CLA_MAP_BIT ? DC_BITS : DC_MAP);
}
constexpr int DC_ROWS = 64;            // (256 / 128 / 64 rows on 250,001 x 500: 346 / 319 / 310 us)
constexpr int DC_WARPS = 16;
constexpr int64_t DC_CELLS = 4 << 20, DC_FIRST = 20 << 20;  // cells of a call; of the block, for its first call
constexpr size_t DC_TBL = 100 * 1024;  // table bytes of a CTA
constexpr size_t DC_CELLBUF = 16 * 32 * 8;  // and of a warp with lists or runs to walk, sixteen rows of a column per lane
constexpr size_t DC_SMEM = 113 * 1024;      // of both, for two CTAs on an SM
__global__ void __launch_bounds__(DC_WARPS * 32, 2) k_decomp_cols(const DecCol* __restrict__ cols, double* __restrict__ out, size_t ld, int r0, int r1,
                                                     int nRows, int nCols, int exactSdc, int cellsAt) {
  extern __shared__ double dct[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nW = blockDim.x >> 5;
  const int c = (blockIdx.y * nW + warp) * 32 + lane;
  const int rb = r0 + blockIdx.x * DC_ROWS, re = min(r1, rb + DC_ROWS), blk = rb / SKIP_ROWS, nBlocks = (nRows + SKIP_ROWS - 1) / SKIP_ROWS;
  DecCol d;
  d.kind = -1;
  if (c < nCols) d = cols[c];
  const double cst = c < nCols ? d.cst : 0.0;
  double* T = dct;
  if (d.kind == DC_BYTES || d.kind == DC_BITS) {
    T = dct + d.tbl + lane;
    for (int k = 0; k < d.nVals; k++) T[k * 32] = cst + d.dict[(size_t)k * d.stride];
  }
  double* o = out + (size_t)(rb - r0) * ld + c;
  if (d.kind == DC_BYTES || d.kind == DC_BITS) {  // (a lane reads only what it wrote itself)
    for (int r = rb; r < re; r += 16, o += 16 * ld) {
      if (r + 16 <= re) {
        uint32_t w[4];
        if (d.kind == DC_BYTES) {
          const uint4 v = __ldg((const uint4*)((const uint8_t*)d.a + r));
          w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
        } else {
          const uint32_t bits = (uint32_t)(((const unsigned long long*)d.a)[r >> 6] >> (r & 63));
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const uint32_t x = bits >> (4 * q);
            w[q] = (x & 1u) | ((x & 2u) << 7) | ((x & 4u) << 14) | ((x & 8u) << 21);
          }
        }
#pragma unroll
        for (int i = 0; i < 16; i++) o[i * ld] = T[((w[i >> 2] >> (8 * (i & 3))) & 0xFF) * 32];
      } else
        for (int i = 0; r + i < re; i++) o[i * ld] = T[map_get(d.mapType, d.a, nullptr, r + i) * 32];
    }
  } else if (d.kind == DC_UNC) {
    const double* x = d.dict + (size_t)rb * d.stride;
    const size_t xs = d.stride;
    for (int r = rb; r < re; r += 16, o += 16 * ld, x += 16 * xs) {
      if (r + 16 <= re) {
        double v[16];
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = __ldcs(x + i * xs);
#pragma unroll
        for (int i = 0; i < 16; i++) o[i * ld] = cst + v[i];
      } else
        for (int i = 0; r + i < re; i++) o[i * ld] = cst + x[i * xs];
    }
  } else if (d.kind == DC_SDC) {
    const uint32_t* items = (const uint32_t*)d.a;
    const SdcSkip* sk = (const SdcSkip*)d.b;
    const int64_t end = blk + 1 < nBlocks ? (int64_t)sk[blk + 1].elem : d.n;
    int64_t p = sk[blk].elem, hi = end;
    const uint32_t first = (uint32_t)(rb & (SKIP_ROWS - 1));
    while (p < hi) {  // first item at or behind row rb
      const int64_t mid = (p + hi) >> 1;
      if ((items[mid] & 1023u) < first) p = mid + 1;
      else hi = mid;
    }
    const int base = blk * SKIP_ROWS;
    auto value = [&](uint32_t it) { return exactSdc ? d.dict[(size_t)(it >> 10) * d.stride] : cst + d.dict[(size_t)(it >> 10) * d.stride]; };
    // the next listed row and its value, and the item behind it
    uint32_t it = p < end ? items[p] : 0u, ahead = p + 1 < end ? items[p + 1] : 0u;
    int row = p < end ? base + (int)(it & 1023u) : INT_MAX;
    double val = p < end ? value(it) : 0.0;
    auto advance = [&]() {
      p++;
      row = p < end ? base + (int)(ahead & 1023u) : INT_MAX;
      if (p < end) val = value(ahead);
      ahead = p + 1 < end ? items[p + 1] : 0u;
    };
    double* cells = dct + cellsAt + warp * 512 + lane;
    for (int r = rb; r < re; r += 16) {
#pragma unroll
      for (int i = 0; i < 16; i++) cells[i * 32] = cst;
      for (; (uint32_t)(row - r) < 16u; advance()) cells[(row - r) * 32] = val;
#pragma unroll
      for (int i = 0; i < 16; i++, o += ld)
        if (r + i < re) *o = cells[i * 32];
    }
  } else if (d.kind == DC_RLE) {
    const RleRun* runs = (const RleRun*)d.a;
    int64_t ri = ((const int32_t*)d.b)[blk];
    int start = INT_MAX, end = INT_MAX;  // the current or next run
    double val = 0.0;
    auto next = [&]() {
      if (ri < d.n) {
        const RleRun run = runs[ri++];
        start = run.start;
        end = run.start + (int)run.len;
        val = cst + d.dict[(size_t)run.k * d.stride];
      } else
        start = end = INT_MAX;
    };
    next();
    double* cells = dct + cellsAt + warp * 512 + lane;
    for (int r = rb; r < re; r += 16) {
      uint32_t set = 0;
      auto change = [&](int i, double x) {
        cells[i * 32] = x;
        set |= 1u << i;
      };
      for (; start - r < 16; next())
        if (end > r) {
          change(max(start - r, 0), val);
          if (end - r > 16) break;
          if (end - r < 16) change(end - r, cst);
        }
      double v = cst;
#pragma unroll
      for (int i = 0; i < 16; i++, o += ld) {
        if (set >> i & 1) v = cells[i * 32];
        if (r + i < re) *o = v;
      }
    }
  } else if (d.kind == DC_MAP) {
    for (int r = rb; r < re; r++, o += ld) *o = cst + d.dict[(size_t)map_get(d.mapType, d.a, d.b, r) * d.stride];
  } else if (d.kind == DC_CONST) {
    for (int r = rb; r < re; r++, o += ld) *o = cst;
  }
}

// The same walk, sixteen rows at a time, into digit planes (cla_split.cu) instead of doubles: tables hold the digits, and a value is split
// where it changes. halves: of 16 rows, those behind the last row are zeros. Two CTAs of sixteen warps' worth of registers on an SM
// hide more of the chains than the 75 registers it would take (t(X) X of 200,000 x 250 mixed 297 -> 290 us, of 50,000 x 400 260 -> 237).
template <bool GUARD>
__global__ void __launch_bounds__(DC_WARPS * 32, 2)
k_split_cols(const DecCol* __restrict__ cols, const int32_t* __restrict__ expo, int64_t halves, uint8_t* __restrict__ planes, int r0, int r1,
             int nRows, int nCols, int exactSdc, int cellsAt, int32_t* __restrict__ refused) {
  extern __shared__ double dct[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nW = blockDim.x >> 5;
  const int c = (blockIdx.y * nW + warp) * 32 + lane;
  if (c >= nCols) return;
  const int rb = r0 + blockIdx.x * DC_ROWS, re = min(r1, rb + DC_ROWS), blk = rb / SKIP_ROWS, nBlocks = (nRows + SKIP_ROWS - 1) / SKIP_ROWS;
  const DecCol d = cols[c];
  const double cst = d.cst, scale = split_scale(expo[c]);
  uint8_t* o = planes + ((size_t)(c / SP_COLS) * halves + (size_t)blockIdx.x * (DC_ROWS / 16)) * SP_HALF;
  bool bad = false;
  const unsigned long long base = split_pack<GUARD>(cst, scale, bad);
  auto value = [&](size_t k) {
    const double x = d.dict[k * d.stride];
    return split_pack<GUARD>(d.kind == DC_SDC && exactSdc ? x : cst + x, scale, bad);
  };
  unsigned long long v[16];
  // the groups of 16 rows; cell(i, row) gives the digits
  auto walk = [&](auto&& cell) {
    for (int g = 0; g < DC_ROWS / 16; g++) {
      const int r = rb + g * 16;
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = r + i < re ? cell(r + i) : 0ull;
      split_store<GUARD>(o + (size_t)g * SP_HALF, c, v);
    }
  };
  if (rb >= r1) walk([&](int) { return 0ull; });
  else if (d.kind == DC_BYTES || d.kind == DC_BITS) {
    unsigned long long* T = (unsigned long long*)dct + d.tbl + lane;
    for (int k = 0; k < d.nVals; k++) T[k * 32] = value(k);
    for (int g = 0; g < DC_ROWS / 16; g++) {
      const int r = rb + g * 16;
      if (r + 16 <= re) {
        uint32_t w[4];
        if (d.kind == DC_BYTES) {
          const uint4 q = __ldg((const uint4*)((const uint8_t*)d.a + r));
          w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
        } else {
          const uint32_t bits = (uint32_t)(((const unsigned long long*)d.a)[r >> 6] >> (r & 63));
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const uint32_t x = bits >> (4 * q);
            w[q] = (x & 1u) | ((x & 2u) << 7) | ((x & 4u) << 14) | ((x & 8u) << 21);
          }
        }
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = T[((w[i >> 2] >> (8 * (i & 3))) & 0xFF) * 32];
      } else
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = r + i < re ? T[map_get(d.mapType, d.a, nullptr, r + i) * 32] : 0ull;
      split_store<GUARD>(o + (size_t)g * SP_HALF, c, v);
    }
  } else if (d.kind == DC_UNC) {
    const double* x = d.dict + (size_t)rb * d.stride;
    const size_t xs = d.stride;
    for (int g = 0; g < DC_ROWS / 16; g++, x += 16 * xs) {
      double y[16];
#pragma unroll
      for (int i = 0; i < 16; i++) y[i] = rb + g * 16 + i < re ? __ldcs(x + i * xs) : 0.0;
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = rb + g * 16 + i < re ? split_pack<GUARD>(cst + y[i], scale, bad) : 0ull;
      split_store<GUARD>(o + (size_t)g * SP_HALF, c, v);
    }
  } else if (d.kind == DC_SDC) {
    const uint32_t* items = (const uint32_t*)d.a;
    const SdcSkip* sk = (const SdcSkip*)d.b;
    const int64_t end = blk + 1 < nBlocks ? (int64_t)sk[blk + 1].elem : d.n;
    int64_t p = sk[blk].elem, hi = end;
    const uint32_t first = (uint32_t)(rb & (SKIP_ROWS - 1));
    while (p < hi) {  // first item at or behind row rb
      const int64_t mid = (p + hi) >> 1;
      if ((items[mid] & 1023u) < first) p = mid + 1;
      else hi = mid;
    }
    const int at = blk * SKIP_ROWS;
    uint32_t it = p < end ? items[p] : 0u, ahead = p + 1 < end ? items[p + 1] : 0u;
    int row = p < end ? at + (int)(it & 1023u) : INT_MAX;
    unsigned long long val = p < end ? value(it >> 10) : 0ull;
    auto advance = [&]() {
      p++;
      row = p < end ? at + (int)(ahead & 1023u) : INT_MAX;
      if (p < end) val = value(ahead >> 10);
      ahead = p + 1 < end ? items[p + 1] : 0u;
    };
    unsigned long long* cells = (unsigned long long*)dct + cellsAt + warp * 512 + lane;  // (see k_decomp_cols)
    for (int g = 0; g < DC_ROWS / 16; g++) {
      const int r = rb + g * 16;
      uint32_t set = 0;
      for (; (uint32_t)(row - r) < 16u; advance()) {
        cells[(row - r) * 32] = val;
        set |= 1u << (row - r);
      }
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = set >> i & 1 ? cells[i * 32] : (r + i < re ? base : 0ull);
      split_store<GUARD>(o + (size_t)g * SP_HALF, c, v);
    }
  } else if (d.kind == DC_RLE) {
    const RleRun* runs = (const RleRun*)d.a;
    int64_t ri = ((const int32_t*)d.b)[blk];
    int start = INT_MAX, end = INT_MAX;  // the current or next run
    unsigned long long val = 0;
    auto next = [&]() {
      if (ri < d.n) {
        const RleRun run = runs[ri++];
        start = run.start;
        end = run.start + (int)run.len;
        val = value(run.k);
      } else
        start = end = INT_MAX;
    };
    next();
    unsigned long long* cells = (unsigned long long*)dct + cellsAt + warp * 512 + lane;
    for (int g = 0; g < DC_ROWS / 16; g++) {
      const int r = rb + g * 16;
      uint32_t set = 0;
      auto change = [&](int i, unsigned long long x) {
        cells[i * 32] = x;
        set |= 1u << i;
      };
      for (; start - r < 16; next())
        if (end > r) {
          change(max(start - r, 0), val);
          if (end - r > 16) break;
          if (end - r < 16) change(end - r, base);
        }
      unsigned long long x = base;
#pragma unroll
      for (int i = 0; i < 16; i++) {
        if (set >> i & 1) x = cells[i * 32];
        v[i] = r + i < re ? x : 0ull;
      }
      split_store<GUARD>(o + (size_t)g * SP_HALF, c, v);
    }
  } else if (d.kind == DC_MAP) {
    walk([&](int r) { return value(map_get(d.mapType, d.a, d.b, r)); });
  } else
    walk([&](int) { return base; });
  if (GUARD && bad) *refused = 1;
}

// The records of k_decomp_cols, filled by CTAs of the shape it will have.
__global__ void __launch_bounds__(DC_WARPS * 32)
k_dec_cols(const DevGroup* __restrict__ groups, const int32_t* __restrict__ colSrc, const double* __restrict__ constV,
           const uint32_t* __restrict__ sdcItems, DecCol* __restrict__ cols, int nCols, int exactSdc) {
  __shared__ int deep[DC_WARPS];  // longest table of every 32 columns
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * blockDim.x + threadIdx.x;
  DecCol d = {};
  d.kind = DC_CONST;
  if (c < nCols) {
    d.cst = constV ? constV[c] : 0.0;
    const int gi = colSrc[2 * c], j = colSrc[2 * c + 1];
    if (gi >= 0) {
      const DevGroup& g = groups[gi];
      d.kind = dc_kind(g);
      d.stride = g.gCols;
      d.nVals = g.nVals;
      d.mapType = g.mapType;
      d.dict = (d.kind == DC_UNC ? g.dense : (d.kind == DC_SDC && exactSdc ? g.dictRaw : g.dict)) + j;
      d.a = d.kind == DC_SDC ? (const void*)(sdcItems + g.listAt) : (d.kind == DC_RLE ? (const void*)g.runs : g.map);
      d.b = d.kind == DC_SDC ? (const void*)g.skip : (d.kind == DC_RLE ? (const void*)g.runSkip : g.mapHi);
      d.n = d.kind == DC_SDC ? g.nOff : g.nRuns;
    }
  }
  const int most = __reduce_max_sync(0xffffffffu, d.kind == DC_BYTES || d.kind == DC_BITS ? d.nVals : 0);
  if (lane == 0) deep[warp] = most;
  __syncthreads();
  for (int w = 0; w < warp; w++) d.tbl += deep[w] * 32;
  if (c < nCols) cols[c] = d;
}

// Warps of a CTA for n stretches of 32 columns. CTAs of five to eight warps overlap better than wider ones, whose warps all wait for
// the slowest walk; of those the width that leaves the fewest warps without columns, which hold their CTA's registers. Decompress mixed, us, this
// width and one CTA of n (or 16): 300,001 x 352 233 (6) and 252, 250,001 x 384 197 (6) and 223, 100,003 x 416 102 (7) and 108, x 480 99 (5) and 120, x 544 117 (6)
// and 142, 40,001 x 400 47 (7) and 49, 250,001 x 500 273 (8) and 292; 100,003 x 288 74 (5) and 74, 30,001 x 352 34 and 34. t(X) X mixed,
// 60,000 rows: x 288 155 and 156, x 352 169 and 178, x 400 277 and 281, x 480 271 and 295.
static int dec_warps(int n) {
  int best = std::min(n, 8);
  for (int w = best; w >= 5; w--)
    if ((n + w - 1) / w * w < (n + best - 1) / best * best) best = w;  // (warps of a row of CTAs)
  return best;
}

// Whether k_decomp_cols is the better kernel for the block's columns (m->dec.warps, 0: the tile kernel is) and how many
// warps a CTA has. Part of the upload, whose pass over the columns has everything at hand: finding it out at the first call
// took longer than that call saves on small blocks.
void decomp_shape(Matrix* m, const int32_t* colSrc) {
  int scattered = 0, kinds = 0;
  bool walks = false;
  std::vector<int> deep((m->nCols + 31) / 32, 0);
  for (int c0 = 0; c0 < m->nCols; c0 += 32) {
    unsigned seen = 0;
    for (int c = c0; c < std::min(m->nCols, c0 + 32); c++) {
      const int gi = colSrc[2 * c], k = gi < 0 ? DC_CONST : dc_kind(m->groups[gi]);
      scattered += k == DC_MAP;
      walks |= k == DC_SDC || k == DC_RLE;
      seen |= 1u << (k == DC_BITS ? DC_BYTES : k);
      if (k == DC_BYTES || k == DC_BITS) deep[c0 / 32] = std::max(deep[c0 / 32], m->groups[gi].nVals);
    }
    kinds += __builtin_popcount(seen);
  }
  // A lane-private gather from a large dictionary touches 32 lines per row, and a warp whose columns are of several kinds
  // walks its rows once per kind: matrices with many such columns keep the tile kernel (1M x 60 with four kinds in two
  // warps: 280 us there, 342 here).
  if (scattered * 16 > m->nCols || kinds * 5 > (int)deep.size() * 7) return;
  // tables: 256 bytes per tuple of the deepest small dictionary of every 32 columns; fewer columns per CTA if they are deep
  for (int warps = dec_warps((int)deep.size()); warps >= 1; warps /= 2) {
    const size_t cells = walks ? warps * DC_CELLBUF : 0;
    size_t most = 0;
    for (size_t w = 0; w < deep.size(); w += warps) {
      size_t b = 0;
      for (size_t i = w; i < std::min(deep.size(), w + warps); i++) b += (size_t)deep[i] * 256;
      most = std::max(most, b);
    }
    if (most <= DC_TBL && (warps <= 4 || most + cells <= DC_SMEM)) {
      m->dec.warps = warps;
      m->dec.tables = most;
      m->dec.smem = most + cells;
      return;
    }
  }
}

// The records of k_decomp_cols and the items of the SDC columns, m->dec.cols; without them the tile kernel runs. m->dec.warps becomes 0
// where there is no room for them. The device fills them, no host copy; they are complete when the handle has them, so that a
// call on any stream may use them.
static int64_t ensure_dec(Matrix* m, cudaStream_t s) {
  DecPlan& D = m->dec;
  if (D.cols || D.warps == 0) return CLA_OK;
  const int warps = D.warps;
  // (a call that is being captured runs nothing yet, so it cannot build a plan)
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &capture) != cudaSuccess) {
    cudaGetLastError();
    return CLA_OK;
  }
  if (capture != cudaStreamCaptureStatusNone) return CLA_OK;
  const int64_t itemBytes = m->sdcItemsOk ? 0 : sdc_items_bytes(m);
  const size_t at = ((size_t)m->nCols * sizeof(DecCol) + 255) & ~(size_t)255;
  void* p = nullptr;
  D.warps = 0;
  if (itemBytes < 0 || plan_alloc(m, &p, at + (size_t)itemBytes) < 0) return CLA_OK;
  uint32_t* items = m->sdcItemsOk ? m->sdcItems : (uint32_t*)((char*)p + at);
  if (!m->sdcItemsOk) launch_sdc_items(m, items, s);
  k_dec_cols<<<(m->nCols + warps * 32 - 1) / (warps * 32), warps * 32, 0, s>>>(
      m->dGroups, m->dColSrc, m->hasConst ? m->dConstV : nullptr, items, (DecCol*)p, m->nCols, m->multiCover ? 0 : 1);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  CLA_CUDA(cudaStreamSynchronize(s));
  m->sdcItems = items;
  m->sdcItemsOk = true;
  D.cols = p;
  D.warps = warps;
  return CLA_OK;
}

// r0 must be a multiple of SKIP_ROWS; a row of dOut is ld doubles wide
int64_t launch_decompress_range(Matrix* m, int r0, int r1, double* dOut, cudaStream_t s, size_t ld) {
  if (ld == 0) ld = (size_t)m->nCols;
  const int64_t n = (int64_t)(r1 - r0) * m->nCols;
  if (n <= 0) return CLA_OK;
  if (m->colSrcValid) {  // no column held by two groups: one pass, every cell written once
    const int64_t rf = fast_decompress(m, r0, r1, dOut, s, ld);  // byte-map matrices: straight from the column-per-lane layout
    if (rf != 0) return rf < 0 ? rf : CLA_OK;
    int64_t rc;
    // Below DC_CELLS both kernels take the same time (8,400 x 500: 32 us). Records and items cost a call 30 to 40 us,
    // which a block's first call makes up for from DC_FIRST on (24 million cells: 147 us as with the tile kernel, 33: 177 against
    // 183, 125: 403 against 534); a smaller block gets them when it is decompressed again (12 million: 58 against 66 from then on).
    bool byCols = n >= DC_CELLS;
    if (byCols && !m->dec.cols) {
      byCols = m->dec.again || (int64_t)m->nRows * m->nCols >= DC_FIRST;
      m->dec.again = true;
    }
    if (byCols && (rc = ensure_dec(m, s)) < 0) return rc;
    if (byCols && m->dec.cols) {
      static OncePerDevice once;
      if (const int64_t e = allow_smem(once, m->device, DC_TBL + 4 * DC_CELLBUF, k_decomp_cols); e < 0) return e;
      dim3 grid((r1 - r0 + DC_ROWS - 1) / DC_ROWS, (m->nCols + m->dec.warps * 32 - 1) / (m->dec.warps * 32));
      k_decomp_cols<<<grid, m->dec.warps * 32, m->dec.smem, s>>>(
          (const DecCol*)m->dec.cols, dOut, ld, r0, r1, m->nRows, m->nCols, m->multiCover ? 0 : 1, (int)(m->dec.tables / 8));
      m->stats.kernel_launches++;
      CLA_CUDA(cudaGetLastError());
      return CLA_OK;
    }
    const size_t smem = (size_t)DB_COLS * DB_LD * sizeof(double);
    static OncePerDevice once;
    if (const int64_t e = allow_smem(once, m->device, smem, k_decomp_block); e < 0) return e;
    dim3 grid((r1 - r0 + DB_ROWS - 1) / DB_ROWS, (m->nCols + DB_COLS - 1) / DB_COLS);
    k_decomp_block<<<grid, DB_WARPS * 32, smem, s>>>(m->dGroups, m->dColSrc, m->hasConst ? m->dConstV : nullptr, dOut, ld, r0, r1, m->nCols,
                                           m->multiCover ? 0 : 1);
    m->stats.kernel_launches++;
    CLA_CUDA(cudaGetLastError());
    return CLA_OK;
  }
  // overlapping groups: constants first, then every group adds its values (the reference's list-order summation)
  k_decomp_init<<<grid_for(n, 256), 256, 0, s>>>(dOut, ld, m->hasConst ? m->dConstV : nullptr, r1 - r0, m->nCols);
  m->stats.kernel_launches++;
  for (auto& g : m->groups) {
    if (g.type == GT_DDC || g.type == GT_UNC)
      k_decomp_dense<<<grid_for((int64_t)(r1 - r0) * g.gCols, 256), 256, 0, s>>>(g, dOut, r0, r1, ld);
    else if (g.type == GT_SDC) {
      const int nb = (r1 - r0 + SKIP_ROWS - 1) / SKIP_ROWS;
      k_decomp_sdc<<<(nb * 32 + 255) / 256, 256, 0, s>>>(g, dOut, r0, r1, ld);
    } else if (g.type == GT_RLE && g.nRuns)
      k_decomp_rle<<<64, 256, 0, s>>>(g, dOut, r0, r1, ld);
    m->stats.kernel_launches++;
  }
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

bool split_cols_covers(Matrix* m, cudaStream_t s) {
  // (fewer warps than four a CTA: deep tables, better read once to doubles)
  return m->colSrcValid && m->dec.warps >= 4 && ensure_dec(m, s) >= 0 && m->dec.cols;
}
int64_t launch_split_cols(Matrix* m, int r0, int r1, const int32_t* expo, int64_t halves, uint8_t* planes, int32_t* refused, cudaStream_t s) {
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, DC_TBL + 4 * DC_CELLBUF, k_split_cols<false>, k_split_cols<true>); e < 0) return e;
  dim3 grid((unsigned)((halves * 16 + DC_ROWS - 1) / DC_ROWS), (m->nCols + m->dec.warps * 32 - 1) / (m->dec.warps * 32));
  const DecCol* cols = (const DecCol*)m->dec.cols;
  const int exact = m->multiCover ? 0 : 1, threads = m->dec.warps * 32;
  if (refused) k_split_cols<true><<<grid, threads, m->dec.smem, s>>>(cols, expo, halves, planes, r0, r1, m->nRows, m->nCols, exact, (int)(m->dec.tables / 8), refused);
  else k_split_cols<false><<<grid, threads, m->dec.smem, s>>>(cols, expo, halves, planes, r0, r1, m->nRows, m->nCols, exact, (int)(m->dec.tables / 8), nullptr);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

int64_t launch_decompress(Matrix* m, double* dOut, cudaStream_t s) {
  return launch_decompress_range(m, 0, m->nRows, dOut, s);
}

// --------------------------------------------------------------------------------------------------
// LMM
// --------------------------------------------------------------------------------------------------
constexpr int LMM_THREADS = 256;
constexpr int LMM_QT = 4;                 // left rows per pass (the reference's rowBlockSize)
constexpr int LMM_HIST_MAX = 6144;        // doubles of shared histogram (48 KB)

// grid: (row chunks, dictionary groups, q tiles). A: [totalVals x q]
__global__ void __launch_bounds__(LMM_THREADS)
k_lmm_preagg(const DevGroup* __restrict__ groups, int nRows, int rowsPerChunk, const double* __restrict__ Yt, int q,
             double* __restrict__ A, int skipFast) {
  __shared__ double hist[LMM_HIST_MAX];
  const DevGroup& g = groups[blockIdx.y];
  if (g.type == GT_UNC || (skipFast && g.inFast)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ra = blockIdx.x * rowsPerChunk, rb = min(nRows, ra + rowsPerChunk);
  if (ra >= rb) return;
  const int q0 = blockIdx.z * LMM_QT, qt = min(LMM_QT, q - q0);
  const int nv = g.nVals;
  const bool useShared = (int64_t)nv * qt <= LMM_HIST_MAX;
  double* Ag = A + g.valOff * q;
  if (useShared) {
    for (int e = tid; e < nv * qt; e += LMM_THREADS) hist[e] = 0.0;
    __syncthreads();
  }
  auto add = [&](int id, int i, double v) {
    if (useShared) atomicAdd(&hist[i * nv + id], v);
    else atomicAdd(&Ag[(size_t)id * q + q0 + i], v);
  };
  if (g.type == GT_DDC) {
    for (int r = ra + tid; r < rb; r += LMM_THREADS) {
      const int id = map_get(g.mapType, g.map, g.mapHi, r);
      for (int i = 0; i < qt; i++) add(id, i, Yt[(size_t)(q0 + i) * nRows + r]);
    }
  } else if (g.type == GT_SDC) {
    for (int b = ra + warp * SKIP_ROWS; b < rb; b += (LMM_THREADS / 32) * SKIP_ROWS) {
      sdc_walk_block(g, b, min(rb, b + SKIP_ROWS), [&](int row, int e) {
        const int id = g.single ? 0 : map_get(g.mapType, g.map, g.mapHi, e);
        for (int i = 0; i < qt; i++) add(id, i, Yt[(size_t)(q0 + i) * nRows + row]);
      });
    }
  } else if (g.type == GT_RLE) {
    // one warp per run: sum the left values over the run, then one add per left row
    for (int64_t ri = g.runSkip[ra / SKIP_ROWS] + warp; ri < g.nRuns; ri += LMM_THREADS / 32) {
      const RleRun run = g.runs[ri];
      if (run.start >= rb) break;
      const int a = max(run.start, ra), b = min(run.start + (int)run.len, rb);
      for (int i = 0; i < qt; i++) {
        double sum = 0;
        for (int r = a + lane; r < b; r += 32) sum += Yt[(size_t)(q0 + i) * nRows + r];
        for (int d = 16; d; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d);
        if (lane == 0 && a < b) add(run.k, i, sum);
      }
    }
  }
  if (useShared) {
    __syncthreads();
    for (int e = tid; e < nv * qt; e += LMM_THREADS) {
      const double v = hist[e];
      if (v != 0.0) {
        const int i = e / nv, id = e - i * nv;
        atomicAdd(&Ag[(size_t)id * q + q0 + i], v);
      }
    }
  }
}

// out[i, cols_g[c]] += sum_k A_g[k, i] * D_g[k, c]; one block per group
__global__ void k_lmm_post(const DevGroup* __restrict__ groups, const double* __restrict__ A, int q, int nCols,
                           double* __restrict__ out, int skipFast) {
  const DevGroup& g = groups[blockIdx.x];
  if (g.type == GT_UNC || (skipFast && g.inFast)) return;
  const double* Ag = A + g.valOff * q;
  for (int e = threadIdx.x; e < q * g.gCols; e += blockDim.x) {
    const int i = e / g.gCols, c = e - i * g.gCols;
    double s = 0;
    for (int k = 0; k < g.nVals; k++) s += Ag[(size_t)k * q + i] * g.dict[(size_t)k * g.gCols + c];
    atomicAdd(&out[(size_t)i * nCols + g.cols[c]], s);
  }
}

// uncompressed group: out[i, cols[c]] += sum_r Yt[i, r] * dense[r, c]. A thread owns one column c (threads along
// the columns read a dense row contiguously) and one of `ry` row phases; the block covers a chunk of rows.
__global__ void k_lmm_unc(DevGroup g, int nRows, int rowsPerChunk, const double* __restrict__ Yt, int q, int nCols,
                          double* __restrict__ out) {
  extern __shared__ double red[];  // [ry][gCols]
  const int ra = blockIdx.x * rowsPerChunk, rb = min(nRows, ra + rowsPerChunk);
  const int gc = g.gCols;
  const int cx = threadIdx.x % gc, ry = threadIdx.x / gc, nry = blockDim.x / gc;
  for (int i = 0; i < q; i++) {
    double s = 0;
    if (ry < nry)
      for (int r = ra + ry; r < rb; r += nry) s += Yt[(size_t)i * nRows + r] * g.dense[(size_t)r * gc + cx];
    if (ry < nry) red[ry * gc + cx] = s;
    __syncthreads();
    if (ry == 0) {
      for (int k = 1; k < nry; k++) s += red[k * gc + cx];
      atomicAdd(&out[(size_t)i * nCols + g.cols[cx]], s);
    }
    __syncthreads();
  }
}

__global__ void k_lmm_unc_wide(DevGroup g, int nRows, int rowsPerChunk, const double* __restrict__ Yt, int q, int nCols,
                               double* __restrict__ out) {
  const int ra = blockIdx.x * rowsPerChunk, rb = min(nRows, ra + rowsPerChunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = blockDim.x >> 5;
  // more columns than a block has threads: each warp owns output cells (i, c) round robin; lanes stride over rows
  for (int e = warp; e < q * g.gCols; e += nWarps) {
    const int i = e / g.gCols, c = e - i * g.gCols;
    double s = 0;
    for (int r = ra + lane; r < rb; r += 32) s += Yt[(size_t)i * nRows + r] * g.dense[(size_t)r * g.gCols + c];
    for (int d = 16; d; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
    if (lane == 0) atomicAdd(&out[(size_t)i * nCols + g.cols[c]], s);
  }
}

__global__ void k_row_sums(const double* __restrict__ Yt, int nRows, int q, double* __restrict__ sums) {
  const int i = blockIdx.y;
  double s = 0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nRows; r += (int64_t)gridDim.x * blockDim.x)
    s += Yt[(size_t)i * nRows + r];
  for (int d = 16; d; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
  if ((threadIdx.x & 31) == 0) atomicAdd(&sums[i], s);
}
__global__ void k_lmm_const(const double* __restrict__ sums, const double* __restrict__ constV, int q, int nCols,
                            double* __restrict__ out) {
  const int64_t n = (int64_t)q * nCols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    out[e] += sums[e / nCols] * constV[e % nCols];
}

int64_t launch_lmm_const(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s);

int64_t launch_lmm(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s, bool afterFast) {
  if (q == 0 || m->nCols == 0) return CLA_OK;
  if (!afterFast) CLA_CUDA(cudaMemsetAsync(dOut, 0, sizeof(double) * (size_t)q * m->nCols, s));
  if (m->nRows == 0) return CLA_OK;
  int64_t rc;
  if (m->nDev > 0 && (afterFast || !fast_plan_partial(m))) {  // (without the specialised kernels' part only where they leave no group)
    if ((rc = rest_lmm(m, dYt, q, dOut, s)) < 0) return rc;
    if (rc == 1) return afterFast ? CLA_OK : launch_lmm_const(m, dYt, q, dOut, s);
  }
  const size_t aBytes = (size_t)std::max<int64_t>(m->totalVals, 1) * q * sizeof(double);
  const size_t sOff = (aBytes + 255) & ~(size_t)255;
  if ((rc = ensure_scratch(m, sOff + (size_t)q * sizeof(double))) < 0) return rc;
  double* A = (double*)m->scratch;
  double* sums = (double*)((char*)m->scratch + sOff);
  CLA_CUDA(cudaMemsetAsync(A, 0, sOff + (size_t)q * sizeof(double), s));
  if (m->nDev > 0) {
    const int target = std::max(1, (8 * m->smCount) / std::max(1, m->nDev));
    int rowsPerChunk = (int)(((int64_t)m->nRows + target - 1) / target);
    rowsPerChunk = std::max(SKIP_ROWS * 4, ((rowsPerChunk + SKIP_ROWS - 1) / SKIP_ROWS) * SKIP_ROWS);
    const int chunks = (m->nRows + rowsPerChunk - 1) / rowsPerChunk;
    dim3 grid(chunks, m->nDev, (q + LMM_QT - 1) / LMM_QT);
    prof_begin(m, s);
    k_lmm_preagg<<<grid, LMM_THREADS, 0, s>>>(m->dGroups, m->nRows, rowsPerChunk, dYt, q, A, afterFast ? 1 : 0);
    prof_end(m, s);
    k_lmm_post<<<m->nDev, 128, 0, s>>>(m->dGroups, A, q, m->nCols, dOut, afterFast ? 1 : 0);
    m->stats.kernel_launches += 2;
    for (auto& g : m->groups)
      if (g.type == GT_UNC) {
        const int rpc = std::max(2048, (int)(((int64_t)m->nRows + 8 * m->smCount - 1) / (8 * m->smCount)));
        if (g.gCols <= 512) {
          const int threads = std::max(g.gCols, (512 / g.gCols) * g.gCols);  // whole multiples of the column count
          k_lmm_unc<<<(m->nRows + rpc - 1) / rpc, threads, (size_t)threads * sizeof(double), s>>>(g, m->nRows, rpc, dYt, q,
                                                                                              m->nCols, dOut);
        } else
          k_lmm_unc_wide<<<(m->nRows + rpc - 1) / rpc, 256, 0, s>>>(g, m->nRows, rpc, dYt, q, m->nCols, dOut);
        m->stats.kernel_launches++;
      }
  }
  if (m->hasConst && !afterFast) {
    dim3 grid(grid_for(m->nRows, 256, 4 * m->smCount), q);
    k_row_sums<<<grid, 256, 0, s>>>(dYt, m->nRows, q, sums);
    k_lmm_const<<<grid_for((int64_t)q * m->nCols, 256), 256, 0, s>>>(sums, m->dConstV, q, m->nCols, dOut);
    m->stats.kernel_launches += 2;
  }
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

// out += rowSums(Yt) (x) constV into a caller-provided vector of q sums
int64_t launch_lmm_const_with(Matrix* m, const double* dYt, int q, double* dOut, double* sums, cudaStream_t s) {
  if (!m->hasConst || q == 0 || m->nRows == 0) return CLA_OK;
  CLA_CUDA(cudaMemsetAsync(sums, 0, (size_t)q * sizeof(double), s));
  dim3 grid(grid_for(m->nRows, 256, 4 * m->smCount), q);
  k_row_sums<<<grid, 256, 0, s>>>(dYt, m->nRows, q, sums);
  k_lmm_const<<<grid_for((int64_t)q * m->nCols, 256), 256, 0, s>>>(sums, m->dConstV, q, m->nCols, dOut);
  m->stats.kernel_launches += 2;
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

// out += rowSums(Yt) (x) constV, for callers that computed the group part themselves
int64_t launch_lmm_const(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s) {
  if (!m->hasConst || q == 0 || m->nRows == 0) return CLA_OK;
  int64_t rc;
  if ((rc = ensure_small(m, (size_t)q * sizeof(double) + 256)) < 0) return rc;
  return launch_lmm_const_with(m, dYt, q, dOut, (double*)m->small_, s);
}

}  // namespace cla
