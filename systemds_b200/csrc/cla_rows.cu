// Row-oriented forms of the column groups, built once per handle on first use.
//
// Column plan: every column of every group as one flat record, so that a kernel needs one coalesced read per column
// instead of a group record and its column list.
//
// Row lists: the SDC and RLE groups store, per group, which rows hold which tuple. A product that forms a row's sum
// wants the opposite direction, so the groups are turned into
//   * per row: the table rows of the listed SDC tuples (a CSR over the rows; 4 B per listed row + 4 B per row), and
//   * per 64-row window: the table rows of the RLE runs that cover the window entirely, and for the others the
//     piece of the window they cover.
// Both are in the groups' list order within a row / window, so that sums over them have one fixed order. A CTA builds
// the lists of one 1024-row block (the granularity of the groups' skip indexes): a first pass counts, a scan turns
// counts into positions, a second pass fills. Rows are filled by atomics on the row's cursor and then sorted (a row
// holds at most one item per SDC group); windows are filled by a warp with a prefix sum over the groups, in order
// from the start.
#include "cla_common.cuh"
#include <algorithm>
#include <climits>
#include <cstring>
#include <cub/cub.cuh>

namespace cla {

constexpr int RL_WIN = SKIP_ROWS / WIN_ROWS;  // windows per block
constexpr int RL_THREADS = 256;

int64_t plan_alloc(Matrix* m, void** p, size_t bytes, bool needed) {
  *p = nullptr;
  if (!needed && m->planLimit >= 0 && m->planBytes + (int64_t)bytes > m->planLimit)
    return fail(CLA_ERR_NOMEM, "the handle's plan limit has no room for " + std::to_string(bytes) + " bytes");
  cudaError_t e = dev_malloc(m, p, std::max<size_t>(bytes, 16));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CLA_ERR_NOMEM, std::string("cudaMalloc row plan: ") + cudaGetErrorString(e));
  }
  m->allocs.push_back(*p);
  if (!needed) m->planBytes += (int64_t)bytes;
  m->deviceBytes += (int64_t)bytes;
  m->stats.device_bytes = m->deviceBytes;
  return CLA_OK;
}
void plan_release(Matrix* m, void* p, size_t bytes) {
  m->allocs.erase(std::remove(m->allocs.begin(), m->allocs.end(), p), m->allocs.end());
  dev_free(m, p);
  m->planBytes -= (int64_t)bytes;
  m->deviceBytes -= (int64_t)bytes;
  m->stats.device_bytes = m->deviceBytes;
}

int64_t ensure_col_plan(Matrix* m) {
  ColPlan& cp = m->cols;
  if (cp.tried) return CLA_OK;
  std::vector<ColRef> dense, all;
  for (size_t hi = 0; hi < m->hg.size(); hi++) {
    const int gi = m->regToDev[hi];
    if (gi < 0) continue;
    const DevGroup& g = m->groups[gi];
    for (int j = 0; j < g.gCols; j++) {
      ColRef r;
      r.map = g.map;
      r.mapHi = g.mapHi;
      r.src = (g.type == GT_UNC ? g.dense : g.dict) + j;
      r.kind = g.type;
      r.mapType = g.mapType;
      r.stride = g.gCols;
      r.col = m->hg[hi].cols[j];
      r.group = gi;
      r.pad = 0;
      all.push_back(r);
      if (g.type == GT_DDC || g.type == GT_UNC) dense.push_back(r);
    }
  }
  std::stable_sort(all.begin(), all.end(), [](const ColRef& a, const ColRef& b) { return a.col < b.col; });
  std::vector<int32_t> ptr((size_t)m->nCols + 1, 0);
  for (auto& r : all) ptr[r.col + 1]++;
  for (int c = 0; c < m->nCols; c++) ptr[c + 1] += ptr[c];
  // one allocation, one copy
  const size_t bd = dense.size() * sizeof(ColRef), ba = all.size() * sizeof(ColRef), bp = ptr.size() * sizeof(int32_t);
  std::vector<char> blob(bd + ba + bp);
  if (bd) memcpy(blob.data(), dense.data(), bd);
  if (ba) memcpy(blob.data() + bd, all.data(), ba);
  memcpy(blob.data() + bd + ba, ptr.data(), bp);
  void* d = nullptr;
  if (plan_alloc(m, &d, blob.size()) < 0) {
    cp.tried = true;
    return CLA_OK;
  }
  CLA_CUDA(cudaMemcpy(d, blob.data(), blob.size(), cudaMemcpyHostToDevice));
  cp.dense = (ColRef*)d;
  cp.refs = (ColRef*)((char*)d + bd);
  cp.refPtr = (int32_t*)((char*)d + bd + ba);
  cp.nDense = (int)dense.size();
  cp.nRefs = (int)all.size();
  cp.tried = cp.ok = true;
  return CLA_OK;
}

__global__ void k_sparse_vals(const DevGroup* __restrict__ groups, const int32_t* __restrict__ svOff, SparseVal* __restrict__ sv) {
  const DevGroup& g = groups[blockIdx.x];
  if (g.type != GT_SDC && g.type != GT_RLE) return;
  const int o = svOff[blockIdx.x];
  for (int k = threadIdx.x; k < g.nVals; k += blockDim.x) {
    SparseVal v;
    v.val = g.dict[(size_t)k * g.gCols];
    v.col = g.gCols == 1 ? g.cols[0] : -1;
    v.group = blockIdx.x;
    sv[o + k] = v;
  }
}

// FILL = false counts the items of every row and window, FILL = true places them (the pointers then hold positions).
template <bool FILL>
__global__ void __launch_bounds__(RL_THREADS)
k_row_lists(const DevGroup* __restrict__ groups, const int32_t* __restrict__ list, int nSdc, int nRle, int nRows,
            const int32_t* __restrict__ svOff, uint32_t* __restrict__ rowPtr, uint32_t* __restrict__ rowItems,
            uint32_t* __restrict__ fullPtr, uint32_t* __restrict__ fullItems, uint32_t* __restrict__ partPtr,
            uint2* __restrict__ partItems, uint32_t* __restrict__ sdcItems) {
  __shared__ uint32_t cnt[SKIP_ROWS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int blk = blockIdx.x, b0 = blk * SKIP_ROWS, b1 = min(nRows, b0 + SKIP_ROWS);
  if (nSdc) {
    for (int i = tid; i < SKIP_ROWS; i += RL_THREADS) cnt[i] = FILL ? rowPtr[b0 + i] : 0u;
    __syncthreads();
    for (int i = warp; i < nSdc; i += RL_THREADS / 32) {
      const int gi = list[i];
      const DevGroup& g = groups[gi];
      const uint32_t o = (uint32_t)svOff[gi];
      sdc_walk_block(g, b0, b1, [&](int row, int e) {
        const uint32_t p = atomicAdd(&cnt[row - b0], 1u);
        if (FILL) {
          const uint32_t id = (uint32_t)(g.single ? 0 : map_get(g.mapType, g.map, g.mapHi, e));
          rowItems[p] = o + id;
          if (sdcItems) sdcItems[g.listAt + e] = (uint32_t)(row - b0) | (id << 10);
        }
      });
      __syncwarp();
    }
    __syncthreads();
    if (!FILL)
      for (int i = tid; i < SKIP_ROWS; i += RL_THREADS) rowPtr[b0 + i] = cnt[i];
    else
      for (int i = tid; i < SKIP_ROWS; i += RL_THREADS) {  // list order within the row
        const uint32_t p0 = rowPtr[b0 + i], p1 = cnt[i];
        for (uint32_t a = p0 + 1; a < p1; a++) {
          const uint32_t v = rowItems[a];
          uint32_t b = a;
          for (; b > p0 && rowItems[b - 1] > v; b--) rowItems[b] = rowItems[b - 1];
          rowItems[b] = v;
        }
      }
  }
  if (nRle)
    for (int w = warp; w < RL_WIN; w += RL_THREADS / 32) {
      const int w0 = b0 + w * WIN_ROWS, w1 = min(b1, w0 + WIN_ROWS), wi = blk * RL_WIN + w;
      uint32_t nf = FILL ? fullPtr[wi] : 0u, np = FILL ? partPtr[wi] : 0u;
      for (int i0 = 0; i0 < nRle; i0 += 32) {
        // this lane's group: its runs that reach into the window
        const int i = i0 + lane;
        uint32_t f = 0, p = 0;
        int64_t ra = 0, rb = 0;
        const DevGroup* g = nullptr;
        if (i < nRle && w0 < w1) {
          g = &groups[list[nSdc + i]];
          ra = g->runSkip[blk];
          while (ra < g->nRuns && g->runs[ra].start + (int)g->runs[ra].len <= w0) ra++;
          for (rb = ra; rb < g->nRuns; rb++) {
            const RleRun R = g->runs[rb];
            if (R.start >= w1) break;
            const int a = max(R.start, w0), b = min(R.start + (int)R.len, w1);
            if (a < b) (b - a == WIN_ROWS ? f : p)++;
          }
        }
        uint32_t sf = f, sp = p;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t tf = __shfl_up_sync(0xffffffffu, sf, d), tp = __shfl_up_sync(0xffffffffu, sp, d);
          if (lane >= d) sf += tf, sp += tp;
        }
        if (FILL && g) {
          uint32_t pf = nf + sf - f, pp = np + sp - p;
          const uint32_t o = (uint32_t)svOff[list[nSdc + i]];
          for (int64_t r = ra; r < rb; r++) {
            const RleRun R = g->runs[r];
            const int a = max(R.start, w0), b = min(R.start + (int)R.len, w1);
            if (a >= b) continue;
            if (b - a == WIN_ROWS) fullItems[pf++] = o + R.k;
            else partItems[pp++] = make_uint2(o + R.k, (uint32_t)(a - w0) | ((uint32_t)(b - w0) << 8));
          }
        }
        nf += __shfl_sync(0xffffffffu, sf, 31);
        np += __shfl_sync(0xffffffffu, sp, 31);
      }
      if (!FILL && lane == 0) {
        fullPtr[wi] = nf;
        partPtr[wi] = np;
      }
    }
}

// The items alone, where nothing needs the rows' lists: a warp per group and 1024-row block. An item's place follows from
// the group's element number, so there is no counting pass.
constexpr int SDC_ITEM_VALS = 1 << 22;  // an item holds 22 bits of tuple
__global__ void __launch_bounds__(RL_THREADS) k_sdc_items(const DevGroup* __restrict__ groups, int nDev, int nRows, uint32_t* __restrict__ items) {
  const int perBlock = (nDev + RL_THREADS / 32 - 1) / (RL_THREADS / 32), blk = blockIdx.x / perBlock;
  const int gi = (blockIdx.x - blk * perBlock) * (RL_THREADS / 32) + (threadIdx.x >> 5);
  if (gi >= nDev || groups[gi].type != GT_SDC) return;
  const DevGroup& g = groups[gi];
  const int b0 = blk * SKIP_ROWS;
  uint32_t* to = items + g.listAt;
  sdc_walk_block(g, b0, min(nRows, b0 + SKIP_ROWS), [&](int row, int e) {
    to[e] = (uint32_t)(row - b0) | ((uint32_t)(g.single ? 0 : map_get(g.mapType, g.map, g.mapHi, e)) << 10);
  });
}

// -1: a group's tuples do not fit an item
int64_t sdc_items_bytes(const Matrix* m) {
  int64_t n = 0;
  for (auto& g : m->groups)
    if (g.type == GT_SDC && g.nOff > 0) {
      if (g.nVals > SDC_ITEM_VALS) return -1;
      n += g.nOff;
    }
  return n * 4;
}
void launch_sdc_items(Matrix* m, uint32_t* items, cudaStream_t s) {
  if (sdc_items_bytes(m) <= 0) return;
  const unsigned grid = (unsigned)((m->nRows + SKIP_ROWS - 1) / SKIP_ROWS) * (unsigned)((m->nDev + RL_THREADS / 32 - 1) / (RL_THREADS / 32));
  k_sdc_items<<<grid, RL_THREADS, 0, s>>>(m->dGroups, m->nDev, m->nRows, items);
  m->stats.kernel_launches++;
}

int64_t ensure_row_lists(Matrix* m, cudaStream_t s) {
  RowLists& L = m->rows;
  if (L.tried) return CLA_OK;
  L.tried = true;
  std::vector<int32_t> sdc, rle, off((size_t)std::max(m->nDev, 1), 0);
  int64_t nSv = 0;
  for (int gi = 0; gi < m->nDev; gi++) {
    const DevGroup& g = m->groups[gi];
    if (g.type == GT_SDC && g.nOff > 0) sdc.push_back(gi);
    if (g.type == GT_RLE && g.nRuns > 0) rle.push_back(gi);
    if (g.type == GT_SDC || g.type == GT_RLE) {
      off[gi] = (int32_t)std::min<int64_t>(nSv, INT32_MAX);
      nSv += g.nVals;
    }
  }
  L.nSdc = (int)sdc.size();
  L.nRle = (int)rle.size();
  L.nSv = nSv;
  if (m->nRows == 0 || (L.nSdc == 0 && L.nRle == 0)) {
    L.ok = true;
    return CLA_OK;
  }
  {  // positions are 32-bit
    int64_t listed = 0, pieces = ((int64_t)m->nRows / WIN_ROWS + 1) * L.nRle;
    for (int gi : sdc) listed += m->groups[gi].nOff;
    for (int gi : rle) pieces += 2 * m->groups[gi].nRuns;
    if (nSv > INT32_MAX || listed > INT32_MAX || pieces > INT32_MAX) return CLA_OK;
  }
  const int nBlocks = (m->nRows + SKIP_ROWS - 1) / SKIP_ROWS;
  const int64_t nRowPtr = (int64_t)nBlocks * SKIP_ROWS + 1, nWinPtr = (int64_t)nBlocks * RL_WIN + 1;
  std::vector<int32_t> list(sdc);
  list.insert(list.end(), rle.begin(), rle.end());
  // pointers, group list, table-row numbering and values in one allocation
  for (int gi : sdc)
    if (m->groups[gi].nVals > SDC_ITEM_VALS) return CLA_OK;
  const size_t bOff = ((size_t)m->nDev * 4 + 15) & ~(size_t)15, bList = (list.size() * 4 + 15) & ~(size_t)15;
  const size_t bSv = (size_t)std::max<int64_t>(nSv, 1) * sizeof(SparseVal);
  const size_t bRow = (L.nSdc ? (size_t)nRowPtr * 4 : 0), bWin = (L.nRle ? (size_t)nWinPtr * 4 : 0);
  size_t tb1 = 0, tb2 = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, tb1, (uint32_t*)nullptr, (uint32_t*)nullptr, (int)nRowPtr, s);
  cub::DeviceScan::ExclusiveSum(nullptr, tb2, (uint32_t*)nullptr, (uint32_t*)nullptr, (int)nWinPtr, s);
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  void* base = nullptr;
  const size_t bytes = al(bOff) + al(bList) + al(bSv) + al(bRow) + 2 * al(bWin) + std::max(tb1, tb2);
  if (plan_alloc(m, &base, bytes) < 0) return CLA_OK;
  char* p = (char*)base;
  L.svOff = (int32_t*)p; p += al(bOff);
  int32_t* dList = (int32_t*)p; p += al(bList);
  L.sv = (SparseVal*)p; p += al(bSv);
  if (L.nSdc) L.rowPtr = (uint32_t*)p;
  p += al(bRow);
  if (L.nRle) L.fullPtr = (uint32_t*)p;
  p += al(bWin);
  if (L.nRle) L.partPtr = (uint32_t*)p;
  p += al(bWin);
  void* tmp = p;
  CLA_CUDA(cudaMemcpyAsync(L.svOff, off.data(), (size_t)m->nDev * 4, cudaMemcpyHostToDevice, s));
  CLA_CUDA(cudaMemcpyAsync(dList, list.data(), list.size() * 4, cudaMemcpyHostToDevice, s));
  k_sparse_vals<<<m->nDev, 128, 0, s>>>(m->dGroups, L.svOff, L.sv);
  k_row_lists<false><<<nBlocks, RL_THREADS, 0, s>>>(m->dGroups, dList, L.nSdc, L.nRle, m->nRows, L.svOff, L.rowPtr, nullptr,
                                                   L.fullPtr, nullptr, L.partPtr, nullptr, nullptr);
  uint32_t tot[3] = {0, 0, 0};
  if (L.nSdc) {
    CLA_CUDA(cudaMemsetAsync(L.rowPtr + nRowPtr - 1, 0, 4, s));
    cub::DeviceScan::ExclusiveSum(tmp, tb1, L.rowPtr, L.rowPtr, (int)nRowPtr, s);
    CLA_CUDA(cudaMemcpyAsync(&tot[0], L.rowPtr + nRowPtr - 1, 4, cudaMemcpyDeviceToHost, s));
  }
  if (L.nRle) {
    CLA_CUDA(cudaMemsetAsync(L.fullPtr + nWinPtr - 1, 0, 4, s));
    CLA_CUDA(cudaMemsetAsync(L.partPtr + nWinPtr - 1, 0, 4, s));
    cub::DeviceScan::ExclusiveSum(tmp, tb2, L.fullPtr, L.fullPtr, (int)nWinPtr, s);
    cub::DeviceScan::ExclusiveSum(tmp, tb2, L.partPtr, L.partPtr, (int)nWinPtr, s);
    CLA_CUDA(cudaMemcpyAsync(&tot[1], L.fullPtr + nWinPtr - 1, 4, cudaMemcpyDeviceToHost, s));
    CLA_CUDA(cudaMemcpyAsync(&tot[2], L.partPtr + nWinPtr - 1, 4, cudaMemcpyDeviceToHost, s));
  }
  CLA_CUDA(cudaStreamSynchronize(s));
  void* items = nullptr;
  const size_t i0 = al((size_t)tot[0] * 4), i1 = al((size_t)tot[1] * 4), i2 = al((size_t)tot[2] * 8);
  const bool own = !m->sdcItemsOk;  // (the decompress may have built them already)
  if (plan_alloc(m, &items, (own ? 2 : 1) * i0 + i1 + i2) < 0) {
    plan_release(m, base, bytes);
    L.svOff = nullptr, L.sv = nullptr, L.rowPtr = L.fullPtr = L.partPtr = nullptr;
    return CLA_OK;
  }
  uint32_t* sdcItems = own ? (uint32_t*)((char*)items + i0 + i1 + i2) : nullptr;
  L.rowItems = (uint32_t*)items;
  L.fullItems = (uint32_t*)((char*)items + i0);
  L.partItems = (uint2*)((char*)items + i0 + i1);
  k_row_lists<true><<<nBlocks, RL_THREADS, 0, s>>>(m->dGroups, dList, L.nSdc, L.nRle, m->nRows, L.svOff, L.rowPtr, L.rowItems,
                                                  L.fullPtr, L.fullItems, L.partPtr, L.partItems, sdcItems);
  CLA_CUDA(cudaGetLastError());
  CLA_CUDA(cudaStreamSynchronize(s));
  if (own) {
    m->sdcItems = sdcItems;
    m->sdcItemsOk = true;
  }
  L.ok = true;
  return CLA_OK;
}

}  // namespace cla
