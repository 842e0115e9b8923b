// Shared declarations of the CLA device library: device-side group records, the host-side
// matrix object behind a cla_handle, and helpers used by every translation unit.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <memory>
#include <functional>
#include <mutex>
#include <string>
#include <vector>
#include "../../include/systemds_cla.h"
#include "cla_once.h"

namespace cla {

constexpr int SKIP_ROWS = 1024;  // granularity of the SDC / RLE skip indexes (AOffset's skip list uses ~1000)
constexpr int BITMAP_BLOCK_SZ = 65535;

enum GroupType : int { GT_DDC = 0, GT_SDC = 1, GT_RLE = 2, GT_OLE = 3, GT_UNC = 4, GT_CONST = 5, GT_EMPTY = 6 };

// Start state for decoding an offset stream at a row-block boundary: the first listed row at or
// after the boundary, its position in the map (AIterator.getDataIndex), and the stream position
// right behind it.
struct SdcSkip {
  int32_t elem;  // index of that element (== nOff when there is none)
  int32_t row;   // its row
  int64_t pos;   // index of the next delta to read
};

// One run of a value, in absolute rows (decoded from the (gap, len) pairs and merged over values).
struct RleRun {
  int32_t start;
  uint16_t len;
  uint16_t k;
};

// Device-visible record of one column group. All pointers are device addresses.
struct DevGroup {
  int32_t type;      // how products treat it: GT_DDC (also transcoded OLE), GT_SDC, GT_RLE, GT_UNC
  int32_t origType;  // the registered type
  int32_t gCols, nVals;
  int32_t mapType;
  int32_t single;  // SDCSingle*: every listed row holds tuple 0
  int32_t offType, first, last;
  int32_t inFast;  // 1: the specialised vector kernels cover this group (general kernels skip it on their request)
  int64_t mapSize, offLen, nOff, nRuns, dataLen;
  int64_t valOff;  // first row of this group's table in the per-call value arenas (sum of nVals before it)
  int64_t listAt;  // SDC: first of its listed rows in Matrix::sdcItems (sum of nOff of the SDC groups before it)
  const int32_t* cols;
  const double* dict;  // effective dictionary (default tuple subtracted), [nVals x gCols]
  const double* dictRaw;  // the dictionary as registered (== dict unless a default tuple was folded into constV)
  const void* map;
  const void* mapHi;
  const void* offData;
  const SdcSkip* skip;
  const RleRun* runs;
  const int32_t* runSkip;  // per SKIP_ROWS block: first run whose end lies behind the block start
  const int32_t* ptr;      // RLE / OLE as registered
  const uint16_t* data;
  const double* dense;  // UNC [nRows x gCols]
};

// Read one cell of a map in the reference's storage layout.
__device__ __forceinline__ int map_get(int mapType, const void* __restrict__ map, const void* __restrict__ mapHi,
                                       int64_t r) {
  switch (mapType) {
    case CLA_MAP_ZERO: return 0;
    case CLA_MAP_BIT: return (int)((((const unsigned long long*)map)[r >> 6] >> (r & 63)) & 1ULL);
    case CLA_MAP_UBYTE:
    case CLA_MAP_BYTE: return ((const uint8_t*)map)[r];
    case CLA_MAP_CHAR: return ((const uint16_t*)map)[r];
    case CLA_MAP_CHAR_BYTE: return (int)((const uint16_t*)map)[r] + ((int)((const uint8_t*)mapHi)[r] << 16);
    default: return ((const int32_t*)map)[r];
  }
}

// Warp-level decode of one SKIP_ROWS block of an offset stream: deltas are read 32 at a time,
// a warp scan turns them into rows, a ballot numbers the elements (continuation deltas carry none).
// f(row, elemIndex) is called for every listed row in [rowBegin, rowEnd).
template <class F>
__device__ __forceinline__ void sdc_walk_block(const DevGroup& g, int rowBegin, int rowEnd, F&& f) {
  const int lane = threadIdx.x & 31;
  if (g.nOff == 0) return;
  if (g.offType == CLA_OFF_SINGLE || g.offType == CLA_OFF_TWO) {
    if (lane == 0) {
      if (g.first >= rowBegin && g.first < rowEnd) f(g.first, 0);
      if (g.offType == CLA_OFF_TWO && g.last >= rowBegin && g.last < rowEnd) f(g.last, 1);
    }
    return;
  }
  const SdcSkip sk = g.skip[rowBegin / SKIP_ROWS];
  int row = sk.row;
  int elem = sk.elem;
  int64_t pos = sk.pos;
  if (elem >= g.nOff || row >= rowEnd) return;
  if (lane == 0 && row >= rowBegin) f(row, elem);
  const int maxV = g.offType == CLA_OFF_BYTE ? 255 : 65535;
  while (pos < g.offLen) {
    const int64_t i = pos + lane;
    int d = 0;
    if (i < g.offLen) d = g.offType == CLA_OFF_BYTE ? (int)((const uint8_t*)g.offData)[i] : (int)((const uint16_t*)g.offData)[i];
    const bool inb = i < g.offLen;
    int inc = inb ? (d == 0 ? maxV : d) : 0;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, inc, s);
      if (lane >= s) inc += t;
    }
    const bool isElem = inb && d != 0;
    const unsigned bal = __ballot_sync(0xffffffffu, isElem);
    const int myRow = row + inc;
    const int myElem = elem + __popc(bal & ((2u << lane) - 1u));
    if (isElem && myRow >= rowBegin && myRow < rowEnd) f(myRow, myElem);
    row += __shfl_sync(0xffffffffu, inc, 31);
    elem += __popc(bal);
    pos += 32;
    if (row >= rowEnd) break;
  }
}

// Host-side group as registered (arrays copied from the caller).
struct HostGroup {
  int type = GT_DDC;
  std::vector<int32_t> cols;
  int nVals = 0;
  std::vector<double> dict;
  std::vector<double> def;  // default tuple (empty = zeros)
  int mapType = CLA_MAP_ZERO;
  int64_t mapSize = 0;
  std::vector<uint8_t> map, mapHi;  // raw bytes
  bool single = false;
  int offType = CLA_OFF_EMPTY, first = 0, last = 0;
  int64_t offLen = 0, nOff = 0;
  std::vector<uint8_t> offData;
  std::vector<int32_t> ptr;
  std::vector<uint16_t> data;
  std::vector<double> dense;
  // Groups registered from device memory (cla_add_group_ddc_dev / cla_add_group_uncompressed_dev): the caller's
  // buffer, read once at cla_finalize and copied device to device.
  const void* devMap = nullptr;
  const double* devDense = nullptr;
  int devSrcDevice = -1;
};

struct FastPlan;  // plans of the specialised DDC kernels (cla_fast.cu)

// One column of one product group, flat (built once per handle, cla_rows.cu).
struct ColRef {
  const void* map;
  const void* mapHi;
  const double* src;  // dictionary (or dense block) + position of the column inside the group
  int32_t kind;       // GT_DDC, GT_UNC, GT_SDC or GT_RLE
  int32_t mapType;
  int32_t stride;     // columns of the group
  int32_t col;        // matrix column
  int32_t group;      // device group index
  int32_t pad;
};
// The tuples of the SDC / RLE groups are numbered through ("sparse table rows", list order, svOff[group] first).
struct SparseVal {
  double val;     // the dictionary value, single-column groups
  int32_t col;    // their matrix column; -1: a group of several columns
  int32_t group;  // device group index
};
// Row-oriented forms of the SDC and RLE groups (cla_rows.cu).
constexpr int WIN_ROWS = 64;
struct RowLists {
  bool tried = false, ok = false;
  int nSdc = 0, nRle = 0;           // groups with listed rows / with runs
  int64_t nSv = 0;                  // sparse table rows
  int32_t* svOff = nullptr;         // [nDev]
  SparseVal* sv = nullptr;          // [nSv]
  uint32_t* rowPtr = nullptr;       // [nBlocks * 1024 + 1]: first item of a row; items = table rows of its listed SDC tuples
  uint32_t* rowItems = nullptr;
  uint32_t* fullPtr = nullptr;      // [nBlocks * 16 + 1]: runs that cover a whole 64-row window: their table rows
  uint32_t* fullItems = nullptr;
  uint32_t* partPtr = nullptr;      // runs that cover part of a window: table row, first row | end row << 8 in the window
  uint2* partItems = nullptr;
};
// One column of a group the column-per-lane kernels do not take, as the left product walks it (cla_rest.cu).
struct RestTask {
  const double* src;   // dictionary + position of the column
  const void* a;       // SDC: items; RLE: runs; dense map: map
  const void* b;       // SDC: skip entries; RLE: first run of every block; dense map: high bytes
  int64_t n;           // SDC: listed rows; RLE: runs; dense map: tuples
  int32_t kind, mapType, stride, col;
};
struct RestPlan {
  bool tried = false, ok = false;
  int nTasks = 0, nUnc = 0, nDense = 0;
  int nTable = 0, tableVals = 0;  // 16-bit map columns whose tables fit shared memory (the last tasks), longest table
  RestTask* tasks = nullptr;      // SDC, RLE and remaining dense-map columns
  ColRef* dense = nullptr;        // the remaining dense-map columns, list order
  std::vector<int> unc;           // device group indices of the uncompressed groups
};
struct DecPlan {  // column-per-lane decompress (cla_generic.cu)
  int warps = 0;  // of a CTA; 0: the tile kernel is the better one
  bool again = false;    // the block has been decompressed before
  void* cols = nullptr;  // records, built on first use
  size_t tables = 0, smem = 0;  // bytes of tables, and with the cells behind them
};
struct ColPlan {
  bool tried = false, ok = false;
  int nDense = 0, nRefs = 0;
  ColRef* dense = nullptr;     // dense-map and uncompressed columns, list order
  ColRef* refs = nullptr;      // every column of every group, sorted by matrix column (list order within a column)
  int32_t* refPtr = nullptr;   // [nCols + 1]
};
// Where a host-buffer call's result goes when it is small: pinned memory the kernels write straight into.
struct alignas(16) Mailbox {  // one 16-byte store: the flag never arrives before what it stands for
  volatile uint32_t flag;
  int32_t err;
  unsigned long long nnz;
};
constexpr size_t MAIL_HEAD = 256, MAIL_IN = 64 * 1024, MAIL_OUT = 128 * 1024;
// Given to the last kernel of a small host-buffer call: it counts the non-zeros and raises the flag.
struct Finish {
  Mailbox* box = nullptr;             // null: not wanted
  unsigned long long* nnz = nullptr;  // device counters, zero between calls
  unsigned int* ticket = nullptr;
  int32_t* err = nullptr;             // the handle's self-check word
  uint32_t seq = 0;
};
struct WidePlan;  // plan of the wide right product (cla_wide.cu)
struct SplitPlan; // of the self product in 8-bit digits (cla_split.cu)
struct HostStage; // pinned ring for operands in pageable host memory (cla_hostcopy.cu)

struct Matrix;
struct Matrix {
  // A block returned by cla_rmm_overlapping shares the index structures of the block it was computed from; it
  // keeps that block alive (parent), and a parent destroyed before its children only leaves the handle table: its
  // device memory is released with the last child (children, zombie; both guarded by the parent's mutex).
  std::shared_ptr<Matrix> parent;
  int children = 0;
  bool zombie = false;
  int32_t nRows = 0, nCols = 0;
  bool overlapping = false;
  bool finalized = false;
  int device = -1;
  std::mutex mu;
  std::vector<HostGroup> hg;   // cleared after finalize (records kept, arrays dropped)
  std::vector<DevGroup> groups;  // host copy of the device records (product groups only)
  std::vector<int> regToDev;     // registered group index -> index in groups (-1: const / empty)
  DevGroup* dGroups = nullptr;
  int nDev = 0;
  int64_t totalVals = 0;         // sum of nVals over dictionary groups
  std::vector<double> constV;    // host copy
  std::vector<double> colMin, colMax;  // per-column extrema over the compressed groups, dictionary-based (cla_agg.cu)
  bool multiCover = false;             // some column is held by more than one registered group (e.g. FOR group + reference)
  double* dConstV = nullptr;     // [nCols]
  void* dDenseCols = nullptr;    // list of dense-operand columns for the tensor-core RMM (built on first use)
  int nDenseCols = 0;
  bool denseColsBuilt = false;
  int32_t* dSparseIdx = nullptr;  // device group indices of the SDC groups with listed rows and RLE groups with runs, list order
  int nSparse = 0;
  // the other groups by kind, list order: dense-map groups (all, then those the specialised kernels do not take), uncompressed
  int32_t* dDdcIdx = nullptr;
  int32_t* dDdcRestIdx = nullptr;
  int32_t* dUncIdx = nullptr;
  int nDdc = 0, nDdcRest = 0, nUnc = 0;
  bool sparseListBuilt = false;
  int32_t* dColSrc = nullptr;    // [nCols][2]: dense-map / uncompressed group holding the column and the position in it (-1: none)
  bool colSrcValid = false;      // false when some column is held by more than one such group (overlapping input)
  bool hasConst = false;
  std::vector<void*> allocs;     // everything cudaMalloc'ed for the groups
  int64_t deviceBytes = 0, indexBytes = 0;
  int64_t planBytes = 0, planLimit = -1;  // plans built on first use: bytes held, bytes allowed (-1: no limit)
  // growable scratch (value arenas, partial results, host staging)
  void* scratch = nullptr;
  size_t scratchBytes = 0;
  void* scratch2 = nullptr;
  size_t scratch2Bytes = 0;
  void* small_ = nullptr;  // small per-call vectors (row sums of the left operand)
  size_t smallBytes = 0;
  void* io = nullptr;  // device staging for host-buffer calls
  size_t ioBytes = 0;
  int32_t* dErr = nullptr;  // device self-check word
  cudaStream_t stream = nullptr;
  cudaStream_t copyStream = nullptr;  // uploads overlapped with kernels in the host-buffer left product
  cudaEvent_t copyDone[16] = {};  // one per row range of the pipelined host-buffer left product
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // Every product call uses the handle's one set of scratch buffers. A call that arrives on another stream than
  // the previous one first waits for `lastDone` (recorded when the previous call had enqueued its work), so two
  // calls on one handle never overlap on the GPU even when their streams would allow it.
  cudaEvent_t lastDone = nullptr;
  cudaStream_t lastStream = nullptr;
  bool lastValid = false;
  FastPlan* fast = nullptr;
  // listed rows of the SDC groups, group by group in element order: row in its 1024-row block | tuple << 10
  uint32_t* sdcItems = nullptr;
  bool sdcItemsOk = false;
  RowLists rows;
  ColPlan cols;
  RestPlan rest;
  DecPlan dec;
  WidePlan* wide = nullptr;
  SplitPlan* split = nullptr;
  HostStage* hostStage = nullptr;
  char* mail = nullptr;          // pinned: Mailbox, inputs, outputs (small host-buffer calls)
  unsigned long long* dFin = nullptr;  // device counters of Finish
  uint32_t mailSeq = 0;
  bool elapsedPending = false;   // ev0 / ev1 bracket the last host-buffer call
  bool profile = false;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> profEvents;  // ring of event pairs
  size_t profUsed = 0;
  cla_stats stats{};
  int smCount = 148;
};

// error plumbing --------------------------------------------------------------------------------
void set_error(const std::string& msg);
int64_t fail(int64_t code, const std::string& msg);
#define CLA_CUDA(expr)                                                                              \
  do {                                                                                              \
    cudaError_t e_ = (expr);                                                                        \
    if (e_ != cudaSuccess)                                                                          \
      return ::cla::fail(CLA_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_));         \
  } while (0)

// Lets kernels take `bytes` of dynamic shared memory; `device` is the current device.
template <class... K>
inline int64_t allow_smem(OncePerDevice& once, int device, size_t bytes, K... kernels) {
  return once(device, [&]() -> int64_t {
    cudaError_t e = cudaSuccess;
    ((e == cudaSuccess ? (void)(e = cudaFuncSetAttribute(kernels, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)) : (void)0), ...);
    return e == cudaSuccess ? CLA_OK : fail(CLA_ERR_CUDA, std::string("shared memory of a kernel: ") + cudaGetErrorString(e));
  });
}

// profiling brackets around the dominant kernel of a product call (no-ops unless m->profile)
void prof_begin(Matrix* m, cudaStream_t s);
void prof_end(Matrix* m, cudaStream_t s);
void prof_collect(Matrix* m);

int64_t order_begin(Matrix* m, cudaStream_t s);  // see Matrix::lastDone
int64_t order_end(Matrix* m, cudaStream_t s);
// device memory of a handle, from the device's pool (cla_finalize.cu); free only what no stream uses any more
cudaError_t dev_malloc(const Matrix* m, void** p, size_t bytes);
void dev_free(const Matrix* m, void* p);
int64_t ensure_scratch(Matrix* m, size_t bytes);
int64_t ensure_scratch2(Matrix* m, size_t bytes);
int64_t ensure_io(Matrix* m, size_t bytes);
int64_t ensure_small(Matrix* m, size_t bytes);
// Transfers between pageable host memory and the device through the handle's pinned ring (cla_hostcopy.cu).
// host_copy_staged: whether a transfer of `bytes` at `host` should take them (large, pageable, ring available).
bool host_copy_staged(Matrix* m, const void* host, size_t bytes);
int64_t host_to_device_staged(Matrix* m, void* dDst, const void* host, size_t bytes, cudaStream_t cs,
                              const std::function<int64_t(size_t)>& enqueued);
int64_t device_to_host_staged(Matrix* m, void* host, const void* dSrc, size_t bytes, cudaStream_t s);
void host_stage_free(Matrix* m);
int64_t ensure_sparse_list(Matrix* m);  // Matrix::dSparseIdx (cla_generic.cu)

int64_t ensure_col_plan(Matrix* m);                        // Matrix::cols; cols.ok tells whether it exists
int64_t sdc_items_bytes(const Matrix* m);                  // size of Matrix::sdcItems; -1: they cannot exist
void launch_sdc_items(Matrix* m, uint32_t* items, cudaStream_t s);  // fills them into `items`
int64_t ensure_row_lists(Matrix* m, cudaStream_t s);       // Matrix::rows and sdcItems; rows.ok tells whether they exist
// The groups the specialised kernels leave (cla_rest.cu): 1 = done, 0 = not covered (the general kernels then run)
int64_t rest_rmm(Matrix* m, const double* dV, double* dOut, const double* dW, cudaStream_t s, bool addTo);
int64_t rest_lmm(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s);
// Device memory of a plan built on first use, kept until the handle goes. CLA_ERR_NOMEM where the device or the handle's
// limit has no room: the product then takes the kernels that need no plan. `needed`: no kernel does without it, no limit.
int64_t plan_alloc(Matrix* m, void** p, size_t bytes, bool needed = false);
void plan_release(Matrix* m, void* p, size_t bytes);  // gives one back early; no stream may still use it
int64_t wide_rmm(Matrix* m, const double* dV, int vCols, double* dOut, cudaStream_t s);  // cla_wide.cu: 1 = done, 0 = not covered
void wide_plan_free(Matrix* m);
// t(X) X of many columns in 8-bit digits (cla_split.cu): 1 = done, 0 = not covered
int64_t split_tsmm(Matrix* m, double* dOut, cudaStream_t s);
void split_plan_free(Matrix* m);
// Rows [r0, r1) straight to digit planes, a thread per column (cla_generic.cu); whether the block's columns suit that. refused: the
// planes are the guard's, and the word is set where a value has no digits
bool split_cols_covers(Matrix* m, cudaStream_t s);
int64_t launch_split_cols(Matrix* m, int r0, int r1, const int32_t* expo, int64_t halves, uint8_t* planes, int32_t* refused, cudaStream_t s);
// Short blocks (cla_small.cu): one kernel per product, every group type. 1 = done, 0 = not covered
bool small_block(const Matrix* m);
int64_t small_rmm(Matrix* m, const double* dV, int vCols, double* dOut, const double* dW, cudaStream_t s, const Finish& fin,
                  const double* hostV = nullptr);
int64_t small_lmm(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s, const Finish& fin);
int64_t launch_finish(Matrix* m, const double* d, int n, double* out, cudaStream_t s, const Finish& fin);
// Pinned mailboxes for small host-buffer calls, shared by all handles (cla_hostcopy.cu); null when none can be had
char* mailbox_take();
void mailbox_give(char* p);

// launchers implemented in the kernel translation units; all enqueue on `s` and return CLA_OK or an error.
// X v over the groups the specialised kernels leave (all without them), scaled by dW (null: not)
int64_t launch_rmm(Matrix* m, const double* dV, const double* dW, double* dOut, cudaStream_t s, bool afterFast = false);
int64_t launch_rmm_dmma(Matrix* m, const double* dV, int vCols, double* dOut, cudaStream_t s);
int64_t launch_lmm(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s, bool afterFast = false);
void minmax_of_group(const HostGroup& hg, int nRows, std::vector<double>& colMin, std::vector<double>& colMax);
int64_t col_minmax(Matrix* m, std::vector<double>& lo, std::vector<double>& hi, cudaStream_t s);
int64_t row_minmax(Matrix* m, int wantMax, double* dOut, cudaStream_t s);
int64_t launch_tsmm(Matrix* m, double* dOut, cudaStream_t s);
int64_t launch_tmm(Matrix* left, Matrix* right, double* dOut, cudaStream_t s);  // t(left) %*% right, both compressed
// products on the dictionaries of two all-dense-map operands (cla_pairs.cu)
bool pairs_eligible(const Matrix* L, const Matrix* R, bool self);
int64_t launch_pairs(Matrix* L, Matrix* R, bool self, double* dOut, cudaStream_t s);
int64_t launch_decompress(Matrix* m, double* dOut, cudaStream_t s);
void decomp_shape(Matrix* m, const int32_t* colSrc);  // Matrix::dec; colSrc: [nCols][2], host copy of Matrix::dColSrc
// X %*% V kept compressed: fills `child` (fresh Matrix) with groups that alias m's index structures (cla_generic.cu)
int64_t make_overlapping(Matrix* m, Matrix* child, const double* dV, int vCols, cudaStream_t s);
int64_t init_device_state(Matrix* m);  // stream, events, error word of a Matrix whose device is set (cla_finalize.cu)
int64_t launch_decompress_range(Matrix* m, int r0, int r1, double* dOut, cudaStream_t s, size_t ld = 0);  // ld 0: nCols
int64_t launch_group_decode(Matrix* m, int devGroup, int32_t* dIds, cudaStream_t s);
int64_t launch_group_counts(Matrix* m, int devGroup, unsigned long long* dCounts, cudaStream_t s);
int64_t launch_count_nnz(Matrix* m, const double* d, int64_t n, unsigned long long* dCount, cudaStream_t s);
int64_t launch_scale_rows(Matrix* m, double* dU, const double* dW, int64_t n, cudaStream_t s);

// finalize-time device work (cla_finalize.cu)
int64_t finalize_device(Matrix* m);
// fast paths (cla_fast.cu): return 1 if they handled the whole product, 2 if they handled the groups marked inFast
// (the caller then runs the general launcher with afterFast = true), 0 if not applicable, <0 on error
int64_t fast_plan_build(Matrix* m);
void fast_plan_free(Matrix* m);
bool fast_plan_ok(const Matrix* m);       // some or all groups are covered by the specialised kernels
bool fast_plan_partial(const Matrix* m);  // ... some but not all
// dW: null, or factors applied to the rows (0 is returned where the plan does not cover every group)
int64_t fast_rmm_vec(Matrix* m, const double* dV, double* dOut, const double* dW, cudaStream_t s, int64_t stride = 1);
int64_t fast_chain(Matrix* m, const double* dV, const double* dW, double* dOut, double* dU, cudaStream_t s);
int64_t fast_lmm_vec(Matrix* m, const double* dY, double* dOut, cudaStream_t s);
int64_t fast_lmm_rows(Matrix* m, const double* dY, size_t pitch, int q, double* dOut, cudaStream_t s);  // q left rows
int64_t fast_decompress(Matrix* m, int r0, int r1, double* dOut, cudaStream_t s, size_t ld);  // 1 = done, 0 = not covered
int64_t fast_lmm_vec_host(Matrix* m, const double* hostY, double* dY, double* dOut, cudaStream_t s);
int64_t fast_lmm_vec_noalloc(Matrix* m, const double* dY, double* dOut, cudaStream_t s);

}  // namespace cla
