// Specialised vector products for matrices whose product groups are (all or in part) dense-map (DDC) groups with
// at most 256 dictionary tuples and one byte per map cell -- the shape of the headline workloads
// (X %*% v, t(y) %*% X and the two passes of t(X) %*% (X %*% v)).
//
// The kernels are bound by shared-memory lookups (one 8-byte read per lookup, 16 per clock and SM), so the layout makes
// those reads bank-conflict free: a lane owns a *column slot*, not rows. Tables are interleaved 16 slots wide, one such
// "unit" after the other (entry k of slot s of a unit at byte k*128 + s*8), so lane s only ever touches bank pair s
// whatever the ids are. The two half-warps work on different 16-row blocks of the same slots. The maps are kept in a
// second, interleaved form (16 slots x 16 rows of ids: one 128-bit load per lane and block), and the address of an
// entry is one dp4a of the id word (byte * 128 + table base).
//
//  * k_lmm_vec: t(y) X, slot = matrix column, table = its dictionary column.
//  * k_rmm_vec<false>: X v, the same slots and tables; the lane multiplies by its column's v on the fly.
//  * k_chain_vec: t(X) (w * (X v)) in one pass over the maps, for matrices of up to 112 columns.
//  * k_rmm_vec<true>: X v on joint slots, when dictionaries are small: several groups share a slot whose one-byte map
//    holds their joint id (mixed radix, at most 256 joint tuples; combined once at plan time) and whose table, built by
//    each CTA from v, holds the sum of their terms: one byte of map and one lookup for two to eight cells.
//
// Dictionary tables are staged into shared memory with TMA bulk copies (cp.async.bulk + mbarrier, no multicast).
#include "cla_common.cuh"
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>

namespace cla {

int64_t launch_lmm_const(Matrix* m, const double* dYt, int q, double* dOut, cudaStream_t s);  // cla_generic.cu
int64_t launch_lmm_const_with(Matrix* m, const double* dYt, int q, double* dOut, double* sums, cudaStream_t s);

constexpr int FAST_MIN_ROWS = 4096;
constexpr int SMEM_MAX = 227 * 1024;

// ---- plan ----
// Warps per CTA (one CTA per SM). k_lmm_vec: 12 where a CTA has five units or more (10M x 200, 7 + 6 units: 8 / 10 / 12 / 14 / 16 warps
// 615 / 609 / 562 / 658 / 577 us; 16 and 14 leave 128 registers), 16 where fewer (300,001 x 60, 4 units: 16.4 against 17.0 with 12).
__host__ __device__ constexpr int lmm_warps(int units) { return units > 4 ? 12 : 16; }
constexpr int LMM_MAXW = 16;
// k_rmm_vec: 8 warps, whose 255 registers hold the next step's ids as well (1,250,000 x 1000: 402 us; 16 warps without them 409, 10 / 12 / 16 with
// them 679 / 474 / 563, they spill; 2M x 112: 72.9, 77.3 with 16). On joint slots 16 warps (1M x 100 of 16 values: 32 us; with the next
// step's ids 39).
constexpr int RB_W = 8, RBJ_W = 16;
constexpr int LMM_MAX_UNITS = 7;      // 16-column table units per CTA (7 x 32 KB at 256 tuples)
constexpr int LMM_PART = LMM_MAX_UNITS * 16;  // partial sums a CTA writes
constexpr int LMM_STEP = 64;          // rows per warp step (32 per half-warp)

struct LmmChunk {
  int unit0, nUnits;     // units of 16 column slots
  int nk[LMM_MAX_UNITS]; // table depth (max tuples) of each unit
  int64_t tblOff;        // offset in the table image (doubles)
  int tblDoubles;
  int cta0, nCta;        // CTA range of the launch that works on this chunk
};

// A joint slot: groups g0..gm-1 of a row with ids a0..am-1 address entry a0 + n0 * (a1 + n1 * (...)).
constexpr int JS_MAX = 8;
struct JointSlot {
  int32_t n;              // groups (0: unused slot)
  int32_t total;          // joint tuples
  int32_t split, nLo;     // groups 0..split-1 are the low part of the joint id, nLo tuples
  int32_t group[JS_MAX];  // device group indices
  int32_t nv[JS_MAX];
};
// One term D_g[a] v of a slot's table, its groups one after the other: a value times v[col], or for a group of several
// columns (gCols > 0) the tuple at dict.
struct JointTerm {
  union {
    double val;
    const double* dict;
  };
  union {
    int64_t col;  // -1: behind the slot's last term
    const int32_t* cols;
  };
};
constexpr int JOINT_UNITS = 6;  // units per chunk, at most
// So many slots behind the last whole unit go by rows instead of taking a unit. 1M rows of 16 values, us, by rows / as a unit: 98 columns (a tail of one) 37.5 / 38.9, 100 (two)
// 38.3 / 38.9, 36 (two) 26.6 / 28.7, 102 (three) 38.9 / 38.9, 104 (four) 38.9 / 38.9, 108 (six) 39.2 / 38.9, 112 (eight) 40.5 / 38.9.
constexpr int JOINT_TAIL = 4;
struct FastPlan {
  bool ok = false;
  bool partial = false;      // only some groups are covered; the general kernels add the rest
  bool uniqueCols = true;    // no column in two slots
  int nUnits = 0, nSlots = 0;  // column slots in use; padded to whole units
  int nU16 = 0;                // units of 16 slots
  std::vector<LmmChunk> lchunks;       // decompress: units per CTA fixed at plan time
  LmmChunk* dLChunks = nullptr;
  int lmmGrid = 0;
  std::vector<int> unitNk;             // table depth of each unit
  std::vector<int64_t> unitOff;        // its table in the image (doubles)
  int2* dUnits = nullptr;              // {offset / 16, depth} of each unit
  const uint8_t** dSlotMap = nullptr;  // [nSlots] column-major byte maps (plan order)
  uint8_t* dLmmMaps = nullptr;         // the same maps interleaved (see k_lmm_interleave)
  int64_t nRB = 0;                     // 16-row blocks per slot in that layout (padded to whole 64-row steps)
  int* dSlotCol = nullptr;             // [nSlots] output column or -1
  int* dBareCols = nullptr;            // columns without a slot
  int nBare = 0;
  double* dLmmTables = nullptr;        // image of all tables
  size_t imageDoubles = 0;
  // X v on joint slots
  int nJU16 = 0;                       // 0: not worth it, the column slots serve X v too
  int jTail = 0;                       // slots of the last unit that go by rows (0: it is a unit like the others)
  int jParts = 0;                      // sums of parts of a slot, at most
  JointSlot* dJSlots = nullptr;        // [nJU16 * 16]
  JointTerm* dJTerms = nullptr;        // [nJU16][jTerms][16]
  int* dJTermCols = nullptr;           // the same places: columns of the group, 0: one
  int jTerms = 0, jJoinTerms = 0;      // terms of a slot, of one of two or more groups, at most
  std::vector<int> jNk;
  int2* dJUnits = nullptr;
  uint8_t* dJMaps = nullptr;
  std::vector<void*> allocs;
};

// --------------------------------------------------------------------------------------------------
// TMA bulk copy global -> shared, completion on an mbarrier; bounded wait.
// --------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Copies `bytes` (multiple of 16, both addresses 16-byte aligned) and waits. Returns false on timeout.
__device__ __forceinline__ bool tma_load_to_smem(void* dst, const void* src, uint32_t bytes, uint64_t* mbar) {
  const uint32_t bar = smem_u32(mbar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    const uint32_t CH = 32768;
    for (uint32_t off = 0; off < bytes; off += CH) {
      const uint32_t sz = min(CH, bytes - off);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       smem_u32((char*)dst + off)),
                   "l"((const char*)src + off), "r"(sz), "r"(bar)
                   : "memory");
    }
  }
  uint32_t done = 0;
  for (int it = 0; it < (1 << 22) && !done; it++) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(0u)
        : "memory");
  }
  // one verdict for the whole CTA (also the barrier that publishes the data to every thread)
  return __syncthreads_and(done != 0) != 0;
}

// The same copy for kernels that reload the buffer several times: the barrier is initialised once and each use
// waits on the next phase parity. The caller must have synchronised the CTA (all reads of the old contents done)
// before calling; the issuing thread then orders those generic-proxy reads before the async-proxy writes.
__device__ __forceinline__ void tma_barrier_init(uint64_t* mbar) {
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
}
__device__ __forceinline__ bool tma_reload(void* dst, const void* src, uint32_t bytes, uint64_t* mbar, uint32_t parity) {
  const uint32_t bar = smem_u32(mbar);
  if (threadIdx.x == 0) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    const uint32_t CH = 32768;
    for (uint32_t off = 0; off < bytes; off += CH) {
      const uint32_t sz = min(CH, bytes - off);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       smem_u32((char*)dst + off)),
                   "l"((const char*)src + off), "r"(sz), "r"(bar)
                   : "memory");
    }
  }
  uint32_t done = 0;
  for (int it = 0; it < (1 << 22) && !done; it++) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
  }
  return __syncthreads_and(done != 0) != 0;
}

// bytes (a multiple of 16) from p (aligned to 16) to L2
__device__ __forceinline__ void l2_fetch(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes));
}

__device__ __forceinline__ double lds_f64(uint32_t addr) {
  double v;
  asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr));
  return v;
}
// Address of the table entry of byte i of an id word: base + id * 128, one instruction. (Shift, mask and add took three;
// with 16 lookups per clock and SM the issue slots were the next limit.)
// (As asm: the intrinsic with a constant operand is turned back into byte extractions, hoisted and spilled.)
__device__ __forceinline__ uint32_t entry_at(uint32_t w, int i, uint32_t base) {
  uint32_t a;
  asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(a) : "r"(w), "r"(0x80u << (8 * i)), "r"(base));
  return a;
}

__device__ __forceinline__ uint32_t byte_x128(uint32_t w, int i) {  // (byte i of w) << 7
  return i == 0 ? (w << 7) & 0x7F80u : (i == 3 ? (w >> 17) & 0x7F80u : (w >> (8 * i - 7)) & 0x7F80u);
}

__device__ __forceinline__ void dmma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

constexpr int VSTEP = 32;  // rows of a warp step: one 16-row block per half-warp

// --------------------------------------------------------------------------------------------------
// LMM: t(y) X. The grid is cut into chunks of U units; a chunk's CTAs split the rows. A lane needs the y of every row of its
// half-warp's block, multiplied into NU accumulators. It loads those of the rows 4 j + t and the FP64 tensor core, idle otherwise, hands them
// round: m8n8k4 with A[m][k] = y of row 4 j + k of the half-warp of m and a 0 / 1 matrix that picks two k's gives two rows to every lane.
// Eight bytes to 32 lanes are two wavefronts of the pipe that bounds this kernel, so loads of every row (128 bits, uniform per
// half-warp) were 32 of the 284 wavefronts of a step of seven units, eight now. The CTA's partial sums go to `partial`.
// k_lmm_final adds them up in a fixed order, a CTA per 16 columns, resident before the last CTA ends (programmatic
// dependent launch), and stores the result: nothing to clear beforehand. (Left to the last CTA of a chunk, without a second
// launch: 18.2 instead of 14.3 us for the chain on 50,000 x 100, 17.6 instead of 14.2 for t(y) X on 250,000 x 40 -- one
// CTA reads 148 partial rows too slowly.)
// Measured (10M x 200, 256 values): 562 us, 3.7 TB/s, 577 with 16 warps; 634 with y loaded row by row, 685 for the one-row-step form before that, with
// three instructions per address, a clear and a separately launched sum. 625,000 x 1000: 208 -> 187.
// 100,000 x 500: 36.9 -> 30.5 us, 5000 x 500: 15.4 -> 10.4.
// --------------------------------------------------------------------------------------------------
struct LmmArgs {
  const int2* units;           // {table offset / 16, depth}
  const uint8_t* imaps;
  int64_t nRB;
  const double* tables;
  const int* slotCol;
  const double* y;
  int nRows, nU16, U, nChunks;
  int ctaFull, ctaLast;        // CTAs of a chunk of U units, of the last chunk
  int64_t stepBegin, stepEnd;  // warp steps of this launch
  double* partial;             // [parts][gridDim.x][LMM_PART + 1] (the last: sum of y)
  int part, parts;             // this launch's part; parts > 0: it is the last one, k_lmm_final follows
  const double* constV;        // null: none
  const int* bareCols;
  int nBare;
  int addTo;                   // columns may repeat: add with atomics to a cleared result
  double* out;
  int32_t* err;
};

// Adds up the partial sums of unit `u` of a chunk, by one CTA of LMM_FT threads: 32 groups of 16 lanes (a lane per
// column) take every 32nd partial sum, then a tree over the groups: a fixed order.
constexpr int LMM_FT = 512;
constexpr int LMM_FIN = (LMM_FT / 16) * 17 + LMM_FT / 32;  // doubles of shared memory it needs
__device__ __forceinline__ void lmm_finish(const LmmArgs& A, int chunk, int cta0, int nCta, int grid, int u, bool withBare,
                                           double* sm) {
  double(*red)[17] = (double(*)[17])sm;
  double* yred = sm + (LMM_FT / 16) * 17;
  const int tid = threadIdx.x, col = tid & 15, sub = tid >> 4;
  const int n = A.parts * nCta;
  double s = 0.0, ys = 0.0;
  for (int i = sub; i < n; i += LMM_FT / 16) {
    const int p = i / nCta, b = i - p * nCta;
    s += __ldcg(A.partial + ((size_t)p * grid + cta0 + b) * (LMM_PART + 1) + u * 16 + col);
  }
  red[sub][col] = s;
  if (A.constV) {
    for (int i = tid; i < n; i += LMM_FT) {
      const int p = i / nCta, b = i - p * nCta;
      ys += __ldcg(A.partial + ((size_t)p * grid + cta0 + b) * (LMM_PART + 1) + LMM_PART);
    }
    for (int d = 16; d; d >>= 1) ys += __shfl_xor_sync(0xffffffffu, ys, d);
    if ((tid & 31) == 0) yred[tid >> 5] = ys;
  }
  __syncthreads();
  for (int h = LMM_FT / 32; h; h >>= 1) {
    if (sub < h) red[sub][col] += red[sub + h][col];
    __syncthreads();
  }
  if (A.constV) {
    ys = 0.0;
    for (int w = 0; w < LMM_FT / 32; w++) ys += yred[w];
  }
  if (tid < 16) {
    const int c = A.slotCol[(chunk * A.U + u) * 16 + tid];
    if (c >= 0) {
      if (A.addTo) atomicAdd(&A.out[c], red[0][tid]);
      else A.out[c] = A.constV ? fma(ys, A.constV[c], red[0][tid]) : red[0][tid];
    }
  }
  if (withBare && chunk == 0 && !A.addTo)  // columns of constant groups, and those the general kernels will add to
    for (int i = tid; i < A.nBare; i += LMM_FT) {
      const int c = A.bareCols[i];
      A.out[c] = A.constV ? ys * A.constV[c] : 0.0;
    }
}

// grid: units
__global__ void __launch_bounds__(LMM_FT) k_lmm_final(const __grid_constant__ LmmArgs A, int grid) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int chunk = blockIdx.x / A.U, u = blockIdx.x - chunk * A.U;
  __shared__ double sm[LMM_FIN];
  lmm_finish(A, chunk, chunk * A.ctaFull, chunk == A.nChunks - 1 ? A.ctaLast : A.ctaFull, grid, u, u == 0, sm);
}

template <int NU, int LMM_W>
__device__ __forceinline__ void lmm_vec_body(const LmmArgs& A, int chunk, int cta0, int nCta, unsigned char* smraw, uint64_t* mbar) {
  constexpr int LMM_T = LMM_W * 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int slot = lane & 15, half = lane >> 4;
  const int unit0 = chunk * A.U;
  double* mine = A.partial + ((size_t)A.part * gridDim.x + blockIdx.x) * (LMM_PART + 1);
  const int2 first = A.units[unit0], last = A.units[unit0 + NU - 1];
  const uint32_t bytes = (uint32_t)(last.x + last.y - first.x) * 128u;
  bool ok = tma_load_to_smem(smraw, A.tables + (size_t)first.x * 16, bytes, mbar);
  if (!ok) {
    // the tables never arrived: flag it, and make the failure visible in the result as well (a device-buffer caller
    // only sees the error word at its next cla_stats_get)
    if (tid == 0) atomicExch(A.err, 101);
    for (int u = tid; u <= LMM_PART; u += LMM_T) mine[u] = __longlong_as_double(0x7ff8000000000000ll);
  } else {
    uint32_t tb[NU];
#pragma unroll
    for (int u = 0; u < NU; u++) tb[u] = smem_u32(smraw) + (uint32_t)(A.units[unit0 + u].x - first.x) * 128u + slot * 8;
    const uint8_t* mp = A.imaps + (size_t)unit0 * A.nRB * 256 + half * 256 + slot * 16;
    const size_t ustr = (size_t)A.nRB * 256;
    double acc[NU], ysum = 0.0;
#pragma unroll
    for (int u = 0; u < NU; u++) acc[u] = 0.0;
    const int64_t nSteps = A.stepEnd - A.stepBegin;
    const int c = blockIdx.x - cta0;
    const int64_t s0 = A.stepBegin + nSteps * c / nCta, s1 = A.stepBegin + nSteps * (c + 1) / nCta;
    const int g = lane >> 2, t = lane & 3;
    const double even = t == (g & 1) ? 1.0 : 0.0, odd = t == 2 + (g & 1) ? 1.0 : 0.0;  // rows 0, 1 and 2, 3 of four
    uint4 m[NU];
    double y[4];
    auto load_y = [&](int64_t k) {  // rows 4 j + t of this half-warp's block
      const double* ys = A.y + k * VSTEP + half * 16 + t;
#pragma unroll
      for (int j = 0; j < 4; j++) y[j] = k * VSTEP + VSTEP <= A.nRows ? __ldg(ys + 4 * j) : 0.0;
    };
    int64_t st = s0 + warp;
    if (st < s1) {
#pragma unroll
      for (int u = 0; u < NU; u++) m[u] = __ldg((const uint4*)(mp + u * ustr + st * 512));
      load_y(st);
    }
    for (; st < s1; st += LMM_W) {
      const int64_t nxt = st + LMM_W;
      const double four = (y[0] + y[1]) + (y[2] + y[3]);
      // (a product with 0 would carry an Inf or NaN into other rows: such steps go row by row, like the ragged last one)
      if (st * VSTEP + VSTEP <= A.nRows && !__any_sync(0xffffffffu, !isfinite(four))) {
        ysum += four;
        double yv[16];
#pragma unroll
        for (int i = 0; i < 16; i++) yv[i] = 0.0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          dmma884(yv[4 * j], yv[4 * j + 1], y[j], even);
          dmma884(yv[4 * j + 2], yv[4 * j + 3], y[j], odd);
        }
        if (nxt < s1) load_y(nxt);  // in flight until the next step, and the ids likewise
#pragma unroll
        for (int u = 0; u < NU; u++) {
          const uint4 w = m[u];
          if (nxt < s1) m[u] = __ldg((const uint4*)(mp + u * ustr + nxt * 512));
          const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int i = 0; i < 16; i++) acc[u] = fma(yv[i], lds_f64(entry_at(ww[i >> 2], i & 3, tb[u])), acc[u]);
        }
      } else {
        const int64_t r0 = st * VSTEP + half * 16;
        for (int i = 0; i < 16 && r0 + i < A.nRows; i++) {
          const double yy = A.y[r0 + i];
          if (t == 0) ysum += yy;
#pragma unroll
          for (int u = 0; u < NU; u++) acc[u] = fma(yy, lds_f64(tb[u] + 128u * mp[u * ustr + st * 512 + i]), acc[u]);
        }
        if (nxt < s1) {
#pragma unroll
          for (int u = 0; u < NU; u++) m[u] = __ldg((const uint4*)(mp + u * ustr + nxt * 512));
          load_y(nxt);
        }
      }
    }
    // combine the two half-warps (same slots, different rows), then the warps through shared memory
    __syncthreads();  // tables no longer needed
    double* red = (double*)smraw;  // [LMM_W][NU * 16 + 1]
#pragma unroll
    for (int u = 0; u < NU; u++) {
      double a = acc[u];
      a += __shfl_xor_sync(0xffffffffu, a, 16);
      if (half == 0) red[warp * (NU * 16 + 1) + u * 16 + slot] = a;
    }
    for (int d = 1; d < 32; d = d == 2 ? 16 : 2 * d) ysum += __shfl_xor_sync(0xffffffffu, ysum, d);  // (a lane's rows are those of its t)
    if (lane == 0) red[warp * (NU * 16 + 1) + NU * 16] = ysum;
    __syncthreads();
    for (int u = tid; u <= NU * 16; u += LMM_T) {
      double s = 0;
      for (int w = 0; w < LMM_W; w++) s += red[w * (NU * 16 + 1) + u];
      mine[u < NU * 16 ? u : LMM_PART] = s;
    }
  }
}

template <int W>
__global__ void __launch_bounds__(W * 32, 1) k_lmm_vec(const __grid_constant__ LmmArgs A) {
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  const int chunk = min((int)blockIdx.x / A.ctaFull, A.nChunks - 1), cta0 = chunk * A.ctaFull;
  const int nCta = chunk == A.nChunks - 1 ? A.ctaLast : A.ctaFull;
  if (A.parts) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#define LMM_CASE(N) case N: if constexpr (lmm_warps(N) >= W) lmm_vec_body<N, W>(A, chunk, cta0, nCta, smraw, &mbar); break;
  switch (min(A.U, A.nU16 - chunk * A.U)) {
    LMM_CASE(1) LMM_CASE(2) LMM_CASE(3) LMM_CASE(4) LMM_CASE(5) LMM_CASE(6) LMM_CASE(7)
  }
#undef LMM_CASE
}

// --------------------------------------------------------------------------------------------------
// LMM with Q left rows at once (Q = 2 or 4; the reference's left-multiply blocks four rows too,
// lib/CLALibLeftMultBy.java:731-819). Same layout and lookups as k_lmm_vec, but a dictionary value fetched for a
// cell multiplies the cell's Q left values: one pass over the maps and one lookup per cell serve Q rows, where Q
// passes of the one-row kernel would fetch each value Q times. partial: [gridDim.x][Q][LMM_PART].
// --------------------------------------------------------------------------------------------------
constexpr int LQ_W = 12;              // warps per CTA (Q x NU accumulators per lane: up to 170 registers)
constexpr int LQ_T = LQ_W * 32;

template <int NU, int Q>
__device__ __forceinline__ void lmmq_body(const LmmChunk& ch, const uint8_t* __restrict__ imaps, int64_t nRB,
                                          const double* __restrict__ tablesImg, const double* __restrict__ y, size_t pitch,
                                          int nRows, double* __restrict__ partial, unsigned char* smraw, uint64_t* mbar,
                                          int32_t* err) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int slot = lane & 15, half = lane >> 4;
  if (!tma_load_to_smem(smraw, tablesImg + ch.tblOff, (uint32_t)ch.tblDoubles * 8u, mbar)) {
    if (tid == 0) atomicExch(err, 105);
    for (int u = tid; u < Q * LMM_PART; u += LQ_T) partial[(size_t)blockIdx.x * Q * LMM_PART + u] = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  const unsigned char* tbase[NU];
  const uint8_t* mp[NU];
  {
    size_t off = 0;
#pragma unroll
    for (int u = 0; u < NU; u++) {
      tbase[u] = smraw + off + slot * 8;
      off += (size_t)ch.nk[u] * 128;
      mp[u] = imaps + (size_t)(ch.unit0 + u) * nRB * 256 + slot * 16;
    }
  }
  double acc[NU][Q];
#pragma unroll
  for (int u = 0; u < NU; u++)
#pragma unroll
    for (int q = 0; q < Q; q++) acc[u][q] = 0.0;
  const int ctaInChunk = blockIdx.x - ch.cta0;
  const int64_t nSteps = ((int64_t)nRows + LMM_STEP - 1) / LMM_STEP;
  const int64_t s0 = nSteps * ctaInChunk / ch.nCta, s1 = nSteps * (ctaInChunk + 1) / ch.nCta;
  for (int64_t st = s0 + warp; st < s1; st += LQ_W) {
    const int64_t r0 = st * LMM_STEP + half * 32;
    if (st * LMM_STEP + LMM_STEP <= nRows) {
#pragma unroll 1
      for (int sub = 0; sub < 2; sub++) {
        uint4 m[NU];
#pragma unroll
        for (int u = 0; u < NU; u++) m[u] = __ldg((const uint4*)(mp[u] + ((r0 >> 4) + sub) * 256));
        const double* yr = y + r0 + sub * 16;
#pragma unroll
        for (int i = 0; i < 16; i += 2) {  // two rows per 128-bit load of every left row
          double2 yq[Q];
#pragma unroll
          for (int q = 0; q < Q; q++) yq[q] = __ldg((const double2*)(yr + q * pitch + i));
#pragma unroll
          for (int u = 0; u < NU; u++) {
            const uint32_t w = (i >> 2) == 0 ? m[u].x : ((i >> 2) == 1 ? m[u].y : ((i >> 2) == 2 ? m[u].z : m[u].w));
            const double t0 = *(const double*)(tbase[u] + byte_x128(w, i & 3));
            const double t1 = *(const double*)(tbase[u] + byte_x128(w, (i & 3) + 1));
#pragma unroll
            for (int q = 0; q < Q; q++) acc[u][q] = fma(yq[q].y, t1, fma(yq[q].x, t0, acc[u][q]));
          }
        }
      }
    } else {  // ragged last step
      for (int64_t r = r0; r < min((int64_t)nRows, r0 + 32); r++) {
#pragma unroll
        for (int u = 0; u < NU; u++) {
          const double t = *(const double*)(tbase[u] + 128 * (int)mp[u][(r >> 4) * 256 + (r & 15)]);
#pragma unroll
          for (int q = 0; q < Q; q++) acc[u][q] = fma(y[q * pitch + r], t, acc[u][q]);
        }
      }
    }
  }
  __syncthreads();  // tables no longer needed
  double* red = (double*)smraw;  // [LQ_W][Q][NU*16]
#pragma unroll
  for (int u = 0; u < NU; u++)
#pragma unroll
    for (int q = 0; q < Q; q++) {
      double a = acc[u][q];
      a += __shfl_xor_sync(0xffffffffu, a, 16);
      if (half == 0) red[(warp * Q + q) * (NU * 16) + u * 16 + slot] = a;
    }
  __syncthreads();
  for (int e = tid; e < Q * NU * 16; e += LQ_T) {
    const int q = e / (NU * 16), u = e - q * (NU * 16);
    double s = 0;
    for (int w = 0; w < LQ_W; w++) s += red[(w * Q + q) * (NU * 16) + u];
    partial[((size_t)blockIdx.x * Q + q) * LMM_PART + u] = s;
  }
}

template <int Q>
__global__ void __launch_bounds__(LQ_T, 1)
k_lmm_vecq_u8(const LmmChunk* __restrict__ chunks, int nChunks, const uint8_t* __restrict__ imaps, int64_t nRB,
              const double* __restrict__ tablesImg, const double* __restrict__ y, size_t pitch, int nRows,
              double* __restrict__ partial, int32_t* err) {
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ LmmChunk ch;
  if (threadIdx.x == 0) {
    int c = 0;
    while (c + 1 < nChunks && (int)blockIdx.x >= chunks[c].cta0 + chunks[c].nCta) c++;
    ch = chunks[c];
  }
  __syncthreads();
#define LQ_CASE(N) case N: lmmq_body<N, Q>(ch, imaps, nRB, tablesImg, y, pitch, nRows, partial, smraw, &mbar, err); break;
  switch (ch.nUnits) {
    LQ_CASE(1) LQ_CASE(2) LQ_CASE(3) LQ_CASE(4) LQ_CASE(5) LQ_CASE(6)
    default: lmmq_body<7, Q>(ch, imaps, nRB, tablesImg, y, pitch, nRows, partial, smraw, &mbar, err); break;
  }
#undef LQ_CASE
}

// out[q][col] += sum over the chunk's CTAs of partial[cta][q][slot]; blockIdx.z = q
__global__ void k_lmm_vecq_final(const LmmChunk* __restrict__ chunks, int nChunks, const int* __restrict__ slotCol,
                                 const double* __restrict__ partial, double* __restrict__ out, int Q, int nCols) {
  const int c = blockIdx.x, q = blockIdx.z;
  if (c >= nChunks) return;
  const LmmChunk ch = chunks[c];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nWarps = (blockDim.x >> 5) * gridDim.y;
  for (int u = blockIdx.y * (blockDim.x >> 5) + warp; u < ch.nUnits * 16; u += nWarps) {
    const int col = slotCol[ch.unit0 * 16 + u];
    if (col < 0) continue;
    double s = 0;
    for (int i = lane; i < ch.nCta; i += 32) s += partial[((size_t)(ch.cta0 + i) * Q + q) * LMM_PART + u];
#pragma unroll
    for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (lane == 0) atomicAdd(&out[(size_t)q * nCols + col], s);
  }
}

// --------------------------------------------------------------------------------------------------
// LMM with two to eight left rows at once, on the FP64 tensor core: m8n8k4 with A = left rows x matrix rows, B = matrix
// rows x eight column slots. Lane (g, t) looks up slot g's values of rows 4 t .. 4 t + 3 of a 16-row block (one word of
// ids), the four products of the block taking one of them each, so a lookup serves all left rows and nothing is staged.
// Four lanes share a slot, so its table is kept four times: entry k of slot s for lane t at (k * 16 + (s & 3) * 4 + t) * 8,
// which gives each of the 16 lanes of a half-warp a bank pair of its own.
// Bound: the FP64 rate, 16 clocks of the tensor pipe per 16 rows and eight slots (half of it with four left rows or fewer
// wasted), against 8 for the lookups, 1 for the ids and 8 for the left values of all the CTA's slots. (FMA on scalar
// accumulators, four left rows per lookup, took 47 us per pass of four rows over 500k x 100 columns of four tuples.)
// --------------------------------------------------------------------------------------------------
constexpr int LR_W = 16;
constexpr int LR_T = LR_W * 32;
constexpr int LR_MAXT = 8;                    // tiles of eight slots per CTA
constexpr int LR_PART = LR_MAXT * 64 + 8;     // partial sums of a CTA: [slot][left row], then the sums of the left rows
constexpr int LR_SMEM = 220 * 1024;
struct LmmRowsArgs {
  const int2* units;           // {table offset / 16, depth} of a unit = two tiles
  const uint8_t* imaps;
  int64_t nRB;
  const double* tables;
  const int* slotCol;
  const double* y;
  size_t pitch;
  int q, nRows, nTiles, nChunks, grid;
  // chunk c: tiles [tile0(c), tile0(c + 1)), even to one tile, and CTAs in proportion
  __host__ __device__ int tile0(int c) const { return (int)((int64_t)nTiles * c / nChunks); }
  __host__ __device__ int cta0(int c) const { return (int)((int64_t)grid * tile0(c) / nTiles); }
  __host__ __device__ int chunk_of(int cta) const {
    int c = (int)((int64_t)cta * nChunks / grid);
    while (c > 0 && cta0(c) > cta) c--;
    while (c + 1 < nChunks && cta0(c + 1) <= cta) c++;
    return c;
  }
  double* partial;             // [gridDim.x][LR_PART]
  const double* constV;        // null: none
  const int* bareCols;
  int nBare, nCols, addTo;
  double* out;
};

template <int NT>
__device__ __forceinline__ void lmm_rows_body(const LmmRowsArgs& A, int chunk, int cta0, int nCta, double* sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int tile0 = A.tile0(chunk);
  uint32_t tb[NT];
  {
    uint32_t at = 0;  // entries of 128 bytes
#pragma unroll
    for (int u = 0; u < NT; u++) {
      const int2 un = A.units[(tile0 + u) >> 1];
      const double* src = A.tables + (size_t)un.x * 16 + ((tile0 + u) & 1) * 8;
      double* dst = sm + (size_t)at * 16;
      for (int e = tid; e < un.y * 32; e += LR_T) {  // entry, quad, slot of the quad, copy
        const int k = e >> 5, quad = (e >> 4) & 1, s = (e >> 2) & 3;
        dst[((size_t)quad * un.y + k) * 16 + (e & 15)] = src[(size_t)k * 16 + quad * 4 + s];
      }
      tb[u] = smem_u32(sm) + (at + (uint32_t)((g >> 2) * un.y)) * 128u + (uint32_t)((g & 3) * 4 + t) * 8u;
      at += 2u * un.y;
    }
  }
  __syncthreads();
  double c[NT][2], ys = 0.0;
#pragma unroll
  for (int u = 0; u < NT; u++) c[u][0] = c[u][1] = 0.0;
  const bool live = g < A.q;
  const double* yr = A.y + (size_t)(live ? g : 0) * A.pitch + 4 * t;
  const size_t ustr = (size_t)A.nRB * 256;
  // tile tl: slots (tl & 1) * 8 .. + 8 of unit tl >> 1
  auto ids_at = [&](int u, int64_t blk) {
    const int tl = tile0 + u;
    return __ldg((const uint32_t*)(A.imaps + (size_t)(tl >> 1) * ustr + blk * 256 + ((tl & 1) * 8 + g) * 16 + 4 * t));
  };
  const int64_t nBlk = ((int64_t)A.nRows + 15) / 16, whole = A.nRows / 16;
  const int ci = blockIdx.x - cta0;
  const int64_t b0 = nBlk * ci / nCta, b1 = nBlk * (ci + 1) / nCta;
  // NB blocks per turn, the next turn's loads in flight during this one's lookups: with few tiles a block is little work,
  // and the left values come from L2
  constexpr int NB = NT <= 4 ? 2 : 1;
  uint32_t id[NB][NT];
  double2 ya[NB], yb[NB];
  auto load = [&](int64_t k0) {
#pragma unroll
    for (int n = 0; n < NB; n++) {
      const int64_t k = min(k0 + n, nBlk - 1);
#pragma unroll
      for (int u = 0; u < NT; u++) id[n][u] = ids_at(u, k);
      if (k < whole) {
        ya[n] = __ldg((const double2*)(yr + k * 16));
        yb[n] = __ldg((const double2*)(yr + k * 16) + 1);
      }
    }
  };
  int64_t blk = b0 + warp * NB;
  if (blk < b1) load(blk);
  for (; blk < b1; blk += LR_W * NB) {
    uint32_t w[NB][NT];
    double yv[NB][4];
#pragma unroll
    for (int n = 0; n < NB; n++) {
#pragma unroll
      for (int u = 0; u < NT; u++) w[n][u] = id[n][u];
      yv[n][0] = ya[n].x, yv[n][1] = ya[n].y, yv[n][2] = yb[n].x, yv[n][3] = yb[n].y;
    }
    if (blk + LR_W * NB < b1) load(blk + LR_W * NB);
#pragma unroll
    for (int n = 0; n < NB; n++) {
      if (blk + n >= b1) break;
      if (blk + n < whole) {
#pragma unroll
        for (int u = 0; u < NT; u++) {
          double x[4];
#pragma unroll
          for (int i = 0; i < 4; i++) x[i] = lds_f64(entry_at(w[n][u], i, tb[u]));
#pragma unroll
          for (int i = 0; i < 4; i++) dmma884(c[u][0], c[u][1], yv[n][i], x[i]);
        }
      } else {  // the last rows: nothing of the padding enters the products
        const int64_t r0 = (blk + n) * 16 + 4 * t;
#pragma unroll
        for (int i = 0; i < 4; i++) yv[n][i] = r0 + i < A.nRows ? yr[(blk + n) * 16 + i] : 0.0;
#pragma unroll
        for (int u = 0; u < NT; u++)
#pragma unroll
          for (int i = 0; i < 4; i++)
            dmma884(c[u][0], c[u][1], yv[n][i], r0 + i < A.nRows ? lds_f64(entry_at(w[n][u], i, tb[u])) : 0.0);
      }
      if (A.constV) ys += (yv[n][0] + yv[n][1]) + (yv[n][2] + yv[n][3]);
    }
  }
  __syncthreads();  // tables no longer needed
  // c: left row g, slots 2 t, 2 t + 1; the warps through shared memory
  double* red = sm;  // [LR_W][NT * 64 + 8]
  constexpr int N = NT * 64 + 8;
#pragma unroll
  for (int u = 0; u < NT; u++)
#pragma unroll
    for (int e = 0; e < 2; e++) red[warp * N + (u * 8 + 2 * t + e) * 8 + g] = c[u][e];
  ys += __shfl_xor_sync(0xffffffffu, ys, 1);
  ys += __shfl_xor_sync(0xffffffffu, ys, 2);
  if (t == 0) red[warp * N + NT * 64 + g] = ys;
  __syncthreads();
  double* mine = A.partial + (size_t)blockIdx.x * LR_PART;
  for (int e = tid; e < N; e += LR_T) {
    double s = 0.0;
    for (int k = 0; k < LR_W; k++) s += red[k * N + e];
    mine[e < NT * 64 ? e : LR_MAXT * 64 + e - NT * 64] = s;
  }
}

__global__ void __launch_bounds__(LR_T, 1) k_lmm_rows(const __grid_constant__ LmmRowsArgs A) {
  extern __shared__ __align__(128) double lrsm[];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int chunk = A.chunk_of(blockIdx.x), cta0 = A.cta0(chunk), nCta = A.cta0(chunk + 1) - cta0;
#define LR_CASE(N) case N: lmm_rows_body<N>(A, chunk, cta0, nCta, lrsm); break;
  switch (A.tile0(chunk + 1) - A.tile0(chunk)) {
    LR_CASE(1) LR_CASE(2) LR_CASE(3) LR_CASE(4) LR_CASE(5) LR_CASE(6) LR_CASE(7)
    default: lmm_rows_body<LR_MAXT>(A, chunk, cta0, nCta, lrsm); break;
  }
#undef LR_CASE
}

// Adds up the partial sums of one tile (64 cells by 8 threads each, a fixed order) and stores the results. grid: tiles
__global__ void __launch_bounds__(512) k_lmm_rows_final(const __grid_constant__ LmmRowsArgs A) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ double red[8][64], yred[8][8];
  int chunk = (int)((int64_t)blockIdx.x * A.nChunks / A.nTiles);  // this tile's chunk
  while (chunk > 0 && A.tile0(chunk) > (int)blockIdx.x) chunk--;
  while (chunk + 1 < A.nChunks && A.tile0(chunk + 1) <= (int)blockIdx.x) chunk++;
  const int u = blockIdx.x - A.tile0(chunk), cta0 = A.cta0(chunk), nCta = A.cta0(chunk + 1) - cta0;
  const int cell = threadIdx.x & 63, sub = threadIdx.x >> 6;
  double s = 0.0, ys = 0.0;
#pragma unroll 4
  for (int i = sub; i < nCta; i += 8) {
    const double* p = A.partial + (size_t)(cta0 + i) * LR_PART;
    s += __ldcg(p + u * 64 + cell);
    if (A.constV && cell < 8) ys += __ldcg(p + LR_MAXT * 64 + cell);
  }
  red[sub][cell] = s;
  if (cell < 8) yred[sub][cell] = ys;
  __syncthreads();
  auto row_sum = [&](int g) {
    double x = 0.0;
    for (int k = 0; k < 8; k++) x += yred[k][g];
    return x;
  };
  if (sub == 0) {
    for (int k = 1; k < 8; k++) s += red[k][cell];
    const int g = cell & 7, col = A.slotCol[blockIdx.x * 8 + (cell >> 3)];
    if (g < A.q && col >= 0) {
      double* o = A.out + (size_t)g * A.nCols + col;
      if (A.addTo) atomicAdd(o, s);
      else *o = A.constV ? fma(row_sum(g), A.constV[col], s) : s;
    }
  }
  if (blockIdx.x == 0 && !A.addTo)  // columns of constant groups, and those the general kernels will add to
    for (int e = threadIdx.x; e < A.nBare * A.q; e += 512) {
      const int g = e / A.nBare, col = A.bareCols[e - g * A.nBare];
      A.out[(size_t)g * A.nCols + col] = A.constV ? row_sum(g) * A.constV[col] : 0.0;
    }
}

// --------------------------------------------------------------------------------------------------
// Decompress from the column-per-lane layout.
//
// Interleaved maps and table images of k_lmm_vec, chunks of units fixed at plan time: lane s of a half-warp owns column slot s of a
// unit, loads 16 rows of its ids with one 128-bit load, reads each value from its own bank pair of the unit's
// table and stores it. The 16 slots of a unit are 16 neighbouring output columns (the plan orders the slots by
// column), so a warp store writes two full 128-byte pieces of two rows: no transposition through shared memory,
// no bank conflicts, no gathers from global memory. Per 32 cells the L1 data pipe sees 2 wavefronts of lookups,
// 2 of stores and 1/4 of map loads (the tile kernel in cla_generic.cu needs about 20, most of them for the gather
// of dictionary values through L1), which puts the bound on the output stream. Every cell is written exactly once
// with the same operation as the tile kernel (column constant + dictionary value).
// --------------------------------------------------------------------------------------------------
constexpr int DEC_W = 12;  // warps per CTA (measured 8 / 10 / 12 / 14 / 16 / 20 / 24: 12 writes the most, 4.2-4.5 TB/s)
constexpr int DEC_T = DEC_W * 32;
constexpr int DEC_NP = (LMM_MAX_UNITS + 1) / 2;  // unit pairs of a chunk: a warp store covers 32 neighbouring columns

__global__ void __launch_bounds__(DEC_T, 1)
k_decomp_fast(const LmmChunk* __restrict__ chunks, int nChunks, const uint8_t* __restrict__ imaps, int64_t nRB,
              const double* __restrict__ tablesImg, const int* __restrict__ slotCol, const double* __restrict__ constV,
              double* __restrict__ out, size_t ld, int r0, int r1, int32_t* err) {
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ LmmChunk ch;
  __shared__ int unitOff[LMM_MAX_UNITS];
  __shared__ int sCol[LMM_MAX_UNITS * 16];
  __shared__ double sCst[LMM_MAX_UNITS * 16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int slot = lane & 15, half = lane >> 4;
  if (tid == 0) {
    int c = 0;
    while (c + 1 < nChunks && (int)blockIdx.x >= chunks[c].cta0 + chunks[c].nCta) c++;
    ch = chunks[c];
    int off = 0;
    for (int u = 0; u < ch.nUnits; u++) {
      unitOff[u] = off;
      off += ch.nk[u] * 128;
    }
  }
  __syncthreads();
  if (tid < ch.nUnits * 16) {
    const int col = slotCol[ch.unit0 * 16 + tid];
    sCol[tid] = col;
    sCst[tid] = (constV && col >= 0) ? constV[col] : 0.0;
  }
  const int NU = ch.nUnits;
  const int ctaInChunk = blockIdx.x - ch.cta0;
  const int64_t stepBegin = r0 / LMM_STEP, stepEnd = ((int64_t)r1 + LMM_STEP - 1) / LMM_STEP;  // r0 is a multiple of LMM_STEP
  const int64_t nSteps = stepEnd - stepBegin;
  const int64_t s0 = stepBegin + nSteps * ctaInChunk / ch.nCta, s1 = stepBegin + nSteps * (ctaInChunk + 1) / ch.nCta;
  if (!tma_load_to_smem(smraw, tablesImg + ch.tblOff, (uint32_t)ch.tblDoubles * 8u, &mbar)) {
    // the tables never arrived: flag it, and make the failure visible in this CTA's cells as well (a device-buffer
    // caller only sees the error word at its next cla_stats_get)
    if (tid == 0) atomicExch(err, 102);
    const int64_t rb = s0 * LMM_STEP, re = min((int64_t)r1, s1 * LMM_STEP);
    const int w = NU * 16;
    for (int64_t i = tid; i < (re - rb) * w; i += DEC_T) {
      const int col = sCol[(int)(i % w)];
      if (col >= 0) out[(size_t)(rb + i / w - r0) * ld + col] = __longlong_as_double(0x7ff8000000000000ll);
    }
    return;
  }
  // This lane's column of every unit pair: unit 2p + half, slot lane & 15
  int toff[DEC_NP];   // byte offset of the lane's table column in shared memory
  double cst[DEC_NP];
  int colOf[DEC_NP];
#pragma unroll
  for (int p = 0; p < DEC_NP; p++) {
    const int u = 2 * p + half;
    const bool ok = u < NU;
    colOf[p] = ok ? sCol[u * 16 + slot] : -1;
    cst[p] = ok ? sCst[u * 16 + slot] : 0.0;
    toff[p] = (ok ? unitOff[u] : 0) + slot * 8;
  }
  // ids of this lane's column of pair p, 16-row block b: units lie nRB * 256 bytes apart, a missing last unit reads unit 0's
  const uint8_t* mbase = imaps + (size_t)ch.unit0 * nRB * 256 + slot * 16;
  const size_t pairStride = (size_t)2 * nRB * 256, halfOff = (size_t)half * nRB * 256;
  auto ids_at = [&](int p, int64_t b) {
    const size_t uo = (2 * p + half < NU) ? p * pairStride + halfOff : 0;
    return __ldg((const uint4*)(mbase + uo + b * 256));
  };
  // A warp owns 16-row blocks; it writes them a row at a time, 256 contiguous bytes per store and the chunk's columns
  // of a row one after the other: runs of consecutive addresses are what the memory system turns into full-rate
  // writes (the same cells written as 128-byte pieces of many rows reach about 0.9 of this order's rate). The ids of
  // the next block are loaded before the current one is looked up.
  const int64_t b0 = s0 * (LMM_STEP / 16), b1 = s1 * (LMM_STEP / 16);
  uint4 w[DEC_NP], nw[DEC_NP];
  int64_t blk = b0 + warp;
  if (blk < b1) {
#pragma unroll
    for (int p = 0; p < DEC_NP; p++) w[p] = ids_at(p, blk);
  }
  for (; blk < b1; blk += DEC_W) {
    if (blk + DEC_W < b1) {
#pragma unroll
      for (int p = 0; p < DEC_NP; p++) nw[p] = ids_at(p, blk + DEC_W);
    }
    const int64_t row0 = blk * 16;
    double* o = out + (size_t)(row0 - r0) * ld;
    const bool whole = row0 + 16 <= r1;
#pragma unroll 1
    for (int j = 0; j < 4; j++) {  // four rows per round (one id word per unit pair): 4 x DEC_NP lookups in flight
      uint32_t word[DEC_NP];
#pragma unroll
      for (int p = 0; p < DEC_NP; p++) word[p] = j == 0 ? w[p].x : (j == 1 ? w[p].y : (j == 2 ? w[p].z : w[p].w));
      double* orow = o + (size_t)(4 * j) * ld;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (whole || row0 + 4 * j + i < r1) {
#pragma unroll
          for (int p = 0; p < DEC_NP; p++)
            if (colOf[p] >= 0) orow[colOf[p]] = cst[p] + *(const double*)(smraw + toff[p] + byte_x128(word[p], i));
        }
        orow += ld;
      }
    }
#pragma unroll
    for (int p = 0; p < DEC_NP; p++) w[p] = nw[p];
  }
}

// --------------------------------------------------------------------------------------------------
// RMM: X v. A CTA owns a contiguous range of rows and walks chunks of up to seven units one after the other, reloading
// the tables; the first chunk stores its partial sums, later chunks add to them (the CTA owns the rows: no atomics,
// one summation order). Within a chunk a lane accumulates 16 rows over its slots; the sums over the 16 lanes of the
// half-warps are then formed by the FP64 tensor core, which is idle otherwise: ten m8n8k4 products with 0 / 1 matrices
// per eight rows of both half-warps. (As shuffles the reduction was 30 of 280 wavefronts of the data pipe that bounds this kernel and a
// third of its instructions.) A product with 0 would carry an Inf or NaN of one row into its neighbours, so a warp that
// sees a non-finite result forms its sums again with shuffles.
// --------------------------------------------------------------------------------------------------
// 1.0 where a == b, else 0.0; volatile: formed where it is used (kept in registers across the main loop, the nine
// coefficients below pushed the kernel into spilling).
__device__ __forceinline__ double one_if(int a, int b) {
  double r;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, %2;\n\tselp.f64 %0, 0d3FF0000000000000, 0d0000000000000000, p;\n\t}" : "=d"(r) : "r"(a), "r"(b));
  return r;
}
// Sums acc[i] over the 16 lanes of each half-warp, over quads of lanes by products with 0 / 1 matrices (C[m][n] = sum over the four
// lanes of quad n of acc[m]: B = acc[i], A_i = 1 in row i; the lower half-warp's quads are 0..3) and over two pairs of quads by one shuffle: lane
// 4 g + t returns row g of the lower half-warp where t < 2, of the upper one otherwise.
__device__ __forceinline__ double half_warp_sums(const double (&acc)[8]) {
  const int g = (threadIdx.x & 31) >> 2;
  double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};  // two chains of four products
#pragma unroll
  for (int i = 0; i < 4; i++) {
    dmma884(c[0][0], c[0][1], one_if(g, i), acc[i]);
    dmma884(c[1][0], c[1][1], one_if(g, i + 4), acc[i + 4]);
  }
  const double s = (c[0][0] + c[0][1]) + (c[1][0] + c[1][1]);
  return s + __shfl_xor_sync(0xffffffffu, s, 1);
}
// The row of a step of 32 whose sum this lane holds afterwards: t odd for the second eight rows of a block.
__device__ __forceinline__ int sum_row() {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  return (t >> 1) * 16 + (t & 1) * 8 + g;
}

struct RmmArgs {
  const int2* units;       // {table offset / 16, depth}
  const uint8_t* imaps;
  int64_t nRB;
  const double* tables;    // column slots
  const int* slotCol;
  const JointSlot* joint;  // joint slots
  const JointTerm* terms;
  const int* termCols;     // null: all groups have one column
  int nTerms, joinTerms;   // terms of a slot, of one of two or more groups, at most
  int U;                   // units per chunk
  int tail;                // slots behind them that go by rows
  int partRows, pairs;     // see joint_tables: rows of 32 slots before their tables, at most; pairs of units that have room for them
  const double* v;
  const double* constV;    // null: none
  int nCols;
  int nRows, nU16;
  const double* rowScale;  // null, or a factor per row applied at the end
  int64_t stride;          // of v and out (column of a row-major matrix)
  double* out;
  int32_t* err;
};

// The sums of step `st` again, for a warp that saw an Inf or NaN: every row by itself, with shuffles. v null: joint slots.
__device__ __noinline__ double rmm_step_by_rows(const uint8_t* mp, size_t ustr, const int2* units, const int* slotCol,
                                                const double* v, int64_t stride, int nu, uint32_t table0) {
  const int lane = threadIdx.x & 31, slot = lane & 15, row = sum_row();
  double r = 0.0;
  for (int i = 0; i < 16; i++) {
    double a = 0.0;
    for (int u = 0; u < nu; u++) {
      const double x = lds_f64(table0 + (uint32_t)(units[u].x - units[0].x) * 128u + slot * 8 + 128u * mp[u * ustr + i]);
      if (!v) a += x;
      else if (const int col = slotCol[u * 16 + slot]; col >= 0) a = fma(x, v[col * stride], a);
    }
    for (int d = 1; d < 16; d <<= 1) a += __shfl_xor_sync(0xffffffffu, a, d);
    const double other = __shfl_xor_sync(0xffffffffu, a, 16);
    if (i == (row & 15)) r = (lane >> 4) == (row >> 4) ? a : other;
  }
  return r;
}

// Row sums of one step from its id words, this lane's as sum_row says. JOINT: the terms are the table entries themselves.
// (Joint slots with a reduction of shuffles alone: 30 of the 150 wavefronts of a step of three units; 40.4 against 38.0 us for 1M x 100 of
// 16 values, cold.)
template <int NU, bool JOINT, int UNROLL_ROWS, class F>
__device__ __forceinline__ double step_sums(const uint4 (&m)[NU], const uint32_t (&tb)[NU], const double (&v)[NU], F&& used) {
  double r = 0.0;
#pragma unroll UNROLL_ROWS
  for (int h = 0; h < 2; h++) {  // rows 0..7 and 8..15 of each half-warp's block
    double acc[8];
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i] = 0.0;
#pragma unroll
    for (int u = 0; u < NU; u++) {
      const uint32_t w0 = h ? m[u].z : m[u].x, w1 = h ? m[u].w : m[u].y;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const double x = lds_f64(entry_at(i < 4 ? w0 : w1, i & 3, tb[u]));
        acc[i] = JOINT ? acc[i] + x : fma(x, v[u], acc[i]);
      }
      if (h == 1) used(u);
    }
    const double s = half_warp_sums(acc);
    if ((threadIdx.x & 1) == h) r = s;
  }
  return r;
}

// Ids of units [unit0, unit0 + nu) for the steps [from, from + n), clipped to s1, to L2: warp u takes unit u.
__device__ __forceinline__ void rmm_fetch(const RmmArgs& A, int unit0, int nu, int64_t from, int64_t n, int64_t s1) {
  const int warp = threadIdx.x >> 5;
  n = min(n, s1 - from);
  if (warp < nu && (threadIdx.x & 31) == 0 && n > 0)
    l2_fetch(A.imaps + ((size_t)(unit0 + warp) * A.nRB + (size_t)from * 2) * 256, (uint32_t)n * 512u);
}
// Turns of the warps whose ids are on their way to L2: about 100 KB per SM, what the memory's latency takes. (1,250,000 x 1000, 16 warps: 430 us
// without, 409 with, 413 and 433 with two and four times as many.)
__host__ __device__ constexpr int rmm_ahead(int nu) { return 14 / nu; }

template <int NU, bool JOINT>
__device__ __forceinline__ void rmm_rows(const RmmArgs& A, int unit0, int64_t s0, int64_t s1, double init, bool first, bool last,
                                         uint32_t table0, uint32_t tail0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = lane & 15, half = lane >> 4, rowOf = sum_row();
  uint32_t tb[NU];
  double v[NU];
#pragma unroll
  for (int u = 0; u < NU; u++) {
    tb[u] = table0 + (uint32_t)(A.units[unit0 + u].x - A.units[unit0].x) * 128u + slot * 8;
    v[u] = 0.0;
    if (!JOINT) {
      const int col = A.slotCol[(unit0 + u) * 16 + slot];
      v[u] = col >= 0 ? A.v[col * A.stride] : 0.0;
    }
  }
  const uint8_t* mp = A.imaps + (size_t)unit0 * A.nRB * 256 + half * 256 + slot * 16;
  const size_t ustr = (size_t)A.nRB * 256;
  constexpr int W = JOINT ? RBJ_W : RB_W;
  uint4 m[NU];
  auto load = [&](int64_t st) {
#pragma unroll
    for (int u = 0; u < NU; u++) m[u] = __ldg((const uint4*)(mp + u * ustr + st * 512));
  };
  if (!JOINT && s0 + warp < s1) load(s0 + warp);
  for (int64_t st = s0 + warp; st < s1; st += W) {
    if (JOINT) load(st);
    auto used = [&](int u) {  // a unit's ids of the next step, as soon as this step's are used up
      if (!JOINT && st + W < s1) m[u] = __ldg((const uint4*)(mp + u * ustr + (st + W) * 512));
    };
    rmm_fetch(A, unit0, NU, st - warp + rmm_ahead(NU) * W, W, s1);
    const int64_t row = st * VSTEP + rowOf;
    const bool mine = row < A.nRows;
    uint32_t tailId[JOINT_TAIL];
    if (JOINT && last)
#pragma unroll
      for (int b = 0; b < JOINT_TAIL; b++)
        if (b < A.tail) tailId[b] = __ldg(A.imaps + ((size_t)(unit0 + NU) * A.nRB + (size_t)st * 2 + (rowOf >> 4)) * 256 + b * 16 + (rowOf & 15));
    double o = init;  // what this row holds from the chunks before
    if (!first) o = mine ? A.out[row * A.stride] : 0.0;
    double r = step_sums<NU, JOINT, 2>(m, tb, v, used);
    if (__any_sync(0xffffffffu, !isfinite(r)))
      r = rmm_step_by_rows(mp + st * 512, ustr, A.units + unit0, A.slotCol + unit0 * 16, JOINT ? nullptr : A.v, A.stride, NU, table0);
    if (JOINT && last)
#pragma unroll
      for (int b = 0; b < JOINT_TAIL; b++)
        if (b < A.tail) r += lds_f64(tail0 + (uint32_t)b * 2048u + tailId[b] * 8u);
    r += o;
    if (last && A.rowScale && mine) r *= A.rowScale[row];
    if (mine) A.out[row * A.stride] = r;
  }
}

// Tables of the joint slots of `nu` units, and of `tail` slots behind them whose entries lie side by side (tailTbl): first the terms
// D_g v of their groups, then the sums of the low and of the high groups of every slot, then the tables as sums of the two. A lane works
// for one slot, its entries are spread over warps; as many pairs of units at once as have room for what comes before the tables.
// Bound: the latency of the first loads. (Group after group with a barrier after each, two units at a time, each term behind the load of its
// group's record: 1M x 100 of 16 values, inputs changing from call to call, 43.0 us; 34.9 now, with the slots by rows and the ids brought to L2;
// 41.5 with the ids asked for before the terms.)
template <class F>
__device__ __forceinline__ void joint_tables(const RmmArgs& A, int unit0, int nu, int tail, double* tbl, double* tailTbl, double* parts, F&& loaded) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, all = nu + (tail > 0), nPairs = (all + 1) / 2;
  for (int p0 = 0; p0 < nPairs; p0 += A.pairs) {
    const int np = min(A.pairs, nPairs - p0), wp = RBJ_W / np;  // warps per pair
    const int pair = p0 + warp / wp, r = warp % wp, u = 2 * pair + (lane >> 4), sl = lane & 15, slot = (unit0 + u) * 16 + sl;
    const bool on = warp < wp * np && u < all && (u < nu || sl < tail);
    JointSlot js;
    js.n = 0;
    if (on) js = A.joint[slot];
    const int n = js.n;
    double* P = parts + (size_t)(pair - p0) * A.partRows * 32 + lane;
    double* T = u < nu ? tbl + (size_t)(on ? A.units[unit0 + u].x - A.units[unit0].x : 0) * 16 + sl : tailTbl + sl * 256;
    const int str = u < nu ? 16 : 1, depth = on && u < nu ? A.units[unit0 + u].y : 0;
    // (the records of the terms lie side by side, so that nothing but v hangs on a load before)
    if (on) {
      const size_t at = ((size_t)(unit0 + u) * A.nTerms) * 16 + sl;
#pragma unroll 4
      for (int e = r; e < A.nTerms; e += wp) {
        const JointTerm t = A.terms[at + (size_t)e * 16];
        const int gc = A.termCols ? A.termCols[at + (size_t)e * 16] : 0;
        double x = 0.0;
        if (gc > 0)
          for (int h = 0; h < gc; h++) x += t.dict[h] * A.v[t.cols[h] * A.stride];
        else if (t.col >= 0) x = t.val * A.v[t.col * A.stride];
        if (n > 1 && e < A.joinTerms) P[(size_t)e * 32] = x;
        else if (n == 1 && e < js.total) T[(size_t)e * str] = x;
      }
    }
    for (int k = (n > 0 ? js.total : 0) + r; k < depth; k += wp) T[(size_t)k * str] = 0.0;
    __syncthreads();
    if (p0 == 0) loaded();
    // low and high part: the terms themselves where it is one group, behind the terms otherwise
    const int nLo = n > 1 ? js.nLo : 0, nHi = n > 1 ? js.total / js.nLo : 0;
    const double *L = P, *H = P;
    if (n > 1) {
      int at = 0;
#pragma unroll
      for (int i = 0; i < JS_MAX; i++)
        if (i < js.split) at += js.nv[i];
      H = P + (size_t)at * 32;  // first term of the high groups
      double* free = P + (size_t)A.joinTerms * 32;
      auto sums = [&](const double* src, int g0, int g1, int count) {
        for (int e = r; e < count; e += wp) {
          const double* q = src;
          double x = 0.0;
          int k = e;
#pragma unroll
          for (int i = 0; i < JS_MAX; i++)
            if (i >= g0 && i < g1) {
              const int d = (int)(((float)k + 0.5f) / (float)js.nv[i]);  // k / nv: half a step from any whole number
              x += q[(size_t)(k - d * js.nv[i]) * 32];
              q += (size_t)js.nv[i] * 32;
              k = d;
            }
          free[(size_t)e * 32] = x;
        }
        const double* res = free;
        free += (size_t)count * 32;
        return res;
      };
      if (js.split > 1) L = sums(P, 0, js.split, nLo);
      if (n - js.split > 1) H = sums(H, js.split, n, nHi);
    }
    __syncthreads();
    if (n > 1) {
      // few low tuples: warps side by side along the high ones
      const int side = max(1, wp / nLo), l0 = nLo >= wp ? r : r % nLo, h0 = nLo >= wp ? 0 : r / nLo;
      if (h0 < side)
        for (int k = l0; k < nLo; k += wp) {
          const double x = L[(size_t)k * 32];
#pragma unroll 4
          for (int h = h0; h < nHi; h += side) T[(size_t)(k + nLo * h) * str] = x + H[(size_t)h * 32];
        }
    }
    __syncthreads();
  }
}

template <bool JOINT>
__global__ void __launch_bounds__((JOINT ? RBJ_W : RB_W) * 32, 1) k_rmm_vec(const __grid_constant__ RmmArgs A) {
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  constexpr int W = JOINT ? RBJ_W : RB_W;
  __shared__ double cred[W];
  const int64_t nSteps = ((int64_t)A.nRows + VSTEP - 1) / VSTEP;
  const int64_t s0 = nSteps * blockIdx.x / gridDim.x, s1 = nSteps * (blockIdx.x + 1) / gridDim.x;
  double init = 0.0;
  if (A.constV) {
    for (int c = threadIdx.x; c < A.nCols; c += W * 32) init = fma(A.constV[c], A.v[c * A.stride], init);
    for (int d = 16; d; d >>= 1) init += __shfl_xor_sync(0xffffffffu, init, d);
    if ((threadIdx.x & 31) == 0) cred[threadIdx.x >> 5] = init;
    __syncthreads();
    init = 0.0;
    for (int w = 0; w < W; w++) init += cred[w];
  }
  tma_barrier_init(&mbar);
  const int U = A.U;
  for (int unit0 = 0, c = 0; unit0 < A.nU16; unit0 += U, c++) {
    const int nu = min(U, A.nU16 - unit0);
    const bool last = unit0 + nu == A.nU16;
    uint32_t tail0 = 0;
    auto fetch = [&] { rmm_fetch(A, unit0, nu, s0, rmm_ahead(nu) * W, s1); };
    if (!JOINT) fetch();
    __syncthreads();  // everyone is done with the previous chunk's tables
    if (JOINT) {
      const int rows = A.units[unit0 + nu - 1].x + A.units[unit0 + nu - 1].y - A.units[unit0].x;
      double* tails = (double*)smraw + (size_t)rows * 16;
      const int tail = last ? A.tail : 0;
      tail0 = smem_u32(tails);
      joint_tables(A, unit0, nu, tail, (double*)smraw, tails, tails + tail * 256, fetch);  // (the ids behind the terms, which the tables wait for)
    } else {
      const int2 f = A.units[unit0], l = A.units[unit0 + nu - 1];
      if (!tma_reload(smraw, A.tables + (size_t)f.x * 16, (uint32_t)(l.x + l.y - f.x) * 128u, &mbar, (uint32_t)(c & 1))) {
        if (threadIdx.x == 0) atomicExch(A.err, 102);
        return;
      }
    }
    const uint32_t t0 = smem_u32(smraw);
#define RB_CASE(N) case N: rmm_rows<N, JOINT>(A, unit0, s0, s1, init, c == 0, last, t0, tail0); break;
    switch (nu) {
      RB_CASE(1) RB_CASE(2) RB_CASE(3) RB_CASE(4) RB_CASE(5) RB_CASE(6)
      default: rmm_rows<7, JOINT>(A, unit0, s0, s1, init, c == 0, last, t0, tail0); break;
    }
#undef RB_CASE
  }
}

// --------------------------------------------------------------------------------------------------
// t(X) (w * (X v)) in one kernel, for up to seven units of column slots (112 columns), whose tables fit one SM: a step's
// row sums are formed as in k_rmm_vec, scaled, put in shared memory, and multiplied into the column sums as in
// k_lmm_vec with the id words still in registers (row loops not unrolled: the compiler would hoist a step's worth of
// lookups and spill). The maps are read once instead of twice, the tables are staged once,
// and u = X v never leaves the SM (it is stored only if the caller gave a buffer for it). With a step's row sums by eight products and a
// shuffle per eight rows instead of ten products: 2M x 100 142.7 -> 141.4 us, 2M x 40 98.3 -> 93.9, 300,000 x 100 30.7 -> 30.3, 50,000 x 100 14.3 as before.
// --------------------------------------------------------------------------------------------------
constexpr int CH_W = 11;         // what fits next to seven units of 256 tuples
constexpr int CH_T = CH_W * 32;
constexpr int CH_STATIC = 3072;  // static shared memory of the kernel, at most
struct ChainArgs {
  LmmArgs L;            // y unused
  const double* v;
  const double* w;      // null: no weights
  double* u;            // null: not wanted
  int nCols;
};

template <int NU>
__device__ __forceinline__ void chain_body(const ChainArgs& C, unsigned char* smraw, uint64_t* mbar, double* ubuf, double init) {
  const LmmArgs& A = C.L;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int slot = lane & 15, half = lane >> 4, rowOf = sum_row();
  double* mine = A.partial + (size_t)blockIdx.x * (LMM_PART + 1);
  const int2 first = A.units[0], last = A.units[NU - 1];
  if (!tma_load_to_smem(smraw, A.tables, (uint32_t)(last.x + last.y - first.x) * 128u, mbar)) {
    if (tid == 0) atomicExch(A.err, 103);
    for (int u = tid; u <= LMM_PART; u += CH_T) mine[u] = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  const uint32_t table0 = smem_u32(smraw);
  uint32_t tb[NU];
  double v[NU], acc[NU], ysum = 0.0;
#pragma unroll
  for (int u = 0; u < NU; u++) {
    tb[u] = table0 + (uint32_t)(A.units[u].x - first.x) * 128u + slot * 8;
    const int col = A.slotCol[u * 16 + slot];
    v[u] = col >= 0 ? C.v[col] : 0.0;
    acc[u] = 0.0;
  }
  const uint8_t* mp = A.imaps + half * 256 + slot * 16;
  const size_t ustr = (size_t)A.nRB * 256;
  double* ub = ubuf + warp * 32;
  const int64_t s0 = A.stepEnd * blockIdx.x / gridDim.x, s1 = A.stepEnd * (blockIdx.x + 1) / gridDim.x;
  for (int64_t st = s0 + warp; st < s1; st += CH_W) {
    uint4 m[NU];
#pragma unroll
    for (int u = 0; u < NU; u++) m[u] = __ldg((const uint4*)(mp + u * ustr + st * 512));
    const int64_t row = st * VSTEP + rowOf;
    const bool in = row < A.nRows;
    const double wt = C.w && in ? C.w[row] : 1.0;
    double r = step_sums<NU, false, 1>(m, tb, v, [](int) {});
    if (__any_sync(0xffffffffu, !isfinite(r))) r = rmm_step_by_rows(mp + st * 512, ustr, A.units, A.slotCol, C.v, 1, NU, table0);
    r = (r + init) * wt;
    if (C.u && in) C.u[row] = r;
    ub[rowOf] = r;
    __syncwarp();
    if (st * VSTEP + VSTEP <= A.nRows) {
#pragma unroll 1
      for (int b = 0; b < 4; b++) {
        double y[4];
        const double2 ya = *(const double2*)&ub[half * 16 + b * 4], yb = *(const double2*)&ub[half * 16 + b * 4 + 2];
        y[0] = ya.x, y[1] = ya.y, y[2] = yb.x, y[3] = yb.y;
        if (A.constV) ysum += (y[0] + y[1]) + (y[2] + y[3]);
#pragma unroll
        for (int u = 0; u < NU; u++) {
          const uint32_t w = b == 0 ? m[u].x : (b == 1 ? m[u].y : (b == 2 ? m[u].z : m[u].w));
#pragma unroll
          for (int i = 0; i < 4; i++) acc[u] = fma(y[i], lds_f64(entry_at(w, i, tb[u])), acc[u]);
        }
      }
    } else {  // ragged last step
      for (int i = 0; i < 16 && st * VSTEP + half * 16 + i < A.nRows; i++) {
        const double yy = ub[half * 16 + i];
        ysum += yy;
#pragma unroll
        for (int u = 0; u < NU; u++) acc[u] = fma(yy, lds_f64(tb[u] + 128u * mp[u * ustr + st * 512 + i]), acc[u]);
      }
    }
    __syncwarp();
  }
  __syncthreads();  // tables no longer needed
  double* red = (double*)smraw;  // [CH_W][NU * 16 + 1]
#pragma unroll
  for (int u = 0; u < NU; u++) {
    double a = acc[u];
    a += __shfl_xor_sync(0xffffffffu, a, 16);
    if (half == 0) red[warp * (NU * 16 + 1) + u * 16 + slot] = a;
  }
  ysum += __shfl_xor_sync(0xffffffffu, ysum, 16);
  if (lane == 0) red[warp * (NU * 16 + 1) + NU * 16] = ysum;
  __syncthreads();
  for (int u = tid; u <= NU * 16; u += CH_T) {
    double s = 0;
    for (int w = 0; w < CH_W; w++) s += red[w * (NU * 16 + 1) + u];
    mine[u < NU * 16 ? u : LMM_PART] = s;
  }
}

__global__ void __launch_bounds__(CH_T, 1) k_chain_vec(const __grid_constant__ ChainArgs C) {
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ __align__(16) double ubuf[CH_W * 32];
  __shared__ double cred[CH_W];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  double init = 0.0;
  if (C.L.constV) {
    for (int c = threadIdx.x; c < C.nCols; c += CH_T) init = fma(C.L.constV[c], C.v[c], init);
    for (int d = 16; d; d >>= 1) init += __shfl_xor_sync(0xffffffffu, init, d);
    if ((threadIdx.x & 31) == 0) cred[threadIdx.x >> 5] = init;
    __syncthreads();
    init = 0.0;
    for (int w = 0; w < CH_W; w++) init += cred[w];
  }
#define CH_CASE(N) case N: chain_body<N>(C, smraw, &mbar, ubuf, init); break;
  switch (C.L.nU16) {
    CH_CASE(1) CH_CASE(2) CH_CASE(3) CH_CASE(4) CH_CASE(5) CH_CASE(6)
    default: chain_body<7>(C, smraw, &mbar, ubuf, init); break;
  }
#undef CH_CASE
}

// Maps are handed to the interleave kernels as tagged addresses: bit 0 set = MapToBit words, else one byte per row.
__device__ __forceinline__ uint4 ids16(const uint8_t* tagged, int64_t r, int nRows) {
  const uintptr_t p = (uintptr_t)tagged & ~(uintptr_t)1;
  uint4 v = make_uint4(0, 0, 0, 0);
  if (r >= nRows) return v;
  if ((uintptr_t)tagged & 1) {  // r is a multiple of 16: the 16 bits lie in one word
    uint32_t bits = (uint32_t)(((const unsigned long long*)p)[r >> 6] >> (r & 63)) & 0xFFFFu;
    if (r + 16 > nRows) bits &= (1u << (nRows - r)) - 1u;
    auto four = [](uint32_t x) { return (x & 1u) | ((x & 2u) << 7) | ((x & 4u) << 14) | ((x & 8u) << 21); };
    return make_uint4(four(bits), four(bits >> 4), four(bits >> 8), four(bits >> 12));
  }
  if (r + 16 <= nRows) return *(const uint4*)(p + r);
  __align__(16) uint8_t tmp[16];
  for (int i = 0; i < 16; i++) tmp[i] = (r + i < nRows) ? ((const uint8_t*)p)[r + i] : 0;
  return *(const uint4*)tmp;
}

// Device layout of the maps for the column-per-lane kernels: [unit of 16 slots][16-row block][slot][16 ids].
// A half-warp (one lane per slot) then reads 256 contiguous bytes per 128-bit load instead of 16 scattered
// lines. Built once at plan time; unused slots and rows past the end hold id 0.
__global__ void k_lmm_interleave(const uint8_t* const* __restrict__ slotMap, int nSlots, int nUnits, int nRows,
                                 int64_t nRB, uint8_t* __restrict__ out) {
  const int64_t total = (int64_t)nSlots * nRB;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < total; g += (int64_t)gridDim.x * blockDim.x) {
    const int slot = (int)(g & 15);
    const int64_t rb = (g >> 4) % nRB, slab = (g >> 4) / nRB;
    const int unit = (int)slab * 16 + slot;
    ((uint4*)out)[g] = unit < nUnits ? ids16(slotMap[unit], rb * 16, nRows) : make_uint4(0, 0, 0, 0);
  }
}

// Joint ids of the slots in the same layout.
__global__ void k_joint_interleave(const JointSlot* __restrict__ slots, const uint8_t* const* __restrict__ groupMap, int nSlots,
                                   int nRows, int64_t nRB, uint8_t* __restrict__ out) {
  const int64_t total = (int64_t)nSlots * nRB;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < total; g += (int64_t)gridDim.x * blockDim.x) {
    const int slot = (int)(g & 15);
    const int64_t rb = (g >> 4) % nRB, slab = (g >> 4) / nRB;
    const JointSlot& js = slots[slab * 16 + slot];
    // joint ids stay below 256, so the bytes of a word never carry into each other
    uint4 id = make_uint4(0, 0, 0, 0);
    uint32_t stride = 1;
    for (int k = 0; k < js.n; k++) {
      const uint4 w = ids16(groupMap[js.group[k]], rb * 16, nRows);
      id.x += stride * w.x, id.y += stride * w.y, id.z += stride * w.z, id.w += stride * w.w;
      stride *= js.nv[k];
    }
    ((uint4*)out)[g] = id;
  }
}

// --------------------------------------------------------------------------------------------------
// plan
// --------------------------------------------------------------------------------------------------
void fast_plan_free(Matrix* m) {
  if (!m->fast) return;
  for (void* p : m->fast->allocs) dev_free(m, p);
  delete m->fast;
  m->fast = nullptr;
}

static int64_t plan_malloc(Matrix* m, FastPlan* fp, void** p, size_t bytes) {
  *p = nullptr;
  cudaError_t e = dev_malloc(m, p, std::max<size_t>(bytes, 16));
  if (e != cudaSuccess) return fail(CLA_ERR_NOMEM, std::string("cudaMalloc plan: ") + cudaGetErrorString(e));
  fp->allocs.push_back(*p);
  return CLA_OK;
}

// Host arrays of the plan, uploaded with one allocation and one copy.
struct PlanBlob {
  std::vector<char> host;
  template <typename T>
  size_t add(const std::vector<T>& v) {
    const size_t at = (host.size() + 255) & ~(size_t)255;
    host.resize(at + std::max<size_t>(v.size() * sizeof(T), 1));
    if (!v.empty()) memcpy(host.data() + at, v.data(), v.size() * sizeof(T));
    return at;
  }
};

int64_t fast_plan_build(Matrix* m) {
  FastPlan* fp = new FastPlan();
  m->fast = fp;
  if (m->nRows < FAST_MIN_ROWS || m->nDev == 0) return CLA_OK;
  // the groups these kernels cover: dense maps, at most 256 tuples, one byte (or bit) per cell
  struct Sel { int dev, reg; };
  std::vector<Sel> sel;
  int nUnitsSel = 0;
  for (size_t hi = 0; hi < m->hg.size(); hi++) {
    const int gi = m->regToDev[hi];
    if (gi < 0) continue;
    const DevGroup& g = m->groups[gi];
    if (g.type != GT_DDC || g.nVals > 256 || g.nVals < 1) continue;
    if (g.mapType != CLA_MAP_UBYTE && g.mapType != CLA_MAP_BYTE && g.mapType != CLA_MAP_BIT) continue;
    sel.push_back({gi, (int)hi});
    nUnitsSel += g.gCols;
  }
  const bool all = (int)sel.size() == m->nDev;
  if (sel.empty() || (!all && nUnitsSel < 16)) return CLA_OK;  // too few columns to be worth a separate pass
  fp->partial = !all;
  const int nG = (int)sel.size();
  int64_t rc;
  auto G = [&](int i) -> const DevGroup& { return m->groups[sel[i].dev]; };
  auto tagged = [&](int i) { return (const uint8_t*)((uintptr_t)G(i).map | (G(i).mapType == CLA_MAP_BIT ? 1u : 0u)); };
  fp->nRB = (((int64_t)m->nRows + LMM_STEP - 1) / LMM_STEP) * (LMM_STEP / 16);

  // ---- column slots: one per (group, column), in output-column order; 16 slots per unit ----
  // (in column order the 16 slots of a unit are neighbours in a decompressed row)
  struct Unit { int g, j, nv, col; };
  std::vector<Unit> units;
  for (int i = 0; i < nG; i++)
    for (int j = 0; j < G(i).gCols; j++) units.push_back({i, j, G(i).nVals, m->hg[sel[i].reg].cols[j]});
  std::stable_sort(units.begin(), units.end(), [](const Unit& a, const Unit& b) { return a.col < b.col; });
  fp->nUnits = (int)units.size();
  const int nU16 = fp->nU16 = (fp->nUnits + 15) / 16;
  fp->nSlots = nU16 * 16;
  std::vector<const uint8_t*> slotMap(fp->nSlots, nullptr);
  std::vector<int> slotCol(fp->nSlots, -1);
  fp->unitNk.assign(nU16, 1);
  fp->unitOff.assign(nU16, 0);
  std::vector<uint8_t> held(m->nCols, 0);
  for (int u = 0; u < fp->nUnits; u++) {
    slotMap[u] = tagged(units[u].g);
    slotCol[u] = units[u].col;
    if (held[units[u].col]) fp->uniqueCols = false;
    held[units[u].col] = 1;
    fp->unitNk[u / 16] = std::max(fp->unitNk[u / 16], units[u].nv);
  }
  std::vector<int> bare;
  for (int c = 0; c < m->nCols; c++)
    if (!held[c]) bare.push_back(c);
  fp->nBare = (int)bare.size();
  // table image, unit after unit
  std::vector<int2> unitRec(nU16);
  int64_t imgD = 0;
  for (int q = 0; q < nU16; q++) {
    fp->unitOff[q] = imgD;
    unitRec[q] = make_int2((int)(imgD / 16), fp->unitNk[q]);
    imgD += (int64_t)fp->unitNk[q] * 16;
  }
  std::vector<double> image(imgD, 0.0);
  for (int u = 0; u < fp->nUnits; u++) {
    const HostGroup& hg = m->hg[sel[units[u].g].reg];
    const int gc = (int)hg.cols.size(), nv = hg.nVals;  // (an OLE group's extra "no tuple" entry stays zero)
    double* T = image.data() + fp->unitOff[u / 16] + (u & 15);
    for (int k = 0; k < nv; k++) T[(size_t)k * 16] = hg.dict[(size_t)k * gc + units[u].j];
  }
  fp->imageDoubles = image.size();
  // chunks of up to LMM_MAX_UNITS units for the kernels that fix them at plan time (several left rows, decompress):
  // CTAs per chunk in proportion to its cost in L1 data-pipe wavefronts per 64-row step: 64 per unit for the dictionary
  // reads, 8 for the map loads and 64 for the left vector
  {
    LmmChunk lc{};
    for (int q = 0; q < nU16; q++) {
      if (lc.nUnits == LMM_MAX_UNITS) {
        fp->lchunks.push_back(lc);
        lc = LmmChunk{};
      }
      if (lc.nUnits == 0) {
        lc.unit0 = q;
        lc.tblOff = fp->unitOff[q];
      }
      lc.nk[lc.nUnits++] = fp->unitNk[q];
      lc.tblDoubles += fp->unitNk[q] * 16;
    }
    fp->lchunks.push_back(lc);
    const int totalCta = std::max(m->smCount, (int)fp->lchunks.size());
    double totalCost = 0;
    auto chunkCost = [](const LmmChunk& c) { return 72.0 * c.nUnits + 64.0; };
    for (auto& c : fp->lchunks) totalCost += chunkCost(c);
    const int64_t nSteps = ((int64_t)m->nRows + LMM_STEP - 1) / LMM_STEP;
    std::vector<int> share(fp->lchunks.size());
    int used = 0, cta = 0;
    for (size_t i = 0; i < fp->lchunks.size(); i++) {
      share[i] = std::max(1, (int)(totalCta * chunkCost(fp->lchunks[i]) / totalCost));
      used += share[i];
    }
    for (size_t i = 0; used < totalCta; i = (i + 1) % fp->lchunks.size(), used++) share[i]++;  // hand out the remainder
    for (size_t i = 0; i < fp->lchunks.size(); i++) {
      auto& c = fp->lchunks[i];
      const int n = (int)std::min<int64_t>(share[i], nSteps);
      c.cta0 = cta;
      c.nCta = n;
      cta += n;
    }
    fp->lmmGrid = cta;
  }

  // ---- joint slots for X v: the smallest dictionaries first, as many groups per slot as 256 joint tuples allow ----
  std::vector<JointSlot> js;
  std::vector<const uint8_t*> groupMap(m->nDev, nullptr);
  {
    std::vector<int> byNv(nG);
    std::iota(byNv.begin(), byNv.end(), 0);
    std::stable_sort(byNv.begin(), byNv.end(), [&](int a, int b) { return G(a).nVals < G(b).nVals; });
    for (int i : byNv) {
      const int nv = G(i).nVals;
      if (js.empty() || js.back().n == JS_MAX || js.back().total * nv > 256) {
        JointSlot s{};
        s.total = 1;
        js.push_back(s);
      }
      JointSlot& s = js.back();
      s.group[s.n] = sel[i].dev;
      s.nv[s.n++] = nv;
      s.total *= nv;
      groupMap[sel[i].dev] = tagged(i);
    }
    // a second copy of the maps pays from a quarter fewer lookups on
    if (js.size() * 4 > (size_t)fp->nUnits * 3) js.clear();
    for (auto& x : js) {  // low and high part: the split with the fewest terms
      x.split = x.n;
      x.nLo = x.total;
      int lo = 1, best = x.total + 1;
      for (int k = 1; k < x.n; k++) {
        lo *= x.nv[k - 1];
        const int hi = x.total / lo;
        if (lo + hi < best) best = lo + hi, x.split = k, x.nLo = lo;
      }
      if (x.n > 1) {
        fp->jParts = std::max(fp->jParts, (x.split > 1 ? x.nLo : 0) + (x.n - x.split > 1 ? x.total / x.nLo : 0));
      }
      int terms = 0;
      for (int k = 0; k < x.n; k++) terms += x.nv[k];
      fp->jTerms = std::max(fp->jTerms, terms);
      if (x.n > 1) fp->jJoinTerms = std::max(fp->jJoinTerms, terms);
    }
    std::stable_sort(js.begin(), js.end(), [](const JointSlot& a, const JointSlot& b) { return a.total > b.total; });
    fp->nJU16 = (int)(js.size() + 15) / 16;
    fp->jTail = js.size() > 16 && js.size() % 16 <= JOINT_TAIL ? (int)(js.size() % 16) : 0;
    js.resize((size_t)fp->nJU16 * 16, JointSlot{});
  }
  std::vector<JointTerm> jt(js.size() * fp->jTerms);
  std::vector<int> jtCols, regOf(m->nDev, 0);
  for (auto& x : sel) regOf[x.dev] = x.reg;
  for (auto& t : jt) t.val = 0.0, t.col = -1;
  for (size_t i = 0; i < js.size(); i++)
    for (int k = 0, e = 0; k < js[i].n; k++) {
      const DevGroup& g = m->groups[js[i].group[k]];
      const HostGroup* hg = &m->hg[regOf[js[i].group[k]]];
      for (int a = 0; a < js[i].nv[k]; a++, e++) {
        const size_t at = ((i / 16) * fp->jTerms + e) * 16 + i % 16;
        if (g.gCols == 1) {  // (an OLE group's extra "no tuple" entry is zero)
          jt[at].val = a < (int)hg->dict.size() ? hg->dict[a] : 0.0;
          jt[at].col = hg->cols[0];
        } else {
          jt[at].dict = g.dict + (size_t)a * g.gCols;
          jt[at].cols = g.cols;
          jtCols.resize(jt.size(), 0);
          jtCols[at] = g.gCols;
        }
      }
    }
  std::vector<int2> jRec(fp->nJU16);
  fp->jNk.assign(fp->nJU16, 1);
  int jAt = 0;
  for (int q = 0; q < fp->nJU16; q++) {
    for (int s = 0; s < 16; s++) fp->jNk[q] = std::max(fp->jNk[q], js[q * 16 + s].total);
    jRec[q] = make_int2(jAt, fp->jNk[q]);
    jAt += fp->jNk[q];
  }

  PlanBlob blob;
  const size_t oChunks = blob.add(fp->lchunks), oMap = blob.add(slotMap), oCol = blob.add(slotCol), oBare = blob.add(bare);
  const size_t oUnits = blob.add(unitRec), oImage = blob.add(image);
  const size_t oJs = blob.add(js), oJt = blob.add(jt), oJtCols = blob.add(jtCols), oJRec = blob.add(jRec), oGMap = blob.add(groupMap);
  const size_t mapBytes = (size_t)fp->nSlots * fp->nRB * 16, jMapBytes = (size_t)fp->nJU16 * 16 * fp->nRB * 16;
  void *d = nullptr, *maps = nullptr;
  if ((rc = plan_malloc(m, fp, &d, blob.host.size())) < 0 || (rc = plan_malloc(m, fp, &maps, mapBytes + jMapBytes)) < 0) return rc;
  CLA_CUDA(cudaMemcpyAsync(d, blob.host.data(), blob.host.size(), cudaMemcpyHostToDevice, m->stream));
  char* base = (char*)d;
  fp->dLChunks = (LmmChunk*)(base + oChunks);
  fp->dSlotMap = (const uint8_t**)(base + oMap);
  fp->dSlotCol = (int*)(base + oCol);
  fp->dBareCols = (int*)(base + oBare);
  fp->dUnits = (int2*)(base + oUnits);
  fp->dLmmTables = (double*)(base + oImage);
  fp->dJSlots = (JointSlot*)(base + oJs);
  fp->dJTerms = (JointTerm*)(base + oJt);
  fp->dJTermCols = jtCols.empty() ? nullptr : (int*)(base + oJtCols);
  fp->dJUnits = (int2*)(base + oJRec);
  fp->dLmmMaps = (uint8_t*)maps;
  fp->dJMaps = (uint8_t*)maps + mapBytes;
  m->deviceBytes += (int64_t)(mapBytes + jMapBytes + blob.host.size());
  k_lmm_interleave<<<m->smCount * 8, 256, 0, m->stream>>>(fp->dSlotMap, fp->nSlots, fp->nUnits, m->nRows, fp->nRB, fp->dLmmMaps);
  if (fp->nJU16)
    k_joint_interleave<<<m->smCount * 8, 256, 0, m->stream>>>(fp->dJSlots, (const uint8_t* const*)(base + oGMap), fp->nJU16 * 16,
                                                             m->nRows, fp->nRB, fp->dJMaps);
  CLA_CUDA(cudaStreamSynchronize(m->stream));
  static OncePerDevice once, onceDecomp;
  if ((rc = allow_smem(once, m->device, SMEM_MAX - 1024, k_lmm_vec<12>, k_lmm_vec<16>, k_rmm_vec<false>, k_rmm_vec<true>)) < 0) return rc;
  if ((rc = allow_smem(onceDecomp, m->device, SMEM_MAX - 2048, k_decomp_fast)) < 0) return rc;
  if (fp->partial) {  // tell the general kernels which groups are taken care of
    for (auto& x : sel) m->groups[x.dev].inFast = 1;
    CLA_CUDA(cudaMemcpy(m->dGroups, m->groups.data(), sizeof(DevGroup) * m->groups.size(), cudaMemcpyHostToDevice));
  }
  fp->ok = true;
  return CLA_OK;
}

// --------------------------------------------------------------------------------------------------
// launchers
// --------------------------------------------------------------------------------------------------
bool fast_plan_ok(const Matrix* m) { return m->fast && m->fast->ok; }
bool fast_plan_partial(const Matrix* m) { return m->fast && m->fast->ok && m->fast->partial; }

// Rows [r0, r1) of the decompressed matrix into dOut (row r0 first) when every column is a slot of the plan and no
// column belongs to two groups; 0 = not covered (the caller takes the tile kernel).
int64_t fast_decompress(Matrix* m, int r0, int r1, double* dOut, cudaStream_t s, size_t ld) {
  FastPlan* fp = m->fast;
  if (!fp || !fp->ok || fp->partial || !fp->dLmmMaps || !m->colSrcValid || fp->nUnits != m->nCols || (r0 % LMM_STEP)) return 0;
  static const bool off = getenv("CLA_DECOMP_TILES") != nullptr;
  if (off) return 0;
  size_t smem = 0;
  for (auto& c : fp->lchunks) smem = std::max(smem, (size_t)c.tblDoubles * 8);
  k_decomp_fast<<<fp->lmmGrid, DEC_T, smem, s>>>(fp->dLChunks, (int)fp->lchunks.size(), fp->dLmmMaps, fp->nRB, fp->dLmmTables,
                                                fp->dSlotCol, m->hasConst ? m->dConstV : nullptr, dOut, ld, r0, r1,
                                                m->dErr);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  return 1;
}

int64_t fast_rmm_vec(Matrix* m, const double* dV, double* dOut, const double* dW, cudaStream_t s, int64_t stride) {
  FastPlan* fp = m->fast;
  if (!fp || !fp->ok || (dW && fp->partial)) return 0;
  // (short matrices: building the joint tables takes longer than the lookups they save)
  const bool joint = fp->nJU16 > 0 && m->nRows >= 300000;
  RmmArgs A{};
  A.units = joint ? fp->dJUnits : fp->dUnits;
  A.imaps = joint ? fp->dJMaps : fp->dLmmMaps;
  A.nRB = fp->nRB;
  A.tables = fp->dLmmTables;
  A.slotCol = fp->dSlotCol;
  A.joint = fp->dJSlots;
  A.terms = fp->dJTerms;
  A.termCols = fp->dJTermCols;
  A.nTerms = fp->jTerms;
  A.joinTerms = fp->jJoinTerms;
  A.v = dV;
  A.constV = m->hasConst ? m->dConstV : nullptr;
  A.nCols = m->nCols;
  A.nRows = m->nRows;
  A.nU16 = joint ? fp->nJU16 : fp->nU16;
  A.rowScale = dW;
  A.stride = stride;
  A.out = dOut;
  A.err = m->dErr;
  const std::vector<int>& nk = joint ? fp->jNk : fp->unitNk;
  if (joint && fp->jTail) {
    A.tail = fp->jTail;
    A.nU16--;
  }
  // units per chunk, evenly: what fits, the joint slots' with room for what comes before the tables of a pair of units
  A.partRows = std::max(1, fp->jJoinTerms + fp->jParts);
  const size_t parts = joint ? (size_t)A.partRows * 256 : 0, tails = (size_t)A.tail * 2048, room = SMEM_MAX - 1024;
  size_t tables = 1024;
  for (int most = joint ? JOINT_UNITS : LMM_MAX_UNITS; most >= 1; most--) {
    const int nChunks = (A.nU16 + most - 1) / most;
    A.U = (A.nU16 + nChunks - 1) / nChunks;
    tables = 1024;
    for (int q = 0; q < A.nU16; q += A.U) {
      size_t b = 0;
      for (int i = q; i < std::min(A.nU16, q + A.U); i++) b += (size_t)nk[i] * 128;
      tables = std::max(tables, b);
    }
    if (tables + tails + parts <= room) break;
  }
  A.pairs = joint ? std::max(1, std::min((A.U + 2) / 2, (int)((room - tables - tails) / parts))) : 1;
  const size_t smem = tables + tails + A.pairs * parts;
  const int64_t nSteps = ((int64_t)m->nRows + VSTEP - 1) / VSTEP;
  const int grid = (int)std::min<int64_t>(m->smCount, nSteps);
  prof_begin(m, s);
  if (joint) k_rmm_vec<true><<<grid, RBJ_W * 32, smem, s>>>(A);
  else k_rmm_vec<false><<<grid, RB_W * 32, smem, s>>>(A);
  prof_end(m, s);
  m->stats.kernel_launches++;
  CLA_CUDA(cudaGetLastError());
  return fp->partial ? 2 : 1;
}

// Units per chunk of k_lmm_vec: with few rows per CTA, staging the tables (32 KB per unit) costs more than the rows, so
// the columns are spread over more CTAs; with many, wide chunks read y less often. Clocks, from the pipe's
// wavefronts: 512 per unit staged, 1.13 per unit and row and 1 for the rest, and at least one round of steps. (0.3 for the rest, what y takes
// there now, changes little but 100,000 x 200: 18.9 instead of 16.8 us.)
static int lmm_chunk_units(const FastPlan* fp, int nRows, int sm) {
  int best = 1;
  double bestCost = 1e300;
  for (int U = 1; U <= LMM_MAX_UNITS; U++) {
    const int nChunks = (fp->nU16 + U - 1) / U, u = (fp->nU16 + nChunks - 1) / nChunks;
    if (nChunks > sm && U < LMM_MAX_UNITS) continue;
    const double ctas = std::max(1.0, (double)sm / nChunks), rows = nRows / ctas, waves = std::ceil((double)nChunks / sm);
    const double rounds = std::ceil(rows / (VSTEP * lmm_warps(u)));
    const double cost = waves * (512.0 * u + std::max(rows * (1.13 * u + 1.0), rounds * (600.0 + 40.0 * u)));
    if (cost < bestCost) bestCost = cost, best = u;
  }
  return best;
}

static size_t lmm_args(Matrix* m, FastPlan* fp, LmmArgs& A, int* grid) {
  A.units = fp->dUnits;
  A.imaps = fp->dLmmMaps;
  A.nRB = fp->nRB;
  A.tables = fp->dLmmTables;
  A.slotCol = fp->dSlotCol;
  A.nRows = m->nRows;
  A.nU16 = fp->nU16;
  A.U = lmm_chunk_units(fp, m->nRows, m->smCount);
  A.nChunks = (fp->nU16 + A.U - 1) / A.U;
  A.addTo = fp->uniqueCols ? 0 : 1;
  A.constV = (m->hasConst && fp->uniqueCols) ? m->dConstV : nullptr;
  A.bareCols = fp->dBareCols;
  A.nBare = fp->nBare;
  A.err = m->dErr;
  A.part = 0;
  A.parts = 1;
  A.stepBegin = 0;
  A.stepEnd = ((int64_t)m->nRows + VSTEP - 1) / VSTEP;
  const int uLast = fp->nU16 - (A.nChunks - 1) * A.U;
  const double w = 1.13 * A.U + 1.0, wl = 1.13 * uLast + 1.0, all = (A.nChunks - 1) * w + wl;
  const int steps = (int)std::min<int64_t>(A.stepEnd, 1 << 20);
  A.ctaFull = std::max(1, std::min(steps, (int)(m->smCount * w / all + 0.5)));
  if (A.nChunks > 1 && A.ctaFull * (A.nChunks - 1) >= m->smCount) A.ctaFull = std::max(1, (m->smCount - 1) / (A.nChunks - 1));
  A.ctaLast = std::max(1, std::min(steps, m->smCount - A.ctaFull * (A.nChunks - 1)));
  *grid = A.ctaFull * (A.nChunks - 1) + A.ctaLast;
  size_t smem = (size_t)LMM_MAXW * (LMM_PART + 1) * 8;
  for (int q = 0; q < fp->nU16; q += A.U) {
    size_t b = 0;
    for (int i = q; i < std::min(fp->nU16, q + A.U); i++) b += (size_t)fp->unitNk[i] * 128;
    smem = std::max(smem, b);
  }
  return smem;
}

// k_lmm_final behind a kernel that lets it start early
static int64_t launch_lmm_final(Matrix* m, const LmmArgs& A, int grid, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)A.nU16);
  cfg.blockDim = dim3(LMM_FT);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CLA_CUDA(cudaLaunchKernelEx(&cfg, k_lmm_final, A, grid));
  m->stats.kernel_launches++;
  return CLA_OK;
}
// The product's last (or only) launch of k_lmm_vec and what finishes it
static int64_t launch_lmm_vec(Matrix* m, const LmmArgs& A, int grid, size_t smem, cudaStream_t s) {
  const int W = lmm_warps(A.U);
  if (W == 12) k_lmm_vec<12><<<grid, 12 * 32, smem, s>>>(A);
  else k_lmm_vec<16><<<grid, 16 * 32, smem, s>>>(A);
  m->stats.kernel_launches++;
  if (A.parts) return launch_lmm_final(m, A, grid, s);
  return CLA_OK;
}

// t(X) (w * (X v)) where one kernel can do it (see k_chain_vec); 0: not covered
int64_t fast_chain(Matrix* m, const double* dV, const double* dW, double* dOut, double* dU, cudaStream_t s) {
  FastPlan* fp = m->fast;
  if (!fp || !fp->ok || fp->partial || !fp->uniqueCols || fp->nU16 > LMM_MAX_UNITS) return 0;
  // many rows of small dictionaries: X v by joint slots and t(X) u by themselves take fewer lookups
  if (fp->nJU16 > 0 && fp->nJU16 * 2 <= fp->nU16 && m->nRows >= (1 << 20)) return 0;
  ChainArgs C{};
  int grid;
  lmm_args(m, fp, C.L, &grid);
  C.L.U = fp->nU16;
  C.L.nChunks = 1;
  grid = (int)std::min<int64_t>(m->smCount, C.L.stepEnd);
  C.L.ctaFull = C.L.ctaLast = grid;
  size_t smem = (size_t)CH_W * (LMM_PART + 1) * 8, b = 0;
  for (int nk : fp->unitNk) b += (size_t)nk * 128;
  smem = std::max(smem, b);
  if (smem > SMEM_MAX - CH_STATIC) return 0;
  int64_t rc;
  if ((rc = ensure_scratch(m, (size_t)grid * (LMM_PART + 1) * 8 + 256)) < 0) return rc;
  C.L.partial = (double*)m->scratch;
  C.L.out = dOut;
  C.v = dV;
  C.w = dW;
  C.u = dU;
  C.nCols = m->nCols;
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, SMEM_MAX - CH_STATIC, k_chain_vec); e < 0) return e;
  prof_begin(m, s);
  k_chain_vec<<<grid, CH_T, smem, s>>>(C);
  m->stats.kernel_launches++;
  if ((rc = launch_lmm_final(m, C.L, grid, s)) < 0) return rc;
  prof_end(m, s);
  CLA_CUDA(cudaGetLastError());
  return 1;
}

int64_t fast_lmm_vec(Matrix* m, const double* dY, double* dOut, cudaStream_t s) {
  FastPlan* fp = m->fast;
  if (!fp || !fp->ok || ((uintptr_t)dY & 15)) return 0;  // 128-bit loads of the left vector need alignment
  LmmArgs A{};
  int grid;
  const size_t smem = lmm_args(m, fp, A, &grid);
  int64_t rc;
  if ((rc = ensure_scratch(m, (size_t)grid * (LMM_PART + 1) * 8 + 256)) < 0) return rc;
  A.partial = (double*)m->scratch;
  A.y = dY;
  A.out = dOut;
  if (A.addTo) CLA_CUDA(cudaMemsetAsync(dOut, 0, sizeof(double) * (size_t)m->nCols, s));
  prof_begin(m, s);
  if ((rc = launch_lmm_vec(m, A, grid, smem, s)) < 0) return rc;
  prof_end(m, s);
  if (m->hasConst && !A.constV)
    if ((rc = launch_lmm_const(m, dY, 1, dOut, s)) < 0) return rc;
  CLA_CUDA(cudaGetLastError());
  return fp->partial ? 2 : 1;
}

// Q = 2 or 4 left rows (rows q of y at y + q * pitch, 16-byte aligned) in one pass; same return values as fast_lmm_vec.
template <int Q>
static int64_t fast_lmm_rows_t(Matrix* m, FastPlan* fp, const double* dY, size_t pitch, double* dOut, cudaStream_t s) {
  int64_t rc;
  const size_t partBytes = (size_t)fp->lmmGrid * Q * LMM_PART * 8;
  if ((rc = ensure_scratch(m, partBytes + 256)) < 0) return rc;
  double* partial = (double*)m->scratch;
  CLA_CUDA(cudaMemsetAsync(dOut, 0, sizeof(double) * (size_t)Q * m->nCols, s));
  size_t smem = (size_t)LQ_W * Q * LMM_PART * 8;
  for (auto& c : fp->lchunks) smem = std::max(smem, (size_t)c.tblDoubles * 8);
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, SMEM_MAX - 1024, k_lmm_vecq_u8<Q>); e < 0) return e;
  prof_begin(m, s);
  k_lmm_vecq_u8<Q><<<fp->lmmGrid, LQ_T, smem, s>>>(fp->dLChunks, (int)fp->lchunks.size(), fp->dLmmMaps, fp->nRB, fp->dLmmTables, dY,
                                                  pitch, m->nRows, partial, m->dErr);
  prof_end(m, s);
  k_lmm_vecq_final<<<dim3((unsigned)fp->lchunks.size(), LMM_MAX_UNITS, Q), 512, 0, s>>>(fp->dLChunks, (int)fp->lchunks.size(),
                                                                                       fp->dSlotCol, partial, dOut, Q, m->nCols);
  m->stats.kernel_launches += 2;
  if (m->hasConst)
    for (int q = 0; q < Q; q++)
      if ((rc = launch_lmm_const(m, dY + q * pitch, 1, dOut + (size_t)q * m->nCols, s)) < 0) return rc;
  CLA_CUDA(cudaGetLastError());
  return fp->partial ? 2 : 1;
}
// Up to eight left rows on the tensor core; NOT_HERE: k_lmm_vecq is the better one.
constexpr int64_t NOT_HERE = 3;
static int64_t lmm_rows_tensor(Matrix* m, FastPlan* fp, const double* dY, size_t pitch, int q, double* dOut, cudaStream_t s) {
  LmmRowsArgs A{};
  A.units = fp->dUnits;
  A.imaps = fp->dLmmMaps;
  A.nRB = fp->nRB;
  A.tables = fp->dLmmTables;
  A.slotCol = fp->dSlotCol;
  A.y = dY;
  A.pitch = pitch;
  A.q = q;
  A.nRows = m->nRows;
  A.nTiles = (fp->nUnits + 7) / 8;
  A.constV = (m->hasConst && fp->uniqueCols) ? m->dConstV : nullptr;
  A.bareCols = fp->dBareCols;
  A.nBare = fp->nBare;
  A.nCols = m->nCols;
  A.addTo = fp->uniqueCols ? 0 : 1;
  A.out = dOut;
  auto bytes_of = [&](int t0, int n) {
    size_t b = 0;
    for (int i = t0; i < std::min(A.nTiles, t0 + n); i++) b += (size_t)fp->unitNk[i >> 1] * 256;
    return b;
  };
  // Tiles per chunk: what fits, and by the same balance as lmm_chunk_units -- clocks per 16 rows 16 a tile and 10 for the
  // left values, 2 per tuple of a staged tile, at least one round of blocks.
  size_t smem = 0;
  int fits = 0;
  double bestCost = 1e300;
  const int64_t nBlk = ((int64_t)m->nRows + 15) / 16;
  for (int U = 1; U <= LR_MAXT; U++) {
    LmmRowsArgs T = A;
    T.nChunks = (A.nTiles + U - 1) / U;
    size_t most = (size_t)LR_W * (std::min(U, A.nTiles) * 64 + 8) * 8, stage = 0;
    for (int c = 0; c < T.nChunks; c++) stage = std::max(stage, bytes_of(T.tile0(c), T.tile0(c + 1) - T.tile0(c)));
    most = std::max(most, stage);
    if (most > (size_t)LR_SMEM) continue;
    fits = U;
    const double ctas = std::max(1.0, (double)m->smCount / T.nChunks), blocks = nBlk / ctas, waves = std::ceil((double)T.nChunks / m->smCount);
    const double cost = waves * (stage / 128.0 + std::max(blocks * (16.0 * U + 10.0), std::ceil(blocks / LR_W) * (700.0 + 60.0 * U)));
    if (cost < bestCost) {
      bestCost = cost;
      A.nChunks = T.nChunks;
      smem = most;
    }
  }
  if (A.nChunks == 0) return fail(CLA_ERR_STATE, "left product: a table does not fit shared memory");
  // Up to four rows on deep tables: half of the products would be wasted, and with few tiles per CTA the left values are
  // read too often for that (1M x 200, 256 values, 2 / 3 / 4 rows: 199 / 207 / 215 us here, 121 / 197 / 154 in passes of
  // k_lmm_vecq; at 100 values and eight tiles, 100k x 500, three rows, 50 against 74).
  if (q <= 4 && fits < 6 && A.nTiles > fits) return NOT_HERE;
  // at least one CTA for every chunk, however the shares round; no more than four blocks of rows justify
  const int64_t most = std::max<int64_t>((int64_t)2 * A.nChunks, ((nBlk + 3) / 4) * A.nChunks);
  const int grid = A.grid = (int)std::min<int64_t>(most, 2 * A.nChunks > m->smCount ? 2 * A.nChunks : m->smCount);
  int64_t rc;
  if ((rc = ensure_scratch(m, (size_t)grid * LR_PART * 8 + 256)) < 0) return rc;
  A.partial = (double*)m->scratch;
  if (A.addTo) CLA_CUDA(cudaMemsetAsync(dOut, 0, sizeof(double) * (size_t)q * m->nCols, s));
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, LR_SMEM, k_lmm_rows); e < 0) return e;
  prof_begin(m, s);
  k_lmm_rows<<<grid, LR_T, smem, s>>>(A);
  prof_end(m, s);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)A.nTiles);
  cfg.blockDim = dim3(512);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CLA_CUDA(cudaLaunchKernelEx(&cfg, k_lmm_rows_final, A));
  m->stats.kernel_launches += 2;
  if (m->hasConst && !A.constV)
    for (int i = 0; i < q; i++)
      if ((rc = launch_lmm_const(m, dY + i * pitch, 1, dOut + (size_t)i * m->nCols, s)) < 0) return rc;
  CLA_CUDA(cudaGetLastError());
  return fp->partial ? 2 : 1;
}

// q left rows (row i at y + i * pitch, 16-byte aligned); same return values as fast_lmm_vec.
int64_t fast_lmm_rows(Matrix* m, const double* dY, size_t pitch, int q, double* dOut, cudaStream_t s) {
  FastPlan* fp = m->fast;
  if (!fp || !fp->ok || ((uintptr_t)dY & 15) || (pitch & 1)) return 0;
  int64_t rc = 0;
  for (int i = 0; i < q;) {
    const double* y = dY + (size_t)i * pitch;
    double* o = dOut + (size_t)i * m->nCols;
    int n = std::min(8, q - i);
    rc = n == 1 ? NOT_HERE : lmm_rows_tensor(m, fp, y, pitch, n, o, s);
    if (rc == NOT_HERE) {
      n = n == 4 ? 4 : std::min(2, n);
      rc = n == 4 ? fast_lmm_rows_t<4>(m, fp, y, pitch, o, s) : (n == 2 ? fast_lmm_rows_t<2>(m, fp, y, pitch, o, s) : fast_lmm_vec(m, y, o, s));
    }
    if (rc <= 0) return rc;
    i += n;
  }
  return rc;
}

// Host-buffer t(y) %*% X with the upload of y overlapped with the product: y is copied in up to LMM_PIPE_MAX row ranges
// on a second stream, and the kernel for a range starts as soon as its slice has arrived. Returns 0 if the
// specialised kernel does not cover the matrix (the caller then copies y whole and takes the normal path).
constexpr int LMM_PIPE_MAX = 16;  // = the handle's copyDone events
static int lmm_pipe_depth() {
  static const int d = [] {
    const char* e = getenv("CLA_LMM_PIPE");
    const int v = e ? atoi(e) : 8;
    return v < 1 ? 1 : (v > LMM_PIPE_MAX ? LMM_PIPE_MAX : v);
  }();
  return d;
}
int64_t fast_lmm_vec_host(Matrix* m, const double* hostY, double* dY, double* dOut, cudaStream_t s) {
  FastPlan* fp = m->fast;
  if (!fp || !fp->ok || fp->partial || ((uintptr_t)dY & 15) || m->nRows < (1 << 20)) return 0;
  LmmArgs A{};
  int grid;
  const size_t smem = lmm_args(m, fp, A, &grid);
  int64_t rc;
  const int LMM_PIPE = lmm_pipe_depth();
  if ((rc = ensure_scratch(m, (size_t)LMM_PIPE * grid * (LMM_PART + 1) * 8 + 256)) < 0) return rc;
  if (!m->copyStream) {
    CLA_CUDA(cudaStreamCreateWithFlags(&m->copyStream, cudaStreamNonBlocking));
    for (int i = 0; i < LMM_PIPE_MAX; i++) CLA_CUDA(cudaEventCreateWithFlags(&m->copyDone[i], cudaEventDisableTiming));
  }
  A.partial = (double*)m->scratch;
  A.y = dY;
  A.out = dOut;
  if (A.addTo) CLA_CUDA(cudaMemsetAsync(dOut, 0, sizeof(double) * (size_t)m->nCols, s));
  const int64_t nSteps = A.stepEnd;
  // the copy stream must not run ahead of work already queued on s that still reads dY
  CLA_CUDA(cudaEventRecord(m->ev1, s));
  CLA_CUDA(cudaStreamWaitEvent(m->copyStream, m->ev1, 0));
  // Row ranges of decreasing size (weights n, n - 1, ..., 1): the copy engine is the slower side, so every kernel has
  // finished before the next range has arrived, and what is left after the last byte has landed is the product over
  // the smallest range only.
  const int64_t wSum = (int64_t)LMM_PIPE * (LMM_PIPE + 1) / 2;
  auto range_start = [&](int i) { return nSteps * ((int64_t)i * (2 * LMM_PIPE - i + 1) / 2) / wSum; };  // i ranges: n + ... + (n - i + 1)
  auto range_rows = [&](int i, int64_t& sb, int64_t& se, int64_t& rb, int64_t& re) {
    sb = range_start(i), se = i + 1 == LMM_PIPE ? nSteps : range_start(i + 1);
    rb = sb * VSTEP, re = std::min<int64_t>(m->nRows, se * VSTEP);
  };
  // the kernel of row range i, once that range of y is on the copy stream
  auto launch_range = [&](int i) -> int64_t {
    int64_t sb, se, rb, re;
    range_rows(i, sb, se, rb, re);
    CLA_CUDA(cudaEventRecord(m->copyDone[i], m->copyStream));
    CLA_CUDA(cudaStreamWaitEvent(s, m->copyDone[i], 0));
    if (i == 0) prof_begin(m, s);
    A.stepBegin = sb;
    A.stepEnd = se;
    A.part = i;
    A.parts = i == LMM_PIPE - 1 ? LMM_PIPE : 0;  // the last range's launch adds up all ranges' partial sums
    const int64_t r = launch_lmm_vec(m, A, grid, smem, s);
    if (r < 0) return r;
    if (i == LMM_PIPE - 1) prof_end(m, s);
    return CLA_OK;
  };
  if (host_copy_staged(m, hostY, (size_t)m->nRows * 8)) {
    // y lives in pageable memory: host threads move it through the pinned ring, and every row range starts as soon
    // as its last slice is on the copy stream
    int nextRange = 0;
    rc = host_to_device_staged(m, dY, hostY, (size_t)m->nRows * 8, m->copyStream, [&](size_t bytesQueued) -> int64_t {
      while (nextRange < LMM_PIPE) {
        int64_t sb, se, rb, re;
        range_rows(nextRange, sb, se, rb, re);
        if ((size_t)re * 8 > bytesQueued) break;
        const int64_t r = launch_range(nextRange++);
        if (r < 0) return r;
      }
      return CLA_OK;
    });
    if (rc < 0) return rc;
    while (nextRange < LMM_PIPE)
      if ((rc = launch_range(nextRange++)) < 0) return rc;
  } else {
    for (int i = 0; i < LMM_PIPE; i++) {
      int64_t sb, se, rb, re;
      range_rows(i, sb, se, rb, re);
      if (re > rb) CLA_CUDA(cudaMemcpyAsync(dY + rb, hostY + rb, (size_t)(re - rb) * 8, cudaMemcpyHostToDevice, m->copyStream));
      if ((rc = launch_range(i)) < 0) return rc;
    }
  }
  if (m->hasConst && !A.constV)
    if ((rc = launch_lmm_const(m, dY, 1, dOut, s)) < 0) return rc;
  CLA_CUDA(cudaGetLastError());
  return 1;
}

// --------------------------------------------------------------------------------------------------
// t(y) %*% X without any device allocation.
//
// Some hosts may not allocate device memory when they call in: a runtime that has handed the whole GPU to
// its own memory pool (SystemDS's GPU memory manager works that way), or a service loop that must not hit
// cudaMalloc because the driver synchronises the device inside it. For them the per-CTA partial sums and the
// row sum of the left vector live in this fixed array instead of the handle's growable scratch. Every GPU
// whose context loads the library holds the array (about 450 KB) until the process exits.
// --------------------------------------------------------------------------------------------------
constexpr int NOALLOC_MAX_CTAS = 512;  // partial-sum rows available; one CTA per SM is launched, more only with > 148 column chunks
constexpr size_t NOALLOC_PARTIAL_DOUBLES = (size_t)NOALLOC_MAX_CTAS * (LMM_PART + 1);
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_PARTIAL_DOUBLES + 32];

static std::mutex g_noallocMu;
static double* g_noallocAddr[64] = {};  // device address of the array, per device ordinal

// The name g_noalloc_scratch is only a handle on the host; kernels need the address the device sees.
// Looked up once per device, with that device current.
static int64_t noalloc_address(int device, double** out) {
  if (device < 0 || device >= 64) return fail(CLA_ERR_BAD_ARG, "device ordinal out of range");
  std::lock_guard<std::mutex> lk(g_noallocMu);
  if (!g_noallocAddr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p)
      return fail(CLA_ERR_CUDA, std::string("cudaGetSymbolAddress(g_noalloc_scratch): ") + cudaGetErrorString(e));
    g_noallocAddr[device] = (double*)p;
  }
  *out = g_noallocAddr[device];
  return CLA_OK;
}

int64_t fast_lmm_vec_noalloc(Matrix* m, const double* dY, double* dOut, cudaStream_t s) {
  FastPlan* fp = m->fast;
  if (!fp || !fp->ok || fp->partial)
    return fail(CLA_ERR_UNSUPPORTED, "no-allocation product: needs dense-map groups with at most 256 tuples and byte maps");
  if ((uintptr_t)dY & 15) return fail(CLA_ERR_BAD_ARG, "no-allocation product: the left vector must be 16-byte aligned");
  LmmArgs A{};
  int grid;
  const size_t smem = lmm_args(m, fp, A, &grid);
  if (grid > NOALLOC_MAX_CTAS)
    return fail(CLA_ERR_UNSUPPORTED, "no-allocation product: the matrix needs " + std::to_string(grid) +
                                         " partial-sum rows, the fixed scratch holds " + std::to_string(NOALLOC_MAX_CTAS));
  double* scratch = nullptr;
  int64_t rc = noalloc_address(m->device, &scratch);
  if (rc < 0) return rc;
  m->stats.calls_lmm++;
  A.partial = scratch;                                 // fully rewritten by every launch
  double* rowSum = scratch + NOALLOC_PARTIAL_DOUBLES;  // accumulated with atomics: cleared below before use
  A.y = dY;
  A.out = dOut;
  if (A.addTo) CLA_CUDA(cudaMemsetAsync(dOut, 0, sizeof(double) * (size_t)m->nCols, s));
  if ((rc = launch_lmm_vec(m, A, grid, smem, s)) < 0) return rc;
  if (m->hasConst && !A.constV)
    if ((rc = launch_lmm_const_with(m, dY, 1, dOut, rowSum, s)) < 0) return rc;
  CLA_CUDA(cudaGetLastError());
  return CLA_OK;
}

}  // namespace cla
