// X %*% V for two or more columns of V, every group type, on the FP64 tensor cores.
//
// The columns of the dense-map (DDC, transcoded OLE) and uncompressed groups are one dense operand, multiplied with V by
// m16n8k8: this replaces dictionary pre-aggregation + decompress-and-sum (lib/CLALibRightMultBy.java:208-258) for those
// groups. SDC and RLE groups are added from their tables P_g = D_g * V[cols_g, :]
// (colgroup/ADictBasedColGroup.java:246-275) by way of the row lists (cla_rows.cu).
//
// k_rmm_wide: a warp owns 32 rows x 8 NT result columns in registers and needs no other warp. The A fragments are not
// staged: lane (g, t) looks up the values of its rows 4 g .. 4 g + 3 and columns t, t + 4 itself, four ids per load from the
// registered maps, the values from the columns' tables in shared memory, which hold a chunk of columns next to the
// matching rows of V for as long as the CTA walks its rows. With the values going straight into the fragments the L1 data
// pipe sees one random lookup per cell (about three wavefronts per 16 lanes) where decode -> stage -> fragment took
// three passes, and 32 rows share every V fragment. SDC / RLE table rows are added to the accumulators themselves: the
// four lanes of a row read its table row in 64-byte pieces.
// Bounds per 32 rows and eight columns: 32 NT clocks of the tensor pipe against about 50 (random lookups) + 14 + 4 NT of the
// L1 data pipe, so from 24 result columns on the tensor pipe is the limit.
#include "cla_common.cuh"
#include <algorithm>
#include <climits>
#include <cstring>

namespace cla {

constexpr int WD_WARPS = 16;  // (8 / 12 / 16 warps: 2212 / 1691 / 1523 us on 1M x 500 mixed, 64 columns)
constexpr int WD_T = WD_WARPS * 32;
constexpr size_t WD_SMEM = 228 * 1000;  // columns, tables and V of a chunk
constexpr int WD_TABLE = 4096;          // tuples of a table kept in shared memory, at most

__device__ __forceinline__ void dmma1688(double (&c)[4], double a0, double a1, double a2, double a3, double b0, double b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}
__device__ __forceinline__ double lds_at(uint32_t addr) {
  double v;
  asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr));
  return v;
}
// base + 8 * byte i of w, base + 8 * half i of w: one instruction each
__device__ __forceinline__ uint32_t at_byte(uint32_t w, int i, uint32_t base) {
  uint32_t a;
  asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(a) : "r"(w), "r"(8u << (8 * i)), "r"(base));
  return a;
}
__device__ __forceinline__ uint32_t at_half(uint32_t w, int i, uint32_t base) {
  uint32_t a;
  asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(a) : "r"(w), "r"(8u << (8 * i)), "r"(base));
  return a;
}

// A column of a chunk. src: dictionary (or dense block) + position in the group, for columns without a table here.
struct WideCol {
  const void* map;
  const void* mapHi;
  const double* src;
  int64_t imgAt;      // its values in the table image (doubles), -1: none
  int32_t tbl;        // byte offset of its table in the chunk's shared memory (-1: none)
  int32_t mapType, stride, vrow, nVals, pad;
};
struct WideChunk {
  int col0;            // first column
  int n[4];            // byte maps, 16-bit maps, other maps, uncompressed columns, in this order; kinds start at multiples of 8
  int nPad;            // columns with each kind rounded up to eights
  int tblBytes;        // tables
  int64_t img;         // their image (doubles)
};
// A sparse table row (tuple of an SDC / RLE group of one column): its value and where its row of V lies.
struct WideSv {
  double val;
  uint32_t at;  // bytes from the first sparse row of V in shared memory
  uint32_t pad;
};
struct WidePlanNT {
  bool tried = false, ok = false;
  int nSp = 0;                // rows of V kept for the SDC / RLE columns in the first chunk's CTAs; 0: tables P instead
  int32_t* spCols = nullptr;  // [nSp] matrix columns
  WideSv* sv = nullptr;       // [sparse table rows]
  std::vector<WideChunk> chunks;
  WideCol* cols = nullptr;
  double* image = nullptr;
  size_t smem = 0;
};
struct WidePlan {
  WidePlanNT nt[5];
};

struct WideArgs {
  const WideCol* cols;
  const double* image;
  WideChunk ch;
  int first, last;       // first / last chunk of the product
  int nRows, vCols;
  const double* V;
  // sparse groups (first chunk)
  const double* P;       // [table rows][vCols]
  const uint32_t *rowPtr, *rowItems, *fullPtr, *fullItems, *partPtr;
  const uint2* partItems;
  int nSp;               // > 0: the sparse groups from values and rows of V in shared memory, not from P
  const int32_t* spCols;
  const WideSv* sv;
  const double* constRow;
  double* out;
  int32_t* err;
  int vec2;              // rows of out and P are 16-byte aligned in pairs of columns
};

// image[at ...] = the column's dictionary values, contiguous
__global__ void k_wide_image(const WideCol* __restrict__ cols, int n, double* __restrict__ image) {
  if ((int)blockIdx.x >= n) return;
  const WideCol c = cols[blockIdx.x];
  if (c.imgAt < 0) return;
  for (int k = threadIdx.x; k < c.nVals; k += blockDim.x) image[c.imgAt + k] = c.src[(size_t)k * c.stride];
}
__global__ void k_wide_sv(const SparseVal* __restrict__ sv, int64_t nSv, const int32_t* __restrict__ slotOf, uint32_t rowBytes,
                          WideSv* __restrict__ out) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nSv; p += (int64_t)gridDim.x * blockDim.x) {
    const int slot = sv[p].col >= 0 ? slotOf[sv[p].col] : -1;
    out[p] = WideSv{sv[p].val, (uint32_t)max(slot, 0) * rowBytes, 0u};  // (groups without rows have no slot, and no items)
  }
}
// P[p][j] for every sparse table row
__global__ void k_wide_terms(const SparseVal* __restrict__ sv, int64_t nSv, const DevGroup* __restrict__ groups,
                             const int32_t* __restrict__ svOff, const double* __restrict__ V, int vCols, double* __restrict__ P) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nSv * vCols; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = e / vCols;
    const int j = (int)(e - p * vCols);
    const SparseVal s = sv[p];
    double x = 0.0;
    if (s.col >= 0) x = s.val * V[(size_t)s.col * vCols + j];
    else {
      const DevGroup& g = groups[s.group];
      const double* d = g.dict + (size_t)(p - svOff[s.group]) * g.gCols;
      for (int h = 0; h < g.gCols; h++) x += d[h] * V[(size_t)g.cols[h] * vCols + j];
    }
    P[e] = x;
  }
}
__global__ void k_wide_const(const double* __restrict__ constV, int nCols, const double* __restrict__ V, int vCols,
                             double* __restrict__ constRow) {
  const int j = blockIdx.x;  // a warp per result column
  double s = 0;
  for (int c = threadIdx.x; c < nCols; c += 32) s += constV[c] * V[(size_t)c * vCols + j];
  for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  if (threadIdx.x == 0) constRow[j] = s;
}

template <int NT>
__global__ void __launch_bounds__(WD_T, 1) k_rmm_wide(const __grid_constant__ WideArgs A) {
  constexpr int TN = NT * 8, LDB = TN + 4;  // = 4 mod 8: the V fragment loads are conflict free
  extern __shared__ __align__(128) unsigned char wsm[];
  __shared__ __align__(8) uint64_t mbar;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int j0 = blockIdx.y * TN, vc = min(TN, A.vCols - j0);
  // shared memory: tables | V rows [nPad][LDB] | map pointers [nPad] | table addresses [nPad]
  double* Vs = (double*)(wsm + A.ch.tblBytes);
  const void** mapOf = (const void**)(Vs + (size_t)A.ch.nPad * LDB);
  uint32_t* tblOf = (uint32_t*)(mapOf + A.ch.nPad);
  double* spV = (double*)(tblOf + ((A.ch.nPad + 3) & ~3));  // [nSp][LDB]
  const char* spB = (const char*)spV;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(wsm);
  if (A.ch.tblBytes) {
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&mbar);
    if (tid == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)A.ch.tblBytes) : "memory");
      for (uint32_t off = 0; off < (uint32_t)A.ch.tblBytes; off += 32768) {
        const uint32_t sz = min(32768u, (uint32_t)A.ch.tblBytes - off);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(base + off),
                     "l"((const char*)(A.image + A.ch.img) + off), "r"(sz), "r"(bar)
                     : "memory");
      }
    }
  }
  for (int e = tid; e < A.ch.nPad * TN; e += WD_T) {
    const int k = e / TN, n = e - k * TN;
    const int vr = A.cols[A.ch.col0 + k].vrow;
    Vs[k * LDB + n] = (vr >= 0 && n < vc) ? A.V[(size_t)vr * A.vCols + j0 + n] : 0.0;
  }
  for (int e = tid; e < A.nSp * TN; e += WD_T) {
    const int k = e / TN, n = e - k * TN;
    spV[k * LDB + n] = n < vc ? A.V[(size_t)A.spCols[k] * A.vCols + j0 + n] : 0.0;
  }
  for (int k = tid; k < A.ch.nPad; k += WD_T) {
    const WideCol& c = A.cols[A.ch.col0 + k];
    mapOf[k] = c.mapType < 0 ? (const void*)c.src : c.map;
    tblOf[k] = c.mapType < 0 ? (c.vrow >= 0 ? (uint32_t)c.stride : 0u) : (c.tbl >= 0 ? base + (uint32_t)c.tbl : 0u);
  }
  __syncthreads();
  if (A.ch.tblBytes) {
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&mbar);
    uint32_t done = 0;
    for (int it = 0; it < (1 << 22) && !done; it++)
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(done)
                   : "r"(bar), "r"(0u)
                   : "memory");
    if (!__syncthreads_and(done != 0)) {
      if (tid == 0) atomicExch(A.err, 110);
      return;
    }
  }
  const int nWin = (A.nRows + WIN_ROWS - 1) / WIN_ROWS;
  const int kC = (A.ch.n[0] + 7) / 8, kO = kC + (A.ch.n[1] + 7) / 8, kU = kO + (A.ch.n[2] + 7) / 8, kE = kU + (A.ch.n[3] + 7) / 8;
  // windows are dealt to the SMs first, then to their warps: short matrices use every SM
  for (int w = warp * gridDim.x + blockIdx.x; w < nWin; w += gridDim.x * WD_WARPS) {
    double full[2] = {0.0, 0.0};  // runs over the whole window: lane = result column
    if (A.fullPtr && A.nSp) {
      const uint32_t q1 = A.fullPtr[w + 1];
      for (uint32_t p = A.fullPtr[w]; p < q1; p += 32) {  // a lane per item, then every item by all lanes
        WideSv mine = {0.0, 0u, 0u};
        if (p + lane < q1) mine = A.sv[A.fullItems[p + lane]];
        const int n = (int)min(32u, q1 - p);
        for (int u = 0; u < n; u++) {
          const double x = __shfl_sync(0xffffffffu, mine.val, u);
          const uint32_t at = __shfl_sync(0xffffffffu, mine.at, u);
          if (lane < TN) full[0] = fma(x, *(const double*)(spB + at + lane * 8), full[0]);
        }
      }
    } else if (A.fullPtr && lane < vc) {
      const uint32_t q1 = A.fullPtr[w + 1];
      for (uint32_t p = A.fullPtr[w]; p < q1; p += 8) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = p + u < q1 ? A.P[(size_t)A.fullItems[p + u] * A.vCols + j0 + lane] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; u++) full[0] += x[u];
      }
    }
    if (A.constRow && A.last && lane < vc) full[1] = A.constRow[j0 + lane];
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
      const int row0 = w * WIN_ROWS + half * 32, row = row0 + 4 * g;
      if (row0 >= A.nRows) break;
      const bool whole = row0 + 32 <= A.nRows;
      double c[2][NT][4];  // tile i: rows 4 g + 2 i (c[0], c[1]) and 4 g + 2 i + 1 (c[2], c[3]), columns 8 n + 2 t + {0, 1}
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
          for (int u = 0; u < 4; u++) {
            c[i][n][u] = 0.0;
            if (!A.first) {
              const int r = row + 2 * i + (u >> 1), j = n * 8 + 2 * t + (u & 1);
              if (r < A.nRows && j < vc) c[i][n][u] = A.out[(size_t)r * A.vCols + j0 + j];
            }
          }
      auto multiply = [&](int ks, const double (&x0)[4], const double (&x1)[4]) {
        const double* v0 = Vs + (ks * 8 + t) * LDB + g;
#pragma unroll
        for (int n = 0; n < NT; n++) {
          const double b0 = v0[n * 8], b1 = v0[n * 8 + 4 * LDB];
          dmma1688(c[0][n], x0[0], x0[1], x1[0], x1[1], b0, b1);
          dmma1688(c[1][n], x0[2], x0[3], x1[2], x1[3], b0, b1);
        }
      };
      int ks = 0;
      if (whole) {
        // byte maps: the ids of the next eight columns are in flight while these are looked up and multiplied
        uint32_t w0 = 0, w1 = 0;
        if (kC > 0) {
          w0 = __ldg((const uint32_t*)((const uint8_t*)mapOf[t] + row));
          w1 = __ldg((const uint32_t*)((const uint8_t*)mapOf[4 + t] + row));
        }
        for (; ks < kC; ks++) {
          const uint32_t a0 = w0, a1 = w1;
          if (ks + 1 < kC) {
            w0 = __ldg((const uint32_t*)((const uint8_t*)mapOf[ks * 8 + 8 + t] + row));
            w1 = __ldg((const uint32_t*)((const uint8_t*)mapOf[ks * 8 + 12 + t] + row));
          }
          const uint32_t t0 = tblOf[ks * 8 + t], t1 = tblOf[ks * 8 + 4 + t];
          double x0[4], x1[4];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            x0[i] = lds_at(at_byte(a0, i, t0));
            x1[i] = lds_at(at_byte(a1, i, t1));
          }
          multiply(ks, x0, x1);
        }
        // 16-bit maps
        uint2 h0 = make_uint2(0, 0), h1 = h0;
        if (kC < kO) {
          h0 = __ldg((const uint2*)((const uint16_t*)mapOf[kC * 8 + t] + row));
          h1 = __ldg((const uint2*)((const uint16_t*)mapOf[kC * 8 + 4 + t] + row));
        }
        for (; ks < kO; ks++) {
          const uint2 a0 = h0, a1 = h1;
          if (ks + 1 < kO) {
            h0 = __ldg((const uint2*)((const uint16_t*)mapOf[ks * 8 + 8 + t] + row));
            h1 = __ldg((const uint2*)((const uint16_t*)mapOf[ks * 8 + 12 + t] + row));
          }
          const uint32_t t0 = tblOf[ks * 8 + t], t1 = tblOf[ks * 8 + 4 + t];
          double x0[4], x1[4];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            x0[i] = lds_at(at_half(i < 2 ? a0.x : a0.y, i & 1, t0));
            x1[i] = lds_at(at_half(i < 2 ? a1.x : a1.y, i & 1, t1));
          }
          multiply(ks, x0, x1);
        }
      }
      // other maps, and every map in the last rows of the matrix (rows past the end repeat the last one and are not stored)
      for (; ks < kU; ks++) {
        double x[2][4];
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const int k = ks * 8 + 4 * q + t;
          const WideCol& cd = A.cols[A.ch.col0 + k];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            x[q][i] = 0.0;
            if (cd.vrow >= 0) {
              const int id = map_get(cd.mapType, cd.map, cd.mapHi, min(row + i, A.nRows - 1));
              x[q][i] = cd.tbl >= 0 ? lds_at(tblOf[k] + 8u * id) : cd.src[(size_t)id * cd.stride];
            }
          }
        }
        multiply(ks, x[0], x[1]);
      }
      // uncompressed columns
      for (; ks < kE; ks++) {
        double x[2][4];
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const int k = ks * 8 + 4 * q + t;
          const uint32_t stride = tblOf[k];  // columns of the group (0: padding)
          const double* s = (const double*)mapOf[k];
#pragma unroll
          for (int i = 0; i < 4; i++) x[q][i] = stride ? __ldcs(s + (size_t)min(row + i, A.nRows - 1) * stride) : 0.0;
        }
        multiply(ks, x[0], x[1]);
      }
      // SDC: the listed tuples of the lane's rows; the four lanes of a row read 64 bytes of a table row per n
      if (A.rowPtr && A.nSp) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int r = row + i;
          uint32_t p = 0, p1 = 0;
          if (r < A.nRows) {
            p = A.rowPtr[r];
            p1 = A.rowPtr[r + 1];
          }
          for (; p < p1; p += 4) {  // four items in flight
            WideSv e[4];
#pragma unroll
            for (int u = 0; u < 4; u++) e[u] = p + u < p1 ? A.sv[A.rowItems[p + u]] : WideSv{0.0, 0u, 0u};
#pragma unroll
            for (int u = 0; u < 4; u++)
              if (p + u < p1) {
                const char* q = spB + e[u].at + 2 * t * 8;
#pragma unroll
                for (int n = 0; n < NT; n++) {
                  const double2 v = *(const double2*)(q + n * 64);
                  double* d = &c[i >> 1][n][(i & 1) * 2];
                  d[0] = fma(e[u].val, v.x, d[0]);
                  d[1] = fma(e[u].val, v.y, d[1]);
                }
              }
          }
        }
      } else if (A.rowPtr) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int r = row + i;
          uint32_t p = 0, p1 = 0;
          if (r < A.nRows) {
            p = A.rowPtr[r];
            p1 = A.rowPtr[r + 1];
          }
          for (; p < p1; p += 2) {
            const double* q0 = A.P + (size_t)A.rowItems[p] * A.vCols + j0 + 2 * t;
            const bool two = p + 1 < p1;
            const double* q1 = two ? A.P + (size_t)A.rowItems[p + 1] * A.vCols + j0 + 2 * t : q0;
            double2 u0[NT], u1[NT];
            if (A.vec2) {
#pragma unroll
              for (int n = 0; n < NT; n++) {
                const bool in = n * 8 + 2 * t < vc;  // vc is even
                u0[n] = in ? *(const double2*)(q0 + n * 8) : make_double2(0.0, 0.0);
                u1[n] = (in && two) ? *(const double2*)(q1 + n * 8) : make_double2(0.0, 0.0);
              }
            } else {
#pragma unroll
              for (int n = 0; n < NT; n++) {
                const bool x = n * 8 + 2 * t < vc, y = n * 8 + 2 * t + 1 < vc;
                u0[n] = make_double2(x ? q0[n * 8] : 0.0, y ? q0[n * 8 + 1] : 0.0);
                u1[n] = make_double2(x && two ? q1[n * 8] : 0.0, y && two ? q1[n * 8 + 1] : 0.0);
              }
            }
#pragma unroll
            for (int n = 0; n < NT; n++) {
              double* d = &c[i >> 1][n][(i & 1) * 2];
              d[0] = (d[0] + u0[n].x) + u1[n].x;
              d[1] = (d[1] + u0[n].y) + u1[n].y;
            }
          }
        }
      }
      // RLE: pieces of the window, then the runs over all of it and the constants
      if (A.fullPtr) {
        const uint32_t q1 = A.partPtr[w + 1];
        for (uint32_t p = A.partPtr[w]; p < q1; p++) {
          const uint2 it = A.partItems[p];
          const int ra = (int)(it.y & 0xFF) - half * 32, rb = (int)(it.y >> 8) - half * 32;
          if (rb <= 0 || ra >= 32) continue;
          const double* q = A.P + (size_t)it.x * A.vCols + j0 + 2 * t;
          WideSv e = {0.0, 0u, 0u};
          if (A.nSp) e = A.sv[it.x];
#pragma unroll
          for (int n = 0; n < NT; n++) {
            double x, y;
            if (A.nSp) {
              const double2 v = *(const double2*)(spB + e.at + (2 * t + n * 8) * 8);
              x = e.val * v.x, y = e.val * v.y;
            } else {
              x = n * 8 + 2 * t < vc ? q[n * 8] : 0.0;
              y = n * 8 + 2 * t + 1 < vc ? q[n * 8 + 1] : 0.0;
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
              if (4 * g + i >= ra && 4 * g + i < rb) {
                c[i >> 1][n][(i & 1) * 2] += x;
                c[i >> 1][n][(i & 1) * 2 + 1] += y;
              }
          }
        }
      }
      if (A.fullPtr || (A.constRow && A.last)) {
        const double add = full[0] + full[1];
#pragma unroll
        for (int n = 0; n < NT; n++) {
          const double x = __shfl_sync(0xffffffffu, add, n * 8 + 2 * t), y = __shfl_sync(0xffffffffu, add, n * 8 + 2 * t + 1);
#pragma unroll
          for (int i = 0; i < 2; i++) {
            c[i][n][0] += x, c[i][n][2] += x;
            c[i][n][1] += y, c[i][n][3] += y;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int r = row + i;
        if (r < A.nRows) {
          double* o = A.out + (size_t)r * A.vCols + j0 + 2 * t;
#pragma unroll
          for (int n = 0; n < NT; n++) {
            const double x = c[i >> 1][n][(i & 1) * 2], y = c[i >> 1][n][(i & 1) * 2 + 1];
            if (A.vec2) {
              if (n * 8 + 2 * t < vc) *(double2*)(o + n * 8) = make_double2(x, y);
            } else {
              if (n * 8 + 2 * t < vc) o[n * 8] = x;
              if (n * 8 + 2 * t + 1 < vc) o[n * 8 + 1] = y;
            }
          }
        }
      }
    }
  }
}

// --------------------------------------------------------------------------------------------------
// plan: columns by kind, cut into chunks that fit shared memory next to their rows of V
// --------------------------------------------------------------------------------------------------
void wide_plan_free(Matrix* m) {
  delete m->wide;
  m->wide = nullptr;
}

static int64_t ensure_wide(Matrix* m, int NT, cudaStream_t s) {
  if (!m->wide) m->wide = new WidePlan();
  if (m->wide->nt[NT].tried) return CLA_OK;
  WidePlanNT W;  // takes its place in the handle when it is complete (after an error the next call tries again)
  W.tried = true;
  std::vector<WideCol> kind[4];
  for (size_t hi = 0; hi < m->hg.size(); hi++) {
    const int gi = m->regToDev[hi];
    if (gi < 0) continue;
    const DevGroup& g = m->groups[gi];
    if (g.type != GT_DDC && g.type != GT_UNC) continue;
    for (int j = 0; j < g.gCols; j++) {
      WideCol c{};
      c.map = g.map;
      c.mapHi = g.mapHi;
      c.src = (g.type == GT_UNC ? g.dense : g.dict) + j;
      c.mapType = g.type == GT_UNC ? -1 : g.mapType;
      c.stride = g.gCols;
      c.vrow = m->hg[hi].cols[j];
      c.nVals = g.nVals;
      c.tbl = -1;
      c.imgAt = -1;
      const bool resident = g.type == GT_DDC && g.nVals <= WD_TABLE;
      if (resident) c.tbl = 0;
      const bool bytes = g.mapType == CLA_MAP_UBYTE || g.mapType == CLA_MAP_BYTE;
      kind[g.type == GT_UNC ? 3 : (resident && bytes ? 0 : (resident && g.mapType == CLA_MAP_CHAR ? 1 : 2))].push_back(c);
    }
  }
  const size_t perCol = (size_t)(NT * 8 + 4) * 8 + 12;
  auto cost = [&](const WideCol& c) { return perCol + (c.tbl >= 0 ? (((size_t)c.nVals * 8 + 15) & ~(size_t)15) : 0); };
  // Rows of V of the SDC / RLE columns, next to the first chunk, where they take at most half of it and every such group
  // has one column: reading table rows P = D V (eight tuples and 64 columns: 4 KB a column) from L2 instead was 3.8 GB per
  // product on 1M x 500 mixed, 64 columns of V (1.51 ms; 1.41 ms so).
  std::vector<int32_t> spCols, slotOf(m->nCols, -1);
  bool single = true;
  for (size_t hi = 0; hi < m->hg.size(); hi++) {
    const int gi = m->regToDev[hi];
    if (gi < 0) continue;
    const DevGroup& g = m->groups[gi];
    if (!((g.type == GT_SDC && g.nOff > 0) || (g.type == GT_RLE && g.nRuns > 0))) continue;
    single &= g.gCols == 1;
    const int c = m->hg[hi].cols[0];
    if (slotOf[c] < 0) {
      slotOf[c] = (int)spCols.size();
      spCols.push_back(c);
    }
  }
  const size_t rowB = (size_t)(NT * 8 + 4) * 8;
  if (!single || spCols.size() * rowB > WD_SMEM / 2) spCols.clear();
  W.nSp = (int)spCols.size();
  const size_t spBytes = spCols.size() * rowB;
  size_t total = spBytes;
  for (auto& k : kind)
    for (auto& c : k) total += cost(c);
  // Kinds are padded to eights. A padding column of the first two kinds reads the map of the matrix' column of that kind
  // with the fewest tuples, but looks its ids up in zeros at the start of the tables (0 times a row of V that is 0).
  WideCol padCol[2];
  int64_t zeroBytes = 16;
  for (int k = 0; k < 2; k++)
    if (!kind[k].empty()) {
      padCol[k] = *std::min_element(kind[k].begin(), kind[k].end(), [](const WideCol& a, const WideCol& b) { return a.nVals < b.nVals; });
      zeroBytes = std::max<int64_t>(zeroBytes, ((int64_t)padCol[k].nVals * 8 + 15) & ~(int64_t)15);
    }
  const size_t room = WD_SMEM - 4 * 8 * perCol - 256 - (size_t)zeroBytes;
  const size_t want = total / std::max<size_t>(1, (total + room - 1) / room) + 4096;  // even chunks
  std::vector<WideCol> cols;
  WideChunk ch{};
  std::vector<WideCol> cur[4];
  int64_t img = 0;
  auto flush = [&]() {
    ch = WideChunk{};
    ch.col0 = (int)cols.size();
    ch.img = img;
    int64_t tb = zeroBytes;
    for (int k = 0; k < 4; k++) {
      ch.n[k] = (int)cur[k].size();
      for (auto& c : cur[k]) {
        if (c.tbl >= 0) {
          c.tbl = (int32_t)tb;
          c.imgAt = img + tb / 8;
          tb += ((int64_t)c.nVals * 8 + 15) & ~(int64_t)15;
        }
        if (k == 3) c.tbl = -1;
        cols.push_back(c);
      }
      while (((int)cols.size() - ch.col0) % 8 != 0) {
        WideCol pad = k < 2 ? padCol[k] : cur[k][0];
        pad.vrow = -1;
        pad.imgAt = -1;
        pad.tbl = k < 2 ? 0 : -1;
        cols.push_back(pad);
      }
      cur[k].clear();
    }
    ch.nPad = (int)cols.size() - ch.col0;
    ch.tblBytes = (int)tb;
    img += tb / 8;
    W.chunks.push_back(ch);
  };
  size_t used = spBytes;
  bool any = false;
  for (int k = 0; k < 4; k++)
    for (auto& c : kind[k]) {
      const size_t b = cost(c);
      if (any && used + b > std::min(want, room)) {
        flush();
        used = 0;
      }
      cur[k].push_back(c);
      any = true;
      used += b;
    }
  flush();
  for (size_t i = 0; i < W.chunks.size(); i++)
    W.smem = std::max(W.smem, (size_t)W.chunks[i].tblBytes + (size_t)W.chunks[i].nPad * perCol + (i == 0 ? spBytes : 0) + 64);
  void* d = nullptr;
  const size_t bc = (cols.size() * sizeof(WideCol) + 255) & ~(size_t)255;
  const size_t bi = ((size_t)img * 8 + 255) & ~(size_t)255, bs = ((size_t)W.nSp * 4 + 255) & ~(size_t)255;
  const size_t bl = ((size_t)m->nCols * 4 + 255) & ~(size_t)255, bv = W.nSp ? (size_t)m->rows.nSv * sizeof(WideSv) : 0;
  if (plan_alloc(m, &d, bc + bi + bs + bl + bv) < 0) {
    m->wide->nt[NT].tried = true;
    return CLA_OK;
  }
  W.spCols = (int32_t*)((char*)d + bc + bi);
  W.sv = (WideSv*)((char*)d + bc + bi + bs + bl);
  if (W.nSp) {
    int32_t* slots = (int32_t*)((char*)d + bc + bi + bs);
    CLA_CUDA(cudaMemcpyAsync(W.spCols, spCols.data(), spCols.size() * 4, cudaMemcpyHostToDevice, s));
    CLA_CUDA(cudaMemcpyAsync(slots, slotOf.data(), slotOf.size() * 4, cudaMemcpyHostToDevice, s));
    k_wide_sv<<<(unsigned)std::min<int64_t>(1024, (m->rows.nSv + 255) / 256), 256, 0, s>>>(m->rows.sv, m->rows.nSv, slots, (uint32_t)rowB, W.sv);
  }
  W.cols = (WideCol*)d;
  W.image = (double*)((char*)d + bc);
  CLA_CUDA(cudaMemsetAsync(W.image, 0, (size_t)img * 8, s));
  CLA_CUDA(cudaMemcpyAsync(W.cols, cols.data(), cols.size() * sizeof(WideCol), cudaMemcpyHostToDevice, s));
  if (!cols.empty()) k_wide_image<<<(unsigned)cols.size(), 128, 0, s>>>(W.cols, (int)cols.size(), W.image);
  CLA_CUDA(cudaGetLastError());
  CLA_CUDA(cudaStreamSynchronize(s));
  W.ok = true;
  m->wide->nt[NT] = std::move(W);
  return CLA_OK;
}

// 1 = done, 0 = not covered (no row lists or no plan: the caller takes the general kernel)
int64_t wide_rmm(Matrix* m, const double* dV, int vCols, double* dOut, cudaStream_t s) {
  if (m->nRows == 0 || vCols == 0) return 1;
  int64_t rc;
  if ((rc = ensure_row_lists(m, s)) < 0) return rc;
  const RowLists& L = m->rows;
  if (!L.ok) return 0;
  const int slices = (vCols + 31) / 32, NT = ((vCols + slices - 1) / slices + 7) / 8;
  if ((rc = ensure_wide(m, NT, s)) < 0) return rc;
  const WidePlanNT& W = m->wide->nt[NT];
  if (!W.ok) return 0;
  const bool sparse = (L.nSdc > 0 || L.nRle > 0) && W.nSp == 0;  // needs the tables P
  const size_t pBytes = sparse ? (((size_t)L.nSv * vCols * sizeof(double) + 255) & ~(size_t)255) : 0;
  if ((rc = ensure_scratch(m, pBytes + (size_t)vCols * sizeof(double) + 256)) < 0) return rc;
  WideArgs A{};
  A.cols = W.cols;
  A.image = W.image;
  A.nRows = m->nRows;
  A.vCols = vCols;
  A.V = dV;
  A.out = dOut;
  A.err = m->dErr;
  A.vec2 = (vCols % 2 == 0 && ((uintptr_t)dOut & 15) == 0) ? 1 : 0;
  A.P = (const double*)m->scratch;
  if (sparse) {
    k_wide_terms<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(4096, (L.nSv * vCols + 255) / 256)), 256, 0, s>>>(
        L.sv, L.nSv, m->dGroups, L.svOff, dV, vCols, (double*)m->scratch);
    m->stats.kernel_launches++;
  }
  if (m->hasConst) {
    A.constRow = (const double*)((char*)m->scratch + pBytes);
    k_wide_const<<<vCols, 32, 0, s>>>(m->dConstV, m->nCols, dV, vCols, (double*)A.constRow);
    m->stats.kernel_launches++;
  }
  static OncePerDevice once;
  if (const int64_t e = allow_smem(once, m->device, WD_SMEM + 1024, k_rmm_wide<1>, k_rmm_wide<2>, k_rmm_wide<3>, k_rmm_wide<4>); e < 0) return e;
  const int gridY = (vCols + NT * 8 - 1) / (NT * 8), nWin = (m->nRows + WIN_ROWS - 1) / WIN_ROWS;
  const dim3 grid((unsigned)std::max(1, std::min(nWin, m->smCount / gridY)), gridY);
  auto kern = NT == 1 ? k_rmm_wide<1> : (NT == 2 ? k_rmm_wide<2> : (NT == 3 ? k_rmm_wide<3> : k_rmm_wide<4>));
  prof_begin(m, s);
  for (size_t i = 0; i < W.chunks.size(); i++) {
    A.ch = W.chunks[i];
    A.first = i == 0;
    A.last = i + 1 == W.chunks.size();
    A.nSp = A.first ? W.nSp : 0;
    A.spCols = W.spCols;
    A.sv = W.sv;
    A.rowPtr = (A.first && L.nSdc) ? L.rowPtr : nullptr;
    A.rowItems = L.rowItems;
    A.fullPtr = (A.first && L.nRle) ? L.fullPtr : nullptr;
    A.fullItems = L.fullItems;
    A.partPtr = L.partPtr;
    A.partItems = L.partItems;
    kern<<<grid, WD_T, W.smem, s>>>(A);
    m->stats.kernel_launches++;
  }
  prof_end(m, s);
  CLA_CUDA(cudaGetLastError());
  return 1;
}

}  // namespace cla
