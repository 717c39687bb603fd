// FP64 refinement of the log-Pfaffian with the pivot order of the FP32 factorisation.
//
// The FP32 kernel (nh_pfaffian.cu) does the part of Parlett-Reid that is latency-bound: the 112
// sequential pivot searches at n = 224.  It records the pivot order it chose (logical index ->
// physical row, plus the parity of the relabelling).  This kernel factorises the same matrix
// again in FP64 with that order held fixed (static pivoting): with no pivot search the
// elimination is blocked into panels of 4 steps (8 logical columns) whose trailing update is a
// rank-8 FP64 product, and it returns the FP64 pivots x_t, so log|pf| = sum_t log|x_t| and
// sign(pf) = item sign x parity x prod_t sign(x_t).  The FP32 pivots bound the multipliers of the
// FP32 matrix by 1, and those of the FP64 one stay there (beyond_bound says how far) unless the
// FP32 run broke down or its last columns were rounding noise, so the fixed order is as stable as
// partial pivoting; the result carries FP64 rounding only, against ~1e-4 for the FP32 factorisation
// of an ill-conditioned block.
//
// The matrix is refined against its own FP32 entries (the bits the FP32 kernel factorised, so
// the result is log|pf| of that FP32 matrix to FP64 accuracy) or against the FP64 matrix
// gathered from FP64 features (images flagged ill-conditioned or cancelling, whose FP32 features
// are not accurate enough).  The gather follows pf_kernel.py:156-166 of the reference:
// F[p, q] = sum_a (Y[p, a] Y[q, a]) Wt[2 s_p + s_q, r(p, q), a], in the same order of operations
// as the FP32 gather so that the FP32 matrix is reproduced bit for bit.
//
// One CTA of 512 threads per SM (two of 256 where the lattice is small).  Phase 1 fills the permuted
// lower triangle in shared memory, stored as 8 x 8 FP64 tiles (tile (I, J <= I) at index
// I (I + 1) / 2 + J; 16-byte chunks swizzled inside a tile, see toff); phase 2 eliminates panels of
// 8 columns: one warp factorises the 8 x 8 pivot block, the panel rows are multiplied by the inverse
// of its unit factor, and the trailing tiles take P W^T, all as m8n8k4 FP64 products.  The next
// panel's column is updated first, so that its pivot block (a serial chain) is factorised by warp 0
// while the other warps update the rest.  n <= kRefineMaxN (224: the tiles take 203 KB); larger
// matrices in refine_big_kernel.
#include <cooperative_groups.h>
#include <limits.h>
#include <math.h>

#include <algorithm>

#include "nh_cnn_item.cuh"
#include "nh_cnn_mma.cuh"
#include "nh_common.cuh"

namespace nh {
namespace {

constexpr int kPW = 8;  // panel width: 4 elimination steps

// Modes 1 and 3 (FP32 entries): row a of a packed lower triangle in the CTA's slice starts at
// roff(a).
__host__ __device__ __forceinline__ int roff(int a) { return (a * (a - 1)) / 2 + a / 2; }
__host__ __device__ __forceinline__ int tile_rows(int n) { return (n + 7) >> 3; }
__host__ __device__ __forceinline__ int tile_base(int I) { return (I * (I + 1)) >> 1; }
// Bytes of the tiles of rows < I.
__host__ __device__ __forceinline__ size_t tile_bytes(int I) { return 512 * (size_t)tile_base(I); }
// Offset of element (r, c) in an 8 x 8 tile: the row's four 16-byte chunks are XOR-ed with the bit
// reversal of r / 2, so that 8 rows of one chunk (the panel solve), 2 rows of all chunks (an MMA
// accumulator) and 4 rows x 4 columns of doubles (an MMA operand) all hit distinct banks.
__device__ __forceinline__ int toff(int r, int c) {
  const int f = (r & 2) | ((r >> 2) & 1);
  return r * 8 + ((((c >> 1) ^ f) << 1) | (c & 1));
}
// Bytes of one CTA's slice: the tiles, the packed FP32 triangle, or an item's rows and modes
// (mode 3), whichever is largest; a multiple of 16.
__host__ __device__ __forceinline__ size_t slice_stride(int n, int d) {
  const size_t tri = tile_bytes(tile_rows(n)), rows = 8 * (size_t)n * d + 4 * (size_t)n;
  return ((tri > rows ? tri : rows) + 15) & ~(size_t)15;
}

struct RefineArgs {
  int n;
  int mode;  // 0: dense FP32 F (items, n, n); 1: gather FP32 (Y, idx by item); 2: gather FP64
             // (Y64, idx64 by slot, Wt64); 3 / 4: FP32 / FP64 features computed in the kernel
             // from the configuration list, then gathered (Wt / Wt64)
  ConfigList cl;       // modes 3, 4
  const float* cnn_w;  // modes 3, 4: packed weights [l][ci][tap][co]
  const float* cnn_b;
  int C, layers;
  const float* F;
  const void* Y;
  const int32_t* idx;
  const void* Wt;
  int Lx, Ly, D;
  bool stage_wt;  // Wt (modes 2, 4: one spin block of it) fits in shared memory with the rows
  const int32_t* list;   // slot -> item
  const int32_t* count;  // device number of slots; beyond [min_count, max_count] nothing is done
  int min_count, max_count;
  const uint16_t* perm;  // per item: perm[0, n) logical -> physical, [n] relabelling parity
  int perm_stride;       // uint16 per item
  const float* item_sign;  // (items,) or null
  float* sign;
  double* logabs;
  int32_t* flags;
  void* slice;  // per CTA: slice_stride(n, D) bytes
  // modes 2, 4 (byte offsets in dynamic shared memory): rows Y, packed modes, one spin block of
  // Wt64 (stage_wt); tiles of rows >= keep overlap them and go through the slice.
  int y_off, info_off, wt_off, keep;
  bool rows_slice;  // mode 4: no room for Y above the CNN, its rows pass through the slice
};

// Phase 1 of modes 1 and 3: logical lower triangle A[p][q] = F[perm p][perm q] of one item, FP32,
// into the CTA's slice.  Warp <-> 32 consecutive logical columns q (their features in registers when
// small), rows p > q in turn (the row's features broadcast); each element reads one Wt row.
template <int D, int TH>
__device__ void gather_permuted(const RefineArgs& a, const float* Yg, const int32_t* ig,
                                const uint16_t* perm, unsigned char* smem, float* slice) {
  const int n = a.n, N = a.Lx * a.Ly;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int DP = D + 4, VK = 4;
  const float* Wg = static_cast<const float*>(a.Wt);
  float* ys = reinterpret_cast<float*>(smem);                    // (n, DP)
  int* info = reinterpret_cast<int*>(ys + n * DP);               // (n) spin << 16 | x << 8 | y
  float* wts = reinterpret_cast<float*>(info + ((n + 3) & ~3));  // (4 N, DP) when staged
  // Row r of the source (D values, 16-byte vectors) to row r of the padded staging copy; several
  // vectors in flight per thread.  Read-only tables (nc) take the non-coherent path; the rows,
  // which mode 3 writes in this kernel, plain loads.
  auto stage = [&](const float* src, float* dst, int rows, bool nc) {
    constexpr int VPR = D / VK;  // vectors per row
    const int nv = rows * VPR;
    for (int v0 = tid; v0 < nv; v0 += 4 * TH) {
      float4 buf[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int v = v0 + u * TH;
        if (v < nv) buf[u] = nc ? __ldg(reinterpret_cast<const float4*>(src) + v)
                                : reinterpret_cast<const float4*>(src)[v];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int v = v0 + u * TH;
        if (v < nv) {
          const int r = v / VPR;
          *reinterpret_cast<float4*>(dst + r * DP + (v - r * VPR) * VK) = buf[u];
        }
      }
    }
  };
  stage(Yg, ys, n, false);
  for (int p = tid; p < n; p += TH) {
    const int m = ig[p];
    const int sp = m >= N ? 1 : 0, site = m - sp * N, x = site / a.Ly;
    info[p] = (sp << 16) | (x << 8) | (site - x * a.Ly);
  }
  if (a.stage_wt) stage(Wg, wts, 4 * N, true);
  __syncthreads();
  int total = 0;
  for (int qb = 0; 32 * qb + 1 < n; ++qb) total += n - 32 * qb - 1;
  int qb = 0, rem = wid, cur = -1, j = 0, infj = 0;
  // The column's features stay in registers when they are small, else they are read per element.
  constexpr bool kRegs = D <= 16;
  float yj[kRegs ? D : 1];
#pragma unroll 1
  for (int u = wid; u < total; u += (TH / 32), rem += (TH / 32)) {
    while (rem >= n - 32 * qb - 1) {
      rem -= n - 32 * qb - 1;
      ++qb;
    }
    const int q = 32 * qb + lane;
    if (qb != cur) {
      cur = qb;
      j = perm[q < n ? q : 0];
      infj = info[j];
      if constexpr (kRegs) {
#pragma unroll
        for (int c = 0; c < D; c += VK)
          *reinterpret_cast<float4*>(yj + c) = *reinterpret_cast<const float4*>(ys + j * DP + c);
      }
    }
    const int p = 32 * qb + 1 + rem;
    if (q >= p) continue;
    const int i = perm[p];
    const int infi = info[i];
    const bool up = i > j;  // row i is the higher physical row
    const int ih = up ? infi : infj, il = up ? infj : infi;
    int dx = ((ih >> 8) & 0xFF) - ((il >> 8) & 0xFF), dy = (ih & 0xFF) - (il & 0xFF);
    dx += dx < 0 ? a.Lx : 0;
    dy += dy < 0 ? a.Ly : 0;
    const int r = (2 * (ih >> 16) + (il >> 16)) * N + dx * a.Ly + dy;
    // yi[c] * yj[c] equals the FP32 gather's row-times-column product bit for bit (the product
    // commutes); the accumulation order over c is the gather's.
    const float* yi = ys + i * DP;
    const float* wr = a.stage_wt ? wts + r * DP : Wg + (size_t)r * D;
    float acc = 0.0f;
#pragma unroll
    for (int c = 0; c < D; c += VK) {
      float vi[VK], vw[VK], vj[VK];
      *reinterpret_cast<float4*>(vi) = *reinterpret_cast<const float4*>(yi + c);
      if (a.stage_wt)
        *reinterpret_cast<float4*>(vw) = *reinterpret_cast<const float4*>(wr + c);
      else
        *reinterpret_cast<float4*>(vw) = __ldg(reinterpret_cast<const float4*>(wr + c));
      if constexpr (kRegs) {
#pragma unroll
        for (int k = 0; k < VK; ++k) vj[k] = yj[c + k];
      } else {
        *reinterpret_cast<float4*>(vj) = *reinterpret_cast<const float4*>(ys + j * DP + c);
      }
#pragma unroll
      for (int k = 0; k < VK; ++k) acc = fma(vi[k] * vj[k], vw[k], acc);
    }
    slice[roff(p) + q] = up ? acc : -acc;
  }
}

// Phase 1 of modes 2 and 4: F[i][j] = sum_a (Y[i, a] Y[j, a]) Wt[2 s_i + s_j, r(i, j), a] of the
// physical pairs i > j, scattered with its sign to the logical tile.  LPR lanes share a pair, each
// with CPL 16-byte chunks of the a; a table row is then read in contiguous pieces (no bank
// conflicts, where one lane per pair read 32 scattered rows), the column's features stay in
// registers, and LPR rows are reduced together.  Lane c takes the rows in the order u ^ c, so
// that the reduction's exchanges need no selection and lane c ends with row c.
// The table is staged one spin block at a time (uu, du, dd: the modes ascend, so rows and columns
// of a block are ranges); unsorted mode lists (a wrong particle number) and lattices whose block
// does not fit read it from global memory.
// gw of nw: this warp among those that share the item.
template <int D, int TH>
__device__ void gather_tiles(const RefineArgs& a, const double* Ys, const int* info,
                             const uint16_t* iperm, int nu, bool sorted, unsigned char* smem,
                             double* S, double* slice, int gw, int nw) {
  constexpr int LPR = D <= 16 ? 4 : 8, CPL = D / (2 * LPR);  // lanes per pair, chunks per lane
  constexpr int GR = 32 / LPR, JW = 2 * GR;                  // column groups, columns per warp
  const int n = a.n, N = a.Lx * a.Ly;
  const int tid = threadIdx.x, lane = tid & 31;
  const int grp = lane / LPR, c = lane % LPR;
  // Offset of chunk x of this lane in a row: with two chunks per lane, odd groups read theirs in
  // the other order, so that the two groups of a quarter-warp use different banks.
  int ch[CPL];
#pragma unroll
  for (int x = 0; x < CPL; ++x) ch[x] = 2 * (c + LPR * (CPL == 2 && LPR == 4 ? x ^ (grp & 1) : x));
  const double* Wg = static_cast<const double*>(a.Wt);
  double* wts = reinterpret_cast<double*>(smem + a.wt_off);
  const bool stage = a.stage_wt && sorted;
  for (int ph = 0; ph < (stage ? 3 : 1); ++ph) {
    // uu, du, dd; without staging every pair at once
    const int i0 = stage && ph > 0 ? nu : 0, i1 = stage && ph == 0 ? nu : n;
    const int j0 = stage && ph == 2 ? nu : 0, j1 = stage && ph < 2 ? nu : n;
    const bool tri = !(stage && ph == 1);
    if (stage) {
      const double2* src =
          reinterpret_cast<const double2*>(Wg + (size_t)(ph == 0 ? 0 : ph + 1) * N * D);
      __syncthreads();  // the previous block's readers are done
      if (i1 > i0 && j1 > j0)
        for (int v0 = tid; v0 < N * (D / 2); v0 += 4 * TH) {
          double2 buf[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (v0 + u * TH < N * (D / 2)) buf[u] = __ldg(src + v0 + u * TH);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (v0 + u * TH < N * (D / 2)) reinterpret_cast<double2*>(wts)[v0 + u * TH] = buf[u];
        }
      __syncthreads();
    }
    const int nr = i1 - i0, nc = j1 - j0;
    if (nr <= 0 || nc <= 0) continue;
    const int nrb = (nr + LPR - 1) / LPR, ncg = (nc + JW - 1) / JW;
    // column groups of row block rb that hold a pair (i > j for the triangular blocks)
    auto groups = [&](int rb) {
      return tri ? min(ncg, (rb * LPR + LPR - 1 + JW - 1) / JW) : ncg;
    };
    int rb = 0, rem = gw;
    for (;; rem += nw) {
      while (rb < nrb && rem >= groups(rb)) {
        rem -= groups(rb);
        ++rb;
      }
      if (rb >= nrb) break;
      int j[2], infj[2];
      double2 yj[2][CPL];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        j[q] = j0 + rem * JW + q * GR + grp;
        const int jj = min(j[q], j1 - 1);
        infj[q] = info[jj];
#pragma unroll
        for (int x = 0; x < CPL; ++x)
          yj[q][x] = *reinterpret_cast<const double2*>(Ys + jj * D + ch[x]);
      }
      const int ib = i0 + rb * LPR;
      double part[2][LPR];
#pragma unroll
      for (int u = 0; u < LPR; ++u) {
        const int i = min(ib + (u ^ c), i1 - 1);
        const int infi = info[i];
        double2 yi[CPL];
#pragma unroll
        for (int x = 0; x < CPL; ++x)
          yi[x] = *reinterpret_cast<const double2*>(Ys + i * D + ch[x]);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          int dx = ((infi >> 8) & 0xFF) - ((infj[q] >> 8) & 0xFF);
          int dy = (infi & 0xFF) - (infj[q] & 0xFF);
          dx += dx < 0 ? a.Lx : 0;
          dy += dy < 0 ? a.Ly : 0;
          const int r = dx * a.Ly + dy;
          double acc = 0.0;
          const int blk = 2 * (infi >> 16) + (infj[q] >> 16);
          const double* wr = stage ? wts + r * D : Wg + (size_t)(blk * N + r) * D;
#pragma unroll
          for (int x = 0; x < CPL; ++x) {
            const double2 w = *reinterpret_cast<const double2*>(wr + ch[x]);
            acc = fma(yi[x].x * yj[q][x].x, w.x, acc);
            acc = fma(yi[x].y * yj[q][x].y, w.y, acc);
          }
          part[q][u] = acc;
        }
      }
      // Sum over the LPR lanes: index u of lane c is row u ^ c, which its partner c ^ h holds at
      // index u ^ h; row c stays.
#pragma unroll
      for (int h = LPR / 2; h; h >>= 1)
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int u = 0; u < h; ++u)
            part[q][u] += __shfl_xor_sync(0xffffffffu, part[q][u + h], h);
      const int i = ib + c;
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (i < i1 && j[q] < j1 && (!tri || i > j[q])) {
          const int p = iperm[i], lq = iperm[j[q]];
          const int hi = max(p, lq), lo = min(p, lq), I = hi >> 3;
          const int o = (tile_base(I) + (lo >> 3)) * 64 + toff(hi & 7, lo & 7);
          const double v = p > lq ? part[q][0] : -part[q][0];
          if (I < a.keep)
            S[o] = v;
          else
            slice[o] = v;
        }
    }
  }
}

// The slice's tiles of rows >= keep into shared memory, once the staged rows and table are dead.
template <int TH>
__device__ void copy_tail(const RefineArgs& a, double* S, const double* slice) {
  const int T = tile_rows(a.n), o0 = tile_base(a.keep) * 32, o1 = tile_base(T) * 32;
  for (int v0 = o0 + threadIdx.x; v0 < o1; v0 += 4 * TH) {
    double2 buf[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v0 + u * TH < o1) buf[u] = reinterpret_cast<const double2*>(slice)[v0 + u * TH];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v0 + u * TH < o1) reinterpret_cast<double2*>(S)[v0 + u * TH] = buf[u];
  }
}

// Modes 3 and 4: the features of the item's configuration (CNN in shared memory) as its occupied
// rows Y (n, d) and modes: mode 3 to the CTA's slice (read back by the gather's staging), mode 4
// to the staging area above the CNN's shared memory.
template <typename T, int TH>
__device__ void features_to(const RefineArgs& a, int item, unsigned char* smem, T* Ydst,
                            int32_t* idst, float* sign_dummy) {
  const int N = a.Lx * a.Ly, C = a.C, M2 = 2 * N, NS = N + 1, d = C / 2;
  const int G = a.cl.G;
  const int c = item / G, g = item - c * G;
  const int smp = a.cl.sample ? a.cl.sample[c] : c;
  const int fr = a.cl.from ? a.cl.from[c] : -1;
  const int to = a.cl.from ? a.cl.to[c] : -1;
  const int8_t* base = a.cl.spins + (int64_t)smp * M2;
  int* simg = reinterpret_cast<int*>(smem);
  int* occl = simg + M2;
  int* wbuf = occl + M2;
  const size_t ints = 4 * (size_t)N + 4 * a.Lx + 32;
  T* actA = reinterpret_cast<T*>(smem + ((sizeof(int) * ints + 15) & ~(size_t)15));
  __syncthreads();
  if constexpr (sizeof(T) == 8) {
    if (cnn_mma_fits(a.Lx, a.Ly, C, TH)) {
      const int PS = mma_plane(a.Lx, a.Ly), W = a.Ly + 2;
      cnn_layers_mma<4, TH>(a.cnn_w, a.cnn_b, a.Lx, a.Ly, a.layers, base, fr, to, g, actA,
                            actA + (size_t)C * PS, simg);
      auto feat = [&](int sg, int aa, int site) {
        const int x = site / a.Ly;
        return actA[(sg * d + aa) * PS + (x + 1) * W + site - x * a.Ly + 1];
      };
      write_occupied_rows<T, decltype(feat), TH>(simg, occl, wbuf, N, a.n, d, g, a.Lx, a.Ly, Ydst,
                                                 idst, sign_dummy, feat);
      __syncthreads();
      return;
    }
  }
  T* actB = actA + C * NS;
  T* wsm = actB + C * NS;
  wsm = reinterpret_cast<T*>((reinterpret_cast<uintptr_t>(wsm) + 15) & ~(uintptr_t)15);
  T* bsm = wsm + C * C * 9;
  const T* in = cnn_layers<T, TH>(a.cnn_w, a.cnn_b, a.Lx, a.Ly, C, a.layers, base, fr, to, g, actA,
                                  actB, wsm, bsm, simg);
  auto feat = [&](int sg, int aa, int site) { return in[(sg * d + aa) * NS + site]; };
  write_occupied_rows<T, decltype(feat), TH>(simg, occl, wbuf, N, a.n, d, g, a.Lx, a.Ly, Ydst, idst,
                                             sign_dummy, feat);
  __syncthreads();
}

// Shared memory of the in-kernel CNN (modes 3, 4) with TH threads.
size_t features_smem(int Lx, int Ly, int C, int elt, int TH) {
  const size_t N = (size_t)Lx * Ly, ints = 4 * N + 4 * Lx + 32;
  const size_t act0 = (sizeof(int) * ints + 15) & ~(size_t)15;
  if (elt == 8 && cnn_mma_fits(Lx, Ly, C, TH)) return act0 + 8 * cnn_mma_doubles(Lx, Ly, C);
  const size_t act = act0 + (size_t)elt * 2 * C * (N + 1);
  return ((act + 15) & ~(size_t)15) + (size_t)elt * ((size_t)C * C * 9 + C);
}

// Largest multiplier |A[i][k] / A[k+1][k]| of an elimination in the FP32 pivot order that still
// counts as pivoted; partial pivoting keeps it at 1.  Where the FP32 factorisation was sound it stays
// there in FP64 too: at n = 240 and 504 at most 1.0001 over blocks of pivot ratio up to 2e7.  It
// leaves 1 where a column of FP32 Schur complements is at its rounding noise (3.6 seen at a ratio of
// 3e10) and is unbounded where the FP32 run met infinities.
__device__ __forceinline__ bool beyond_bound(double m) {  // |m| >= 2 (its high word), or NaN
  constexpr int kMaxMultiplier = 0x40000000;
  return (__double2hiint(m) & 0x7FFFFFFF) >= kMaxMultiplier;
}

// A lane's two elements of a tile in the MMA accumulator layout.
__device__ __forceinline__ double2* acc_ptr(double* t) {
  const int lane = threadIdx.x & 31;
  return reinterpret_cast<double2*>(t + toff(lane >> 2, 2 * (lane & 3)));
}

// Pivot block of a panel (w <= 8 columns) by one warp, two elements per lane: lane (r, q) = 4 r + q
// holds B[r][2q], B[r][2q + 1] (the MMA accumulator layout; only c < r is used).  A step takes
// its columns k, k + 1 from the lanes (r, k / 2) by shuffles; the same row operations applied to
// the identity give the inverse of the block's unit lower factor, which the panel solve uses as
// an MMA operand.  Writes Li (that inverse, a swizzled tile), the reciprocal pivots xinv and the
// pivots to piv[0, w / 2).  d: the lane's two elements.  The loop stays rolled (the code runs on one
// warp).  CHECK: a multiplier beyond the bound sets *grew.
template <bool CHECK>
__device__ __forceinline__ void factor_block(double2 d, int w, double* Li, double* xinv,
                                             double* piv, int* grew = nullptr) {
  const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
  // entries outside the strict lower triangle of the w rows hold no data
  double b0 = (r < w && 2 * q < r) ? d.x : 0.0, b1 = (r < w && 2 * q + 1 < r) ? d.y : 0.0;
  double e0 = r == 2 * q ? 1.0 : 0.0, e1 = r == 2 * q + 1 ? 1.0 : 0.0;
  const unsigned full = 0xffffffffu;
#pragma unroll 1
  for (int t = 0; 2 * t < w; ++t) {
    const double x = -__shfl_sync(full, b0, (2 * t + 1) * 4 + t);  // B[k][k+1] = -B[k+1][k]
    const double inv = 1.0 / x;
    // B[r][k], B[r][k+1] of this row and of the rows 2q, 2q + 1 (this lane's columns)
    const double xr = __shfl_sync(full, b0, (lane & 28) + t);
    const double yr = __shfl_sync(full, b1, (lane & 28) + t);
    const double x0 = __shfl_sync(full, b0, 8 * q + t), y0 = __shfl_sync(full, b1, 8 * q + t);
    const double x1 = __shfl_sync(full, b0, 8 * q + 4 + t), y1 = __shfl_sync(full, b1, 8 * q + 4 + t);
    const double f0 = __shfl_sync(full, e0, 8 * t + q), f1 = __shfl_sync(full, e1, 8 * t + q);
    const double g0 = __shfl_sync(full, e0, 8 * t + 4 + q), g1 = __shfl_sync(full, e1, 8 * t + 4 + q);
    const double yi = yr * inv, xi = xr * inv;
    if (r >= 2 * t + 2) {
      if (CHECK && r < w && beyond_bound(xi)) *grew = 1;
      if (2 * q >= 2 * t + 2) {
        b0 = fma(yi, x0, fma(-xi, y0, b0));
        b1 = fma(yi, x1, fma(-xi, y1, b1));
      }
      e0 = fma(-yi, f0, fma(xi, g0, e0));
      e1 = fma(-yi, f1, fma(xi, g1, e1));
    }
    if (lane == 0) {
      piv[t] = x;
      xinv[t] = inv;
    }
  }
  *reinterpret_cast<double2*>(Li + toff(r, 2 * q)) = make_double2(e0, e1);
}

// Tile update C += P W^T: P and W are 8 x 8 tiles (rows x panel columns).
struct Operand {
  double k0, k1;
};
__device__ __forceinline__ Operand load_operand(const double* t) {
  const int lane = threadIdx.x & 31;
  return Operand{t[toff(lane >> 2, lane & 3)], t[toff(lane >> 2, 4 + (lane & 3))]};
}
__device__ __forceinline__ double2 tile_mma(double2 v, const Operand& p, const Operand& w) {
  double c[2] = {v.x, v.y};
  mma_f64(c, p.k0, w.k0);
  mma_f64(c, p.k1, w.k1);
  return make_double2(c[0], c[1]);
}

// The item's sign, log|pf| and flags from its n / 2 pivots, by one warp: log|pf| = sum of log|x_t| as
// one product per lane (mantissa and exponent), then a butterfly.  check: an item whose order failed
// (grew, or a zero or non-finite pivot) is marked kFlagRepivot.
template <typename Piv>
__device__ __forceinline__ void write_result(const RefineArgs& a, int item, int swapped, Piv pivot,
                                             bool check = false, bool grew = false) {
  const int lane = threadIdx.x & 31;
  double mant = 1.0;
  int expo = 0, neg = 0, bad = 0;
  for (int t = lane; t < a.n / 2; t += 32) {
    const double x = pivot(t);
    if (x < 0.0) neg ^= 1;
    const double ax = fabs(x);
    if (!(ax > 0.0) || !isfinite(ax)) bad |= ax == 0.0 ? NH_FLAG_ZERO_PIVOT : NH_FLAG_NONFINITE;
    int e;
    mant = frexp(mant * ax, &e);
    expo += e;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {  // 32 mantissas in [1/2, 1]: no underflow
    mant *= __shfl_xor_sync(0xffffffffu, mant, o);
    expo += __shfl_xor_sync(0xffffffffu, expo, o);
    neg ^= __shfl_xor_sync(0xffffffffu, neg, o);
    bad |= __shfl_xor_sync(0xffffffffu, bad, o);
  }
  if (lane == 0) {
    float s = a.item_sign ? a.item_sign[item] : 1.0f;
    if (swapped) s = -s;
    if (neg) s = -s;
    int f = a.flags ? a.flags[item] : 0;
    f &= ~(kFlagNeedRefine | NH_FLAG_ZERO_PIVOT | NH_FLAG_NONFINITE);
    double la = log(mant) + (double)expo * 0.6931471805599453;
    if (isnan(s)) f |= NH_FLAG_NONFINITE;
    if (bad & NH_FLAG_ZERO_PIVOT) {
      s = 0.0f;
      la = -INFINITY;
    }
    if (!isfinite(la) && s != 0.0f) bad |= NH_FLAG_NONFINITE;
    f |= bad | NH_FLAG_REFINED;
    if (check && (grew || bad)) f |= kFlagRepivot;
    a.sign[item] = s;
    a.logabs[item] = s == 0.0f ? -INFINITY : la;
    if (a.flags) a.flags[item] = f;
  }
}

// MODE is a.mode as a template argument, so that each instance holds only its own phase-1 code
// (the register allocation of the elimination is then not shaped by the other modes).
template <int D, int MODE, int TH>
__global__ void __launch_bounds__(TH, TH <= 256 ? 2 : 1) refine_kernel(RefineArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint16_t perm_s[kRefineMaxN];  // logical -> physical (modes 2, 4: physical -> logical)
  __shared__ __align__(16) double Li[kPW * kPW];  // inverse unit factor of the current pivot block
  __shared__ double xinv[kPW / 2];                // reciprocals of its pivots
  __shared__ int nu_s;                      // up modes of the item; bit 31: list not sorted by spin
  constexpr int WARPS = TH / 32;
  const int n = a.n, T = tile_rows(n);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double* S = reinterpret_cast<double*>(smem);
  double* Wb = S + (size_t)tile_base(T) * 64;  // W tiles of the current panel, one per tile row
  const int n_work = *a.count;
  if (n_work < a.min_count || n_work > a.max_count) return;
  for (int slot = blockIdx.x; slot < n_work; slot += gridDim.x) {
    const int item = a.list[slot];
    const uint16_t* pr = a.perm + (size_t)item * a.perm_stride;
    __syncthreads();
    for (int p = tid; p < n; p += TH) {
      const int v = pr[p];
      if (MODE == 2 || MODE == 4)
        perm_s[v < n ? v : 0] = (uint16_t)p;
      else
        perm_s[p] = (uint16_t)v;
    }
    if (tid == 0) nu_s = 0;
    __syncthreads();
    // Phase 1: the permuted lower triangle in FP64 tiles.
    unsigned char* slb =
        static_cast<unsigned char*>(a.slice) + (size_t)blockIdx.x * slice_stride(n, D);
    if constexpr (MODE == 0) {
      const float* F = a.F + (size_t)item * n * n;
      for (int p = wid; p < n; p += WARPS) {
        const int i = perm_s[p];
        for (int q = lane; q < p; q += 32) {
          const int j = perm_s[q];
          S[(tile_base(p >> 3) + (q >> 3)) * 64 + toff(p & 7, q & 7)] =
              i > j ? (double)__ldg(F + (size_t)i * n + j) : -(double)__ldg(F + (size_t)j * n + i);
        }
      }
    } else if constexpr (MODE == 1 || MODE == 3) {
      float* sl = reinterpret_cast<float*>(slb);
      const float* Yg = static_cast<const float*>(a.Y) + (size_t)item * n * D;
      const int32_t* ig = a.idx + (size_t)item * n;
      if constexpr (MODE == 3) {  // the item's FP32 features, rows and modes to the slice
        features_to<float, TH>(a, item, smem, sl, reinterpret_cast<int32_t*>(sl + n * D),
                               reinterpret_cast<float*>(xinv));
        Yg = sl;
        ig = reinterpret_cast<const int32_t*>(sl + n * D);
      }
      gather_permuted<D, TH>(a, Yg, ig, perm_s, smem, sl);
      __syncthreads();  // slice written; the staging area is dead
      for (int p = wid; p < n; p += WARPS)
        for (int q = lane; q < p; q += 32)
          S[(tile_base(p >> 3) + (q >> 3)) * 64 + toff(p & 7, q & 7)] = (double)sl[roff(p) + q];
    } else {
      double* Ys = reinterpret_cast<double*>(smem + a.y_off);
      int* info = reinterpret_cast<int*>(smem + a.info_off);
      const int N = a.Lx * a.Ly;
      const double* Yg = static_cast<const double*>(a.Y) + (size_t)slot * n * D;
      const int32_t* ig = a.idx + (size_t)slot * n;
      if constexpr (MODE == 4) {
        double* Yd = a.rows_slice ? reinterpret_cast<double*>(slb) : Ys;
        int32_t* id = a.rows_slice ? reinterpret_cast<int32_t*>(Yd + n * D) : info;
        features_to<double, TH>(a, item, smem, Yd, id, reinterpret_cast<float*>(xinv));
        Yg = Yd;
        ig = id;
      }
      if (MODE == 2 || a.rows_slice) {
        const double2* src = reinterpret_cast<const double2*>(Yg);
        for (int v = tid; v < n * (D / 2); v += TH) reinterpret_cast<double2*>(Ys)[v] = src[v];
        for (int p = tid; p < n; p += TH) info[p] = ig[p];
        __syncthreads();
      }
      int mode_p = 0, mode_n = 0;
      if (tid < n) {
        mode_p = info[tid];
        mode_n = tid + 1 < n ? info[tid + 1] : 2 * N;
      }
      __syncthreads();
      if (tid < n) {
        const int sp = mode_p >= N ? 1 : 0, site = mode_p - sp * N, x = site / a.Ly;
        info[tid] = (sp << 16) | (x << 8) | (site - x * a.Ly);
        if (sp == 0) atomicAdd(&nu_s, 1);
        if (sp == 1 && mode_n < N) atomicOr(&nu_s, (int)0x80000000);
      }
      __syncthreads();
      const int nus = nu_s;
      double* sl = reinterpret_cast<double*>(slb);
      gather_tiles<D, TH>(a, Ys, info, perm_s, nus & 0x7FFFFFFF, nus >= 0, smem, S, sl, wid, WARPS);
      __syncthreads();
      copy_tail<TH>(a, S, sl);
    }
    __syncthreads();

    // Phase 2: static-pivot blocked elimination.  The pivots of panel p are kept in the W tile of
    // tile row p, which no later step reads or writes.
    if (wid == 0) factor_block<false>(*acc_ptr(S), min(kPW, n), Li, xinv, Wb);
    __syncthreads();
    for (int p = 0; p + 1 < T; ++p) {
      // (1) tile rows I > p: W_I = -S_(I, p) Li^T (the forward substitution of every row as one
      // product); the dead tile (I, p) then holds P[c][2t] = W[c][2t+1] / x_t, P[c][2t+1] =
      // -W[c][2t] / x_t, both columns in this lane.
      {
        const Operand li = load_operand(Li);
        const double inv = xinv[lane & 3];
        for (int I = p + 1 + wid; I < T; I += WARPS) {
          double* sc = S + (size_t)(tile_base(I) + p) * 64;
          const double2 w = tile_mma(make_double2(0.0, 0.0), load_operand(sc), li);
          __syncwarp();  // every lane has read its operand
          *acc_ptr(sc) = make_double2(-w.y * inv, w.x * inv);
          *acc_ptr(Wb + I * 64) = make_double2(-w.x, -w.y);
        }
      }
      __syncthreads();
      // (2) the next panel's column of tiles.
      {
        const Operand w = load_operand(Wb + (p + 1) * 64);
        for (int I = p + 1 + wid; I < T; I += WARPS) {
          double* row = S + (size_t)tile_base(I) * 64;
          double2* cp = acc_ptr(row + (p + 1) * 64);
          *cp = tile_mma(*cp, load_operand(row + p * 64), w);
        }
      }
      __syncthreads();
      // (3) warp 0: the next pivot block; the others: the remaining tiles, 2 x 2 at a time.
      if (wid == 0) {
        factor_block<false>(*acc_ptr(S + (size_t)(tile_base(p + 1) + p + 1) * 64),
                            min(kPW, n - 8 * (p + 1)), Li, xinv, Wb + (p + 1) * 64);
      } else if (wid & 3) {
        // not the warps of warp 0's scheduler, whose chain would queue behind their products
        constexpr int NW = WARPS - WARPS / 4;
        const int R = T - (p + 2), SR = (R + 1) >> 1;
        int si = 0, rem = wid - 1 - (wid >> 2);
        for (;; rem += NW) {
          while (si < SR && rem > si) {
            rem -= si + 1;
            ++si;
          }
          if (si >= SR) break;
          const int I0 = p + 2 + 2 * si, J0 = p + 2 + 2 * rem;
          const bool i2 = I0 + 1 < T, up = rem < si;  // second row; tile (I0, J0 + 1) exists
          double* r0 = S + (size_t)tile_base(I0) * 64;
          double* r1 = S + (size_t)tile_base(i2 ? I0 + 1 : I0) * 64;
          const bool c2 = up || i2;  // column J0 + 1 is needed
          const Operand a0 = load_operand(r0 + p * 64), a1 = load_operand(r1 + p * 64);
          const Operand b0 = load_operand(Wb + J0 * 64);
          const Operand b1 = load_operand(Wb + (c2 ? J0 + 1 : J0) * 64);
          double2 *p00 = acc_ptr(r0 + J0 * 64), *p01 = acc_ptr(r0 + (up ? J0 + 1 : J0) * 64);
          double2 *p10 = acc_ptr(r1 + J0 * 64), *p11 = acc_ptr(r1 + (c2 ? J0 + 1 : J0) * 64);
          const double2 v00 = tile_mma(*p00, a0, b0);
          const double2 v01 = tile_mma(*p01, a0, b1);
          const double2 v10 = tile_mma(*p10, a1, b0);
          const double2 v11 = tile_mma(*p11, a1, b1);
          *p00 = v00;
          if (up) *p01 = v01;
          if (i2) {
            *p10 = v10;
            *p11 = v11;
          }
        }
      }
      __syncthreads();
    }
    if (wid == 0)
      write_result(a, item, pr[n] & 1, [&](int t) { return Wb[(t >> 2) * 64 + (t & 3)]; });
  }
}

// ------------------------------------------------------------------ n beyond shared memory
// The same factorisation with the FP64 tiles in global memory (L2), one item per cluster of kBigCl
// CTAs.  CTA r owns the tile rows I = r mod kBigCl: all updates of a row stay in one CTA, only the
// W tiles of a panel travel, written by their owner into every CTA's shared memory (two panels'
// worth, by parity), so a panel costs one cluster barrier.  Every CTA factorises the pivot block
// itself, and every warp forms the one foreign W tile that the next column needs.  The order is the
// FP32 matrix's, so the multipliers of the FP64 one are watched (beyond_bound): an item beyond the
// bound is marked kFlagRepivot and factorised again with pivoting.  What bounds it is the L2 traffic
// of the trailing tiles (1 KB per tile update) and, at the end, the panels' latency.  Replaces the
// pivoted FP64 factorisation with its triangle in global memory, one CTA per item: 44 items at
// n = 896 12.25 -> 2.64 ms, 98 at n = 504 3.33 -> 1.38 ms, of which the check and the launch that
// looks for marked items are 22 and 8 us.
constexpr int kBigTh = 512;
constexpr int kBigCl = 4;
constexpr int kBigWarps = kBigTh / 32;

// Accumulator layout (row r, columns 2q, 2q + 1 in lane 4 r + q) to MMA operand layout.
__device__ __forceinline__ Operand to_operand(const double2& v) {
  const int lane = threadIdx.x & 31, src = (lane & 28) + ((lane & 3) >> 1);
  const double x0 = __shfl_sync(0xffffffffu, v.x, src), y0 = __shfl_sync(0xffffffffu, v.y, src);
  const double x1 = __shfl_sync(0xffffffffu, v.x, src + 2), y1 = __shfl_sync(0xffffffffu, v.y, src + 2);
  return (lane & 1) ? Operand{y0, y1} : Operand{x0, x1};
}
__device__ __forceinline__ double2 ldcg2(const double* p) {
  return __ldcg(reinterpret_cast<const double2*>(p));
}

template <int D>
__global__ void __cluster_dims__(kBigCl, 1, 1) __launch_bounds__(kBigTh, 1)
    refine_big_kernel(RefineArgs a, size_t item_doubles) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) double Li[kPW * kPW];
  __shared__ double xinv[kPW / 2];
  __shared__ double piv[kMaxN / 2];
  __shared__ uint16_t iperm[kMaxN];
  __shared__ int nu_s;
  __shared__ int grew_s;  // rank 0's: a multiplier of the item was beyond the bound
  const int n = a.n, T = tile_rows(n), N = a.Lx * a.Ly;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // Elimination: W tiles of two panels, then this CTA's P tiles (rows rank, rank + kBigCl, ...).
  double* Wl = reinterpret_cast<double*>(smem);
  double* Pl = Wl + 2 * (size_t)T * 64;
  double* Wr[kBigCl];
#pragma unroll
  for (int r = 0; r < kBigCl; ++r) Wr[r] = cluster.map_shared_rank(Wl, r);
  int* grew0 = cluster.map_shared_rank(&grew_s, 0);
  const int clusters = gridDim.x / kBigCl, cid = blockIdx.x / kBigCl;
  double* S = static_cast<double*>(a.slice) + (size_t)cid * item_doubles;
  const int n_work = *a.count;
  for (int slot = cid; slot < n_work; slot += clusters) {
    const int item = a.list[slot];
    const uint16_t* pr = a.perm + (size_t)item * a.perm_stride;
    double* Ys = reinterpret_cast<double*>(smem + a.y_off);
    int* info = reinterpret_cast<int*>(smem + a.info_off);
    const double* Yg = static_cast<const double*>(a.Y) + (size_t)slot * n * D;
    const int32_t* ig = a.idx + (size_t)slot * n;
    __syncthreads();  // the previous item's readers are done
    if (tid == 0) nu_s = grew_s = 0;
    for (int p = tid; p < n; p += kBigTh) {
      const int v = pr[p];
      iperm[v < n ? v : 0] = (uint16_t)p;
    }
    if (!a.rows_slice) {  // rows staged in shared memory
      const double2* src = reinterpret_cast<const double2*>(Yg);
      for (int v = tid; v < n * (D / 2); v += kBigTh)
        reinterpret_cast<double2*>(Ys)[v] = __ldg(src + v);
    }
    __syncthreads();
    for (int p = tid; p < n; p += kBigTh) {
      const int m = ig[p], sp = m >= N ? 1 : 0, site = m - sp * N, x = site / a.Ly;
      info[p] = (sp << 16) | (x << 8) | (site - x * a.Ly);
      if (sp == 0) atomicAdd(&nu_s, 1);
      if (sp == 1 && p + 1 < n && ig[p + 1] < N) atomicOr(&nu_s, (int)0x80000000);
    }
    __syncthreads();
    const int nus = nu_s;
    gather_tiles<D, kBigTh>(a, a.rows_slice ? Yg : Ys, info, iperm, nus & 0x7FFFFFFF, nus >= 0, smem,
                            nullptr, S, rank * kBigWarps + wid, kBigCl * kBigWarps);
    cluster.sync();  // every tile written; the staging areas are dead in every CTA
    const int o = toff(lane >> 2, 2 * (lane & 3));  // this lane's elements of a tile
    if (wid == 0) factor_block<true>(ldcg2(S + o), min(kPW, n), Li, xinv, piv, &grew_s);
    __syncthreads();
    for (int p = 0; p + 1 < T; ++p) {
      double* Wp = Wl + (size_t)(p & 1) * T * 64;
      // (1) this CTA's rows I > p: W_I and P_I from tile (I, p), then tile (I, p + 1).  W of row
      // p + 1 comes from that row's own tile (its owner does not overwrite it).
      {
        const Operand li = load_operand(Li);
        const double inv = xinv[lane & 3];
        const int I0 = p + 1 + ((rank - (p + 1)) & (kBigCl - 1));
        Operand wn{0.0, 0.0};
        if (I0 + kBigCl * wid < T) {
          const double2 w = tile_mma(make_double2(0.0, 0.0),
                                     to_operand(ldcg2(S + (size_t)(tile_base(p + 1) + p) * 64 + o)),
                                     li);
          wn = to_operand(make_double2(-w.x, -w.y));
        }
        for (int I = I0 + kBigCl * wid; I < T; I += kBigCl * kBigWarps) {
          double* row = S + (size_t)tile_base(I) * 64;
          const double2 sv = ldcg2(row + p * 64 + o), cv = ldcg2(row + (p + 1) * 64 + o);
          const double2 w = tile_mma(make_double2(0.0, 0.0), to_operand(sv), li);
          const double2 pv = make_double2(-w.y * inv, w.x * inv);
          if (beyond_bound(pv.y) && 8 * I + (lane >> 2) < n) *grew0 = 1;
          *reinterpret_cast<double2*>(Pl + (I / kBigCl) * 64 + o) = pv;
#pragma unroll
          for (int r = 0; r < kBigCl; ++r)
            *reinterpret_cast<double2*>(Wr[r] + (size_t)(p & 1) * T * 64 + I * 64 + o) =
                make_double2(-w.x, -w.y);
          const double2 nv = tile_mma(cv, to_operand(pv), wn);
          __stcg(reinterpret_cast<double2*>(row + (p + 1) * 64 + o), nv);
        }
      }
      cluster.sync();  // W complete everywhere, column p + 1 updated
      // (2) warp 0: the next pivot block; the others: this CTA's rows over the columns p + 2 .. I,
      // strips of kStrip tiles of one row with all loads in flight.
      if (wid == 0) {
        factor_block<true>(ldcg2(S + (size_t)(tile_base(p + 1) + p + 1) * 64 + o),
                           min(kPW, n - 8 * (p + 1)), Li, xinv, piv + 4 * (p + 1), &grew_s);
      } else {
        constexpr int kStrip = 6, NW = kBigWarps - 1;
        int I = p + 2 + ((rank - (p + 2)) & (kBigCl - 1)), rem = wid - 1;
        for (;; rem += NW) {
          while (I < T && rem >= (I - p - 2) / kStrip + 1) {
            rem -= (I - p - 2) / kStrip + 1;
            I += kBigCl;
          }
          if (I >= T) break;
          const int J0 = p + 2 + rem * kStrip;
          double* row = S + (size_t)tile_base(I) * 64 + o;
          double2 v[kStrip];
#pragma unroll
          for (int u = 0; u < kStrip; ++u)
            if (J0 + u <= I) v[u] = ldcg2(row + (J0 + u) * 64);
          const Operand pa = load_operand(Pl + (I / kBigCl) * 64);
#pragma unroll
          for (int u = 0; u < kStrip; ++u)
            if (J0 + u <= I)
              __stcg(reinterpret_cast<double2*>(row + (J0 + u) * 64),
                     tile_mma(v[u], pa, load_operand(Wp + (J0 + u) * 64)));
        }
      }
      __syncthreads();  // Li ready, this CTA's rows updated
    }
    if (rank == 0 && wid == 0)
      write_result(a, item, pr[n] & 1, [&](int t) { return piv[t]; }, true, grew_s != 0);
    cluster.sync();  // no CTA starts the next item's gather over tiles still being read
  }
}

size_t stage_bytes(int n, int N, int D, int elt, bool wt) {
  const int DP = D + (elt == 4 ? 4 : 2);
  return (size_t)elt * n * DP + sizeof(int) * ((n + 3) & ~3) + (wt ? (size_t)elt * 4 * N * DP : 0);
}

// Shared memory of one launch with TH threads (modes 2, 4: and the staging offsets, where it is at
// most kRefineSmemLimit).
template <int D>
size_t refine_smem(RefineArgs& a, int TH) {
  const int N = a.Lx * a.Ly, n = a.n, T = tile_rows(n);
  const size_t elim = tile_bytes(T) + 512 * (size_t)T;
  size_t smem = elim;
  if (a.mode == 1 || a.mode == 3) {
    a.stage_wt = stage_bytes(n, N, D, 4, true) <= kRefineSmemLimit;
    smem = std::max(smem, stage_bytes(n, N, D, 4, a.stage_wt));
    if (a.mode == 3) smem = std::max(smem, features_smem(a.Lx, a.Ly, a.C, 4, TH));
  } else if (a.mode != 0) {
    const size_t y = 8 * (size_t)n * D, inf = (4 * (size_t)n + 15) & ~(size_t)15;
    const size_t wt = 8 * (size_t)N * D;
    const size_t feat = a.mode == 4 ? (features_smem(a.Lx, a.Ly, a.C, 8, TH) + 15) & ~(size_t)15 : 0;
    if (feat > kRefineSmemLimit) return feat;
    a.rows_slice = feat + y + inf > kRefineSmemLimit;
    smem = std::max(smem, a.rows_slice ? std::max(feat, y + inf) : feat + y + inf);
    // One spin block of the table above the tiles' first rows, where it fits at all.
    a.stage_wt = wt + y + inf <= kRefineSmemLimit;
    if (a.stage_wt) smem = std::max(smem, wt + y + inf);
    smem = (smem + 15) & ~(size_t)15;
    a.info_off = (int)(smem - inf);
    a.y_off = (int)(smem - inf - y);
    a.wt_off = a.stage_wt ? (int)(smem - inf - y - wt) : a.y_off;
    a.keep = T;
    while (a.keep > 0 && tile_bytes(a.keep) > (size_t)a.wt_off) --a.keep;
  }
  return smem;
}

template <int D, int MODE, int TH>
int launch_refine_k(const RefineArgs& a, int max_slots, size_t smem, cudaStream_t st) {
  static const cudaError_t attr =
      cudaFuncSetAttribute(refine_kernel<D, MODE, TH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kRefineSmemLimit);
  if (attr != cudaSuccess) return check_cuda(attr, "refine smem attribute");
  int grid = num_sms() * (TH <= 256 ? 2 : 1);
  if (grid > max_slots) grid = max_slots;
  if (grid <= 0) return NH_OK;
  ProfScope prof_scope(NH_K_REFINE, st);
  refine_kernel<D, MODE, TH><<<grid, TH, smem, st>>>(a);
  return check_launch("refine_kernel");
}

// Two CTAs of 256 threads per SM where shared memory holds both and there are items for them (small
// lattices, whose phases are latency-bound), else one of 512.  In-kernel features on the matrix
// instruction need 512 threads beyond 128 sites.  The scalar network (16 channels) runs with either,
// and there the number of listed items decides on the device, both forms being launched (3 us): 290
// bare images, all listed, whole call with 512 and with 256 threads: 4x4 159 and 118 us, 8x8 200 and
// 159, 12x14 361 and 320; 320 images of 40 projected configurations, a third of them listed: 8x8 167
// and 178, 12x12 270 and 299.
constexpr size_t kTwoCtaSmem = 111 * 1024;  // dynamic, beside the static arrays

template <int D, int MODE>
int launch_refine_m(RefineArgs a, int max_slots, cudaStream_t st) {
  const bool scalar = MODE == 4 && !cnn_mma_fits(a.Lx, a.Ly, a.C, 512);
  const bool small = MODE != 4 || scalar || cnn_mma_fits(a.Lx, a.Ly, a.C, 256);
  const size_t s256 = refine_smem<D>(a, 256);
  a.max_count = INT_MAX;
  if (small && s256 <= kTwoCtaSmem && max_slots > num_sms()) {
    a.min_count = scalar ? num_sms() + 1 : 0;
    const int rc = launch_refine_k<D, MODE, 256>(a, max_slots, s256, st);
    if (rc || !scalar) return rc;
    a.min_count = 0;
    a.max_count = num_sms();
  }
  const size_t s512 = refine_smem<D>(a, 512);
  if (s512 > kRefineSmemLimit)
    return fail(NH_ERR_UNSUPPORTED, "refine: n=%d needs %zu B of shared memory", a.n, s512);
  return launch_refine_k<D, MODE, 512>(a, max_slots, s512, st);
}

// n > kRefineMaxN (mode 2 only): tiles in the scratch q.slice.
template <int D>
int launch_refine_big(RefineArgs a, int max_slots, cudaStream_t st) {
  const int N = a.Lx * a.Ly, n = a.n, T = tile_rows(n);
  const size_t inf = (4 * (size_t)n + 15) & ~(size_t)15, y = 8 * (size_t)n * D;
  const size_t wt = 8 * (size_t)N * D;
  const size_t lim = 200 * 1024;
  a.rows_slice = inf + y > lim;  // rows read from global memory
  a.stage_wt = !a.rows_slice && inf + y + wt <= lim;
  a.info_off = 0;
  a.y_off = (int)inf;
  a.wt_off = (int)(inf + y);
  a.keep = 0;  // every tile in global memory
  size_t smem = 512 * (2 * (size_t)T + (T + kBigCl - 1) / kBigCl);
  smem = std::max(smem, inf + (a.rows_slice ? 0 : y) + (a.stage_wt ? wt : 0));
  static const cudaError_t attr = cudaFuncSetAttribute(
      refine_big_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lim);
  if (attr != cudaSuccess) return check_cuda(attr, "refine smem attribute");
  int clusters = num_sms() / kBigCl;
  if (clusters > max_slots) clusters = max_slots;
  if (clusters <= 0) return NH_OK;
  ProfScope prof_scope(NH_K_PFAFFIAN64, st);
  refine_big_kernel<D><<<clusters * kBigCl, kBigTh, smem, st>>>(a, tile_bytes(T) / 8);
  return check_launch("refine_big_kernel");
}

template <int D>
int launch_refine_d(const RefineArgs& a, int max_slots, cudaStream_t st) {
  switch (a.mode) {
    case 1: return launch_refine_m<D, 1>(a, max_slots, st);
    case 2: return launch_refine_m<D, 2>(a, max_slots, st);
    case 3: return launch_refine_m<D, 3>(a, max_slots, st);
    default: return launch_refine_m<D, 4>(a, max_slots, st);
  }
}

}  // namespace

size_t refine_big_bytes(int n) {
  return n > kRefineMaxN ? (size_t)(num_sms() / kBigCl) * tile_bytes(tile_rows(n)) : 0;
}

size_t refine_slice_bytes(int n, int d) {
  if (n <= 0 || n > kRefineMaxN) return 0;
  // one slice per CTA: two CTAs per SM only where the elimination alone leaves room for both
  const int T = tile_rows(n);
  const size_t per_sm = tile_bytes(T) + 512 * (size_t)T <= kTwoCtaSmem ? 2 : 1;
  return per_sm * num_sms() * slice_stride(n, d < 8 ? 8 : d);
}

int launch_refine(const RefineLaunch& q, cudaStream_t st) {
  const bool big = q.n > kRefineMaxN;  // stored FP64 rows only, tiles in q.slice (refine_big_bytes)
  if (q.n <= 0 || q.n % 2 || q.n > (q.mode == 2 ? kMaxN : kRefineMaxN))
    return fail(NH_ERR_UNSUPPORTED, "refine: n=%d (even, <= %d)", q.n,
                q.mode == 2 ? kMaxN : kRefineMaxN);
  if (q.max_slots <= 0) return NH_OK;
  if (q.mode < 0 || q.mode > 4) return fail(NH_ERR_INVALID, "refine: mode %d", q.mode);
  if (q.mode != 0 && !q.slice) return fail(NH_ERR_INVALID, "refine: gather mode needs the slice");
  RefineArgs a{};
  a.n = q.n;
  a.mode = q.mode;
  a.F = q.F;
  a.Y = q.Y;
  a.idx = q.idx;
  a.Wt = q.Wt;
  a.Lx = q.Lx;
  a.Ly = q.Ly;
  a.D = q.d;
  a.list = q.list;
  a.count = q.count;
  a.perm = q.perm;
  a.perm_stride = q.perm_stride;
  a.item_sign = q.item_sign;
  a.sign = q.sign;
  a.logabs = q.logabs;
  a.flags = q.flags;
  a.slice = q.slice;
  a.cl = q.cl;
  a.cnn_w = q.cnn_w;
  a.cnn_b = q.cnn_b;
  a.C = q.C;
  a.layers = q.layers;
  if (q.mode >= 3 && (!q.cnn_w || !q.cnn_b || q.C % 16 || q.d * 2 != q.C))
    return fail(NH_ERR_INVALID, "refine: in-kernel features need the CNN weights");
  if (q.mode == 0) return launch_refine_m<16, 0>(a, q.max_slots, st);
  if (big) {
    switch (q.d) {
      case 8: return launch_refine_big<8>(a, q.max_slots, st);
      case 16: return launch_refine_big<16>(a, q.max_slots, st);
      case 32: return launch_refine_big<32>(a, q.max_slots, st);
      default: return fail(NH_ERR_UNSUPPORTED, "refine: d=%d (8, 16 or 32)", q.d);
    }
  }
  switch (q.d) {
    case 8: return launch_refine_d<8>(a, q.max_slots, st);
    case 16: return launch_refine_d<16>(a, q.max_slots, st);
    case 32: return launch_refine_d<32>(a, q.max_slots, st);
    default: return fail(NH_ERR_UNSUPPORTED, "refine: d=%d (8, 16 or 32)", q.d);
  }
}

}  // namespace nh
