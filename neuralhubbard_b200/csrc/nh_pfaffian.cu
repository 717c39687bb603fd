// Batched log-Pfaffian (blocked Parlett-Reid LTL^T with partial pivoting), the pairing
// gather, and the combination of symmetry images.
//
// FP32 matrices of n <= 256 run in pf32_kernel, larger ones in pf32_big_kernel (both described
// where they stand); pfaffian_kernel below is the FP64 form for dense matrices, for 224 < n <= 236
// and beyond for the blocks whose FP32 pivot order does not hold in FP64.  One CTA per antisymmetric
// n x n matrix, n even.  The strict lower triangle lives in shared memory (row i at offset
// i (i - 1) / 2) or in a slice of global scratch.  A pivot does not move data: it swaps the logical
// labels of two physical rows, so an elimination step costs two barriers.  Panel columns are formed
// lazily (stored column plus the panel's rank-2 terms U V^T - V U^T); at the end of a panel of NB
// steps the active rows are listed in physical order and the trailing triangle receives the
// rank-2NB update.  The Pfaffian is the product of the pivots A[k, k+1] times the parity of the
// relabelling, accumulated in FP64 as mantissa and exponent.  The ratio of the largest to the
// smallest pivot magnitude estimates the condition number; above cond_tau the item is flagged
// NH_FLAG_GROWTH (near-nodal) for the FP64 recompute.
//
// Replaces fermix.slogpf (code/backflow/models.py:210) and, in the gather mode, the Pallas
// pairing kernel pfsbp_pairing_fwd (code/backflow/pf_kernel.py:156-190) whose formula it
// follows: F[p, q] = sum_a (Y[p, a] Y[q, a]) Wt[2 s_p + s_q, r(p, q), a] with the product of
// the features formed first, so that F[q, p] = -F[p, q] holds bit for bit.
#include <math.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "nh_cnn_item.cuh"
#include "nh_common.cuh"

namespace nh {
namespace {

constexpr int kWarps = kNumThreads / 32;

template <typename T>
struct Vec;
template <>
struct Vec<float> {
  static constexpr int k = 4;
};
template <>
struct Vec<double> {
  static constexpr int k = 2;
};

__device__ __forceinline__ float tfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double tfma(double a, double b, double c) { return fma(a, b, c); }

__device__ __forceinline__ void ldg16(const float* p, float* o) {
  float4 v = __ldg(reinterpret_cast<const float4*>(p));
  o[0] = v.x;
  o[1] = v.y;
  o[2] = v.z;
  o[3] = v.w;
}
__device__ __forceinline__ void ldg16(const double* p, double* o) {
  double2 v = __ldg(reinterpret_cast<const double2*>(p));
  o[0] = v.x;
  o[1] = v.y;
}
__device__ __forceinline__ void lds16(const float* p, float* o) {
  float4 v = *reinterpret_cast<const float4*>(p);
  o[0] = v.x;
  o[1] = v.y;
  o[2] = v.z;
  o[3] = v.w;
}
__device__ __forceinline__ void lds16(const double* p, double* o) {
  double2 v = *reinterpret_cast<const double2*>(p);
  o[0] = v.x;
  o[1] = v.y;
}

struct PfArgs {
  int n;
  int mode;  // 0: F dense FP32 (items, n, n) in global memory; 1: gather from Y / idx / Wt
  const float* F;
  const void* Y;       // (slots, n, D) of T
  const int32_t* idx;  // (slots, n)
  const void* Wt;      // (4, N, D) of T
  const float4* Wc;    // modes 2, 3: the FP32 table in chunks of four a (pair_chunks)
  int Lx, Ly;
  const int32_t* count_dev;  // work count on the device (times count_mult) or null
  int count_mult;
  int n_slots;               // host count, upper bound when count_dev is set
  const int32_t* slot_item;  // slot -> item, null: identity
  const float* item_sign;    // (items,) or null
  float* sign;               // (items,)
  double* logabs;            // (items,)
  int32_t* flags;            // (items,) or null
  double cond_tau;           // flag NH_FLAG_GROWTH when max|piv| > cond_tau min|piv| (0: off)
  int flag_or;               // OR-ed into every written flag
  int only_flag;             // pfaffian_kernel: when set, items without this flag are left alone
  void* tri;                 // large n: per-CTA lower triangles of T in global memory
  uint16_t* perm;            // or null: per item, logical -> physical row, then the parity
  double refine_tau;         // set kFlagNeedRefine when max|piv| > refine_tau min|piv| (0: off)
  float* ratio;              // or null: per item, max|piv| / min|piv| (inf for a zero pivot)
  // mode 2 (features in the kernel): item = c * G + g of the configuration list; the CNN's
  // occupied rows at byte y_off and their modes at idx_off of shared memory; rows >= tail_row
  // of the triangle overlap the rows and are gathered through registers first.
  ConfigList cl;
  const float* cnn_w;   // packed weights [l][ci][tap][co]
  const float* cnn_b;
  int C, layers;
  int y_off, idx_off, tail_row;
  float* item_sign_out;  // (items,) the item signs the CNN phase computes
  int32_t* queue;        // mode 2: work counter (zero before the launch)
};

// Shared-memory layout of the in-kernel CNN phase (mode 2): simg, occl (2N ints each), scan
// scratch (4 Lx + 32 ints), activation planes A and B (C (N + 1) floats each), staged weights
// (C * C * 9) and biases (C).  Returns the end of the activation planes; *end the whole extent.
__host__ __device__ inline size_t cnn_phase_layout(int N, int C, int Lx, size_t* end) {
  const size_t ints = 4 * (size_t)N + 4 * Lx + 32;
  const size_t act0 = (sizeof(int) * ints + 15) & ~(size_t)15;
  const size_t act_end = act0 + sizeof(float) * 2 * (size_t)C * (N + 1);
  const size_t w0 = (act_end + 15) & ~(size_t)15;
  *end = w0 + sizeof(float) * ((size_t)C * C * 9 + C);
  return act_end;
}

// A mode m (spin s = m >= N, site x Ly + y) packed as s << 16 | x << 8 | y for the gather from
// shared memory (no division per element).
__device__ __forceinline__ int pack_mode(int m, int N, int Ly) {
  const int s = m >= N ? 1 : 0, site = m - s * N, x = site / Ly;
  return (s << 16) | (x << 8) | (site - x * Ly);
}

__device__ __forceinline__ int tri_off(int i) { return (i * (i - 1)) >> 1; }

// Pivot-search key of a magnitude: FP32, rounded up so that no non-zero value becomes zero.
__device__ __forceinline__ float to_key_float(double x) { return __double2float_ru(x); }

template <typename T>
__device__ __forceinline__ T aval(const T* Lw, int i, int j) {
  return i > j ? Lw[tri_off(i) + j] : (i < j ? -Lw[tri_off(j) + i] : T(0));
}

template <typename T, int D>
__device__ __forceinline__ T pair_value(const T* yp, int sp, int xp, int ypos,
                                        const T* __restrict__ Yq, int mq, int N, int Lx, int Ly,
                                        const T* __restrict__ Wt) {
  const int sq = mq >= N ? 1 : 0;
  const int siteq = mq - sq * N;
  const int xq = siteq / Ly, yq = siteq - xq * Ly;
  int dx = xp - xq, dy = ypos - yq;
  dx += dx < 0 ? Lx : 0;
  dy += dy < 0 ? Ly : 0;
  const T* wrow = Wt + ((size_t)(2 * sp + sq) * N + dx * Ly + dy) * D;
  T acc = T(0);
#pragma unroll
  for (int a0 = 0; a0 < D; a0 += Vec<T>::k) {
    T w[Vec<T>::k], q[Vec<T>::k];
    ldg16(wrow + a0, w);
    ldg16(Yq + a0, q);
#pragma unroll
    for (int k = 0; k < Vec<T>::k; ++k) acc = tfma(yp[a0 + k] * q[k], w[k], acc);
  }
  return acc;
}

template <typename T, int D, int WARPS = kWarps>
__device__ void gather_lower(T* Lw, int n, const T* __restrict__ Y, const int32_t* __restrict__ idx,
                             const T* __restrict__ Wt, int Lx, int Ly) {
  const int N = Lx * Ly;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int p = wid; p < n; p += WARPS) {
    const int mp = __ldg(idx + p);
    const int sp = mp >= N ? 1 : 0;
    const int sitep = mp - sp * N;
    const int xp = sitep / Ly, ypos = sitep - xp * Ly;
    T yp[D];
#pragma unroll
    for (int a0 = 0; a0 < D; a0 += Vec<T>::k) ldg16(Y + (size_t)p * D + a0, yp + a0);
    T* row = Lw + tri_off(p);
    int q = lane;
    for (; q + 32 < p; q += 64) {  // two independent elements per lane in flight
      const int mq0 = __ldg(idx + q), mq1 = __ldg(idx + q + 32);
      const T v0 = pair_value<T, D>(yp, sp, xp, ypos, Y + (size_t)q * D, mq0, N, Lx, Ly, Wt);
      const T v1 = pair_value<T, D>(yp, sp, xp, ypos, Y + (size_t)(q + 32) * D, mq1, N, Lx, Ly, Wt);
      row[q] = v0;
      row[q + 32] = v1;
    }
    if (q < p)
      row[q] = pair_value<T, D>(yp, sp, xp, ypos, Y + (size_t)q * D, __ldg(idx + q), N, Lx, Ly, Wt);
  }
}

// Load phase of modes 2 and 3 by a TH-thread block: the item's occupied rows Y (n, D) and packed
// modes in shared memory (mode 2: the CNN of its configuration in shared memory,
// write_occupied_rows, item sign to item_sign_out; mode 3: copied from the global rows a.Y / a.idx
// of slot), then the gather of the lower triangle from them.  Rows of the triangle that overlap Y
// (tail_row on) are computed into registers first and stored after a barrier.
constexpr int kTailElems = 4096;

template <int D, int TH>
__device__ void features_to_smem(const PfArgs& a, int item, unsigned char* smem, float* Ys,
                                 int* ids);
template <int D, int TH>
__device__ void gather_from_rows(const PfArgs& a, float* Lw, const float* Ys, const int* ids);

template <int D, int TH>
__device__ void rows_and_gather(const PfArgs& a, int item, int slot, float* Lw,
                                unsigned char* smem) {
  const int n = a.n;
  const int tid = threadIdx.x;
  float* Ys = reinterpret_cast<float*>(smem + a.y_off);
  int* ids = reinterpret_cast<int*>(smem + a.idx_off);
  if (a.mode == 3) {
    const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(a.Y) +
                                                        (size_t)slot * n * D);
    constexpr int K = D / 4;  // 16-byte chunks per row, stored swizzled (swz_index)
    const int nv = n * K;
    for (int v0 = tid; v0 < nv; v0 += 2 * TH) {
      float4 buf[2];
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (v0 + u * TH < nv) buf[u] = __ldg(src + v0 + u * TH);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int v = v0 + u * TH, row = v / K;
        if (v < nv) reinterpret_cast<float4*>(Ys)[row * K + ((v % K) ^ swz_key(row, K))] = buf[u];
      }
    }
    const int N = a.Lx * a.Ly;
    for (int p = tid; p < n; p += TH)
      ids[p] = pack_mode(__ldg(a.idx + (size_t)slot * n + p), N, a.Ly);
    __syncthreads();
  } else {
    features_to_smem<D, TH>(a, item, smem, Ys, ids);
  }
  gather_from_rows<D, TH>(a, Lw, Ys, ids);
}

template <int D, int TH>
__device__ void features_to_smem(const PfArgs& a, int item, unsigned char* smem, float* Ys,
                                 int* ids) {
  const int N = a.Lx * a.Ly, C = a.C, M2 = 2 * N, NS = N + 1;
  const int G = a.cl.G;
  const int c = item / G, g = item - c * G;
  const int smp = a.cl.sample ? a.cl.sample[c] : c;
  const int fr = a.cl.from ? a.cl.from[c] : -1;
  const int to = a.cl.from ? a.cl.to[c] : -1;
  const int8_t* base = a.cl.spins + (int64_t)smp * M2;
  int* simg = reinterpret_cast<int*>(smem);
  int* occl = simg + M2;
  int* wbuf = occl + M2;
  size_t cnn_end;
  const size_t act_end = cnn_phase_layout(N, C, a.Lx, &cnn_end);
  const size_t act0 = act_end - sizeof(float) * 2 * (size_t)C * NS;
  float* actA = reinterpret_cast<float*>(smem + act0);
  float* actB = actA + C * NS;
  float* wsm = reinterpret_cast<float*>(smem + ((act_end + 15) & ~(size_t)15));
  float* bsm = wsm + C * C * 9;
  const float* in = cnn_layers<float, TH>(a.cnn_w, a.cnn_b, a.Lx, a.Ly, C, a.layers, base, fr, to,
                                          g, actA, actB, wsm, bsm, simg);
  const int d = C / 2;
  auto feat = [&](int sg, int aa, int site) { return in[(sg * d + aa) * NS + site]; };
  write_occupied_rows<float, decltype(feat), TH>(simg, occl, wbuf, N, a.n, d, g, a.Lx, a.Ly, Ys,
                                                 ids, a.item_sign_out + item, feat, true);
  __syncthreads();
  for (int p = threadIdx.x; p < a.n; p += TH) ids[p] = pack_mode(ids[p], N, a.Ly);
  __syncthreads();
}

// The features of row p (chunk-swizzled rows, swz_index).
template <int D>
__device__ __forceinline__ void row_features(const float* Ys, int p, float* y) {
#pragma unroll
  for (int a0 = 0; a0 < D; a0 += 4) lds16(Ys + swz_index<float, D>(p, a0), y + a0);
}

// F[p][q] (p > q): sum_a (Y[p, a] Y[q, a]) Wt[2 s_p + s_q, r(p, q), a] in order of a (the
// arithmetic of pair_value: the product of the features commutes).  Wc: the table in chunks,
// Wc[(a / 4) 4 N + row] of four a, so that the lanes' neighbouring rows share cache lines.
// yq: the column's features (a lane's registers, or nullptr to read row q of Ys).
template <int D>
__device__ __forceinline__ float pair_chunks(const float* Ys, int p, int cp, const float* yq, int q,
                                             int cq, int N, int Lx, int Ly,
                                             const float4* __restrict__ Wc) {
  int dx = ((cp >> 8) & 0xff) - ((cq >> 8) & 0xff), dy = (cp & 0xff) - (cq & 0xff);
  dx += dx < 0 ? Lx : 0;
  dy += dy < 0 ? Ly : 0;
  const float4* w4 = Wc + (2 * (cp >> 16) + (cq >> 16)) * N + dx * Ly + dy;
  float acc = 0.0f;
#pragma unroll
  for (int c = 0; c < D / 4; ++c) {
    const float4 w = __ldg(w4 + c * 4 * N);
    float yp[4], yc[4];
    lds16(Ys + swz_index<float, D>(p, 4 * c), yp);
    if (yq) {
#pragma unroll
      for (int x = 0; x < 4; ++x) yc[x] = yq[4 * c + x];
    } else {
      lds16(Ys + swz_index<float, D>(q, 4 * c), yc);
    }
    acc = fmaf(yp[0] * yc[0], w.x, acc);
    acc = fmaf(yp[1] * yc[1], w.y, acc);
    acc = fmaf(yp[2] * yc[2], w.z, acc);
    acc = fmaf(yp[3] * yc[3], w.w, acc);
  }
  return acc;
}

// Lane <-> column (its features in registers over the rows below), the row's features broadcast;
// rows go to the warps in turn.  The shared-memory port bounds this loop: D / 4 broadcasts and
// D / 4 table loads of about ten cache lines per 32 pairs.
template <int D, int TH>
__device__ void gather_from_rows(const PfArgs& a, float* Lw, const float* Ys, const int* ids) {
  const int n = a.n, N = a.Lx * a.Ly;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const float4* Wc = a.Wc;
  int total = 0;  // (column block, row) units over the rows below tail_row
  for (int q0 = 0; q0 + 1 < a.tail_row; q0 += 32) total += a.tail_row - q0 - 1;
  int q0 = 0, rem = wid, cur = -1, cq = 0;
  float yq[D];
#pragma unroll 1
  for (int u = wid; u < total; u += TH / 32, rem += TH / 32) {
    while (rem >= a.tail_row - q0 - 1) {
      rem -= a.tail_row - q0 - 1;
      q0 += 32;
    }
    const int p = q0 + 1 + rem, q = q0 + lane;
    if (q0 != cur) {
      cur = q0;
      const int qq = q < n ? q : n - 1;
      row_features<D>(Ys, qq, yq);
      cq = ids[qq];
    }
    if (q < p)
      Lw[tri_off(p) + q] = pair_chunks<D>(Ys, p, ids[p], yq, q, cq, N, a.Lx, a.Ly, Wc);
  }
  if (a.tail_row < n) {
    // rows tail_row .. n-1 (E elements, at most kTailElems) through registers
    const int t0 = tri_off(a.tail_row);
    const int E = tri_off(n) - t0;
    float v[kTailElems / TH];
#pragma unroll
    for (int k = 0; k < kTailElems / TH; ++k) {
      const int e = tid + k * TH;
      v[k] = 0.0f;
      if (e < E) {
        int p = a.tail_row;
        while (tri_off(p + 1) - t0 <= e) ++p;
        const int q = e - (tri_off(p) - t0);
        v[k] = pair_chunks<D>(Ys, p, ids[p], nullptr, q, ids[q], N, a.Lx, a.Ly, Wc);
      }
    }
    __syncthreads();  // every read of Y is done
#pragma unroll
    for (int k = 0; k < kTailElems / TH; ++k) {
      const int e = tid + k * TH;
      if (e < E) Lw[t0 + e] = v[k];
    }
  }
}

// THREADS = 256: the lower triangle lives in shared memory (n <= 256).  THREADS = 1024 (large
// lattices, n <= 1024): one thread per row as well, the triangle in a per-CTA slice of global
// memory (a.tri; L2-resident up to n ~ 500), shared memory holding only the panel and the
// reduction slots.
template <typename T, int NB, int D, int THREADS = kNumThreads>
__global__ void __launch_bounds__(THREADS, 1) pfaffian_kernel(PfArgs a) {
  static_assert(sizeof(T) == 8, "FP32 matrices have their own kernels");
  static_assert(NB % Vec<T>::k == 0, "panel width must fill 16-byte vectors");
  constexpr int WARPS = THREADS / 32;
  constexpr bool kGlobalTri = THREADS > kNumThreads;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = a.n;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int tri = tri_off(n);
  T* Lw;
  T* Us;  // (n, NB)
  if constexpr (kGlobalTri) {
    Lw = static_cast<T*>(a.tri) + (size_t)blockIdx.x * ((tri + 3) & ~3);
    Us = reinterpret_cast<T*>(smem_raw);
  } else {
    Lw = reinterpret_cast<T*>(smem_raw);
    Us = Lw + ((tri + 3) & ~3);
  }
  T* Vs = Us + n * NB;            // (n, NB)
  // pivs[k/2] = pivot A[k, k+1], negated when that step swapped labels.
  T* rval = Vs + n * NB;                 // (warps) candidate signed value
  T* pivs = rval + WARPS;                // (n / 2) signed pivots, multiplied at the end
  float* rkey = reinterpret_cast<float*>(pivs + ((n / 2 + 3) & ~3));
  int* rt = reinterpret_cast<int*>(rkey + WARPS);  // (warps) trailing update: ballot counts
  int* rlog = rt + WARPS;
  // (warps) packed pivot candidates over rkey and rt: |c| key + 1 (bits 63..32), 0xFFFF - row
  // (31..16), sign of c (15), logical label (14..0): the largest word is the largest |c|, ties
  // to the lowest row.
  unsigned long long* cand = reinterpret_cast<unsigned long long*>(rkey);
  int* alist = rlog + WARPS;                       // (n) active physical rows
  int* misc = alist + n;                            // [0] physical row of logical k

  const int n_work = a.count_dev ? (*a.count_dev) * a.count_mult : a.n_slots;
  const T* Ybase = static_cast<const T*>(a.Y);
  const T* Wt = static_cast<const T*>(a.Wt);
  for (int slot = blockIdx.x; slot < n_work; slot += gridDim.x) {
    const int item = a.slot_item ? a.slot_item[slot] : slot;
    if (a.only_flag && !(a.flags[item] & a.only_flag)) continue;  // the same in all threads
    __syncthreads();
    if (a.mode == 0) {
      const float* F = a.F + (size_t)item * n * n;
      for (int i = wid; i < n; i += WARPS) {
        const float* src = F + (size_t)i * n;
        T* dst = Lw + tri_off(i);
        for (int j = lane; j < i; j += 32) dst[j] = T(__ldg(src + j));
      }
    } else if (a.mode == 1) {
      gather_lower<T, D, WARPS>(Lw, n, Ybase + (size_t)slot * n * D, a.idx + (size_t)slot * n,
                                Wt, a.Lx, a.Ly);
    }
    if (tid == 0) misc[0] = 0;
    __syncthreads();

    int my_log = tid < n ? tid : -1;
    int flag = 0;
    bool zero = false;

    for (int k0 = 0; k0 < n - 1 && !zero; k0 += 2 * NB) {
      const int steps = min(NB, (n - k0) >> 1);
      T myU[NB], myV[NB];
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        myU[j] = T(0);
        myV[j] = T(0);
      }
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        if (j < steps && !zero) {
          const int k = k0 + 2 * j;
          const int ck = misc[0];
          T c = T(0);
          const bool act = my_log > k;
          if (act) {
            c = aval(Lw, tid, ck);
            if (j > 0) {  // row ck's panel values: 16-byte loads (chunk-swizzled rows, swz_index)
              T vr[NB], ur[NB];
#pragma unroll
              for (int q = 0; q < NB; q += Vec<T>::k) {
                lds16(Vs + swz_index<T, NB>(ck, q), vr + q);
                lds16(Us + swz_index<T, NB>(ck, q), ur + q);
              }
#pragma unroll
              for (int p = 0; p < NB; ++p)
                if (p < j) c += myU[p] * vr[p] - myV[p] * ur[p];
            }
          }
          // Warp max of |c| (rounded up to FP32, NaN as +inf), ties to the lowest row, as one
          // integer reduction: non-negative floats order like their bit patterns, and the key
          // bits + 1 leaves 0 for rows that are no longer active.
          const float mag = isnan(c) ? INFINITY : to_key_float(fabs(c));
          const unsigned key = act ? __float_as_uint(mag) + 1u : 0u;
          const unsigned kmax = __reduce_max_sync(0xffffffffu, key);
          const unsigned hit = __ballot_sync(0xffffffffu, key == kmax);
          if (lane == __ffs(hit) - 1) {
            const unsigned lo = ((0xFFFFu - (unsigned)tid) << 16) |
                                (signbit(c) ? 0x8000u : 0u) | ((unsigned)my_log & 0x7FFFu);
            cand[wid] = ((unsigned long long)kmax << 32) | lo;
            rval[wid] = c;
          }
          __syncthreads();  // (1) pivot candidates
          unsigned long long best = 0;
#pragma unroll
          for (int w = 0; w < WARPS; w += 2) {
            const ulonglong2 q2 = *reinterpret_cast<const ulonglong2*>(cand + w);
            best = q2.x > best ? q2.x : best;
            best = q2.y > best ? q2.y : best;
          }
          const unsigned kbest = (unsigned)(best >> 32);
          const float bk = kbest ? __uint_as_float(kbest - 1u) : -1.0f;
          const int r = 0xFFFF - (int)((best >> 16) & 0xFFFFu);
          const int lr = (int)(best & 0x7FFFu);
          const T cr = rval[r >> 5];
          if (!(bk > 0.0f)) {
            zero = true;  // exactly singular (or empty) column: pf = 0
          } else {
            if (tid == r)
              my_log = k + 1;
            else if (my_log == k + 1)
              my_log = lr;  // the row that held label k+1 takes the pivot's old label
            const T piv = -cr;
            const bool live = my_log > k + 1;
            T u = T(0), v = T(0);
            if (live) {
              T dv = aval(Lw, tid, r);
              if (j > 0) {
                T vr[NB], ur[NB];
#pragma unroll
                for (int q = 0; q < NB; q += Vec<T>::k) {
                  lds16(Vs + swz_index<T, NB>(r, q), vr + q);
                  lds16(Us + swz_index<T, NB>(r, q), ur + q);
                }
#pragma unroll
                for (int p = 0; p < NB; ++p)
                  if (p < j) dv += myU[p] * vr[p] - myV[p] * ur[p];
              }
              u = dv;
              v = c * (T(1) / piv);
            }
            myU[j] = u;
            myV[j] = v;
            if (tid < n) {
              Us[swz_index<T, NB>(tid, j)] = u;
              Vs[swz_index<T, NB>(tid, j)] = v;
            }
            if (my_log == k + 2) misc[0] = tid;
            if (tid == 0) pivs[k >> 1] = lr != k + 1 ? -piv : piv;
          }
          __syncthreads();  // (2) panel column written, next column's owner known
        }
      }
      if (zero) break;
      // Trailing update of the active rows: warp <-> row, lane <-> column (32-column blocks).
      const int k_end = k0 + 2 * steps;
      const int m = n - k_end;
      if (m >= 2) {
        const bool on = tid < n && my_log >= k_end;
        const unsigned bal = __ballot_sync(0xffffffffu, on);
        if (lane == 0) rt[wid] = __popc(bal);
        __syncthreads();
        int before = 0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) before += (w < wid) ? rt[w] : 0;
        if (on) alist[before + __popc(bal & ((1u << lane) - 1u))] = tid;
        __syncthreads();  // (3) active list in physical order
        // Work units: (64-column block cb, group of RT consecutive rows below its diagonal);
        // lane l updates columns 64 cb + l and 64 cb + 32 + l, so each row's broadcast U/V
        // serves 64 elements.  All loads of a unit precede its stores (stores may alias loads).
        constexpr int RT = 1;
        int total = 0;
        for (int cb = 0; 64 * cb + 1 < m; ++cb) total += (m - 64 * cb - 1 + RT - 1) / RT;
        int cb = 0, rem = wid, cur_cb = -1, ib0 = 0, ib1 = 0, pb0 = 0, pb1 = 0;
        T ub0[NB], vb0[NB], ub1[NB], vb1[NB];
#pragma unroll
        for (int p = 0; p < NB; ++p) ub0[p] = vb0[p] = ub1[p] = vb1[p] = T(0);
        for (int pi = wid; pi < total; pi += WARPS, rem += WARPS) {
          while (rem >= (m - 64 * cb - 1 + RT - 1) / RT) {
            rem -= (m - 64 * cb - 1 + RT - 1) / RT;
            ++cb;
          }
          const int ia0 = 64 * cb + 1 + rem * RT;
          if (cb != cur_cb) {
            cur_cb = cb;
            ib0 = 64 * cb + lane;
            ib1 = ib0 + 32;
            pb0 = ib0 < m ? alist[ib0] : 0;
            pb1 = ib1 < m ? alist[ib1] : 0;
            // the columns' panel values, 16-byte loads of swizzled rows (conflict-free for
            // consecutive active rows); rows past the end read row 0 and are zeroed
#pragma unroll
            for (int p = 0; p < NB; p += Vec<T>::k) {
              lds16(Us + swz_index<T, NB>(pb0, p), ub0 + p);
              lds16(Vs + swz_index<T, NB>(pb0, p), vb0 + p);
              lds16(Us + swz_index<T, NB>(pb1, p), ub1 + p);
              lds16(Vs + swz_index<T, NB>(pb1, p), vb1 + p);
            }
#pragma unroll
            for (int p = 0; p < NB; ++p) {
              if (ib0 >= m) ub0[p] = vb0[p] = T(0);
              if (ib1 >= m) ub1[p] = vb1[p] = T(0);
            }
          }
          T acc0[RT], acc1[RT], ua[RT][NB], va[RT][NB];
          int off[RT];
          bool ok0[RT], ok1[RT];
#pragma unroll
          for (int rr = 0; rr < RT; ++rr) {
            const int ia = ia0 + rr;
            ok0[rr] = ia < m && ib0 < ia;
            ok1[rr] = ia < m && ib1 < ia;
            const int pa = alist[ia < m ? ia : ia0];
            off[rr] = tri_off(pa);
#pragma unroll
            for (int p = 0; p < NB; p += Vec<T>::k) {
              lds16(Us + swz_index<T, NB>(pa, p), ua[rr] + p);
              lds16(Vs + swz_index<T, NB>(pa, p), va[rr] + p);
            }
          }
#pragma unroll
          for (int rr = 0; rr < RT; ++rr) {
            acc0[rr] = ok0[rr] ? Lw[off[rr] + pb0] : T(0);
            acc1[rr] = ok1[rr] ? Lw[off[rr] + pb1] : T(0);
          }
#pragma unroll
          for (int p = 0; p < NB; ++p) {
            if (p < steps) {
#pragma unroll
              for (int rr = 0; rr < RT; ++rr) {
                acc0[rr] = tfma(ua[rr][p], vb0[p], acc0[rr]);
                acc1[rr] = tfma(ua[rr][p], vb1[p], acc1[rr]);
                acc0[rr] = tfma(-va[rr][p], ub0[p], acc0[rr]);
                acc1[rr] = tfma(-va[rr][p], ub1[p], acc1[rr]);
              }
            }
          }
#pragma unroll
          for (int rr = 0; rr < RT; ++rr) {
            if (ok0[rr]) Lw[off[rr] + pb0] = acc0[rr];
            if (ok1[rr]) Lw[off[rr] + pb1] = acc1[rr];
          }
        }
        __syncthreads();  // (4) trailing triangle updated
      }
    }
    if (tid == 0) {
      // Pfaffian = relabelling parity x product of the pivots, accumulated in FP64 as mantissa
      // and exponent; the pivot ratio flags near-nodal blocks.
      float s = a.item_sign ? a.item_sign[item] : 1.0f;
      double la;
      if (isnan(s)) flag |= NH_FLAG_NONFINITE;  // the CNN could not compute this item
      if (zero) {
        s = 0.0f;
        la = -INFINITY;
        flag |= NH_FLAG_ZERO_PIVOT;
      } else {
        double mant = 1.0;
        int expo = 0;
        double pmin = INFINITY, pmax = 0.0;
        for (int k = 0; k < n / 2; ++k) {
          const double pv = pivs[k];
          if (pv < 0.0) s = -s;
          const double ap = fabs(pv);
          if (!isfinite(ap)) flag |= NH_FLAG_NONFINITE;
          pmin = fmin(pmin, ap);
          pmax = fmax(pmax, ap);
          int e;
          mant = frexp(mant * ap, &e);
          expo += e;
        }
        la = log(mant) + (double)expo * 0.6931471805599453;
        if (!isfinite(la)) flag |= NH_FLAG_NONFINITE;
        if (a.cond_tau > 0.0 && pmax > a.cond_tau * pmin) flag |= NH_FLAG_GROWTH;
      }
      if (s == 0.0f) la = -INFINITY;
      a.sign[item] = s;
      a.logabs[item] = la;
      if (a.flags) a.flags[item] = flag | a.flag_or;
    }
  }
}

template <typename T, int NB, int WARPS = kWarps, bool kGlobalTri = false>
size_t pf_smem(int n) {
  const size_t tri = (size_t)n * (n - 1) / 2;
  return sizeof(T) * ((kGlobalTri ? 0 : ((tri + 3) & ~(size_t)3)) + 2 * (size_t)n * NB +
                      WARPS + ((n / 2 + 3) & ~(size_t)3)) +
         sizeof(float) * WARPS + sizeof(int) * (2 * WARPS + (size_t)n + 2);
}

// Raises a kernel's dynamic shared-memory cap to the largest the launches need, never lowering
// it: the plain and the fused launchers share kernel instantiations, and a cap set lower by one
// would make the other's launch fail.  One cap per kernel, under a lock.
template <typename K>
int raise_smem_cap(K* kernel, size_t smem) {
  static std::mutex mu;
  static std::map<const void*, size_t> caps;
  if (smem <= 48 * 1024) return NH_OK;
  std::lock_guard<std::mutex> g(mu);
  size_t& cap = caps[reinterpret_cast<const void*>(kernel)];
  if (smem <= cap) return NH_OK;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return check_cuda(e, "pfaffian kernel shared-memory attribute");
  cap = smem;
  return NH_OK;
}

// Large lattices: 1024 threads, triangle in a.tri; the panel width that fits shared memory.
constexpr int kBigThreads = 1024;
constexpr int kBigNB = 4;

template <typename T, int NB, int D, int THREADS = kNumThreads>
int launch_pf(const PfArgs& a, cudaStream_t st) {
  constexpr bool kGlobalTri = THREADS > kNumThreads;
  const size_t smem = pf_smem<T, NB, THREADS / 32, kGlobalTri>(a.n);
  if (smem > 227 * 1024)
    return fail(NH_ERR_UNSUPPORTED, "slogpf: n=%d needs %zu B of shared memory", a.n, smem);
  if (kGlobalTri && !a.tri)
    return fail(NH_ERR_UNSUPPORTED, "slogpf: n=%d needs the large-lattice scratch", a.n);
  if (int rc = raise_smem_cap(pfaffian_kernel<T, NB, D, THREADS>, smem)) return rc;
  const int per_sm = (!kGlobalTri && smem <= 113 * 1024) ? 2 : 1;
  int grid = num_sms() * per_sm;
  if (grid > a.n_slots) grid = a.n_slots;
  if (grid <= 0) return NH_OK;
  ProfScope prof_scope(NH_K_PFAFFIAN64, st);
  pfaffian_kernel<T, NB, D, THREADS><<<grid, THREADS, smem, st>>>(a);
  return check_launch("pfaffian_kernel");
}

// ------------------------------------------------------------------ FP32, n <= 256
// The factorisation of pfaffian_kernel (same operations in the same order, so the same bits) for
// the matrices that fit in shared memory, organised around what bounds them.  At n = 224, two CTAs
// per SM, a matrix is resident for 371K cycles: 148K in the panels (112 pivot steps of latency, the
// larger part of the block waiting), 111K in the gather and 109K in the trailing updates (both on
// the shared-memory port, shared with the neighbour), 3K in the tail.
//  * The active rows are compacted at the end of every panel (alist, clog: physical row and
//    logical label in physical order), and a panel is run by ceil(m / 32) warps behind a named
//    barrier of their own: warps without active rows do not repeat the step's work, and the last
//    32 rows need no barrier at all.
//  * The trailing update gives a lane four columns (their U / V in registers) where the row has
//    them, so that a row's broadcast U / V serves 128 elements: a uniform 16-byte shared load costs
//    two cycles of the load port (its register write), which is what bounds this phase.
//  * The pivots are multiplied by one warp in parallel.
constexpr int kPf32NB8MaxN = 224;  // panels of 8 up to here (two CTAs per SM), of 4 beyond

struct Pf32Layout {
  size_t us, vs, pivs, cand, rt, misc, alist, clog, end;  // byte offsets; the triangle is at 0
};
__host__ __device__ inline Pf32Layout pf32_layout(int n, int NB) {
  Pf32Layout L;
  L.us = sizeof(float) * ((((size_t)n * (n - 1)) / 2 + 3) & ~(size_t)3);
  L.vs = L.us + sizeof(float) * (size_t)n * NB;
  L.pivs = L.vs + sizeof(float) * (size_t)n * NB;
  L.cand = (L.pivs + sizeof(float) * (size_t)(n / 2) + 15) & ~(size_t)15;
  L.rt = L.cand + 8 * sizeof(unsigned long long);
  L.misc = L.rt + 12 * sizeof(int);
  L.alist = L.misc + 4 * sizeof(int);
  L.clog = L.alist + n;
  L.end = L.clog + n;
  return L;
}

// Barrier of the PW panel warps (one warp: the warp's own).
__device__ __forceinline__ void panel_sync(int PW) {
  if (PW == 1)
    __syncwarp();
  else
    asm volatile("bar.sync 1, %0;" ::"r"(32 * PW) : "memory");
}

// The panel values of one row: 16-byte loads of a swizzled row.
template <int NB>
__device__ __forceinline__ void panel_load(const float* Us, const float* Vs, int row, float* v,
                                           float* u) {
#pragma unroll
  for (int q = 0; q < NB; q += 4) {
    lds16(Vs + swz_index<float, NB>(row, q), v + q);
    lds16(Us + swz_index<float, NB>(row, q), u + q);
  }
}

// A[ph][q] with the panel's first j terms: panel values past j are zero on both sides.  Branch-free
// but for the uniform half of the terms: both orientations of the element take one load.
template <int NB>
__device__ __forceinline__ float panel_value(const float* Lw, int ph, int off, int q, int j,
                                             const float* U, const float* V, const float* vr,
                                             const float* ur) {
  float c = Lw[ph > q ? off + q : tri_off(q) + ph];
  c = ph < q ? -c : c;
  c = ph == q ? 0.0f : c;
#pragma unroll
  for (int p = 0; p < 4; ++p) c += U[p] * vr[p] - V[p] * ur[p];
  if (NB > 4 && j > 4) {
#pragma unroll
    for (int p = 4; p < NB; ++p) c += U[p] * vr[p] - V[p] * ur[p];
  }
  return c;
}

// Panel of `steps` pivot steps from logical column k0 on the m active rows, one row per thread of
// the first PW warps.  A step is bound by the number of instructions one warp issues in sequence
// (about 150), so the rows are spread over the schedulers, the candidates are compared by
// reductions and the loop stays rolled (unrolled, its code outgrows the instruction cache).
// Measured at n = 224, two CTAs per SM: 1,350 cycles per step; two rows per thread 1,750, and one
// barrier per step, every thread forming the next column's panel values itself, 1,500.  rt[8]
// tells the block whether a column was exactly zero.
template <int NB>
__device__ __forceinline__ void panel_steps(float* Lw, float* Us, float* Vs, float* pivs,
                                            unsigned long long* cand, int* rt, int* misc,
                                            uint8_t* alist, uint8_t* clog, int m, int k0, int steps,
                                            int PW, int& swaps, uint16_t* perm) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const bool has = tid < m;
  const int ph = has ? alist[tid] : 0, off = tri_off(ph);
  int log = has ? clog[tid] : -1;
  if (has) {
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int p = 0; p < NB; p += 4) {
      *reinterpret_cast<float4*>(Us + swz_index<float, NB>(ph, p)) = z;
      *reinterpret_cast<float4*>(Vs + swz_index<float, NB>(ph, p)) = z;
    }
  }
  if (wid == 0 && lane < 8) cand[lane] = 0ull;  // the slots of warps that do not run stay zero
  panel_sync(PW);
  bool zero = false;
#pragma unroll 1
  for (int j = 0; j < steps; ++j) {
    const int k = k0 + 2 * j;
    const int ck = misc[0];
    float U[NB], V[NB], vr[NB], ur[NB];
    panel_load<NB>(Us, Vs, ph, V, U);
    panel_load<NB>(Us, Vs, ck, vr, ur);
    const float c = panel_value<NB>(Lw, ph, off, ck, j, U, V, vr, ur);
    // |c| bits + 1 (NaN as +inf); 0 for rows that are no longer active
    const unsigned mag = min(__float_as_uint(c) & 0x7FFFFFFFu, 0x7F800000u);
    const unsigned key = log > k ? mag + 1u : 0u;
    // Maximum, ties to the lowest physical row (the rows ascend with the thread index).
    unsigned kbest = __reduce_max_sync(0xffffffffu, key);
    const int wl = __ffs(__ballot_sync(0xffffffffu, key == kbest)) - 1;
    unsigned lbest = ((0xFFFFu - (unsigned)ph) << 16) | (signbit(c) ? 0x8000u : 0u) |
                     ((unsigned)log & 0x7FFFu);
    if (PW == 1) {
      lbest = __shfl_sync(0xffffffffu, lbest, wl);
    } else {
      if (lane == wl) cand[wid] = ((unsigned long long)kbest << 32) | lbest;
      panel_sync(PW);  // (1) pivot candidates
      const unsigned long long w = cand[lane & 7];
      const unsigned hi = (unsigned)(w >> 32);
      kbest = __reduce_max_sync(0xffffffffu, hi);
      lbest = __reduce_max_sync(0xffffffffu, hi == kbest ? (unsigned)w : 0u);
    }
    const float bk = kbest ? __uint_as_float(kbest - 1u) : -1.0f;
    if (!(bk > 0.0f)) {  // exactly singular (or empty) column: pf = 0
      zero = true;
      panel_sync(PW);
      break;
    }
    const int r = 0xFFFF - (int)(lbest >> 16);
    const int lr = (int)(lbest & 0x7FFFu);
    const float piv = (lbest & 0x8000u) ? bk : -bk;
    panel_load<NB>(Us, Vs, r, vr, ur);
    const float rp = 1.0f / piv;
    // the row that held label k+1 takes the pivot's old label
    log = has && ph == r ? k + 1 : (log == k + 1 ? lr : log);
    const float u = panel_value<NB>(Lw, ph, off, r, j, U, V, vr, ur);
    if (log > k + 1) {
      const int o = swz_index<float, NB>(ph, j);
      Us[o] = u;
      Vs[o] = c * rp;
    }
    if (log == k + 2) misc[0] = ph;
    if (tid == 0) pivs[k >> 1] = lr != k + 1 ? -piv : piv;
    swaps ^= lr != k + 1 ? 1 : 0;
    panel_sync(PW);  // (2) panel column written, next column's owner known
  }
  // Eliminated rows leave: their order to the record, the others compacted in physical order.
  const int k_end = k0 + 2 * steps;
  const unsigned bal = __ballot_sync(0xffffffffu, log >= k_end);
  if (lane == 0) rt[wid] = __popc(bal);
  if (perm && !zero && log >= 0 && log < k_end) perm[log] = (uint16_t)ph;
  panel_sync(PW);
  if (log >= k_end) {
    int i = __popc(bal & ((1u << lane) - 1u));
    for (int w = 0; w < wid; ++w) i += rt[w];
    alist[i] = (uint8_t)ph;
    clog[i] = (uint8_t)log;
  }
  if (tid == 0) rt[8] = zero ? 1 : 0;
}

// Trailing update of one unit: RT consecutive active rows from ia0, NC columns per lane
// (c0 + lane + 32 i of the active list; physical rows pb, panel values ub / vb).
template <int NB, int RT, int NC, int NCB>
__device__ __forceinline__ void trail_unit(float* Lw, const float* Us, const float* Vs,
                                           const uint8_t* alist, int m, int ia0, int c0,
                                           const int (&pb)[NCB], const float (&ub)[NCB][NB],
                                           const float (&vb)[NCB][NB]) {
  const int lane = threadIdx.x & 31;
  float acc[RT][NC];
  int pa[RT], off[RT];
#pragma unroll
  for (int rr = 0; rr < RT; ++rr) {
    pa[rr] = alist[ia0 + rr < m ? ia0 + rr : ia0];
    off[rr] = tri_off(pa[rr]);
  }
#pragma unroll
  for (int rr = 0; rr < RT; ++rr)
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const bool ok = ia0 + rr < m && c0 + lane + 32 * i < ia0 + rr;
      acc[rr][i] = ok ? Lw[off[rr] + pb[i]] : 0.0f;
    }
#pragma unroll
  for (int h = 0; h < NB; h += 4) {
    float ua[RT][4], va[RT][4];
#pragma unroll
    for (int rr = 0; rr < RT; ++rr) {
      lds16(Us + swz_index<float, NB>(pa[rr], h), ua[rr]);
      lds16(Vs + swz_index<float, NB>(pa[rr], h), va[rr]);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int rr = 0; rr < RT; ++rr) {
#pragma unroll
        for (int i = 0; i < NC; ++i) acc[rr][i] = fmaf(ua[rr][p], vb[i][h + p], acc[rr][i]);
#pragma unroll
        for (int i = 0; i < NC; ++i) acc[rr][i] = fmaf(-va[rr][p], ub[i][h + p], acc[rr][i]);
      }
  }
#pragma unroll
  for (int rr = 0; rr < RT; ++rr)
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const bool ok = ia0 + rr < m && c0 + lane + 32 * i < ia0 + rr;
      if (ok) Lw[off[rr] + pb[i]] = acc[rr][i];
    }
}

// Trailing update of the columns [c0, c0 + 32 NC) of the active list over the rows below;
// done counts the units handed out so far, so that the warps stay evenly loaded across blocks.
template <int NB, int NC, int WARPS>
__device__ __forceinline__ void trail_block(float* Lw, const float* Us, const float* Vs,
                                            const uint8_t* alist, int m, int c0, int& done) {
  constexpr int RT = 2;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int units = (m - c0 - 1 + RT - 1) / RT;
  const int u0 = (wid - done) & (WARPS - 1);
  done += units;
  if (u0 >= units) return;
  int pb[NC];
  float ub[NC][NB], vb[NC][NB];
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int ib = c0 + lane + 32 * i;
    pb[i] = alist[ib < m ? ib : m - 1];
#pragma unroll
    for (int p = 0; p < NB; p += 4) {
      lds16(Us + swz_index<float, NB>(pb[i], p), ub[i] + p);
      lds16(Vs + swz_index<float, NB>(pb[i], p), vb[i] + p);
    }
  }
  for (int u = u0; u < units; u += WARPS) {
    const int ia0 = c0 + 1 + u * RT;
    if (NC == 4 && ia0 + RT - 1 <= c0 + 64)  // no row reaches the upper half of the columns
      trail_unit<NB, RT, NC / 2, NC>(Lw, Us, Vs, alist, m, ia0, c0, pb, ub, vb);
    else
      trail_unit<NB, RT, NC, NC>(Lw, Us, Vs, alist, m, ia0, c0, pb, ub, vb);
  }
}

// The item's results from its n / 2 pivots (negated where the step swapped labels), by one warp:
// Pfaffian = relabelling parity x product of the pivots, accumulated in FP64 as mantissa and
// exponent (one product per lane, then a butterfly); the pivot ratio flags near-nodal blocks.
template <typename Piv>
__device__ __forceinline__ void write_pfaffian(const PfArgs& a, int item, bool zero, int swaps,
                                               uint16_t* perm, const float* item_sign, Piv pivot) {
  const int lane = threadIdx.x & 31;
  int flag = 0, neg = 0, expo = 0;
  double mant = 1.0;
  float pmin = INFINITY, pmax = 0.0f;
  if (!zero)
    for (int k = lane; k < a.n / 2; k += 32) {
      const float pv = pivot(k);
      if (pv < 0.0f) neg ^= 1;
      const float ap = fabsf(pv);
      if (!isfinite(ap)) flag |= NH_FLAG_NONFINITE;
      pmin = fminf(pmin, ap);
      pmax = fmaxf(pmax, ap);
      int e;
      mant = frexp(mant * (double)ap, &e);
      expo += e;
    }
#pragma unroll
  for (int o = 16; o; o >>= 1) {  // 32 mantissas in [1/2, 1]: no underflow
    mant *= __shfl_xor_sync(0xffffffffu, mant, o);
    expo += __shfl_xor_sync(0xffffffffu, expo, o);
    neg ^= __shfl_xor_sync(0xffffffffu, neg, o);
    flag |= __shfl_xor_sync(0xffffffffu, flag, o);
    pmin = fminf(pmin, __shfl_xor_sync(0xffffffffu, pmin, o));
    pmax = fmaxf(pmax, __shfl_xor_sync(0xffffffffu, pmax, o));
  }
  if (lane == 0) {
    float s = item_sign ? item_sign[item] : 1.0f;
    double la;
    if (isnan(s)) flag |= NH_FLAG_NONFINITE;  // the CNN could not compute this item
    if (zero) {
      s = 0.0f;
      la = -INFINITY;
      flag |= NH_FLAG_ZERO_PIVOT;
    } else {
      if (neg) s = -s;
      la = log(mant) + (double)expo * 0.6931471805599453;
      if (!isfinite(la)) flag |= NH_FLAG_NONFINITE;
      if (a.cond_tau > 0.0 && (double)pmax > a.cond_tau * (double)pmin) flag |= NH_FLAG_GROWTH;
      if (a.refine_tau > 0.0 && (double)pmax > a.refine_tau * (double)pmin) flag |= kFlagNeedRefine;
    }
    if (s == 0.0f) la = -INFINITY;
    a.sign[item] = s;
    a.logabs[item] = la;
    if (a.flags) a.flags[item] = flag | a.flag_or;
    if (a.ratio) a.ratio[item] = zero ? INFINITY : (float)((double)pmax / (double)pmin);
    if (perm && !zero) perm[a.n] = (uint16_t)swaps;
  }
}

template <int NB, int D, int TH>
__global__ void __launch_bounds__(TH, 512 / TH) pf32_kernel(PfArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int WARPS = TH / 32;
  const int n = a.n;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const Pf32Layout L = pf32_layout(n, NB);
  float* Lw = reinterpret_cast<float*>(smem_raw);
  float* Us = reinterpret_cast<float*>(smem_raw + L.us);  // (n, NB), swizzled chunks (swz_index)
  float* Vs = reinterpret_cast<float*>(smem_raw + L.vs);
  float* pivs = reinterpret_cast<float*>(smem_raw + L.pivs);  // pivot A[k, k+1], negated on a swap
  unsigned long long* cand = reinterpret_cast<unsigned long long*>(smem_raw + L.cand);
  int* rt = reinterpret_cast<int*>(smem_raw + L.rt);        // compaction counts; [8] zero column
  int* misc = reinterpret_cast<int*>(smem_raw + L.misc);    // [0] row of logical k, [1] item
  uint8_t* alist = smem_raw + L.alist;
  uint8_t* clog = smem_raw + L.clog;

  const int n_work = a.count_dev ? (*a.count_dev) * a.count_mult : a.n_slots;
  for (int slot = blockIdx.x;; slot += gridDim.x) {
    if (a.queue) {  // dynamic schedule: the next item comes off the work counter
      __syncthreads();
      if (tid == 0) misc[1] = atomicAdd(a.queue, 1);
      __syncthreads();
      slot = misc[1];
    }
    if (slot >= n_work) break;
    const int item = a.slot_item ? a.slot_item[slot] : slot;
    __syncthreads();
    if (a.mode >= 2) {
      rows_and_gather<D, TH>(a, item, slot, Lw, smem_raw);
    } else if (a.mode == 0) {
      const float* F = a.F + (size_t)item * n * n;
      for (int i = wid; i < n; i += WARPS) {
        const float* src = F + (size_t)i * n;
        float* dst = Lw + tri_off(i);
        for (int j = lane; j < i; j += 32) dst[j] = __ldg(src + j);
      }
    } else {
      gather_lower<float, D, WARPS>(Lw, n, static_cast<const float*>(a.Y) + (size_t)slot * n * D,
                             a.idx + (size_t)slot * n, static_cast<const float*>(a.Wt), a.Lx, a.Ly);
    }
    __syncthreads();  // the rows in shared memory can overlap the scratch written next
    for (int p = tid; p < n; p += TH) alist[p] = clog[p] = (uint8_t)p;
    if (tid == 0) misc[0] = 0;
    __syncthreads();

    uint16_t* perm = a.perm ? a.perm + (size_t)item * perm_stride(n) : nullptr;
    int swaps = 0;
    bool zero = false;
    for (int k0 = 0; k0 < n - 1; k0 += 2 * NB) {
      const int steps = min(NB, (n - k0) >> 1);
      const int m = n - k0, PW = (m + 31) >> 5;
      if (wid < PW)
        panel_steps<NB>(Lw, Us, Vs, pivs, cand, rt, misc, alist, clog, m, k0, steps, PW, swaps,
                           perm);
      __syncthreads();  // panel written, active rows compacted
      zero = rt[8] != 0;
      if (zero) break;
      const int mt = m - 2 * steps;
      if (mt >= 2) {  // then steps == NB
        int done = 0;
        for (int c0 = 0; c0 + 1 < mt;) {
          if (mt - c0 > 64) {
            trail_block<NB, 4, WARPS>(Lw, Us, Vs, alist, mt, c0, done);
            c0 += 128;
          } else {
            trail_block<NB, 2, WARPS>(Lw, Us, Vs, alist, mt, c0, done);
            c0 += 64;
          }
        }
        __syncthreads();  // trailing triangle updated
      }
    }
    if (wid == 0)
      write_pfaffian(a, item, zero, swaps, perm, a.mode == 2 ? a.item_sign_out : a.item_sign,
                     [&](int k) { return pivs[k]; });
  }
}

// ------------------------------------------------------------------ FP32, n > 256
// The same operations in the same order as pfaffian_kernel with panels of 4 (the same bits), for
// triangles in global memory.  The trailing triangle is the traffic (8 bytes per element and
// update, from L2 or, where 148 triangles exceed it, from HBM), so it is updated once per
// kBbSteps = 16 pivot steps instead of once per 4: the panel values of four panels stay in
// shared memory, a column is brought up to date when it is read (the finished panels' terms as the
// trailing update's chain, then the running panel's), and the trailing update applies all four
// chains to an element in registers.  A negated element takes the two products of a step in the
// other order, so both orientations round alike.  512 threads, up to two rows each; the active
// rows are compacted after every 16 steps.  The next column is loaded while the pivot's is used (its
// owner is published before the step's first barrier).
constexpr int kBbTh = 512;
constexpr int kBbSteps = 16;
constexpr int kBbQuads = kBbSteps / 4;

struct BbLayout {
  size_t us, vs, pivs, cand, rt, misc, offs, alist, clog, end;
};
__host__ __device__ inline BbLayout bb_layout(int n, int D) {
  BbLayout L;
  L.us = 0;
  L.vs = L.us + 16 * (size_t)n * kBbQuads;
  size_t uv = L.vs + 16 * (size_t)n * kBbQuads;
  const size_t rows = 4 * (size_t)n * D + 4 * (size_t)n;  // gather: features and modes
  uv = (uv > rows ? uv : rows) + 15 & ~(size_t)15;
  L.pivs = uv;
  L.cand = (L.pivs + sizeof(float) * (size_t)(n / 2) + 15) & ~(size_t)15;
  L.rt = L.cand + 16 * sizeof(unsigned long long);
  L.misc = L.rt + 36 * sizeof(int);
  L.offs = L.misc + 8 * sizeof(int);
  L.alist = L.offs + sizeof(int) * (size_t)n;
  L.clog = L.alist + 2 * (size_t)n;
  L.end = L.clog + 2 * (size_t)n;
  return L;
}

// Entry (i, q) of the matrix as of step s: the stored element `c` (already negated where the row
// precedes the column), the chains of the finished quads, the running quad's terms.
__device__ __forceinline__ float bb_value(float c, bool gt, int i, int qi, int n, int quad,
                                          const float4* Us, const float4* Vs) {
  for (int b = 0; b < quad; ++b) {
    const float4 u = Us[b * n + i], v = Vs[b * n + i], uq = Us[b * n + qi], vq = Vs[b * n + qi];
    if (gt) {
      c = fmaf(u.x, vq.x, c);
      c = fmaf(-v.x, uq.x, c);
      c = fmaf(u.y, vq.y, c);
      c = fmaf(-v.y, uq.y, c);
      c = fmaf(u.z, vq.z, c);
      c = fmaf(-v.z, uq.z, c);
      c = fmaf(u.w, vq.w, c);
      c = fmaf(-v.w, uq.w, c);
    } else {
      c = fmaf(-v.x, uq.x, c);
      c = fmaf(u.x, vq.x, c);
      c = fmaf(-v.y, uq.y, c);
      c = fmaf(u.y, vq.y, c);
      c = fmaf(-v.z, uq.z, c);
      c = fmaf(u.z, vq.z, c);
      c = fmaf(-v.w, uq.w, c);
      c = fmaf(u.w, vq.w, c);
    }
  }
  const float4 u = Us[quad * n + i], v = Vs[quad * n + i];
  const float4 uq = Us[quad * n + qi], vq = Vs[quad * n + qi];
  c += u.x * vq.x - v.x * uq.x;  // terms past the running step are zero
  c += u.y * vq.y - v.y * uq.y;
  c += u.z * vq.z - v.z * uq.z;
  c += u.w * vq.w - v.w * uq.w;
  return c;
}

// Stored element (ph, q) of the triangle in global memory, negated where ph < q.
__device__ __forceinline__ float bb_stored(const float* Lw, int ph, int off, int q, int qoff) {
  const float c = __ldcg(Lw + (ph > q ? off + q : (ph < q ? qoff + ph : 0)));
  return ph > q ? c : (ph < q ? -c : 0.0f);
}

// Up to 16 pivot steps from logical column k0 on the m active rows by the first PW warps.
__device__ __forceinline__ void bb_panel(const float* Lw, float4* Us, float4* Vs, float* pivs,
                                         unsigned long long* cand, int* rt, int* misc, int* offs,
                                         uint16_t* alist, uint16_t* clog, int n, int m, int k0,
                                         int steps, int PW, int& swaps, uint16_t* perm) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  int ph[2], off[2], log[2];
  float next[2];  // stored entries of the column of the coming step
  const int ck0 = misc[0], ckp0 = alist[ck0], ckoff0 = tri_off(ckp0);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int i = tid + q * kBbTh;
    const bool has = i < m;
    ph[q] = has ? alist[i] : 0;
    log[q] = has ? clog[i] : -1;
    off[q] = tri_off(ph[q]);
    next[q] = has ? bb_stored(Lw, ph[q], off[q], ckp0, ckoff0) : 0.0f;
  }
  if (wid == 0 && lane < 16) cand[lane] = 0ull;
  bool zero = false;
  int ci = ck0;
#pragma unroll 1
  for (int s = 0; s < steps; ++s) {
    const int k = k0 + 2 * s, quad = s >> 2, j = s & 3;
    if (j == 0) {  // a new quad of panel values starts from zeros
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int i = tid + q * kBbTh;
        if (i < m) Us[quad * n + i] = Vs[quad * n + i] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      panel_sync(PW);
    }
    const int ckp = alist[ci];
    float c[2];
    unsigned key[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      key[q] = 0u;
      c[q] = 0.0f;
      if (log[q] > k) {
        c[q] = bb_value(next[q], ph[q] > ckp, tid + q * kBbTh, ci, n, quad, Us, Vs);
        // |c| bits + 1 (NaN as +inf)
        key[q] = min(__float_as_uint(c[q]) & 0x7FFFFFFFu, 0x7F800000u) + 1u;
      }
      if (log[q] == k + 1 || log[q] == k + 2) misc[log[q] - k] = tid + q * kBbTh;
    }
    // Maximum, ties to the lowest physical row (rows ascend with the index, slot 0 before slot 1).
    unsigned kbest = __reduce_max_sync(0xffffffffu, max(key[0], key[1]));
    const unsigned h0 = __ballot_sync(0xffffffffu, key[0] == kbest);
    const unsigned h1 = __ballot_sync(0xffffffffu, key[1] == kbest);
    const int wq = h0 ? 0 : 1, wl = __ffs(h0 ? h0 : h1) - 1;
    // row index, sign, label: 0x3FF - index (10 bits), 1, 10 bits
    const unsigned mine = ((0x3FFu - (unsigned)(tid + wq * kBbTh)) << 11) |
                          (signbit(wq ? c[1] : c[0]) ? 0x400u : 0u) |
                          ((unsigned)(wq ? log[1] : log[0]) & 0x3FFu);
    unsigned lbest;
    if (PW == 1) {
      lbest = __shfl_sync(0xffffffffu, mine, wl);
      __syncwarp();  // misc
    } else {
      if (lane == wl) cand[wid] = ((unsigned long long)kbest << 32) | mine;
      panel_sync(PW);  // (1) pivot candidates, owners of the next labels
      const unsigned long long w = cand[lane & 15];
      const unsigned hi = (unsigned)(w >> 32);
      kbest = __reduce_max_sync(0xffffffffu, hi);
      lbest = __reduce_max_sync(0xffffffffu, hi == kbest ? (unsigned)w : 0u);
    }
    const float bk = kbest ? __uint_as_float(kbest - 1u) : -1.0f;
    if (!(bk > 0.0f)) {  // exactly singular (or empty) column: pf = 0
      zero = true;
      panel_sync(PW);
      break;
    }
    const int ri = 0x3FF - (int)(lbest >> 11), lr = (int)(lbest & 0x3FFu);
    const float piv = (lbest & 0x400u) ? bk : -bk;
    const int rp = alist[ri], roff = tri_off(rp);
    ci = lr == k + 2 ? misc[1] : misc[2];
    const bool more = s + 1 < steps;
    const int cp = more ? alist[ci] : 0, coff = tri_off(cp);
    float dv[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (log[q] <= k) continue;
      // the row that held label k+1 takes the pivot's old label
      log[q] = tid + q * kBbTh == ri ? k + 1 : (log[q] == k + 1 ? lr : log[q]);
      dv[q] = bb_stored(Lw, ph[q], off[q], rp, roff);
      if (more) next[q] = bb_stored(Lw, ph[q], off[q], cp, coff);
    }
    const float rpiv = 1.0f / piv;
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (log[q] > k + 1) {
        const int i = tid + q * kBbTh;
        const float u = bb_value(dv[q], ph[q] > rp, i, ri, n, quad, Us, Vs);
        reinterpret_cast<float*>(Us + quad * n + i)[j] = u;
        reinterpret_cast<float*>(Vs + quad * n + i)[j] = c[q] * rpiv;
      }
    if (tid == 0) pivs[k >> 1] = lr != k + 1 ? -piv : piv;
    swaps ^= lr != k + 1 ? 1 : 0;
    panel_sync(PW);  // (2) panel column written
  }
  // Eliminated rows leave: their order to the record, the others compacted in physical order (with
  // their panel values, which the trailing update reads by the new index).
  const int k_end = k0 + 2 * steps;
  unsigned bal[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    bal[q] = __ballot_sync(0xffffffffu, log[q] >= k_end);
    if (lane == 0) rt[q * 16 + wid] = __popc(bal[q]);
    if (perm && !zero && log[q] >= 0 && log[q] < k_end) perm[log[q]] = (uint16_t)ph[q];
  }
  if (tid == 0) rt[32] = zero ? 1 : 0;
  panel_sync(PW);
  int base = 0, dst[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    int before = base;
    for (int w = 0; w < PW; ++w) {
      before += w < wid ? rt[q * 16 + w] : 0;
      base += rt[q * 16 + w];
    }
    dst[q] = log[q] >= k_end ? before + __popc(bal[q] & ((1u << lane) - 1u)) : -1;
    if (dst[q] >= 0) {
      alist[dst[q]] = (uint16_t)ph[q];
      clog[dst[q]] = (uint16_t)log[q];
      offs[dst[q]] = off[q];
      if (log[q] == k_end) misc[0] = dst[q];
    }
  }
  if (!zero && base > 0) {
#pragma unroll 1
    for (int b = 0; b < kBbQuads; ++b) {
      float4 u[2], v[2];
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (dst[q] >= 0) {
          u[q] = Us[b * n + tid + q * kBbTh];
          v[q] = Vs[b * n + tid + q * kBbTh];
        }
      panel_sync(PW);
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (dst[q] >= 0) {
          Us[b * n + dst[q]] = u[q];
          Vs[b * n + dst[q]] = v[q];
        }
      panel_sync(PW);
    }
  }
}

// One unit of the trailing update: RT rows from ia0 on the lane's two columns (physical rows pb,
// panel values ub / vb).  FULL: every row exists and reaches both columns of every lane.
template <int RT, bool FULL>
__device__ __forceinline__ void bb_unit(float* Lw, const float4* Us, const float4* Vs,
                                        const int* offs, int n, int m, int ia0, int col, const int (&pb)[2],
                                        const float4 (&ub)[2][kBbQuads],
                                        const float4 (&vb)[2][kBbQuads]) {
  float acc[RT][2];
  int off[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    off[r] = offs[FULL ? ia0 + r : min(ia0 + r, m - 1)];
#pragma unroll
    for (int h = 0; h < 2; ++h)
      acc[r][h] = FULL || (ia0 + r < m && col + 32 * h < ia0 + r) ? __ldcg(Lw + off[r] + pb[h])
                                                                  : 0.0f;
  }
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    const int ia = FULL ? ia0 + r : min(ia0 + r, m - 1);
#pragma unroll
    for (int b = 0; b < kBbQuads; ++b) {
      const float4 ua = Us[b * n + ia], va = Vs[b * n + ia];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float x = acc[r][h];
        x = fmaf(ua.x, vb[h][b].x, x);
        x = fmaf(-va.x, ub[h][b].x, x);
        x = fmaf(ua.y, vb[h][b].y, x);
        x = fmaf(-va.y, ub[h][b].y, x);
        x = fmaf(ua.z, vb[h][b].z, x);
        x = fmaf(-va.z, ub[h][b].z, x);
        x = fmaf(ua.w, vb[h][b].w, x);
        x = fmaf(-va.w, ub[h][b].w, x);
        acc[r][h] = x;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (FULL || (ia0 + r < m && col + 32 * h < ia0 + r)) __stcg(Lw + off[r] + pb[h], acc[r][h]);
}

// Trailing update of the m active rows by the 16 steps' panel values: units of 8 rows x 64 columns
// (lane: two columns, their panel values in registers), all loads of a unit in flight together.
// offs: the rows' offsets in the triangle.
__device__ __forceinline__ void bb_trailing(float* Lw, const float4* Us, const float4* Vs,
                                            const uint16_t* alist, const int* offs, int n, int m) {
  constexpr int RT = 8, WARPS = kBbTh / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int done = 0;
#pragma unroll 1
  for (int c0 = 0; c0 + 1 < m; c0 += 64) {
    const int units = (m - c0 - 1 + RT - 1) / RT;
    const int u0 = (wid - done) & (WARPS - 1);
    done += units;
    if (u0 >= units) continue;
    int pb[2];
    float4 ub[2][kBbQuads], vb[2][kBbQuads];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int ib = min(c0 + lane + 32 * h, m - 1);
      pb[h] = alist[ib];
#pragma unroll
      for (int b = 0; b < kBbQuads; ++b) {
        ub[h][b] = Us[b * n + ib];
        vb[h][b] = Vs[b * n + ib];
      }
    }
#pragma unroll 1
    for (int u = u0; u < units; u += WARPS) {
      const int ia0 = c0 + 1 + u * RT;
      if (ia0 >= c0 + 64 && ia0 + RT <= m)
        bb_unit<RT, true>(Lw, Us, Vs, offs, n, m, ia0, c0 + lane, pb, ub, vb);
      else
        bb_unit<RT, false>(Lw, Us, Vs, offs, n, m, ia0, c0 + lane, pb, ub, vb);
    }
  }
}

template <int D>
__global__ void __launch_bounds__(kBbTh, 1) pf32_big_kernel(PfArgs a) {
  constexpr int WARPS = kBbTh / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = a.n, N = a.Lx * a.Ly;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const BbLayout L = bb_layout(n, a.mode == 0 ? 0 : D);
  float4* Us = reinterpret_cast<float4*>(smem_raw + L.us);  // [quad][compact row]
  float4* Vs = reinterpret_cast<float4*>(smem_raw + L.vs);
  float* pivs = reinterpret_cast<float*>(smem_raw + L.pivs);
  unsigned long long* cand = reinterpret_cast<unsigned long long*>(smem_raw + L.cand);
  int* rt = reinterpret_cast<int*>(smem_raw + L.rt);      // compaction counts; [32] zero column
  int* misc = reinterpret_cast<int*>(smem_raw + L.misc);  // compact rows of labels k, k + 1, k + 2
  int* offs = reinterpret_cast<int*>(smem_raw + L.offs);  // triangle offsets of the active rows
  uint16_t* alist = reinterpret_cast<uint16_t*>(smem_raw + L.alist);
  uint16_t* clog = reinterpret_cast<uint16_t*>(smem_raw + L.clog);
  float* Lw = static_cast<float*>(a.tri) + (size_t)blockIdx.x * ((tri_off(n) + 3) & ~3);

  const int n_work = a.count_dev ? (*a.count_dev) * a.count_mult : a.n_slots;
  for (int slot = blockIdx.x; slot < n_work; slot += gridDim.x) {
    const int item = a.slot_item ? a.slot_item[slot] : slot;
    __syncthreads();  // the previous item's readers are done
    if (a.mode == 0) {
      const float* F = a.F + (size_t)item * n * n;
      for (int i = wid; i < n; i += WARPS)
        for (int j = lane; j < i; j += 32) __stcg(Lw + tri_off(i) + j, __ldg(F + (size_t)i * n + j));
    } else {
      float* Ys = reinterpret_cast<float*>(smem_raw);
      int* ids = reinterpret_cast<int*>(Ys + (size_t)n * D);
      const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(a.Y) +
                                                          (size_t)slot * n * D);
      constexpr int K = D / 4;
      for (int v = tid; v < n * K; v += kBbTh) {
        const int row = v / K;
        reinterpret_cast<float4*>(Ys)[row * K + ((v % K) ^ swz_key(row, K))] = __ldg(src + v);
      }
      for (int p = tid; p < n; p += kBbTh)
        ids[p] = pack_mode(__ldg(a.idx + (size_t)slot * n + p), N, a.Ly);
      __syncthreads();
      gather_from_rows<D, kBbTh>(a, Lw, Ys, ids);
    }
    __syncthreads();
    for (int p = tid; p < n; p += kBbTh) alist[p] = clog[p] = (uint16_t)p;
    if (tid == 0) misc[0] = 0;
    __syncthreads();

    uint16_t* perm = a.perm ? a.perm + (size_t)item * perm_stride(n) : nullptr;
    int swaps = 0;
    bool zero = false;
    for (int k0 = 0; k0 < n - 1; k0 += 2 * kBbSteps) {
      const int steps = min(kBbSteps, (n - k0) >> 1);
      const int m = n - k0, PW = min(WARPS, (m + 31) >> 5);
      if (wid < PW)
        bb_panel(Lw, Us, Vs, pivs, cand, rt, misc, offs, alist, clog, n, m, k0, steps, PW, swaps,
                 perm);
      __syncthreads();  // panel values and active rows compacted
      zero = rt[32] != 0;
      if (zero) break;
      const int mt = m - 2 * steps;  // when rows remain, steps == kBbSteps
      if (mt >= 2) {
        bb_trailing(Lw, Us, Vs, alist, offs, n, mt);
        __syncthreads();
      }
    }
    if (wid == 0)
      write_pfaffian(a, item, zero, swaps, perm, a.item_sign, [&](int k) { return pivs[k]; });
  }
}

// Launch with the panel width of n: 8 up to kPf32NB8MaxN, else 4 (the width is part of the
// operation order, so it depends on n alone).
template <int NB, int D, int TH>
int launch_pf32_th(const PfArgs& a, size_t smem, int per_sm, int prof_id, cudaStream_t st) {
  if (int rc = raise_smem_cap(pf32_kernel<NB, D, TH>, smem)) return rc;
  int grid = num_sms() * per_sm;
  if (grid > a.n_slots) grid = a.n_slots;
  if (grid <= 0) return NH_OK;
  ProfScope prof_scope(prof_id, st);
  pf32_kernel<NB, D, TH><<<grid, TH, smem, st>>>(a);
  return check_launch("pf32_kernel");
}

// Two CTAs of 256 threads per SM (one beyond 113 KB), or, where there are items for them, four of
// 128 that shared memory and one row per thread allow: small matrices leave most of 256 threads
// idle, and their steps are latency.
template <int NB, int D>
int launch_pf32_nb(const PfArgs& a, size_t smem, int prof_id, cudaStream_t st) {
  if (smem > 227 * 1024)
    return fail(NH_ERR_UNSUPPORTED, "Pfaffian: n=%d needs %zu B of shared memory", a.n, smem);
  if (smem <= 56 * 1024 && a.n <= 128 && a.n_slots > 2 * num_sms())
    return launch_pf32_th<NB, D, 128>(a, smem, 4, prof_id, st);
  return launch_pf32_th<NB, D, 256>(a, smem, smem <= 113 * 1024 ? 2 : 1, prof_id, st);
}

template <int D>
int launch_pf32(const PfArgs& a, cudaStream_t st) {
  return a.n <= kPf32NB8MaxN
             ? launch_pf32_nb<8, D>(a, pf32_layout(a.n, 8).end, NH_K_PFAFFIAN, st)
             : launch_pf32_nb<4, D>(a, pf32_layout(a.n, 4).end, NH_K_PFAFFIAN, st);
}

template <int D>
int launch_pf32_big(const PfArgs& a, cudaStream_t st) {
  if (!a.tri)
    return fail(NH_ERR_UNSUPPORTED, "Pfaffian: n=%d needs the large-lattice scratch", a.n);
  const size_t smem = bb_layout(a.n, a.mode == 0 ? 0 : D).end;
  if (smem > 227 * 1024)
    return fail(NH_ERR_UNSUPPORTED, "Pfaffian: n=%d needs %zu B of shared memory", a.n, smem);
  if (int rc = raise_smem_cap(pf32_big_kernel<D>, smem)) return rc;
  int grid = num_sms();
  if (grid > a.n_slots) grid = a.n_slots;
  if (grid <= 0) return NH_OK;
  ProfScope prof_scope(NH_K_PFAFFIAN, st);
  pf32_big_kernel<D><<<grid, kBbTh, smem, st>>>(a);
  return check_launch("pf32_big_kernel");
}

// FP32: pf32_kernel up to 256 rows, pf32_big_kernel beyond; FP64: one CTA per SM, beyond shared
// memory (n > 236) the triangle in global memory.
template <typename T, int D>
int launch_pf_pick(const PfArgs& a, cudaStream_t st) {
  if (a.n <= kNumThreads) {
    if constexpr (sizeof(T) == 4) {
      return launch_pf32<D>(a, st);
    } else {
      if (pf_smem<T, 4>(a.n) <= 227 * 1024) return launch_pf<T, 4, D>(a, st);
      if (pf_smem<T, 2>(a.n) <= 227 * 1024) return launch_pf<T, 2, D>(a, st);
    }
  }
  if constexpr (sizeof(T) == 4)
    return launch_pf32_big<D>(a, st);
  else
    return launch_pf<T, kBigNB, D, kBigThreads>(a, st);
}

template <typename T>
int launch_pf_d(const PfArgs& a, int d, cudaStream_t st) {
  switch (d) {
    case 8: return launch_pf_pick<T, 8>(a, st);
    case 16: return launch_pf_pick<T, 16>(a, st);
    case 32: return launch_pf_pick<T, 32>(a, st);
    default: return fail(NH_ERR_UNSUPPORTED, "amplitude: d=%d (8, 16 or 32)", d);
  }
}

// ------------------------------------------------------------------ standalone gather
template <int D>
__global__ void __launch_bounds__(kNumThreads) pairing_kernel(const float* __restrict__ Y,
                                                              const int32_t* __restrict__ idx,
                                                              const float* __restrict__ Wt,
                                                              int Lx, int Ly, int n, int batch,
                                                              float* __restrict__ F) {
  const int N = Lx * Ly;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int item = blockIdx.x; item < batch; item += gridDim.x) {
    const float* Yi = Y + (size_t)item * n * D;
    const int32_t* ii = idx + (size_t)item * n;
    float* Fi = F + (size_t)item * n * n;
    for (int p = wid; p < n; p += kWarps) {
      const int mp = __ldg(ii + p);
      const int sp = mp >= N ? 1 : 0;
      const int sitep = mp - sp * N;
      const int xp = sitep / Ly, ypos = sitep - xp * Ly;
      float yp[D];
#pragma unroll
      for (int a0 = 0; a0 < D; a0 += 4) ldg16(Yi + (size_t)p * D + a0, yp + a0);
      for (int q = lane; q < n; q += 32) {
        float v = 0.0f;
        if (q != p)
          v = pair_value<float, D>(yp, sp, xp, ypos, Yi + (size_t)q * D, __ldg(ii + q), N, Lx, Ly,
                                   Wt);
        Fi[(size_t)p * n + q] = v;
      }
    }
  }
}

// Shared-memory variant: the Wt table is staged once per CTA and each matrix's occupied features
// once per matrix, rows padded to D + 4 floats (16-byte chunks of 8 consecutive rows fall in
// distinct banks); a warp computes two rows per pass so that each feature row it loads serves
// two outputs.  Same per-element arithmetic as pair_value: F is bit-for-bit that of the fused
// gather and exactly antisymmetric.
template <int D>
__global__ void __launch_bounds__(kNumThreads) pairing_smem_kernel(
    const float* __restrict__ Y, const int32_t* __restrict__ idx, const float* __restrict__ Wt,
    int Lx, int Ly, int n, int batch, float* __restrict__ F) {
  constexpr int DP = D + 4;
  extern __shared__ __align__(16) float psm[];
  const int N = Lx * Ly;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  float* wts = psm;            // (4 N, DP)
  float* ys = wts + 4 * N * DP;  // (n, DP)
  int* info = reinterpret_cast<int*>(ys + n * DP);  // (spin << 16) | (x << 8) | y per row
  for (int e = tid; e < 4 * N * D; e += kNumThreads) {
    const int row = e / D;
    wts[row * DP + (e - row * D)] = __ldg(Wt + e);
  }
  for (int item = blockIdx.x; item < batch; item += gridDim.x) {
    const float* Yi = Y + (size_t)item * n * D;
    const int32_t* ii = idx + (size_t)item * n;
    float* Fi = F + (size_t)item * n * n;
    __syncthreads();
    for (int e = tid; e < n * D; e += kNumThreads) {
      const int row = e / D;
      ys[row * DP + (e - row * D)] = __ldg(Yi + e);
    }
    for (int p = tid; p < n; p += kNumThreads) {
      const int m = __ldg(ii + p);
      const int sp = m >= N ? 1 : 0;
      const int site = m - sp * N;
      const int x = site / Ly;
      info[p] = (sp << 16) | (x << 8) | (site - x * Ly);
    }
    __syncthreads();
    for (int p0 = 2 * wid; p0 < n; p0 += 2 * kWarps) {
      const int np = p0 + 1 < n ? 2 : 1;
      float yp[2][D];
      int sp[2], xp[2], ypos[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int p = h < np ? p0 + h : p0;
#pragma unroll
        for (int a0 = 0; a0 < D; a0 += 4) {
          const float4 v = *reinterpret_cast<const float4*>(ys + p * DP + a0);
          yp[h][a0] = v.x;
          yp[h][a0 + 1] = v.y;
          yp[h][a0 + 2] = v.z;
          yp[h][a0 + 3] = v.w;
        }
        const int inf = info[p];
        sp[h] = inf >> 16;
        xp[h] = (inf >> 8) & 0xFF;
        ypos[h] = inf & 0xFF;
      }
      for (int q = lane; q < n; q += 32) {
        float yq[D];
#pragma unroll
        for (int a0 = 0; a0 < D; a0 += 4) {
          const float4 v = *reinterpret_cast<const float4*>(ys + q * DP + a0);
          yq[a0] = v.x;
          yq[a0 + 1] = v.y;
          yq[a0 + 2] = v.z;
          yq[a0 + 3] = v.w;
        }
        const int inf = info[q];
        const int sq = inf >> 16, xq = (inf >> 8) & 0xFF, yqp = inf & 0xFF;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h >= np) continue;
          const int p = p0 + h;
          float acc = 0.0f;
          if (q != p) {
            int dx = xp[h] - xq, dy = ypos[h] - yqp;
            dx += dx < 0 ? Lx : 0;
            dy += dy < 0 ? Ly : 0;
            const float* w = wts + ((2 * sp[h] + sq) * N + dx * Ly + dy) * DP;
#pragma unroll
            for (int a0 = 0; a0 < D; a0 += 4) {
              const float4 wv = *reinterpret_cast<const float4*>(w + a0);
              acc = fmaf(yp[h][a0] * yq[a0], wv.x, acc);
              acc = fmaf(yp[h][a0 + 1] * yq[a0 + 1], wv.y, acc);
              acc = fmaf(yp[h][a0 + 2] * yq[a0 + 2], wv.z, acc);
              acc = fmaf(yp[h][a0 + 3] * yq[a0 + 3], wv.w, acc);
            }
          }
          Fi[(size_t)p * n + q] = acc;
        }
      }
    }
  }
}

size_t pairing_smem_bytes(int N, int n, int D) {
  return sizeof(float) * (4 * (size_t)N + n) * (D + 4) + sizeof(int) * (size_t)n;
}

// ------------------------------------------------------------------ image combination
// Also used with G = 1 to copy the per-item results into the caller's arrays.
// Sum over the images of one configuration in FP64: returns sum_g s_g exp(l_g - m) and sets
// *asum to sum_g |.| and *m to the largest log.
__device__ __forceinline__ double image_sum(const float* __restrict__ sg,
                                           const double* __restrict__ la, int c, int G,
                                           double* m_out, double* asum) {
  double m = -INFINITY;
  for (int g = 0; g < G; ++g) {
    const float s = sg[(size_t)c * G + g];
    const double l = la[(size_t)c * G + g];
    if (s != 0.0f && l > m) m = l;
  }
  double tot = 0.0, a = 0.0;
  if (m > -INFINITY)
    for (int g = 0; g < G; ++g) {
      const float s = sg[(size_t)c * G + g];
      if (s != 0.0f) {
        const double t = exp(la[(size_t)c * G + g] - m);
        tot += (double)s * t;
        a += t;
      }
    }
  *m_out = m;
  *asum = a;
  return tot;
}

// FP64-feature selection for projected amplitudes, before the FP64 list is built.  An image's
// error reaches log|psi_P| weighted by its share w_g = eta_g psi_g / psi_P (sum_g w_g = 1,
// sum_g |w_g| = C), and the error of an image with FP32 (or BF16x3) features grows with its
// pivot ratio r_g.  In a configuration whose images cancel (C > cancel_tau > 0) every image
// with |w_g| > kCancelImageFloor is marked (NH_FLAG_GROWTH | NH_FLAG_CANCEL): an FP32 image
// error (at most ~1e-3) of the others adds < 2e-5.  Otherwise, with weighted set, an image is
// marked exactly when |w_g| r_g > cond_tau (its estimated error, up to the features' relative
// accuracy), and unmarked when not; without weighted (cond_tau <= 1, every image already
// marked) the marks stay.
constexpr double kCancelImageFloor = 2e-2;

__global__ void image_mark_kernel(const float* __restrict__ sg, const double* __restrict__ la,
                                  int32_t* __restrict__ fl, const float* __restrict__ ratio,
                                  int G, int n_cfg, const int32_t* n_cfg_dev, double cancel_tau,
                                  double cond_tau, bool weighted) {
  const int n = n_cfg_dev ? *n_cfg_dev : n_cfg;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    double m, a;
    const double tot = image_sum(sg, la, c, G, &m, &a);
    if (cancel_tau > 0.0 && a > 0.0 && a > cancel_tau * fabs(tot)) {
      for (int g = 0; g < G; ++g) {
        const size_t i = (size_t)c * G + g;
        if (sg[i] != 0.0f && exp(la[i] - m) > kCancelImageFloor * fabs(tot))
          fl[i] |= NH_FLAG_GROWTH | NH_FLAG_CANCEL;
      }
    } else if (weighted && tot != 0.0) {
      for (int g = 0; g < G; ++g) {
        const size_t i = (size_t)c * G + g;
        const int f = fl[i];
        if ((f & (NH_FLAG_NONFINITE | NH_FLAG_ZERO_PIVOT)) || sg[i] == 0.0f) continue;
        const double w = exp(la[i] - m) / fabs(tot);
        fl[i] = w * (double)ratio[i] > cond_tau ? (f | NH_FLAG_GROWTH) : (f & ~NH_FLAG_GROWTH);
      }
    }
  }
}

__global__ void combine_kernel(const float* __restrict__ sg, const double* __restrict__ la,
                               const int32_t* __restrict__ fl, int G, int n_cfg,
                               const int32_t* n_cfg_dev, float* sign, double* logabs,
                               int32_t* flags, double cancel_tau, const int32_t* err) {
  const int n = n_cfg_dev ? *n_cfg_dev : n_cfg;
  const int timeout = (err && *err) ? NH_FLAG_TIMEOUT : 0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    int f = timeout;
    if (fl)
      for (int g = 0; g < G; ++g) f |= fl[(size_t)c * G + g] & kPublicFlags;
    double m, a;
    const double tot = image_sum(sg, la, c, G, &m, &a);
    if (cancel_tau > 0.0 && a > 0.0 && a > cancel_tau * fabs(tot)) f |= NH_FLAG_CANCEL;
    const float so = tot > 0.0 ? 1.0f : (tot < 0.0 ? -1.0f : 0.0f);
    sign[c] = so;
    logabs[c] = so != 0.0f ? log(fabs(tot)) + m - log((double)G) : -INFINITY;
    if (flags) flags[c] = f;
  }
}

// Ordered list of the items whose flags carry a bit of set_mask and none of clear_mask (single
// CTA).
__global__ void __launch_bounds__(1024) flagged_kernel(const int32_t* __restrict__ flags,
                                                       int n_items, const int32_t* count_dev,
                                                       int count_mult, int32_t* list,
                                                       int32_t* count, int set_mask,
                                                       int clear_mask) {
  __shared__ int wsum[32];
  __shared__ int carry;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n = count_dev ? (*count_dev) * count_mult : n_items;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 1024) {
    const int i = base + threadIdx.x;
    const int f = i < n ? flags[i] : 0;
    const int v = (i < n && (f & set_mask) && !(f & clear_mask)) ? 1 : 0;
    const unsigned bal = __ballot_sync(0xffffffffu, v);
    if (lane == 0) wsum[wid] = __popc(bal);
    __syncthreads();
    if (wid == 0) {
      int w = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    if (v) list[carry + (wid ? wsum[wid - 1] : 0) + __popc(bal & ((1u << lane) - 1u))] = i;
    __syncthreads();
    if (threadIdx.x == 0) carry += wsum[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) *count = carry;
}


// ------------------------------------------------------------------ tensor-memory Pfaffian
// The FP32 matrix lives in tensor memory (one matrix per SM: rows 0-127 in lanes 0-127 of
// columns [0, NP), rows 128-255 in columns [NP, 2 NP), NP = n rounded up to 32); thread t owns
// row t and reads pivot columns with tcgen05.ld.  The panel is the same relabelling Parlett-Reid
// as pfaffian_kernel; at the end of each panel of 8 steps the rank-16 update
// A += U V^T - V U^T runs on the tensor cores as 3xTF32 products (X = X_big + X_small, both
// rounded to TF32): U_b V_b^T + U_b V_s^T + U_s V_b^T - V_b U_b^T - V_b U_s^T - V_s U_b^T, six
// kind::tf32 MMAs (M = 128, N = NP, K = 8) per 128-row tile, the minus signs via the A-negate bit
// of the instruction descriptor.  Accuracy: the accumulation into the FP32 matrix in tensor
// memory, not the operand split, limits this form (a three-way split measured no better); at
// n = 224 log|pf| is within about 2e-4 of FP64, against 1e-4 for the CUDA-core kernel.  Rows and columns of eliminated indices carry U = V = 0 and never
// change again.  The occupied block is gathered into a shared-memory lower triangle first and
// copied into tensor memory with tcgen05.st.

constexpr int kTcNB = 8;
constexpr int kTcOpFloats = 4 * 2048 + 2 * kNumThreads * kTcNB;  // operands + FP32 panel copies
constexpr uint32_t kTcCols = 512;
constexpr long long kTcWaitLimit = 1ll << 22;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // sm_100 descriptor version; no swizzle, base offset 0
  return d;
}

// kind::tf32 instruction descriptor: FP32 accumulate, TF32 A and B, K-major, M = 128, N = np.
__device__ __forceinline__ uint32_t tf32_idesc(int np, bool neg_a) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((neg_a ? 1u : 0u) << 13) |
         ((uint32_t)(np >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 1, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc));
}

__device__ __forceinline__ float tmem_ld1(uint32_t taddr) {
  uint32_t r;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(r) : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  return __uint_as_float(r);
}

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, "
      "%29, %30, %31, %32};\n" ::"r"(taddr),
      "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
      "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
      "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])), "r"(__float_as_uint(v[8])),
      "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
      "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])),
      "r"(__float_as_uint(v[15])), "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])),
      "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])), "r"(__float_as_uint(v[20])),
      "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
      "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])),
      "r"(__float_as_uint(v[27])), "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])),
      "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31])));
}

__device__ __forceinline__ float tf32_big(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t a = smem_addr(bar);
  for (long long it = 0; it < kTcWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Operand arrays (K-major, no swizzle): element (row t, k) of a 256 x 8 TF32 matrix at
// (k / 4) * 4096 + (t / 8) * 128 + (t % 8) * 16 + (k % 4) * 4 bytes.
__device__ __forceinline__ int opnd_off(int t, int k) {
  return (k >> 2) * 1024 + (t >> 3) * 32 + (t & 7) * 4 + (k & 3);  // in floats
}

template <int D>
__global__ void __launch_bounds__(kNumThreads, 1) pfaffian_tc_kernel(PfArgs a, int32_t* err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = a.n;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int tri = tri_off(n);
  const int NP = (n + 31) & ~31;
  const int n_tiles = (n + 127) >> 7;
  float* region = reinterpret_cast<float*>(smem_raw);  // staging triangle, later the operands
  const int region_floats = max((tri + 31) & ~31, kTcOpFloats);
  float* Ub = region;               // 4 operand arrays of 256 x 8 TF32 (8 KB each)
  float* Us = region + 2048;
  float* Vb = region + 4096;
  float* Vs = region + 6144;
  float* Uf = region + 8192;        // FP32 copies [row][8] for the in-panel corrections
  float* Vf = Uf + kNumThreads * kTcNB;
  float* pivs = region + region_floats;          // (128) signed pivots
  float* rkey = pivs + 128;                      // (warps)
  int* rt = reinterpret_cast<int*>(rkey + kWarps);
  int* rlog = rt + kWarps;
  int* misc = rlog + kWarps;                     // [0] physical row of logical k, [1] abort
  uint64_t* bar = reinterpret_cast<uint64_t*>(misc + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    misc[1] = 0;
  }
  if (wid == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(tmem_slot)),
                 "r"(kTcCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t my_col0 = tmem + ((uint32_t)(32 * (wid & 3)) << 16) + (uint32_t)((tid >> 7) * NP);
  uint32_t phase = 0;

  const int n_work = a.count_dev ? (*a.count_dev) * a.count_mult : a.n_slots;
  const float* Ybase = static_cast<const float*>(a.Y);
  const float* Wt = static_cast<const float*>(a.Wt);
  for (int slot = blockIdx.x; slot < n_work; slot += gridDim.x) {
    const int item = a.slot_item ? a.slot_item[slot] : slot;
    if (misc[1]) {  // a wait expired earlier: mark the item instead of computing it
      if (tid == 0) {
        a.sign[item] = NAN;
        a.logabs[item] = NAN;
        if (a.flags) a.flags[item] = NH_FLAG_NONFINITE | a.flag_or;
      }
      continue;
    }
    __syncthreads();
    if (a.mode == 0) {
      const float* F = a.F + (size_t)item * n * n;
      for (int i = wid; i < n; i += kWarps) {
        const float* src = F + (size_t)i * n;
        float* dst = region + tri_off(i);
        for (int j = lane; j < i; j += 32) dst[j] = __ldg(src + j);
      }
    } else {
      gather_lower<float, D>(region, n, Ybase + (size_t)slot * n * D, a.idx + (size_t)slot * n,
                             Wt, a.Lx, a.Ly);
    }
    __syncthreads();
    // Full antisymmetric matrix into tensor memory, 32 columns per store; rows >= n are zero.
    for (int b = 0; b < NP / 32; ++b) {
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int q = 32 * b + i;
        float x = 0.0f;
        if (tid < n && q < n) x = q < tid ? region[tri_off(tid) + q] : (q > tid ? -region[tri_off(q) + tid] : 0.0f);
        v[i] = x;
      }
      tmem_st32(my_col0 + 32 * b, v);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // the staging triangle is dead from here: the operand arrays reuse it
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0) misc[0] = 0;
    __syncthreads();

    int my_log = tid < n ? tid : -1;
    int flag = 0, swaps = 0;
    bool zero = false, abort = false;
    for (int k0 = 0; k0 < n - 1 && !zero && !abort; k0 += 2 * kTcNB) {
      const int steps = min(kTcNB, (n - k0) >> 1);
      float myU[kTcNB], myV[kTcNB];
#pragma unroll
      for (int j = 0; j < kTcNB; ++j) {
        myU[j] = 0.0f;
        myV[j] = 0.0f;
        if (j >= steps) {  // columns a short last panel leaves unused must be zero
          const int o = opnd_off(tid, j);
          Ub[o] = Us[o] = Vb[o] = Vs[o] = 0.0f;
        }
      }
#pragma unroll
      for (int j = 0; j < kTcNB; ++j) {
        if (j < steps && !zero) {
          const int k = k0 + 2 * j;
          const int ck = misc[0];
          float c = tmem_ld1(my_col0 + ck);
          const bool act = my_log > k;
          if (act) {
#pragma unroll
            for (int p = 0; p < kTcNB; ++p)
              if (p < j) c += myU[p] * Vf[ck * kTcNB + p] - myV[p] * Uf[ck * kTcNB + p];
          }
          const float mag = act ? (isnan(c) ? INFINITY : fabsf(c)) : -1.0f;
          float wmax = mag;
#pragma unroll
          for (int o = 16; o; o >>= 1) wmax = fmaxf(wmax, __shfl_xor_sync(0xffffffffu, wmax, o));
          const unsigned hit = __ballot_sync(0xffffffffu, mag == wmax);
          if (lane == __ffs(hit) - 1) {
            rkey[wid] = wmax;
            rt[wid] = tid;
            rlog[wid] = my_log | (signbit(c) ? (int)0x80000000 : 0);
          }
          __syncthreads();  // (1) pivot candidates
          float kw[kWarps];
#pragma unroll
          for (int w = 0; w < kWarps; ++w) kw[w] = rkey[w];
          float bk = kw[0];
#pragma unroll
          for (int w = 1; w < kWarps; ++w) bk = fmaxf(bk, kw[w]);
          int w0 = kWarps - 1;
#pragma unroll
          for (int w = kWarps - 2; w >= 0; --w) w0 = kw[w] == bk ? w : w0;
          const int r = rt[w0];
          const int lw = rlog[w0];
          const int lr = lw & 0x7FFFFFFF;
          const float cr = lw < 0 ? -bk : bk;
          if (!(bk > 0.0f)) {
            zero = true;
          } else {
            if (tid == r)
              my_log = k + 1;
            else if (my_log == k + 1)
              my_log = lr;
            const float piv = -cr;
            const bool live = my_log > k + 1;
            float dv = tmem_ld1(my_col0 + r);
            float u = 0.0f, v = 0.0f;
            if (live) {
#pragma unroll
              for (int p = 0; p < kTcNB; ++p)
                if (p < j) dv += myU[p] * Vf[r * kTcNB + p] - myV[p] * Uf[r * kTcNB + p];
              u = dv;
              v = c * (1.0f / piv);
            }
            myU[j] = u;
            myV[j] = v;
            Uf[tid * kTcNB + j] = u;
            Vf[tid * kTcNB + j] = v;
            // Both parts rounded to TF32 here: the tensor cores would truncate an unrounded
            // small part, a bias that accumulates over the pivots.
            const int o = opnd_off(tid, j);
            const float ub = tf32_big(u), vb = tf32_big(v);
            Ub[o] = ub;
            Us[o] = tf32_big(u - ub);
            Vb[o] = vb;
            Vs[o] = tf32_big(v - vb);
            if (my_log == k + 2) misc[0] = tid;
            if (tid == 0) pivs[k >> 1] = lr != k + 1 ? -piv : piv;
            swaps ^= lr != k + 1 ? 1 : 0;
          }
          __syncthreads();  // (2) panel column written, next column's owner known
        }
      }
      if (zero) break;
      if (n - (k0 + 2 * steps) < 2) break;  // nothing left to update
      // Rank-16 trailing update on the tensor cores.
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // Products of the parts: big x big, big x small, small x big.
        const uint32_t u2[2] = {smem_addr(Ub), smem_addr(Us)};
        const uint32_t v2[2] = {smem_addr(Vb), smem_addr(Vs)};
        constexpr int kPa[3] = {0, 0, 1}, kPb[3] = {0, 1, 0};
        const uint32_t lbo = 4096, sbo = 128;
        const uint32_t id_pos = tf32_idesc(NP, false), id_neg = tf32_idesc(NP, true);
        for (int mt = 0; mt < n_tiles; ++mt) {
          const uint32_t d = tmem + (uint32_t)(mt * NP);
          const uint32_t ro = (uint32_t)(mt * 128 / 8 * 128);  // first row group of the tile
#pragma unroll
          for (int t = 0; t < 3; ++t) {  // + U V^T
            mma_tf32(d, tc_desc(u2[kPa[t]] + ro, lbo, sbo), tc_desc(v2[kPb[t]], lbo, sbo), id_pos);
          }
#pragma unroll
          for (int t = 0; t < 3; ++t) {  // - V U^T
            mma_tf32(d, tc_desc(v2[kPa[t]] + ro, lbo, sbo), tc_desc(u2[kPb[t]], lbo, sbo), id_neg);
          }
        }
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_addr(bar))
            : "memory");
      }
      if (!tc_wait(bar, phase)) {
        if (tid == 0) atomicExch(err, 1);
        misc[1] = 1;
      }
      phase ^= 1u;
      __syncthreads();
      abort = misc[1] != 0;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (tid == 0) {
      float s = a.item_sign ? a.item_sign[item] : 1.0f;
      double la, pmax_all = 0.0, pmin_all = 1.0;
      if (isnan(s)) flag |= NH_FLAG_NONFINITE;
      if (abort) {
        s = NAN;
        la = NAN;
        flag |= NH_FLAG_NONFINITE;
      } else if (zero) {
        s = 0.0f;
        la = -INFINITY;
        flag |= NH_FLAG_ZERO_PIVOT;
      } else {
        double mant = 1.0;
        int expo = 0;
        double pmin = INFINITY, pmax = 0.0;
        for (int k = 0; k < n / 2; ++k) {
          const double pv = (double)pivs[k];
          if (pv < 0.0) s = -s;
          const double ap = fabs(pv);
          if (!isfinite(ap)) flag |= NH_FLAG_NONFINITE;
          pmin = fmin(pmin, ap);
          pmax = fmax(pmax, ap);
          int e;
          mant = frexp(mant * ap, &e);
          expo += e;
        }
        la = log(mant) + (double)expo * 0.6931471805599453;
        if (!isfinite(la)) flag |= NH_FLAG_NONFINITE;
        if (a.cond_tau > 0.0 && pmax > a.cond_tau * pmin) flag |= NH_FLAG_GROWTH;
        if (a.refine_tau > 0.0 && pmax > a.refine_tau * pmin) flag |= kFlagNeedRefine;
        pmax_all = pmax;
        pmin_all = pmin;
      }
      if (s == 0.0f) la = -INFINITY;
      a.sign[item] = s;
      a.logabs[item] = la;
      if (a.flags) a.flags[item] = flag | a.flag_or;
      if (a.ratio) a.ratio[item] = (zero || abort) ? INFINITY : (float)(pmax_all / pmin_all);
    }
    if (a.perm && !zero && !abort) {
      uint16_t* pr = a.perm + (size_t)item * perm_stride(n);
      if (tid < n) pr[my_log] = (uint16_t)tid;
      if (tid == 0) pr[n] = (uint16_t)swaps;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (wid == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTcCols)
                 : "memory");
}

size_t pf_tc_smem(int n) {
  const size_t tri = (size_t)n * (n - 1) / 2;
  const size_t region = std::max((tri + 31) & ~(size_t)31, (size_t)kTcOpFloats);
  const size_t need = sizeof(float) * (region + 128 + kWarps) + sizeof(int) * (2 * kWarps + 4) + 32;
  // At least 120 KB, so that two CTAs never share an SM: each allocates all 512 tensor-memory
  // columns, and a second CTA would stall in tcgen05.alloc until the first one exits.
  return std::max(need, (size_t)120 * 1024);
}

template <int D>
int launch_pf_tc(const PfArgs& a, int32_t* err, cudaStream_t st) {
  const size_t smem = pf_tc_smem(a.n);
  // The limit is raised once, to the largest size any n <= 256 needs.
  static const cudaError_t attr = cudaFuncSetAttribute(
      pfaffian_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
      (int)pf_tc_smem(kNumThreads));
  if (attr != cudaSuccess) return check_cuda(attr, "tensor-memory Pfaffian smem attribute");
  int grid = num_sms();
  if (grid > a.n_slots) grid = a.n_slots;
  if (grid <= 0) return NH_OK;
  ProfScope prof_scope(NH_K_PFAFFIAN_TC, st);
  pfaffian_tc_kernel<D><<<grid, kNumThreads, smem, st>>>(a, err);
  return check_launch("pfaffian_tc_kernel");
}
}  // namespace

bool pfaffian64_fits(int n) { return pf_smem<double, 2>(n) <= 227 * 1024; }

bool pfaffian_needs_scratch(int n, bool fp64) {
  return n > kNumThreads || (fp64 && !pfaffian64_fits(n));
}

size_t pfaffian_scratch_bytes(int n) {
  const size_t tri = ((size_t)n * (n - 1) / 2 + 3) & ~(size_t)3;
  return pfaffian_needs_scratch(n, true) ? (size_t)num_sms() * tri * sizeof(double) : 0;
}

int launch_pfaffian_from_F(const float* F, int n, int batch, const int32_t* list,
                           const int32_t* count, bool fp64, double cond_tau, int flag_or,
                           float* sign, double* logabs, int32_t* flags, void* tri,
                           cudaStream_t st, uint16_t* perm, double refine_tau) {
  if (n <= 0 || n % 2 || n > kBigThreads)
    return fail(NH_ERR_UNSUPPORTED, "slogpf: n=%d must be even and <= %d", n, kBigThreads);
  PfArgs a{};
  a.n = n;
  a.mode = 0;
  a.F = F;
  a.n_slots = batch;
  a.count_dev = count;
  a.count_mult = 1;
  a.slot_item = list;
  a.sign = sign;
  a.logabs = logabs;
  a.flags = flags;
  a.cond_tau = cond_tau;
  a.flag_or = flag_or;
  a.tri = tri;
  a.perm = perm;
  a.refine_tau = refine_tau;
  return fp64 ? launch_pf_pick<double, 16>(a, st) : launch_pf_pick<float, 16>(a, st);
}

// Wt (rows, d) to chunks of four a: Wc[(a / 4) rows + row].
__global__ void wt_chunk_kernel(const float4* __restrict__ Wt, int rows, int chunks,
                                float4* __restrict__ Wc) {
  const int step = gridDim.x * blockDim.x;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < rows * chunks; e += step) {
    const int c = e / rows, row = e - c * rows;
    Wc[e] = __ldg(Wt + (size_t)row * chunks + c);
  }
}

static int launch_wt_chunks(const float* Wt, int N, int d, float* Wc, cudaStream_t st) {
  const int total = 4 * N * (d / 4);
  ProfScope prof_scope(NH_K_PACK, st);
  wt_chunk_kernel<<<(total + 255) / 256, 256, 0, st>>>(reinterpret_cast<const float4*>(Wt), 4 * N,
                                                       d / 4, reinterpret_cast<float4*>(Wc));
  return check_launch("wt_chunk_kernel");
}

int launch_pfaffian_gather(const PfGatherArgs& g, cudaStream_t st) {
  if (g.n <= 0 || g.n % 2 || g.n > kBigThreads)
    return fail(NH_ERR_UNSUPPORTED, "amplitude: n=%d must be even and <= %d", g.n, kBigThreads);
  PfArgs a{};
  a.n = g.n;
  a.mode = 1;
  a.Y = g.Y;
  a.idx = g.idx;
  a.Wt = g.Wt;
  a.Lx = g.Lx;
  a.Ly = g.Ly;
  a.count_dev = g.count_dev;
  a.count_mult = g.count_mult;
  a.n_slots = g.n_slots;
  a.slot_item = g.slot_item;
  a.item_sign = g.item_sign;
  a.sign = g.sign;
  a.logabs = g.logabs;
  a.flags = g.flags;
  a.cond_tau = g.cond_tau;
  a.flag_or = g.flag_or;
  a.tri = g.tri;
  a.perm = g.perm;
  a.refine_tau = g.refine_tau;
  a.ratio = g.ratio;
  a.only_flag = g.only_flag;
  if (!g.fp64 && g.n > kNumThreads) {  // pf32_big_kernel gathers from the chunked table
    if (!g.wt_chunks) return fail(NH_ERR_INVALID, "amplitude: n=%d needs the chunked table", g.n);
    if (int rc = launch_wt_chunks(static_cast<const float*>(g.Wt), g.Lx * g.Ly, g.d, g.wt_chunks, st))
      return rc;
    a.Wc = reinterpret_cast<const float4*>(g.wt_chunks);
    a.mode = 3;
    a.tail_row = g.n;
  }
  return g.fp64 ? launch_pf_d<double>(a, g.d, st) : launch_pf_d<float>(a, g.d, st);
}

// Fused features + FP32 Pfaffian (mode 2): shared-memory layout choice and launch.
template <int NB, int D>
int launch_fused_nb(PfArgs a, cudaStream_t st) {
  const int n = a.n, N = a.Lx * a.Ly;
  const Pf32Layout L = pf32_layout(n, NB);
  size_t cnn_end = 0, act_end = 0;  // mode 3 (rows copied from global memory): no CNN phase
  if (a.mode == 2) act_end = cnn_phase_layout(N, a.C, a.Lx, &cnn_end);
  const size_t tri_bytes = L.us, y_bytes = 4 * (size_t)n * D;
  const size_t two_cta = 113 * 1024;
  // A: rows after the triangle and the activation planes, modes after the rows.
  const size_t yA = (std::max(act_end, tri_bytes) + 15) & ~(size_t)15;
  const size_t totA = std::max(std::max(L.end, cnn_end), yA + y_bytes + 4 * (size_t)n);
  // B: rows in the triangle's tail (rows from tail_row gathered through registers), modes at the
  // end of the panel (not yet in use).
  const size_t yB = (tri_bytes - y_bytes) & ~(size_t)15;
  const size_t idsB = L.pivs - 4 * (size_t)n;
  int tail = n;
  if (y_bytes < tri_bytes) {
    const size_t yf = yB / 4;
    tail = 0;
    while (tail < n && (size_t)tail * (tail - 1) / 2 + tail <= yf) ++tail;
  }
  const size_t tail_elems = (size_t)n * (n - 1) / 2 - (size_t)tail * (tail - 1) / 2;
  const size_t totB = std::max(L.end, cnn_end);
  const bool okB = y_bytes < tri_bytes && yB >= act_end && idsB >= act_end &&
                   tail_elems <= (size_t)kTailElems;
  size_t smem;
  if (totA <= two_cta || !okB || totB > two_cta) {
    smem = totA;
    a.y_off = (int)yA;
    a.idx_off = (int)(yA + y_bytes);
    a.tail_row = n;
  } else {
    smem = totB;
    a.y_off = (int)yB;
    a.idx_off = (int)idsB;
    a.tail_row = tail;
  }
  if (smem > 227 * 1024)
    return fail(NH_ERR_UNSUPPORTED, "fused amplitude: n=%d, N=%d needs %zu B of shared memory", n,
                N, smem);
  if (a.queue) {
    cudaError_t e = cudaMemsetAsync(a.queue, 0, sizeof(int32_t), st);
    if (e != cudaSuccess) return check_cuda(e, "fused amplitude: clear work counter");
  }
  return launch_pf32_nb<NB, D>(a, smem, a.mode == 2 ? NH_K_FUSED : NH_K_PFAFFIAN, st);
}

template <int D>
int launch_fused_d(const PfArgs& a, cudaStream_t st) {
  return a.n <= kPf32NB8MaxN ? launch_fused_nb<8, D>(a, st) : launch_fused_nb<4, D>(a, st);
}

int launch_pfaffian_tc(const PfGatherArgs& g, int mode, const float* F, int32_t* err,
                       cudaStream_t st) {
  if (g.n <= 0 || g.n % 2 || g.n > kNumThreads)
    return fail(NH_ERR_UNSUPPORTED, "tensor-memory Pfaffian: n=%d must be even and <= %d", g.n,
                kNumThreads);
  PfArgs a{};
  a.n = g.n;
  a.mode = mode;
  a.F = F;
  a.Y = g.Y;
  a.idx = g.idx;
  a.Wt = g.Wt;
  a.Lx = g.Lx;
  a.Ly = g.Ly;
  a.count_dev = g.count_dev;
  a.count_mult = g.count_mult;
  a.n_slots = g.n_slots;
  a.slot_item = g.slot_item;
  a.item_sign = g.item_sign;
  a.sign = g.sign;
  a.logabs = g.logabs;
  a.flags = g.flags;
  a.cond_tau = g.cond_tau;
  a.flag_or = g.flag_or;
  a.perm = g.perm;
  a.refine_tau = g.refine_tau;
  a.ratio = g.ratio;
  switch (mode == 0 ? 16 : g.d) {
    case 8: return launch_pf_tc<8>(a, err, st);
    case 16: return launch_pf_tc<16>(a, err, st);
    case 32: return launch_pf_tc<32>(a, err, st);
    default: return fail(NH_ERR_UNSUPPORTED, "tensor-memory Pfaffian: d=%d", g.d);
  }
}

template <int D>
int launch_pairing_smem(const float* Y, const int32_t* idx, const float* Wt, int Lx, int Ly, int n,
                        int batch, float* F, size_t smem, cudaStream_t st) {
  static size_t configured = 0;
  if (smem > 48 * 1024 && smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(pairing_smem_kernel<D>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return check_cuda(e, "pairing smem attribute");
    configured = smem;
  }
  int grid = num_sms() * (smem <= 113 * 1024 ? 2 : 1);
  if (grid > batch) grid = batch;
  ProfScope prof_scope(NH_K_PAIRING, st);
  pairing_smem_kernel<D><<<grid, kNumThreads, smem, st>>>(Y, idx, Wt, Lx, Ly, n, batch, F);
  return check_launch("pairing_smem_kernel");
}

bool fused_supported(const nh_backflow_params& p) {
  const int n = p.n_up + p.n_dn, N = p.Lx * p.Ly, d = p.channels / 2;
  return p.net == NH_NET_CNN && n <= kNumThreads && n % 2 == 0 && N % 2 == 0 &&
         p.channels % 16 == 0 && p.channels <= 64 && (d == 8 || d == 16 || d == 32);
}

bool staged_supported(const PfGatherArgs& g) {
  return !g.fp64 && g.n <= kNumThreads && g.n % 2 == 0 && g.d % 4 == 0 && g.d <= 32 && !g.tri &&
         g.wt_chunks;
}

int launch_pfaffian_staged(const PfGatherArgs& g, cudaStream_t st) {
  if (int rc = launch_wt_chunks(static_cast<const float*>(g.Wt), g.Lx * g.Ly, g.d, g.wt_chunks, st))
    return rc;
  PfArgs a{};
  a.Wc = reinterpret_cast<const float4*>(g.wt_chunks);
  a.n = g.n;
  a.mode = 3;
  a.Y = g.Y;
  a.idx = g.idx;
  a.Wt = g.Wt;
  a.Lx = g.Lx;
  a.Ly = g.Ly;
  a.count_dev = g.count_dev;
  a.count_mult = g.count_mult;
  a.n_slots = g.n_slots;
  a.slot_item = g.slot_item;
  a.item_sign = g.item_sign;
  a.sign = g.sign;
  a.logabs = g.logabs;
  a.flags = g.flags;
  a.cond_tau = g.cond_tau;
  a.flag_or = g.flag_or;
  a.perm = g.perm;
  a.refine_tau = g.refine_tau;
  a.ratio = g.ratio;
  switch (g.d) {
    case 8: return launch_fused_d<8>(a, st);
    case 16: return launch_fused_d<16>(a, st);
    case 32: return launch_fused_d<32>(a, st);
    default: return fail(NH_ERR_UNSUPPORTED, "staged Pfaffian: d=%d", g.d);
  }
}

int launch_pfaffian_fused(const FusedLaunch& f, cudaStream_t st) {
  const nh_backflow_params& p = *f.p;
  if (!fused_supported(p)) return fail(NH_ERR_UNSUPPORTED, "fused amplitude: unsupported network");
  if (int rc = launch_wt_chunks(p.Wt, p.Lx * p.Ly, p.channels / 2, f.wt_chunks, st)) return rc;
  PfArgs a{};
  a.Wc = reinterpret_cast<const float4*>(f.wt_chunks);
  a.n = p.n_up + p.n_dn;
  a.mode = 2;
  a.Wt = p.Wt;
  a.Lx = p.Lx;
  a.Ly = p.Ly;
  a.count_dev = f.cl.n_cfg_dev;
  a.count_mult = f.cl.G;
  a.n_slots = f.cl.n_cfg * f.cl.G;
  a.sign = f.sign;
  a.logabs = f.logabs;
  a.flags = f.flags;
  a.cond_tau = p.cond_tau;
  a.perm = f.perm;
  a.refine_tau = p.refine_tau;
  a.ratio = f.ratio;
  a.cl = f.cl;
  a.cnn_w = p.conv_w_packed;
  a.cnn_b = p.conv_b;
  a.C = p.channels;
  a.layers = p.layers;
  a.item_sign_out = f.item_sign;
  a.queue = f.queue;
  switch (p.channels / 2) {
    case 8: return launch_fused_d<8>(a, st);
    case 16: return launch_fused_d<16>(a, st);
    case 32: return launch_fused_d<32>(a, st);
    default: return fail(NH_ERR_UNSUPPORTED, "fused amplitude: d=%d", p.channels / 2);
  }
}

int launch_pairing(const float* Y, const int32_t* idx, const float* Wt, int Lx, int Ly, int d,
                   int n, int batch, float* F, cudaStream_t st) {
  if (batch <= 0) return NH_OK;
  const size_t smem = pairing_smem_bytes(Lx * Ly, n, d);
  if (smem <= 227 * 1024 && Lx < 256 && Ly < 256) {
    switch (d) {
      case 8: return launch_pairing_smem<8>(Y, idx, Wt, Lx, Ly, n, batch, F, smem, st);
      case 16: return launch_pairing_smem<16>(Y, idx, Wt, Lx, Ly, n, batch, F, smem, st);
      case 32: return launch_pairing_smem<32>(Y, idx, Wt, Lx, Ly, n, batch, F, smem, st);
      default: break;
    }
  }
  int grid = num_sms() * 4;
  if (grid > batch) grid = batch;
  ProfScope prof_scope(NH_K_PAIRING, st);
  switch (d) {
    case 8: pairing_kernel<8><<<grid, kNumThreads, 0, st>>>(Y, idx, Wt, Lx, Ly, n, batch, F); break;
    case 16: pairing_kernel<16><<<grid, kNumThreads, 0, st>>>(Y, idx, Wt, Lx, Ly, n, batch, F); break;
    case 32: pairing_kernel<32><<<grid, kNumThreads, 0, st>>>(Y, idx, Wt, Lx, Ly, n, batch, F); break;
    default: return fail(NH_ERR_UNSUPPORTED, "pairing_occ: d=%d (8, 16 or 32)", d);
  }
  return check_launch("pairing_kernel");
}

int launch_combine(const float* sg, const double* la, const int32_t* fl, int G, int n_cfg,
                   const int32_t* n_cfg_dev, float* sign, double* logabs, int32_t* flags,
                   double cancel_tau, const int32_t* err, cudaStream_t st) {
  if (n_cfg <= 0) return NH_OK;
  int grid = (n_cfg + 255) / 256;
  ProfScope prof_scope(NH_K_COMBINE, st);
  combine_kernel<<<grid, 256, 0, st>>>(sg, la, fl, G, n_cfg, n_cfg_dev, sign, logabs, flags,
                                       G > 1 ? cancel_tau : 0.0, err);
  return check_launch("combine_kernel");
}

int launch_image_mark(const float* sg, const double* la, int32_t* fl, const float* ratio, int G,
                      int n_cfg, const int32_t* n_cfg_dev, double cancel_tau, double cond_tau,
                      bool weighted, cudaStream_t st) {
  weighted = weighted && ratio;
  if (n_cfg <= 0 || G <= 1 || (cancel_tau <= 0.0 && !weighted)) return NH_OK;
  int grid = (n_cfg + 255) / 256;
  ProfScope prof_scope(NH_K_COMBINE, st);
  image_mark_kernel<<<grid, 256, 0, st>>>(sg, la, fl, ratio, G, n_cfg, n_cfg_dev, cancel_tau,
                                          cond_tau, weighted);
  return check_launch("image_mark_kernel");
}

int launch_flagged(const int32_t* flags, int n_items, const int32_t* count_dev, int count_mult,
                   int32_t* list, int32_t* count, cudaStream_t st, int set_mask, int clear_mask) {
  ProfScope prof_scope(NH_K_FLAGGED, st);
  flagged_kernel<<<1, 1024, 0, st>>>(flags, n_items, count_dev, count_mult, list, count, set_mask,
                                     clear_mask);
  return check_launch("flagged_kernel");
}

}  // namespace nh
