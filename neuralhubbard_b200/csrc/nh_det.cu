// BCS-backflow amplitude: sign and log|det| of the occupied up x down pairing block
// (code/backflow/models.py:214-302, code/backflow/bcs_kernel.py:1-70),
//
//   F[p, q] = sum_a Yu[p, a] Wt_ud[site_p - site_q, a] Yd[q, a] + delta_d fd(site_p - site_q),
//   psi(s)  = det F (-1)^(n_up (n_up - 1) / 2) x the item sign of the image,
//
// with Wt_ud = block 1 (ud) of the (4, N, d) table of nh_build_wtilde and fd the
// nearest-neighbour d-wave form factor (-1 on x bonds, +1 on y bonds, code/backflow/models.py:
// 80-82).  One matrix per 512-thread CTA, held in registers: thread (warp w, lane c) owns rows
// w + 16 t and columns c + 32 u.  Each thread gathers its own elements: the Wt_ud table sits in
// shared memory in 16-byte chunks [a][displacement] (staged once per CTA), the features in swizzled
// rows, a column's kept in registers (scalar loads of unpadded rows were 16-way bank conflicts:
// 145K of 329K cycles per FP32 block at n_up = 112, 314K of 525K in FP64).  Then an LU elimination
// with implicit partial pivoting runs on the registers: per step each warp gathers column k of its
// rows onto its lanes by shuffles, takes its largest unused entry with two 32-bit warp reductions
// and stores that row and its key as its candidate in shared memory; after the step's one barrier
// every warp reduces the 16 keys, reads the winning candidate as the pivot row, and every unused
// row takes its rank-1 update over the columns not yet eliminated.  det F = parity(pivot order) x
// prod of the pivots; the parity is counted as inversions by all threads, the log-sum of the pivots
// accumulated in FP64 as mantissa and exponent by one warp.
//
// Blocks of up to 128 rows in FP32 need 64 registers per thread, so two CTAs share an SM.
#include <math.h>

#include "nh_common.cuh"

namespace nh {
namespace {

constexpr int kDetThreads = 512;

struct DetArgs {
  const void* Y;       // (slots, n, d): rows [0, nh) the up modes, [nh, 2 nh) the down modes
  const int32_t* idx;  // (slots, n)
  const void* Wt;      // (4, N, d), block 1 read
  int Lx, Ly, nh;
  double delta_d;
  const int32_t* count_dev;  // device work count (times count_mult) or null
  int count_mult;
  int n_slots;
  const int32_t* slot_item;  // slot -> item, null: identity
  const float* item_sign;
  float* sign;
  double* logabs;
  int32_t* flags;
  float* ratio;  // (items,) pivot ratio, or null
  double cond_tau;
  int flag_or;
};

__device__ __forceinline__ unsigned long long det_key(float mag, int row) {
  return ((unsigned long long)__float_as_uint(mag) << 32) | (unsigned)(0x7FFFFFFF - row);
}

__device__ __forceinline__ float key_mag(float x) { return fabsf(x); }
__device__ __forceinline__ float key_mag(double x) { return __double2float_ru(fabs(x)); }

template <typename T>
struct DetVec;
template <>
struct DetVec<float> {
  using V = float4;
};
template <>
struct DetVec<double> {
  using V = double2;
};

template <typename T, int TC>
__global__ void __launch_bounds__(kDetThreads, sizeof(T) == 4 && TC <= 4 ? 2 : 1)
    det_kernel(DetArgs a) {
  constexpr int TR = 2 * TC, NP = 32 * TC;
  constexpr int D = 16, E = 16 / sizeof(T), K = D / E;  // E values per 16-byte chunk, K chunks a row
  using V = typename DetVec<T>::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nh = a.nh, n = 2 * nh, N = a.Lx * a.Ly, Lx = a.Lx, Ly = a.Ly;
  T* ys = reinterpret_cast<T*>(smem_raw);          // (n, D), chunk-swizzled rows (swz_index)
  V* wsm = reinterpret_cast<V*>(ys + (size_t)n * D);  // [K][N] chunks of Wt_ud
  T* colbuf = reinterpret_cast<T*>(wsm + (size_t)K * N);  // [2][NP]
  T* cand = colbuf + 2 * NP;                       // [2][16][NP] each warp's best row of the step
  T* pivs = cand + 32 * NP;                        // [NP]
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(pivs + NP);  // [2][16]
  int* info = reinterpret_cast<int*>(keys + 32);   // (n) spin << 16 | x << 8 | y
  int* rho = info + n;                             // [NP] pivot row of step k
  int* inv_s = rho + NP;                           // [16] inversions of the warps' rows, mod 2
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T* Yb = static_cast<const T*>(a.Y);
  const T* Wud = static_cast<const T*>(a.Wt) + (size_t)N * D;
  const int n_work = a.count_dev ? (*a.count_dev) * a.count_mult : a.n_slots;
  if ((int)blockIdx.x < n_work)
    for (int e = threadIdx.x; e < N * D; e += kDetThreads) {  // scalar: any alignment of the table
      const int row = e / D, c = e - row * D;
      reinterpret_cast<T*>(wsm)[((c / E) * N + row) * E + c % E] = __ldg(Wud + e);
    }

  for (int slot_i = blockIdx.x; slot_i < n_work; slot_i += gridDim.x) {
    const int item = a.slot_item ? a.slot_item[slot_i] : slot_i;
    const V* Yi = reinterpret_cast<const V*>(Yb + (size_t)slot_i * n * D);
    const int32_t* ii = a.idx + (size_t)slot_i * n;
    __syncthreads();  // the previous item's readers are done
    for (int e = threadIdx.x; e < n * K; e += kDetThreads) {
      const int row = e / K;
      *reinterpret_cast<V*>(ys + swz_index<T, D>(row, (e - row * K) * E)) = Yi[e];
    }
    for (int p = threadIdx.x; p < n; p += kDetThreads) {
      int m = __ldg(ii + p);
      if ((unsigned)m >= (unsigned)(2 * N)) m = 0;
      const int sp = m >= N ? 1 : 0, site = m - sp * N, x = site / Ly;
      info[p] = (sp << 16) | (x << 8) | (site - x * Ly);
    }
    __syncthreads();
    // Gather: element (I, J) = F[up row I][down row J].
    T A[TR][TC];
#pragma unroll
    for (int u = 0; u < TC; ++u) {
      const int J = lane + 32 * u, jq = nh + (J < nh ? J : 0);
      T yq[D];
#pragma unroll
      for (int c = 0; c < D; c += E)
        *reinterpret_cast<V*>(yq + c) = *reinterpret_cast<const V*>(ys + swz_index<T, D>(jq, c));
      const int iq = info[jq];
#pragma unroll
      for (int t = 0; t < TR; ++t) {
        const int I = warp + 16 * t;
        T v = (I == J) ? T(1) : T(0);
        if (I < nh && J < nh) {
          const int ip = info[I];
          int dx = ((ip >> 8) & 0xFF) - ((iq >> 8) & 0xFF), dy = (ip & 0xFF) - (iq & 0xFF);
          dx += dx < 0 ? Lx : 0;
          dy += dy < 0 ? Ly : 0;
          const V* w = wsm + dx * Ly + dy;
          T acc = T(0);
#pragma unroll
          for (int c = 0; c < K; ++c) {
            T yp[E], wv[E];
            *reinterpret_cast<V*>(yp) = *reinterpret_cast<const V*>(ys + swz_index<T, D>(I, c * E));
            *reinterpret_cast<V*>(wv) = w[c * N];
#pragma unroll
            for (int x = 0; x < E; ++x) acc += (yp[x] * yq[c * E + x]) * wv[x];
          }
          const int mx = min(dx, Lx - dx), my = min(dy, Ly - dy);
          const T fd = (mx == 1 && my == 0) ? T(-1) : ((mx == 0 && my == 1) ? T(1) : T(0));
          v = acc + T(a.delta_d) * fd;
        }
        A[t][u] = v;
      }
    }
    unsigned used = 0;
#pragma unroll
    for (int t = 0; t < TR; ++t)
      if (warp + 16 * t >= nh) used |= 1u << t;
    int bad = 0;
    // One barrier per step: the column, key and candidate buffers alternate by parity (a warp
    // writes step k + 2's copy only after every warp has passed step k + 1's barrier, so after
    // every read of step k's).
#pragma unroll
    for (int uk = 0; uk < TC; ++uk) {
#pragma unroll 1
      for (int lk = 0; lk < 32; ++lk) {
        const int k = uk * 32 + lk;
        if (k >= nh || bad) break;  // uniform
        const int par = k & 1;
        {
          // Column k of this warp's rows, spread over the lanes (lane t takes row warp + 16 t)
          // so that the pivot proposal runs on TR lanes instead of the one owning the column.
          T cv = T(0);
#pragma unroll
          for (int t = 0; t < TR; ++t) {
            const T v = __shfl_sync(0xffffffffu, A[t][uk], lk);
            if (lane == t) cv = v;
          }
          unsigned long long key = 0ull;
          if (lane < TR) {
            colbuf[par * NP + warp + 16 * lane] = cv;
            if (!((used >> lane) & 1u)) key = det_key(key_mag(cv), warp + 16 * lane);
          }
          // 64-bit warp maximum as two 32-bit reductions: the magnitude bits, then the row
          // tie-break among the lanes holding that magnitude.
          const unsigned hi = (unsigned)(key >> 32);
          const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
          const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)key : 0u);
          key = ((unsigned long long)mh << 32) | ml;
          if (key) {  // this warp's best row goes to its candidate slot
            const int tl = (0x7FFFFFFF - (int)ml) >> 4;
            T* cw = cand + (size_t)(par * 16 + warp) * NP;
#pragma unroll
            for (int t = 0; t < TR; ++t)
              if (t == tl) {
#pragma unroll
                for (int u = uk; u < TC; ++u) cw[lane + 32 * u] = A[t][u];
              }
          }
          if (lane == 0) keys[16 * par + warp] = key;
        }
        __syncthreads();
        const unsigned long long kw = keys[16 * par + (lane & 15)];
        const unsigned wh = __reduce_max_sync(0xffffffffu, (unsigned)(kw >> 32));
        const unsigned wl =
            __reduce_max_sync(0xffffffffu, (unsigned)(kw >> 32) == wh ? (unsigned)kw : 0u);
        const int p = 0x7FFFFFFF - (int)wl;
        const float mag = __uint_as_float(wh);
        if ((wh | wl) == 0u || !(mag > 0.0f && mag <= 3.0e38f)) {
          bad = ((wh | wl) == 0u || mag == 0.0f) ? NH_FLAG_ZERO_PIVOT : NH_FLAG_NONFINITE;
          break;
        }
        if (warp == (p & 15)) used |= 1u << (p >> 4);
        const T piv = colbuf[par * NP + p];
        if (threadIdx.x == 0) {
          rho[k] = p;
          pivs[k] = piv;
        }
        const T* prow = cand + (size_t)(par * 16 + (p & 15)) * NP;
        const T inv = T(1) / piv;
        T r[TC];
#pragma unroll
        for (int u = uk; u < TC; ++u) r[u] = prow[lane + 32 * u] * inv;
#pragma unroll
        for (int t = 0; t < TR; ++t) {
          if ((used >> t) & 1u) continue;  // eliminated rows keep their values (never read)
          const T f = colbuf[par * NP + warp + 16 * t];
#pragma unroll
          for (int u = uk; u < TC; ++u) A[t][u] = fma(-f, r[u], A[t][u]);
        }
      }
    }
    __syncthreads();  // every step's rho and pivs are written
    // Parity of the pivot order: inversions counted by the first rows' threads.
    {
      const int i = threadIdx.x;
      int cnt = 0;
      if (!bad && warp < TC) {
        const int ri = i < nh ? rho[i] : 0;
        for (int j = 0; j < nh; ++j) cnt += (j > i && rho[j] < ri) ? 1 : 0;
        if (i >= nh) cnt = 0;
      }
      const unsigned odd = __ballot_sync(0xffffffffu, cnt & 1);
      if (lane == 0) inv_s[warp] = __popc(odd) & 1;
    }
    __syncthreads();
    if (warp == 0) {
      int flag = bad, par = (lane == 0 ? (nh * (nh - 1) / 2) & 1 : 0), expo = 0;  // (-1)^(n_up ...)
      if (lane < 16) par ^= inv_s[lane];
      double mant = 1.0, pmin = INFINITY, pmax = 0.0;
      if (!bad)
        for (int k = lane; k < nh; k += 32) {
          const double pv = (double)pivs[k];
          if (pv < 0.0) par ^= 1;
          const double ap = fabs(pv);
          if (!isfinite(ap)) flag |= NH_FLAG_NONFINITE;
          pmin = fmin(pmin, ap);
          pmax = fmax(pmax, ap);
          int e;
          mant = frexp(mant * ap, &e);
          expo += e;
        }
#pragma unroll
      for (int o = 16; o; o >>= 1) {  // 32 mantissas in [1/2, 1]: no underflow
        mant *= __shfl_xor_sync(0xffffffffu, mant, o);
        expo += __shfl_xor_sync(0xffffffffu, expo, o);
        par ^= __shfl_xor_sync(0xffffffffu, par, o);
        flag |= __shfl_xor_sync(0xffffffffu, flag, o);
        pmin = fmin(pmin, __shfl_xor_sync(0xffffffffu, pmin, o));
        pmax = fmax(pmax, __shfl_xor_sync(0xffffffffu, pmax, o));
      }
      if (lane == 0) {
        float s = a.item_sign ? a.item_sign[item] : 1.0f;
        double la = -INFINITY, ratio = INFINITY;
        if (isnan(s)) flag |= NH_FLAG_NONFINITE;
        if (bad) {
          s = 0.0f;
        } else {
          if (par) s = -s;
          la = log(mant) + (double)expo * 0.6931471805599453;
          if (!isfinite(la)) flag |= NH_FLAG_NONFINITE;
          ratio = pmax / pmin;
          if (a.cond_tau > 0.0 && pmax > a.cond_tau * pmin) flag |= NH_FLAG_GROWTH;
        }
        if (s == 0.0f) la = -INFINITY;
        a.sign[item] = s;
        a.logabs[item] = la;
        if (a.flags) a.flags[item] = flag | a.flag_or;
        if (a.ratio) a.ratio[item] = (float)ratio;
      }
    }
  }
}

template <typename T, int TC>
size_t det_smem(int nh, int N) {
  constexpr int NP = 32 * TC;
  const size_t n = 2 * (size_t)nh;
  return sizeof(T) * ((n + N) * 16 + 35 * NP) + 32 * sizeof(unsigned long long) +
         sizeof(int) * (n + NP + 16);
}

template <typename T, int TC>
int launch_det_t(const DetArgs& a, cudaStream_t st) {
  const size_t smem = det_smem<T, TC>(a.nh, a.Lx * a.Ly);
  static const cudaError_t attr = cudaFuncSetAttribute(
      det_kernel<T, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (attr != cudaSuccess) return check_cuda(attr, "det smem attribute");
  if (smem > 227 * 1024)
    return fail(NH_ERR_UNSUPPORTED, "BCS determinant: n_up = %d, N = %d", a.nh, a.Lx * a.Ly);
  const int slots = a.n_slots;
  if (slots <= 0) return NH_OK;
  int grid = num_sms() * (sizeof(T) == 4 && TC <= 4 && smem <= 113 * 1024 ? 2 : 1);
  if (grid > slots) grid = slots;
  ProfScope prof_scope(sizeof(T) == 8 ? NH_K_DET64 : NH_K_DET, st);
  det_kernel<T, TC><<<grid, kDetThreads, smem, st>>>(a);
  return check_launch(sizeof(T) == 8 ? "det_kernel<double>" : "det_kernel<float>");
}

}  // namespace

bool det_supported(int nh, int d, bool fp64) {
  return d == 16 && nh >= 1 && nh <= (fp64 ? kDetMaxNh64 : kDetMaxNh);
}

int launch_det(const DetLaunch& q, cudaStream_t st) {
  if (!det_supported(q.nh, q.d, q.fp64))
    return fail(NH_ERR_UNSUPPORTED, "BCS determinant: n_up %d (<= %d FP32, %d FP64), d %d (16)",
                q.nh, kDetMaxNh, kDetMaxNh64, q.d);
  DetArgs a{q.Y, q.idx, q.Wt, q.Lx, q.Ly, q.nh, q.delta_d, q.count_dev, q.count_mult, q.n_slots,
            q.slot_item, q.item_sign, q.sign, q.logabs, q.flags, q.ratio, q.cond_tau,
            q.flag_or};
  const int tc = (q.nh + 31) / 32;
  if (q.fp64) {
    switch (tc) {
      case 1: return launch_det_t<double, 1>(a, st);
      case 2: return launch_det_t<double, 2>(a, st);
      case 3: return launch_det_t<double, 3>(a, st);
      default: return launch_det_t<double, 4>(a, st);
    }
  }
  switch (tc) {
    case 1: return launch_det_t<float, 1>(a, st);
    case 2: return launch_det_t<float, 2>(a, st);
    case 3: return launch_det_t<float, 3>(a, st);
    case 4: return launch_det_t<float, 4>(a, st);
    case 5: return launch_det_t<float, 5>(a, st);
    case 6: return launch_det_t<float, 6>(a, st);
    default: return launch_det_t<float, 7>(a, st);
  }
}

}  // namespace nh
