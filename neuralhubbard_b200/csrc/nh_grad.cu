// Backward of the Pfaffian-backflow amplitude: the per-sample Jacobian
// O_k(s) = d log|psi_P(s)| / d theta_k that SR / AdamSR training consumes
// (code/train_pfaffian_16x16_tpm02.py:100-101), and its two operator-level pieces.
//
// * adjoint_kernel: the cotangent of fermix.slogpf (code/backflow/models.py:210),
//   G = d log|pf F| / dF = 1/2 F^{-T}, from an in-register Gauss-Jordan inverse of F with implicit
//   row pivoting, eight pivot steps at a time (one matrix per 512-thread CTA; thread (warp w,
//   lane c) holds rows w + 16 t and columns c + 32 u).  A per-item scale multiplies G (the image
//   weight of the projection).
// * pairing_vjp_kernel: the custom VJP of the occupied gather (pf_kernel.py:193-320,354-365):
//   dY[p, a] = sum_q (G - G^T)[p, q] Wt[blk(p, q), r(p, q), a] Y[q, a] and
//   dWt[blk, r, a] = sum over the pairs (p, q) with that block and displacement of
//   G[p, q] Y[p, a] Y[q, a].  With several images per sample their dWt are summed in registers and
//   chained through build_wtilde's backward (pf_kernel.py:107-124) into the W and theta columns.
// * cnn_vjp_kernel: the backflow CNN's backward for every image of a sample: the forward is
//   recomputed with the pre-activations kept in shared memory, the features' cotangent is the
//   image's dY scattered to its occupied modes (pf_kernel.py:395), and the convolution weight and
//   bias cotangents of all images are summed into the sample's Jacobian row.
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "nh_cnn_item.cuh"
#include "nh_common.cuh"

namespace nh {
namespace {

constexpr int kAdjThreads = 512;  // 16 row groups (warps) x 32 column groups (lanes)
constexpr int kVjpThreads = 512;

// Weight of item (c, g) in d log|psi_P(c)|: sg_g exp(la_g) / sum_h sg_h exp(la_h) (sg, la: the
// item's signed log-Pfaffian with its fermionic signs folded in); 0 when the sum vanishes.
__device__ double image_weight(const float* sg, const double* la, int item, int G) {
  if (G == 1) return sg[item] != 0.0f ? 1.0 : 0.0;
  const int c = item / G;
  double m = -INFINITY;
  for (int h = 0; h < G; ++h)
    if (sg[c * G + h] != 0.0f && la[c * G + h] > m) m = la[c * G + h];
  if (!(m > -INFINITY)) return 0.0;
  double tot = 0.0;
  for (int h = 0; h < G; ++h)
    if (sg[c * G + h] != 0.0f) tot += (double)sg[c * G + h] * exp(la[c * G + h] - m);
  if (tot == 0.0 || !isfinite(tot) || sg[item] == 0.0f) return 0.0;
  return (double)sg[item] * exp(la[item] - m) / tot;
}

struct AdjArgs {
  const float* F;  // (batch, n, n)
  float* G;        // (batch, n, n), may alias F
  int n, batch;
  const float* pf_sign;     // when set: scale G by the image weight (G = n_img images per sample)
  const double* pf_logabs;
  int n_img;
  int32_t* flags;           // (batch,) or null: NH_FLAG_ZERO_PIVOT / NH_FLAG_NONFINITE
};

// Blocks of kAdjBlock pivot steps.  The buffers of a block and the output tile share one region.
constexpr int kAdjBlock = 8;

template <int TC>
struct AdjLayout {  // float offsets
  static constexpr int TR = 2 * TC, NP = 32 * TC, kFs = ((TR + 3) & ~3) + 4;
  static constexpr int panel = 0, kPs = NP + 4;              // [8][kPs]: the block's columns
  static constexpr int rows = panel + kAdjBlock * kPs;       // [8][NP]: its pivot rows
  static constexpr int scaled = rows + kAdjBlock * NP;       // [8][NP]: row k at step k, / pivot
  static constexpr int mult = scaled + kAdjBlock * NP;       // [8][16][kFs]: -A[i][k] at step k
  static constexpr int cand = mult + kAdjBlock * 16 * kFs;   // [2][TC][8]: candidates' columns
  static constexpr int cross = cand + 2 * TC * kAdjBlock;    // [8][8]: mult of the pivot rows
  static constexpr int mags = cross + kAdjBlock * kAdjBlock;  // [2][8]: their pivots' magnitudes
  static constexpr int total = mags + 16;
  __host__ __device__ static constexpr size_t region(int n) {
    return (size_t)n * (n + 1) > (size_t)total ? (((size_t)n * (n + 1) + 3) & ~(size_t)3) : total;
  }
};

// f(t) for a t in [LO, HI) that is the same in all lanes, as a constant: branches by halves, so that
// an array indexed with it stays in registers.
template <int LO, int HI, typename Fn>
__device__ __forceinline__ void with_row(int t, Fn&& f) {
  if constexpr (HI - LO == 1) {
    f(std::integral_constant<int, LO>{});
  } else {
    constexpr int MID = (LO + HI) / 2;
    if (t < MID)
      with_row<LO, MID>(t, f);
    else
      with_row<MID, HI>(t, f);
  }
}

// Gauss-Jordan inverse in the registers of 512 threads, eight pivot steps at a time.  A step by
// itself is a chain (maximum of a column, pivot row, reciprocal, multipliers) ending in a barrier of
// all warps: 2260 cycles at n = 224, where its 98 products per thread take 390.  Here the chain runs
// on the block's eight columns alone, a row per thread on TC warps; then each thread of those warps
// takes one column of the eight pivot rows through the same steps, and all 512 threads apply the
// eight steps to their elements back to back, two rows per packed instruction.  Every element sees
// the operations of the step-by-step elimination in their order, so the result is bit for bit
// the same.  2048 matrices of n = 224: 2.88 ms (3.73 step by step).  A block of eight steps takes 15K
// cycles there: the chain 5.8K (two warp maxima and a barrier, 720 a step), the products 4.4K of
// 3.1K at the FMA rate, the rest moves columns and pivot rows between registers and shared memory.
template <int TC>
__global__ void __launch_bounds__(kAdjThreads, TC <= 4 ? 2 : 1) adjoint_kernel(AdjArgs a) {
  using L = AdjLayout<TC>;
  constexpr int TR = L::TR, NP = L::NP, KB = kAdjBlock;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = a.n, NS = n + 1;
  float* tile = reinterpret_cast<float*>(smem_raw);  // (n, n + 1): G before the coalesced copy
  float* panel = tile + L::panel;
  float* prows = tile + L::rows;
  float* scaled = tile + L::scaled;
  float* mult = tile + L::mult;
  float* cand = tile + L::cand;
  float* cross = tile + L::cross;
  unsigned* mags = reinterpret_cast<unsigned*>(tile + L::mags);
  int* rho = reinterpret_cast<int*>(tile + L::region(n));  // [NP] pivot row of step k
  int* rhoinv = rho + NP;                                  // [NP]
  float* inv_s = reinterpret_cast<float*>(rhoinv + NP);    // [8] 1 / pivot
  float* scale_s = inv_s + KB;
  int* bad_s = reinterpret_cast<int*>(scale_s + 1);
  int* kb_s = bad_s + 1;  // steps of the block before a bad pivot
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  for (int item = blockIdx.x; item < a.batch; item += gridDim.x) {
    const float* F = a.F + (size_t)item * n * n;
    // A[t][u]: rows warp + 32 t and warp + 32 t + 16, column lane + 32 u
    unsigned long long A[TC][TC];
#pragma unroll
    for (int t = 0; t < TC; ++t) {
      const int i0 = warp + 32 * t, i1 = i0 + 16;
#pragma unroll
      for (int u = 0; u < TC; ++u) {
        const int j = lane + 32 * u;
        const float lo = (i0 < n && j < n) ? __ldg(F + (size_t)i0 * n + j) : (i0 == j ? 1.0f : 0.0f);
        const float hi = (i1 < n && j < n) ? __ldg(F + (size_t)i1 * n + j) : (i1 == j ? 1.0f : 0.0f);
        A[t][u] = pack2(lo, hi);
      }
    }
    bool used = tid >= n;  // row tid is a pivot row already (or padding)
    if (tid == 0) {
      float sc = 0.5f;
      if (a.pf_sign) sc = (float)(0.5 * image_weight(a.pf_sign, a.pf_logabs, item, a.n_img));
      *scale_s = sc;
    }
    int bad = 0;
#pragma unroll 1
    for (int K = 0; K < n; K += KB) {
      const int uk = K >> 5, lk = K & 31;  // the block's columns: lanes lk .. lk + 7, index uk
      // The block's columns to shared memory.  A warp writes and, at the block's end, reads only
      // its own rows of it.
      if (lane >= lk && lane < lk + KB) {
        float* pc = panel + (lane - lk) * L::kPs + warp;
#pragma unroll
        for (int u = 0; u < TC; ++u)
          if (u == uk) {
#pragma unroll
            for (int t = 0; t < TC; ++t) {
              pc[32 * t] = lo2(A[t][u]);
              pc[32 * t + 16] = hi2(A[t][u]);
            }
          }
      }
      __syncthreads();
      // The chain: thread i < NP holds row i of the columns.
      if (warp < TC) {
        float v[KB];
#pragma unroll
        for (int c = 0; c < KB; ++c) v[c] = panel[c * L::kPs + tid];
        const int kb = min(KB, n - K);
        float* mrow = mult + (tid & 15) * L::kFs + (tid >> 4);
        // One body for all steps (eight copies of it run at the speed of the instruction fetch):
        // v[0] is the step's column, and each step moves the columns down by one.
        int done = 0;
#pragma unroll 1
        for (; done < kb; ++done) {
          const int par = done & 1;
          const float cv = v[0];
          const float own_inv = 1.0f / cv;  // every row's, beside the search
          // The warp's largest free row, the first of equals, goes to its candidate slot (|v| >= 0
          // orders like its bit pattern; a warp without a free row proposes 0, as a zero column).
          const unsigned mag = used ? 0u : __float_as_uint(fabsf(cv));
          const unsigned wmag = __reduce_max_sync(0xffffffffu, mag);
          const int wlane = __ffs(__ballot_sync(0xffffffffu, mag == wmag)) - 1;
          if (lane == wlane) {
            float4* cw = reinterpret_cast<float4*>(cand + (par * TC + warp) * KB);
            cw[0] = make_float4(own_inv, v[1] * own_inv, v[2] * own_inv, v[3] * own_inv);
            cw[1] = make_float4(v[4] * own_inv, v[5] * own_inv, v[6] * own_inv, v[7] * own_inv);
            mags[par * 8 + warp] = wmag;
          }
          mrow[done * 16 * L::kFs] = -cv;
          if (TC == 1)
            __syncwarp();
          else
            asm volatile("bar.sync 1, %0;" ::"n"(32 * TC) : "memory");
          const unsigned m = lane < TC ? mags[par * 8 + lane] : 0u;
          const unsigned best = __reduce_max_sync(0xffffffffu, m);
          const int wwarp = __ffs(__ballot_sync(0xffffffffu, m == best)) - 1;
          if (best == 0u || !(__uint_as_float(best) <= 3.0e38f)) {  // zero column, or non-finite
            bad = best == 0u ? NH_FLAG_ZERO_PIVOT : NH_FLAG_NONFINITE;
            break;  // uniform over the TC warps
          }
          const bool pivot = warp == wwarp && lane == wlane;
          const float4* cr = reinterpret_cast<const float4*>(cand + (par * TC + wwarp) * KB);
          const float4 ra = cr[0], rb = cr[1];
          const float r[KB] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
          if (pivot) {
            used = true;
            rho[K + done] = tid;
            inv_s[done] = own_inv;
          }
#pragma unroll
          for (int c = 1; c < KB; ++c) v[c - 1] = pivot ? r[c] : fmaf(-cv, r[c], v[c]);
          v[KB - 1] = pivot ? r[0] : -cv * r[0];
        }
#pragma unroll
        for (int c = 0; c < KB; ++c) panel[((c + done) & (KB - 1)) * L::kPs + tid] = v[c];
        if (tid == 0) {
          *kb_s = done;
          *bad_s = bad;
        }
      }
      __syncthreads();
      const int kb = *kb_s;
      bad = *bad_s;
      // The pivot rows to shared memory, and their multipliers of the block's steps side by side.
      const int pl = lane < kb ? rho[K + lane] : 0;  // lane m: pivot row m
      const unsigned mine = __ballot_sync(0xffffffffu, lane < kb && (pl & 15) == warp);
      for (unsigned left = mine; left; left &= left - 1) {
        const int m = __ffs(left) - 1, t = __shfl_sync(0xffffffffu, pl, m) >> 4;
        float* pr = prows + m * NP + lane;
        with_row<0, TR>(t, [&](auto tc) {
          constexpr int tt = decltype(tc)::value;
#pragma unroll
          for (int u = 0; u < TC; ++u) pr[32 * u] = tt & 1 ? hi2(A[tt / 2][u]) : lo2(A[tt / 2][u]);
        });
      }
      if (tid < KB * KB) {
        const int k = tid >> 3, m = (k + tid) & 7;  // in the order of the loop below
        if (k < kb && m < kb) {
          const int p = rho[K + m];
          cross[tid] = mult[(k * 16 + (p & 15)) * L::kFs + (p >> 4)];
        }
      }
      __syncthreads();
      if (warp < TC) {  // column tid of the pivot rows through the block's steps
        float x[KB];
#pragma unroll
        for (int m = 0; m < KB; ++m) x[m] = prows[m * NP + tid];
#pragma unroll 1
        for (int k = 0; k < kb; ++k) {  // x[0] is row k; each step moves the rows down by one
          const float r = x[0] * inv_s[k];
          const float4* cm = reinterpret_cast<const float4*>(cross + k * KB);
          const float4 ca = cm[0], cb = cm[1];
          const float f[KB] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
          scaled[k * NP + tid] = r;
#pragma unroll
          for (int m = 1; m < KB; ++m) x[m - 1] = fmaf(f[m], r, x[m]);
          x[KB - 1] = r;
        }
#pragma unroll
        for (int m = 0; m < KB; ++m) prows[((m + kb) & (KB - 1)) * NP + tid] = x[m];
      }
      __syncthreads();
      // Every element through the block's steps (the pivot rows and the block's columns too; they
      // are replaced below).
#pragma unroll 1
      for (int k = 0; k < kb; ++k) {
        const float* mk = mult + (k * 16 + warp) * L::kFs;
        const float* sk = scaled + k * NP + lane;
        unsigned long long r[TC];
#pragma unroll
        for (int u = 0; u < TC; ++u) r[u] = pack2(sk[32 * u], sk[32 * u]);
#pragma unroll
        for (int t = 0; t < TC; t += 2) {
          unsigned long long f0, f1 = 0;
          if (t + 1 < TC) {
            const ulonglong2 f = *reinterpret_cast<const ulonglong2*>(mk + 2 * t);
            f0 = f.x, f1 = f.y;
          } else {
            f0 = *reinterpret_cast<const unsigned long long*>(mk + 2 * t);
          }
#pragma unroll
          for (int u = 0; u < TC; ++u) fma2(A[t][u], f0, r[u]);
          if (t + 1 < TC) {
#pragma unroll
            for (int u = 0; u < TC; ++u) fma2(A[t + 1][u], f1, r[u]);
          }
        }
      }
      for (unsigned left = mine; left; left &= left - 1) {
        const int m = __ffs(left) - 1, t = __shfl_sync(0xffffffffu, pl, m) >> 4;
        const float* pr = prows + m * NP + lane;
        with_row<0, TR>(t, [&](auto tc) {
          constexpr int tt = decltype(tc)::value;
#pragma unroll
          for (int u = 0; u < TC; ++u) {
            const float y = pr[32 * u];
            A[tt / 2][u] = tt & 1 ? pack2(lo2(A[tt / 2][u]), y) : pack2(y, hi2(A[tt / 2][u]));
          }
        });
      }
      if (lane >= lk && lane < lk + KB) {
        const float* pc = panel + (lane - lk) * L::kPs + warp;
#pragma unroll
        for (int u = 0; u < TC; ++u)
          if (u == uk) {
#pragma unroll
            for (int t = 0; t < TC; ++t) A[t][u] = pack2(pc[32 * t], pc[32 * t + 16]);
          }
      }
      if (bad) break;  // uniform
      __syncwarp();    // the next block's columns go where other lanes have read
    }
    // The storage holds X = (P F)^{-1} with logical row k in physical row rho[k], so
    // F^{-1}[i][j] = A[rho[i]][rhoinv[j]] and G[p][q] = 1/2 F^{-1}[q][p]: element (I, J) of the
    // storage goes to G[rho[J]][rhoinv[I]].
    if (!bad)
      for (int k = tid; k < n; k += kAdjThreads) rhoinv[rho[k]] = k;
    __syncthreads();
    const float sc = bad ? 0.0f : *scale_s;
#pragma unroll
    for (int t = 0; t < TR; ++t) {
      const int I = warp + 16 * t;
#pragma unroll
      for (int u = 0; u < TC; ++u) {
        const int J = lane + 32 * u;
        if (I < n && J < n) {
          const int dr = bad ? J : rho[J], dc = bad ? I : rhoinv[I];
          tile[dr * NS + dc] = sc * (t & 1 ? hi2(A[t / 2][u]) : lo2(A[t / 2][u]));
        }
      }
    }
    __syncthreads();
    float* Gi = a.G + (size_t)item * n * n;
    for (int e = tid; e < n * n; e += kAdjThreads) {
      const int row = e / n;
      Gi[e] = tile[row * NS + (e - row * n)];
    }
    if (a.flags && tid == 0) a.flags[item] = bad;
    __syncthreads();
  }
}

template <int TC>
size_t adjoint_smem(int n) {
  return sizeof(float) * (AdjLayout<TC>::region(n) + kAdjBlock + 4) +
         sizeof(int) * 2 * AdjLayout<TC>::NP;
}

template <int TC>
int launch_adjoint_t(const AdjArgs& a, cudaStream_t st) {
  const size_t smem = adjoint_smem<TC>(a.n);
  if (smem > 227 * 1024) return fail(NH_ERR_UNSUPPORTED, "pfaffian adjoint: n = %d", a.n);
  static size_t configured = 0;
  if (smem > 48 * 1024 && smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(adjoint_kernel<TC>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return check_cuda(e, "adjoint smem attribute");
    configured = smem;
  }
  int grid = num_sms() * (smem <= 113 * 1024 ? 2 : 1);
  if (grid > a.batch) grid = a.batch;
  ProfScope prof_scope(NH_K_PF_ADJOINT, st);
  adjoint_kernel<TC><<<grid, kAdjThreads, smem, st>>>(a);
  return check_launch("adjoint_kernel");
}

// ------------------------------------------------------------------ pairing VJP
struct VjpArgs {
  const float* G;      // (items, n, n) cotangent of F
  const float* Y;      // (items, n, d)
  const int32_t* idx;  // (items, n)
  const float* Wt;     // (4, N, d)
  const float4* Wc;    // or null: the same table in chunks, Wc[(a / 4) 4 N + row]
  int Lx, Ly, n;
  int n_img;           // images per sample (items = samples * n_img)
  int samples;
  float* dY;           // (items, n, d) or null
  float* dWt;          // mode 0: (items, 4, N, d) per item
  // mode 1: the sample's W / theta cotangent (build_wtilde's backward of the images' summed dWt)
  // into jac[sample * ld + off_w ...], theta at off_w + 3 N d.
  float* jac;
  int64_t ld;
  int64_t off_w;
  float theta;
  int mode;
};

template <int D>
__global__ void __launch_bounds__(kVjpThreads, 1) pairing_vjp_kernel(VjpArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = a.n, N = a.Lx * a.Ly, Lx = a.Lx, Ly = a.Ly, NS = n + 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // Region 0: G (n, n + 1), later the summed dWt (4, N, D); then Y rows (swizzled), modes, inv.
  const size_t reg0 = ((size_t)n * NS > (size_t)4 * N * D ? (size_t)n * NS : (size_t)4 * N * D);
  float* gs = reinterpret_cast<float*>(smem_raw);
  float* ys = gs + ((reg0 + 3) & ~(size_t)3);   // (n, D), 16-byte chunks swizzled
  int* modes = reinterpret_cast<int*>(ys + (size_t)n * D);  // (spin << 16) | (x << 8) | y
  int* inv = modes + n;                                     // (2N) mode -> row or -1
  // dWt ownership: task = pass * kVjpThreads + tid -> (pair, 16-byte chunk c of a); pair ->
  // (sq, r).  A thread keeps the same chunk in every pass (kVjpThreads is a multiple of kCh)
  // and accumulates float4 partial sums per pass and spin of p.
  constexpr int kCh = D / 4;  // also the most passes: 2 N kCh <= kVjpThreads kCh
  const int c_own = tid % kCh;
  int p_base[kCh], p_rx[kCh], p_ry[kCh], p_r[kCh], p_sq[kCh];
  bool p_ok[kCh];
#pragma unroll
  for (int pi = 0; pi < kCh; ++pi) {
    const int pair = (pi * kVjpThreads + tid) / kCh;
    p_ok[pi] = pair < 2 * N;
    p_sq[pi] = p_ok[pi] ? pair / N : 0;
    p_r[pi] = p_ok[pi] ? pair - p_sq[pi] * N : 0;
    p_rx[pi] = p_r[pi] / Ly;
    p_ry[pi] = p_r[pi] - p_rx[pi] * Ly;
    p_base[pi] = p_sq[pi] * N;
  }
  float4 acc0[kCh], acc1[kCh];  // spin of p: up / down
#pragma unroll
  for (int pi = 0; pi < kCh; ++pi) acc0[pi] = acc1[pi] = make_float4(0.f, 0.f, 0.f, 0.f);

  for (int smp = blockIdx.x; smp < a.samples; smp += gridDim.x) {
    for (int g = 0; g < a.n_img; ++g) {
      const size_t item = (size_t)smp * a.n_img + g;
      const float* Gi = a.G + item * n * n;
      const float* Yi = a.Y + item * n * D;
      const int32_t* ii = a.idx + item * n;
      __syncthreads();  // previous item's readers are done
      for (int e = tid; e < n * n; e += kVjpThreads) {
        const int row = e / n;
        gs[row * NS + (e - row * n)] = __ldg(Gi + e);
      }
      for (int e = tid; e < n * D; e += kVjpThreads) {
        const int row = e / D, aa = e - row * D;
        ys[swz_index<float, D>(row, aa)] = __ldg(Yi + e);
      }
      for (int m = tid; m < 2 * N; m += kVjpThreads) inv[m] = -1;
      __syncthreads();
      for (int p = tid; p < n; p += kVjpThreads) {
        int m = __ldg(ii + p);
        if ((unsigned)m >= (unsigned)(2 * N)) m = 0;  // out-of-range mode: read as mode 0
        const int sp = m >= N ? 1 : 0, site = m - sp * N, x = site / Ly;
        modes[p] = (sp << 16) | (x << 8) | (site - x * Ly);
        inv[m] = p;
      }
      __syncthreads();
      // dY: lane <-> row p (R rows per warp; the warp's 32 / R lane groups take alternate q), so that
      // Y[q] is a broadcast, the lanes' neighbouring table rows share cache lines (chunked table) and
      // the sums need few exchanges at the end.  16 rows fill the warps from n = 129 on; below, where
      // the loop over q is latency, fewer rows per warp keep all of them at work (300 matrices of
      // n = 56, d = 16: 87.4 us with 16 rows, 58.9 with 4 and the two changes below).
      if (a.dY) {
        float* dYi = a.dY + item * n * D;
        constexpr int WARPS = kVjpThreads / 32;
        const int R = n <= 4 * WARPS ? 4 : (n <= 8 * WARPS ? 8 : 16);
        for (int p0 = R * warp; p0 < n; p0 += R * WARPS) {
          const int pl = p0 + (lane & (R - 1)), p = pl < n ? pl : n - 1;
          const int mp = modes[p];
          const int sp = mp >> 16, xp = (mp >> 8) & 0xFF, yp = mp & 0xFF;
          float acc[D];
#pragma unroll
          for (int j = 0; j < D; ++j) acc[j] = 0.0f;
#pragma unroll 2
          for (int q = lane / R; q < n; q += 32 / R) {
            const float gh = gs[p * NS + q] - gs[q * NS + p];
            const int mq = modes[q];
            const int sq = mq >> 16;
            int dx = xp - ((mq >> 8) & 0xFF), dy = yp - (mq & 0xFF);
            dx += dx < 0 ? Lx : 0;
            dy += dy < 0 ? Ly : 0;
            const int row = (2 * sp + sq) * N + dx * Ly + dy;
            const float4* w4 =
                a.Wc ? a.Wc + row : reinterpret_cast<const float4*>(a.Wt) + row * (D / 4);
            const int stride = a.Wc ? 4 * N : 1;
#pragma unroll
            for (int c = 0; c < D / 4; ++c) {
              const float4 w = __ldg(w4 + c * stride);
              const float4 y = *reinterpret_cast<const float4*>(ys + swz_index<float, D>(q, 4 * c));
              acc[4 * c + 0] = fmaf(gh * w.x, y.x, acc[4 * c + 0]);
              acc[4 * c + 1] = fmaf(gh * w.y, y.y, acc[4 * c + 1]);
              acc[4 * c + 2] = fmaf(gh * w.z, y.z, acc[4 * c + 2]);
              acc[4 * c + 3] = fmaf(gh * w.w, y.w, acc[4 * c + 3]);
            }
          }
          for (int o = 16; o >= R; o >>= 1)
#pragma unroll
            for (int j = 0; j < D; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
          if (lane < R && pl < n)
#pragma unroll
            for (int j = 0; j < D; ++j) dYi[(size_t)pl * D + j] = acc[j];  // any float alignment
        }
      }
      // dWt: each (pair, chunk) sums over the rows p; partner q = inv[sq, site_p - r].  The loads of
      // an empty partner read row 0 and are not added, so that consecutive rows overlap; passes that
      // hold no pair of this lattice are left out.
      const int passes = (2 * N * kCh + kVjpThreads - 1) / kVjpThreads;
      auto add_row = [&](int p, float4 (&acc)[kCh]) {
        const int mp = modes[p];
        const int xp = (mp >> 8) & 0xFF, yp = mp & 0xFF;
        const float4 y1 = *reinterpret_cast<const float4*>(ys + swz_index<float, D>(p, 4 * c_own));
#pragma unroll
        for (int pi = 0; pi < kCh; ++pi) {
          if (pi >= passes) break;
          int x = xp - p_rx[pi], y = yp - p_ry[pi];
          x += x < 0 ? Lx : 0;
          y += y < 0 ? Ly : 0;
          const int q = p_ok[pi] ? inv[p_base[pi] + x * Ly + y] : -1;
          const int qq = q < 0 ? 0 : q;
          const float gv = gs[p * NS + qq];
          const float4 y2 = *reinterpret_cast<const float4*>(ys + swz_index<float, D>(qq, 4 * c_own));
          if (q >= 0) {
            acc[pi].x = fmaf(gv * y1.x, y2.x, acc[pi].x);
            acc[pi].y = fmaf(gv * y1.y, y2.y, acc[pi].y);
            acc[pi].z = fmaf(gv * y1.z, y2.z, acc[pi].z);
            acc[pi].w = fmaf(gv * y1.w, y2.w, acc[pi].w);
          }
        }
      };
      // rows of one spin in turn (the modes ascend, so there is one run of each); a run's end is
      // found by ballots, as a chain of n loads would be a good part of a small matrix's time
      for (int p = 0; p < n;) {
        const int sp = modes[p] >> 16;
        int end = n;
        for (int b = p; b < n; b += 32) {
          const bool other = b + lane < n && (modes[b + lane] >> 16) != sp;
          const unsigned m = __ballot_sync(0xffffffffu, other);
          if (m) {
            end = b + __ffs(m) - 1;
            break;
          }
        }
        if (sp) {
#pragma unroll 2
          for (; p < end; ++p) add_row(p, acc1);
        } else {
#pragma unroll 2
          for (; p < end; ++p) add_row(p, acc0);
        }
      }
      if (a.mode == 0) {  // per-item dWt
        float* dst = a.dWt + item * 4 * N * D;
#pragma unroll
        for (int pi = 0; pi < kCh; ++pi) {
          if (!p_ok[pi]) continue;
          float* d0 = dst + ((size_t)p_sq[pi] * N + p_r[pi]) * D + 4 * c_own;
          float* d1 = dst + ((size_t)(2 + p_sq[pi]) * N + p_r[pi]) * D + 4 * c_own;
          d0[0] = acc0[pi].x, d0[1] = acc0[pi].y, d0[2] = acc0[pi].z, d0[3] = acc0[pi].w;
          d1[0] = acc1[pi].x, d1[1] = acc1[pi].y, d1[2] = acc1[pi].z, d1[3] = acc1[pi].w;
          acc0[pi] = acc1[pi] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    }
    if (a.mode != 1) continue;
    // Sample done: the summed dWt through build_wtilde's backward.
    __syncthreads();
    float* dw = gs;  // (4, N, D)
#pragma unroll
    for (int pi = 0; pi < kCh; ++pi) {
      if (!p_ok[pi]) continue;
      *reinterpret_cast<float4*>(dw + ((size_t)p_sq[pi] * N + p_r[pi]) * D + 4 * c_own) = acc0[pi];
      *reinterpret_cast<float4*>(dw + ((size_t)(2 + p_sq[pi]) * N + p_r[pi]) * D + 4 * c_own) =
          acc1[pi];
      acc0[pi] = acc1[pi] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    // Envelope pref[r] = exp(-lam D_r) / (N sum exp(-lam D)) and its mean distance, FP64.
    const double th = (double)a.theta;
    const double lam = log1p(exp(-fabs(th))) + fmax(th, 0.0);
    double se = 0.0, sde = 0.0;
    for (int r = tid; r < N; r += kVjpThreads) {
      const int rx = r / Ly, ry = r - rx * Ly;
      const double mx = (double)min(rx, Lx - rx), my = (double)min(ry, Ly - ry);
      const double dist = sqrt(mx * mx + my * my), e = exp(-lam * dist);
      se += e;
      sde += dist * e;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      se += __shfl_xor_sync(0xffffffffu, se, o);
      sde += __shfl_xor_sync(0xffffffffu, sde, o);
    }
    __shared__ double part[2][kVjpThreads / 32];
    if (lane == 0) {
      part[0][warp] = se;
      part[1][warp] = sde;
    }
    __syncthreads();
    double S = 0.0, SD = 0.0;
    for (int w = 0; w < kVjpThreads / 32; ++w) {
      S += part[0][w];
      SD += part[1][w];
    }
    const double mean_d = SD / S;
    float* row = a.jac + (size_t)smp * a.ld + a.off_w;
    double tacc = 0.0;
    for (int e = tid; e < N * D; e += kVjpThreads) {
      const int r = e / D, aa = e - r * D;
      const int rx = r / Ly, ry = r - rx * Ly;
      const int nr = (rx ? Lx - rx : 0) * Ly + (ry ? Ly - ry : 0);
      const double mx = (double)min(rx, Lx - rx), my = (double)min(ry, Ly - ry);
      const double dist = sqrt(mx * mx + my * my);
      const float pref = (float)(exp(-lam * dist) / ((double)N * S));
      const int nrx = nr / Ly, nry = nr - nrx * Ly;
      const double ndist = sqrt((double)min(nrx, Lx - nrx) * min(nrx, Lx - nrx) +
                                (double)min(nry, Ly - nry) * min(nry, Ly - nry));
      const float npref = (float)(exp(-lam * ndist) / ((double)N * S));
      const float d0 = dw[(0 * N + r) * D + aa] * pref, d0n = dw[(0 * N + nr) * D + aa] * npref;
      const float d1 = dw[(1 * N + r) * D + aa] * pref;
      const float d2n = dw[(2 * N + nr) * D + aa] * npref;
      const float d3 = dw[(3 * N + r) * D + aa] * pref, d3n = dw[(3 * N + nr) * D + aa] * npref;
      row[(0 * N + r) * D + aa] = d1 - d2n;
      row[(1 * N + r) * D + aa] = 0.5f * (d0 - d0n);
      row[(2 * N + r) * D + aa] = 0.5f * (d3 - d3n);
      double s4 = 0.0;
#pragma unroll
      for (int b = 0; b < 4; ++b)
        s4 += (double)dw[(b * N + r) * D + aa] * (double)__ldg(a.Wt + (b * N + r) * D + aa);
      tacc += s4 * (mean_d - dist);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) tacc += __shfl_xor_sync(0xffffffffu, tacc, o);
    __syncthreads();
    if (lane == 0) part[0][warp] = tacc;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int w = 0; w < kVjpThreads / 32; ++w) t += part[0][w];
      row[3 * N * D] = (float)(t / (1.0 + exp(-th)));
    }
  }
}

template <int D>
size_t vjp_smem(int n, int N) {
  const size_t reg0 = std::max((size_t)n * (n + 1), (size_t)4 * N * D);
  return sizeof(float) * (((reg0 + 3) & ~(size_t)3) + (size_t)n * D) +
         sizeof(int) * ((size_t)n + 2 * N);
}

template <int D>
int launch_vjp_t(const VjpArgs& a, cudaStream_t st) {
  const int N = a.Lx * a.Ly;
  const size_t smem = vjp_smem<D>(a.n, N);
  if (smem > 227 * 1024 || 2 * N > kVjpThreads)
    return fail(NH_ERR_UNSUPPORTED, "pairing vjp: n = %d, N = %d", a.n, N);
  static size_t configured = 0;
  if (smem > 48 * 1024 && smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(pairing_vjp_kernel<D>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return check_cuda(e, "pairing vjp smem attribute");
    configured = smem;
  }
  int grid = num_sms() * (smem <= 113 * 1024 ? 2 : 1);
  if (grid > a.samples) grid = a.samples;
  ProfScope prof_scope(NH_K_PAIRING_VJP, st);
  pairing_vjp_kernel<D><<<grid, kVjpThreads, smem, st>>>(a);
  return check_launch("pairing_vjp_kernel");
}

// ------------------------------------------------------------------ CNN VJP
constexpr size_t kCvTwoCtaSmem = 113 * 1024;

// One periodic 3x3 cross-correlation of cin planes (stride N + 1) into cout planes, weights
// [ci][tap][co] in shared memory, no bias; epi(co, site, z) stores the result.
template <int TH, typename Epi>
__device__ __forceinline__ void conv_planes(const float* in, int cin, int cout, const float* wsm,
                                            int Lx, int Ly, Epi epi) {
  const int part = Lx * Ly / 2;
  for (int task = threadIdx.x; task < (cout / 8) * part; task += TH) {
    const int grp = task / part;
    const int site[2] = {task - grp * part, task - grp * part + part};
    float acc[2][8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[0][j] = acc[1][j] = 0.0f;
    conv_task<float, 2>(in, cin, cout, wsm, grp, site, Lx, Ly, acc);
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) epi(grp * 8 + j, site[k], acc[k][j]);
  }
}

__device__ __forceinline__ float gelu_tanh_grad_dev(float x) {
  const float k0 = 0.7978845608028654f, c = 0.044715f;
  const float t = tanhf(k0 * (x + c * x * x * x));
  return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * k0 * (1.0f + 3.0f * c * x * x);
}

struct CnnVjpArgs {
  const int8_t* spins;  // (samples, 2N)
  int samples, n_img;
  const float* conv_w;  // OIHW per layer, concatenated
  const float* conv_w_packed;  // [l][ci][tap][co]
  const float* conv_b;
  int Lx, Ly, C, layers, n;
  const float* dY;       // (items, n, d) cotangent of the occupied rows (image weight included)
  const int32_t* idx;    // (items, n) occupied modes of each image configuration
  float* jac;            // (samples, ld): conv weights and biases from column 0
  int64_t ld;
};

// Shared memory: z planes of layers 0 .. L-2 ((L-1) C NS), the input image (2 NS), two cotangent /
// activation buffers (2 C NS) and one layer's weights (C C 9).
template <int TH>
__global__ void __launch_bounds__(TH) cnn_vjp_kernel(CnnVjpArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Lx = a.Lx, Ly = a.Ly, N = Lx * Ly, NS = N + 1, C = a.C, L = a.layers, d = C / 2;
  const int tid = threadIdx.x;
  float* zs = reinterpret_cast<float*>(smem_raw);        // (L-1, C, NS)
  float* img = zs + (size_t)(L - 1) * C * NS;            // (2, NS), padded to 16 bytes
  float* bufA = img + ((2 * NS + 3) & ~3);               // (C, NS)
  float* bufB = bufA + (size_t)C * NS;                   // (C, NS)
  float* wsm = bufB + (size_t)C * NS;                    // (C C 9)

  for (int smp = blockIdx.x; smp < a.samples; smp += gridDim.x) {
    float* row = a.jac + (size_t)smp * a.ld;
    const int8_t* base = a.spins + (size_t)smp * 2 * N;
    for (int g = 0; g < a.n_img; ++g) {
      const size_t item = (size_t)smp * a.n_img + g;
      const int sym = a.n_img == 1 ? 0 : g;
      __syncthreads();
      for (int m = tid; m < 2 * N; m += TH) {
        const int src = sym_map(m, sym, Lx, Ly, N);
        const int ch = m >= N ? 1 : 0;
        img[ch * NS + (m - ch * N)] = base[src] > 0 ? 1.0f : -1.0f;
      }
      // Forward, keeping the pre-activations z_l (l < L - 1); GELU(z) into bufA as next input.
      const float* in = img;
      int cin = 2;
      size_t woff = 0;
      for (int l = 0; l < L - 1; ++l) {
        __syncthreads();
        stage_floats<TH>(wsm, a.conv_w_packed + woff, C * cin * 9);
        __syncthreads();
        float* z = zs + (size_t)l * C * NS;
        const float* bl = a.conv_b + l * C;
        conv_planes<TH>(in, cin, C, wsm, Lx, Ly,
                    [&](int co, int s, float v) { z[co * NS + s] = v + __ldg(bl + co); });
        __syncthreads();
        for (int e = tid; e < C * N; e += TH) {
          const int co = e / N, s = e - co * N;
          bufA[co * NS + s] = gelu_tanh_dev(z[co * NS + s]);
        }
        in = bufA;
        woff += (size_t)C * cin * 9;
        cin = C;
      }
      // Cotangent of the last layer's output: dY scattered to the occupied modes.
      __syncthreads();
      float* dcur = bufB;
      float* dother = bufA;
      for (int e = tid; e < C * NS; e += TH) dcur[e] = 0.0f;
      __syncthreads();
      const float* dYi = a.dY + item * a.n * d;
      const int32_t* ii = a.idx + item * a.n;
      for (int e = tid; e < a.n * d; e += TH) {
        const int p = e / d, aa = e - p * d;
        const int m = __ldg(ii + p);
        const int sg = m >= N ? 1 : 0;
        dcur[(sg * d + aa) * NS + (m - sg * N)] = __ldg(dYi + e);
      }
      // Backward, last layer first.
      size_t wl_off = 0;  // OIHW offset of layer l
      int64_t col = 0;    // Jacobian column of layer l's weights
      // offsets of layer l: layer 0 has cin 2
      for (int l = L - 1; l >= 0; --l) {
        const int lcin = l == 0 ? 2 : C;
        wl_off = l == 0 ? 0 : (size_t)C * 2 * 9 + (size_t)(l - 1) * C * C * 9;
        col = l == 0 ? 0 : (int64_t)(C * 2 * 9 + C) + (int64_t)(l - 1) * (C * C * 9 + C);
        __syncthreads();
        // Layer input activation: the image for l = 0, GELU(z_{l-1}) otherwise (into dother).
        const float* ain = img;
        if (l > 0) {
          const float* z = zs + (size_t)(l - 1) * C * NS;
          for (int e = tid; e < C * N; e += TH) {
            const int ci = e / N, s = e - ci * N;
            dother[ci * NS + s] = gelu_tanh_dev(z[ci * NS + s]);
          }
          ain = dother;
        }
        __syncthreads();
        // Weight cotangent: a task owns (4 output channels, 1 input channel) x 9 taps over a share of
        // the lattice's rows; with fewer tasks than threads (all but very wide layers) the rows
        // are split, and the shares are summed in shared memory (the weights' place, not in use).
        const int pairs = (C / 4) * lcin;
        int split = 1;
        while (2 * split * pairs <= TH && 2 * split <= Lx &&
               (2 * split - 1) * pairs * 36 <= C * C * 9)
          split *= 2;
        for (int t0 = 0; t0 < pairs * split; t0 += TH) {
          const int task = t0 + tid, pr = task % pairs, share = task / pairs;
          const bool on = task < pairs * split;
          const int ci = pr % lcin, cob = pr / lcin;
          float acc[4][9];
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int t = 0; t < 9; ++t) acc[j][t] = 0.0f;
          if (on) {
            const float* ap = ain + ci * NS;
            const float* dp = dcur + (size_t)(cob * 4) * NS;
            for (int x = share; x < Lx; x += split) {
              const float* r0 = ap + (x == 0 ? Lx - 1 : x - 1) * Ly;
              const float* r1 = ap + x * Ly;
              const float* r2 = ap + (x == Lx - 1 ? 0 : x + 1) * Ly;
              // the window's columns y - 1, y, y + 1 slide along the row
              float w0[3] = {r0[Ly - 1], r1[Ly - 1], r2[Ly - 1]}, w1[3] = {r0[0], r1[0], r2[0]};
              for (int y = 0; y < Ly; ++y) {
                const int yp = y == Ly - 1 ? 0 : y + 1, s = x * Ly + y;
                const float w2[3] = {r0[yp], r1[yp], r2[yp]};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float dv = dp[j * NS + s];
#pragma unroll
                  for (int u = 0; u < 3; ++u) {
                    acc[j][3 * u] = fmaf(dv, w0[u], acc[j][3 * u]);
                    acc[j][3 * u + 1] = fmaf(dv, w1[u], acc[j][3 * u + 1]);
                    acc[j][3 * u + 2] = fmaf(dv, w2[u], acc[j][3 * u + 2]);
                  }
                }
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                  w0[u] = w1[u];
                  w1[u] = w2[u];
                }
              }
            }
          }
          if (split > 1) {
            if (on && share > 0) {
              float* part = wsm + (size_t)(share - 1) * pairs * 36 + pr;  // [36][pairs]
#pragma unroll
              for (int q = 0; q < 36; ++q) part[q * pairs] = acc[q / 9][q % 9];
            }
            __syncthreads();
          }
          if (on && share == 0) {
            for (int sh = 1; sh < split; ++sh) {
              const float* part = wsm + (size_t)(sh - 1) * pairs * 36 + pr;
#pragma unroll
              for (int q = 0; q < 36; ++q) acc[q / 9][q % 9] += part[q * pairs];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float* dst = row + col + ((int64_t)(cob * 4 + j) * lcin + ci) * 9;
#pragma unroll
              for (int t = 0; t < 9; ++t) dst[t] = g == 0 ? acc[j][t] : dst[t] + acc[j][t];
            }
          }
        }
        // Bias cotangent: warp per output channel.
        {
          const int lane = tid & 31, warp = tid >> 5;
          for (int co = warp; co < C; co += TH / 32) {
            float s = 0.0f;
            for (int e = lane; e < N; e += 32) s += dcur[co * NS + e];
#pragma unroll
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) {
              float* dst = row + col + (int64_t)C * lcin * 9 + co;
              *dst = g == 0 ? s : *dst + s;
            }
          }
        }
        if (l == 0) break;
        // Input cotangent: transposed convolution with flipped taps, times GELU'(z_{l-1}).
        __syncthreads();
        for (int i = tid; i < C * C * 9; i += TH) {
          const int cj = i % C;        // output channel of the transposed conv = layer input ci
          const int rest = i / C;      // co * 9 + tap'
          const int co = rest / 9, tp = rest - co * 9;
          wsm[i] = __ldg(a.conv_w + wl_off + ((size_t)co * C + cj) * 9 + (8 - tp));
        }
        __syncthreads();
        const float* z = zs + (size_t)(l - 1) * C * NS;
        conv_planes<TH>(dcur, C, C, wsm, Lx, Ly, [&](int ci, int s, float v) {
          dother[ci * NS + s] = v * gelu_tanh_grad_dev(z[ci * NS + s]);
        });
        float* t = dcur;
        dcur = dother;
        dother = t;
      }
    }
  }
}

size_t cnn_vjp_smem(int N, int C, int L) {
  const size_t NS = (size_t)N + 1;
  return sizeof(float) * ((size_t)(L - 1) * C * NS + ((2 * NS + 3) & ~(size_t)3) +
                          2 * (size_t)C * NS + (size_t)C * C * 9);
}

template <int TH>
int launch_cnn_vjp_th(const CnnVjpArgs& a, size_t smem, cudaStream_t st) {
  static size_t configured = 0;
  if (smem > 48 * 1024 && smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(cnn_vjp_kernel<TH>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return check_cuda(e, "cnn vjp smem attribute");
    configured = smem;
  }
  int grid = num_sms() * (smem <= kCvTwoCtaSmem ? 2 : 1);
  if (grid > a.samples) grid = a.samples;
  ProfScope prof_scope(NH_K_CNN_VJP, st);
  cnn_vjp_kernel<TH><<<grid, TH, smem, st>>>(a);
  return check_launch("cnn_vjp_kernel");
}

}  // namespace

// ------------------------------------------------------------------ launchers
int launch_pf_adjoint(const float* F, float* G, int n, int batch, const float* pf_sign,
                      const double* pf_logabs, int n_img, int32_t* flags, cudaStream_t st) {
  if (batch <= 0) return NH_OK;
  AdjArgs a{F, G, n, batch, pf_sign, pf_logabs, n_img, flags};
  const int tc = (n + 31) / 32;
  switch (tc) {
    case 1: return launch_adjoint_t<1>(a, st);
    case 2: return launch_adjoint_t<2>(a, st);
    case 3: return launch_adjoint_t<3>(a, st);
    case 4: return launch_adjoint_t<4>(a, st);
    case 5: return launch_adjoint_t<5>(a, st);
    case 6: return launch_adjoint_t<6>(a, st);
    case 7: return launch_adjoint_t<7>(a, st);
    default: return fail(NH_ERR_UNSUPPORTED, "pfaffian adjoint: n = %d > %d", n, kGradMaxN);
  }
}

int launch_pairing_vjp(const float* G, const float* Y, const int32_t* idx, const float* Wt,
                       const float* wt_chunks, int Lx, int Ly, int d, int n, int n_img,
                       int samples, float* dY, float* dWt, float* jac, int64_t ld, int64_t off_w, float theta,
                       cudaStream_t st) {
  if (samples <= 0) return NH_OK;
  VjpArgs a{G, Y, idx, Wt, reinterpret_cast<const float4*>(wt_chunks), Lx, Ly, n, n_img,
            samples, dY, dWt, jac, ld, off_w, theta, jac ? 1 : 0};
  switch (d) {
    case 8: return launch_vjp_t<8>(a, st);
    case 16: return launch_vjp_t<16>(a, st);
    case 32: return launch_vjp_t<32>(a, st);
    default: return fail(NH_ERR_UNSUPPORTED, "pairing vjp: d = %d (8, 16 or 32)", d);
  }
}

int launch_cnn_vjp(const int8_t* spins, int samples, int n_img, const nh_backflow_params& p,
                   const float* dY, const int32_t* idx, float* jac, int64_t ld, cudaStream_t st) {
  if (samples <= 0) return NH_OK;
  const int N = p.Lx * p.Ly, C = p.channels;
  if (C % 8 || C < 8 || C > 64 || p.layers < 1 || N % 2)
    return fail(NH_ERR_UNSUPPORTED, "cnn vjp: channels %d, layers %d, N %d", C, p.layers, N);
  const size_t smem = cnn_vjp_smem(N, C, p.layers);
  if (smem > 227 * 1024)
    return fail(NH_ERR_UNSUPPORTED, "cnn vjp: N = %d, %d channels, %d layers need %zu B", N, C,
                p.layers, smem);
  CnnVjpArgs a{spins, samples, n_img, p.conv_w, p.conv_w_packed, p.conv_b, p.Lx, p.Ly, C,
               p.layers, p.n_up + p.n_dn, dY, idx, jac, ld};
  // 512 threads leave room for one CTA per SM (registers), so with more samples than SMs two CTAs of
  // 256 that shared memory holds are faster: 250 bare samples, 4 layers of 32 channels, whole call:
  // 3x4 278 -> 232 us, 4x4 322 -> 276, 8x8 487 -> 453, 10x10 721 -> 696; with at most a sample per SM
  // 512 win (148 samples: 192 against 203, 228 / 243, 331 / 347, 471 / 490).
  const bool two = smem <= kCvTwoCtaSmem && samples > num_sms();
  return two ? launch_cnn_vjp_th<256>(a, smem, st) : launch_cnn_vjp_th<512>(a, smem, st);
}

bool cnn_vjp_supported(const nh_backflow_params& p) {
  const int N = p.Lx * p.Ly, C = p.channels;
  return p.net == NH_NET_CNN && C % 8 == 0 && C >= 8 && C <= 64 && N % 2 == 0 && p.layers >= 1 &&
         cnn_vjp_smem(N, C, p.layers) <= 227 * 1024;
}

}  // namespace nh
