// Residual backflow CNN of the released Pfaffian-backflow states (quantax ResConv as built at
// code/backflow/models.py:319-329; network of data/supplement/tableS1_network/
// network_settings.json:21-56, "normal" blocks), forward on CUDA cores in FP32 (FP64 for the
// recompute of flagged items):
//
//   x_0[c, i] = E[c, occ(i)]                       occ = n_up + 2 n_dn (empty, up, down, double)
//   x_{b+1}   = x_b + Conv2(GELU(Conv1(GELU(RMSNorm(x_b)))))   b < blocks
//   y         = x_blocks / sqrt(blocks + 1)        channels [0, d) spin up, [d, 2d) spin down
//
// with 3x3 periodic cross-correlations with bias, RMSNorm over all channels and sites without
// affine parameters (eps kRmsEps inside the root) and tanh-approximated GELU.
//
// One CTA of 256 threads per item (configuration x symmetry image, grid-stride).  The three
// activation planes x, h = GELU(RMSNorm(x)) and u = GELU(Conv1(h)) are channel-major with row
// stride N + 1, in shared memory for FP32 at N <= 256 (197 KB at 64 channels), otherwise in a
// per-CTA slice of global scratch.  A convolution is a tile loop over 256 sites: thread t owns
// 16 output channels (t / 64) of 4 sites (t % 64 + 64 k) as 64 register accumulators; the
// weights stream through shared memory in chunks of 8 input channels ([ci][tap][co], 18 KB in
// FP32), the next chunk held in registers while the current one is used, so that their L2
// latency hides behind the FMAs.  Per (input channel, tap) a thread issues 4 activation loads,
// 4 broadcast 16-byte weight loads and 64 FMAs.  The output rows Y of the occupied modes, their
// indices and the item sign are written by the same epilogue as the plain CNN's.
#include <cooperative_groups.h>
#include <math.h>

#include "nh_cnn_mma.cuh"
#include "nh_common.cuh"

namespace nh {
namespace {

constexpr int kRcThreads = kNumThreads;  // 256
constexpr int kRcC = 64;                 // channels (the released states)
constexpr int kRcCoPerThread = 16;       // output channels per thread
constexpr int kRcSiteLanes = kRcThreads / (kRcC / kRcCoPerThread);                 // 64
constexpr int kRcChunk = 8;              // input channels per staged weight chunk
constexpr int kRcChunkFloats = kRcChunk * 9 * kRcC;                                // 4608
constexpr int kRcChunkVec = kRcChunkFloats / 4;                                    // float4s
constexpr int kRcPrefetch = (kRcChunkVec + kRcThreads - 1) / kRcThreads;          // 5
constexpr double kRmsEps = 1e-6;
static_assert(kRcC % kRcChunk == 0, "chunks must tile the input channels");

// Sites per thread and tile: 4 in FP32 (64 accumulators), 2 in FP64 (the same register count).
template <typename T>
struct RcSpt {
  static constexpr int value = sizeof(T) == 4 ? 4 : 2;
};

__device__ __forceinline__ float tfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double tfma(double a, double b, double c) { return ::fma(a, b, c); }
__device__ __forceinline__ float trsqrt_eps(float ms, double eps) {
  return 1.0f / sqrtf(ms + (float)eps);
}
__device__ __forceinline__ double trsqrt_eps(double ms, double eps) {
  return 1.0 / ::sqrt(ms + eps);
}

__device__ __forceinline__ float gelu_tanh(float x) {
  const float k0 = 0.7978845608028654f;  // sqrt(2 / pi)
  return 0.5f * x * (1.0f + tanhf(k0 * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ double gelu_tanh(double x) {
  const double k0 = 0.7978845608028654;
  return 0.5 * x * (1.0 + tanh(k0 * (x + 0.044715 * x * x * x)));
}

template <typename T>
struct RcArgs {
  ConfigList cl;
  const float* embed;  // packed (4, C): [occ][co]
  const float* wp;     // packed convolutions: per conv [ci][tap][co]
  const float* b;      // (2 blocks, C)
  int Lx, Ly, N, blocks, n;
  int mode;
  const int32_t* slot_item;
  const int32_t* slot_count;
  int max_slots;
  float* feat;
  T* Y;
  int32_t* idx;
  float* item_sign;
  T* act;  // GACT: per-CTA planes (3 C (N + 1))
};

// 16 weights of one (input channel, tap) row for this thread's output channels (broadcast).
__device__ __forceinline__ void ldw16(const float* p, float* w) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 v = reinterpret_cast<const float4*>(p)[q];
    w[4 * q] = v.x;
    w[4 * q + 1] = v.y;
    w[4 * q + 2] = v.z;
    w[4 * q + 3] = v.w;
  }
}
__device__ __forceinline__ void ldw16(const double* p, double* w) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const double2 v = reinterpret_cast<const double2*>(p)[q];
    w[2 * q] = v.x;
    w[2 * q + 1] = v.y;
  }
}

// Registers holding the next weight chunk (kRcPrefetch float4 per thread).
struct ChunkRegs {
  float4 v[kRcPrefetch];
};

__device__ __forceinline__ void chunk_load(ChunkRegs& r, const float* src) {
  const float4* s4 = reinterpret_cast<const float4*>(src);
#pragma unroll
  for (int k = 0; k < kRcPrefetch; ++k) {
    const int i = threadIdx.x + k * kRcThreads;
    if (i < kRcChunkVec) r.v[k] = __ldg(s4 + i);
  }
}

template <typename T>
__device__ __forceinline__ void chunk_store(const ChunkRegs& r, T* dst) {
#pragma unroll
  for (int k = 0; k < kRcPrefetch; ++k) {
    const int i = threadIdx.x + k * kRcThreads;
    if (i < kRcChunkVec) {
      dst[4 * i] = T(r.v[k].x);
      dst[4 * i + 1] = T(r.v[k].y);
      dst[4 * i + 2] = T(r.v[k].z);
      dst[4 * i + 3] = T(r.v[k].w);
    }
  }
}

// One 3x3 periodic convolution C -> C over all sites: dst = epi(conv(src) + bias, dst).
// Entry: pre holds chunk 0 of w; exit: pre holds chunk 0 of w_next (when not null).
// RESID: dst += result; else dst = GELU(result).
template <typename T, bool RESID>
__device__ void conv_pass(const T* src, T* dst, const float* w, const float* w_next,
                          const float* bias, T* wsm, ChunkRegs& pre, int Lx, int Ly, int N) {
  constexpr int SPT = RcSpt<T>::value;
  constexpr int kTile = kRcSiteLanes * SPT;
  const int NS = N + 1;
  const int tid = threadIdx.x;
  const int cg = tid / kRcSiteLanes;  // output-channel group (16 channels)
  const int sl = tid % kRcSiteLanes;  // site lane: sites sl + 64 k of the tile
  constexpr int kChunks = kRcC / kRcChunk;
  const int tiles = (N + kTile - 1) / kTile;
  for (int tile = 0; tile < tiles; ++tile) {
    int nb[SPT][9];
    bool live[SPT];
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
      const int site = tile * kTile + sl + k * kRcSiteLanes;
      live[k] = site < N;
      const int s = live[k] ? site : 0;
      const int x = s / Ly, y = s - x * Ly;
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        int xx = x + u - 1;
        xx = xx < 0 ? xx + Lx : (xx >= Lx ? xx - Lx : xx);
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          int yy = y + v - 1;
          yy = yy < 0 ? yy + Ly : (yy >= Ly ? yy - Ly : yy);
          nb[k][u * 3 + v] = xx * Ly + yy;
        }
      }
    }
    T acc[SPT][kRcCoPerThread];
#pragma unroll
    for (int j = 0; j < kRcCoPerThread; ++j) {
      const T bj = T(__ldg(bias + cg * kRcCoPerThread + j));
#pragma unroll
      for (int k = 0; k < SPT; ++k) acc[k][j] = bj;
    }
#pragma unroll 1
    for (int ch = 0; ch < kChunks; ++ch) {
      __syncthreads();  // every thread is done with the previous chunk in wsm
      chunk_store(pre, wsm);
      __syncthreads();
      const bool last = tile == tiles - 1 && ch == kChunks - 1;
      if (!last) {
        chunk_load(pre, w + (size_t)((ch + 1) % kChunks) * kRcChunkFloats);
      } else if (w_next) {
        chunk_load(pre, w_next);
      }
#pragma unroll 1
      for (int cil = 0; cil < kRcChunk; ++cil) {
        const T* in = src + (ch * kRcChunk + cil) * NS;
        const T* wrow = wsm + cil * 9 * kRcC + cg * kRcCoPerThread;
#pragma unroll
        for (int tap = 0; tap < 9; ++tap) {
          T iv[SPT];
#pragma unroll
          for (int k = 0; k < SPT; ++k) iv[k] = in[nb[k][tap]];
          T wv[kRcCoPerThread];
          ldw16(wrow + tap * kRcC, wv);
#pragma unroll
          for (int k = 0; k < SPT; ++k)
#pragma unroll
            for (int j = 0; j < kRcCoPerThread; ++j) acc[k][j] = tfma(iv[k], wv[j], acc[k][j]);
        }
      }
    }
    // Epilogue: this thread's outputs are read by no other thread of this pass (dst != src).
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
      if (!live[k]) continue;
      const int site = tile * kTile + sl + k * kRcSiteLanes;
#pragma unroll
      for (int j = 0; j < kRcCoPerThread; ++j) {
        T* o = dst + (cg * kRcCoPerThread + j) * NS + site;
        if constexpr (RESID) {
          *o += acc[k][j];
        } else {
          *o = gelu_tanh(acc[k][j]);
        }
      }
    }
  }
}

template <typename T, bool GACT>
__global__ void __launch_bounds__(kRcThreads, 1) resconv_kernel(RcArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = a.N, NS = N + 1, M2 = 2 * N;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int kWarps = kRcThreads / 32;
  T* X;
  T* wsm;  // staged weight chunk [ci][tap][co]
  if constexpr (GACT) {
    X = a.act + (size_t)blockIdx.x * 3 * kRcC * NS;
    wsm = reinterpret_cast<T*>(smem_raw);
  } else {
    X = reinterpret_cast<T*>(smem_raw);
    wsm = X + 3 * kRcC * NS;
  }
  T* H = X + kRcC * NS;
  T* U = H + kRcC * NS;
  T* red = wsm + kRcChunkFloats;                       // (warps) partial sums of x^2
  int* simg = reinterpret_cast<int*>(red + kWarps);    // (2N) +-1 of the image configuration
  int* occl = simg + M2;                                // (2N) occupied modes, ascending
  int* wbuf = occl + M2;                                // 4 Lx + 32 ints of scan scratch

  const int G = a.cl.G;
  const int n_work = a.slot_item ? *a.slot_count
                                 : (a.cl.n_cfg_dev ? *a.cl.n_cfg_dev : a.cl.n_cfg) * G;
  const size_t conv_floats = (size_t)kRcC * 9 * kRcC;
  const T inv_cn = T(1) / T(kRcC * N);
  const T out_scale = trsqrt_eps(T(a.blocks + 1), 0.0);
  ChunkRegs pre;

  for (int slot = blockIdx.x; slot < n_work; slot += gridDim.x) {
    const int item = a.slot_item ? a.slot_item[slot] : slot;
    const int c = item / G, g = item - c * G;
    const int smp = a.cl.sample ? a.cl.sample[c] : c;
    const int fr = a.cl.from ? a.cl.from[c] : -1;
    const int to = a.cl.from ? a.cl.to[c] : -1;
    const int8_t* base = a.cl.spins + (int64_t)smp * M2;
    chunk_load(pre, a.wp);  // chunk 0 of the first convolution

    __syncthreads();  // the previous item's readers of simg / planes are done
    for (int m = tid; m < M2; m += kRcThreads) {
      const int src = sym_map(m, g, a.Lx, a.Ly, N);  // image[m] = s[g(m)] (g is an involution)
      int v = base[src];
      v = move_value(src, v, fr, to);
      simg[m] = v > 0 ? 1 : -1;
    }
    __syncthreads();
    for (int i = tid; i < N; i += kRcThreads) {  // occupation embedding
      const int occ = (simg[i] > 0 ? 1 : 0) + (simg[N + i] > 0 ? 2 : 0);
      const float* e = a.embed + occ * kRcC;
      for (int ch = 0; ch < kRcC; ++ch) X[ch * NS + i] = T(__ldg(e + ch));
    }

    for (int blk = 0; blk < a.blocks; ++blk) {
      __syncthreads();  // x complete
      T ss = T(0);
      for (int ch = 0; ch < kRcC; ++ch)
        for (int i = tid; i < N; i += kRcThreads) {
          const T v = X[ch * NS + i];
          ss = tfma(v, v, ss);
        }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) red[wid] = ss;
      __syncthreads();
      T tot = T(0);
#pragma unroll
      for (int w = 0; w < kWarps; ++w) tot += red[w];
      const T r = trsqrt_eps(tot * inv_cn, kRmsEps);
      for (int ch = 0; ch < kRcC; ++ch)
        for (int i = tid; i < N; i += kRcThreads) H[ch * NS + i] = gelu_tanh(X[ch * NS + i] * r);
      // (the first chunk barrier of conv_pass orders these writes before the reads)
      const float* w1 = a.wp + (size_t)(2 * blk) * conv_floats;
      const float* w2 = w1 + conv_floats;
      conv_pass<T, false>(H, U, w1, w2, a.b + (2 * blk) * kRcC, wsm, pre, a.Lx, a.Ly, N);
      conv_pass<T, true>(U, X, w2, blk + 1 < a.blocks ? w2 + conv_floats : nullptr,
                         a.b + (2 * blk + 1) * kRcC, wsm, pre, a.Lx, a.Ly, N);
    }
    __syncthreads();
    constexpr int d = kRcC / 2;
    if (a.mode == 0) {
      float* dst = a.feat + (int64_t)item * kRcC * N;
      for (int o = tid; o < kRcC * N; o += kRcThreads) {
        const int aa = o % d;
        const int site = (o / d) % N;
        const int sg = o / (N * d);
        dst[o] = (float)(X[(sg * d + aa) * NS + site] * out_scale);
      }
      continue;
    }
    write_occupied_rows(simg, occl, wbuf, N, a.n, d, g, a.Lx, a.Ly,
                        a.Y + (int64_t)slot * a.n * d, a.idx + (int64_t)slot * a.n,
                        a.item_sign + item, [&](int sg, int aa, int site) {
                          return X[(sg * d + aa) * NS + site] * out_scale;
                        });
  }
}

// FP64 features on the FP64 matrix instruction, mode 1 only, lattices up to 256 sites: a cluster of
// two CTAs per item, each with half of the output channels.  The convolutions are the implicit GEMMs
// of nh_cnn_mma.cuh (same products in the same order as conv_pass); both CTAs keep the whole
// input's padded planes in shared memory (166 KB at 16x16) and write their halves of every new
// activation to both.  The residual stream x stays in registers, in the accumulator layout.  The
// weights stream through two 9 KB chunks (4 input channels, in fragment order), the next one in
// registers.  Half an item per CTA also halves the granularity of the last wave: the recompute
// lists are a few items per SM.  478 items of 16 blocks at 16x16: 25.4 ms by conv_pass in FP64 with
// its planes in global memory, 12.2 ms here (the FMA floor, evenly spread, is 7.7 ms).
constexpr int kRmThreads = 512;
constexpr int kRmChunk = 9 * 4 * 32;  // weights of one chunk: 36 k x 32 channels
constexpr int kRmPre = (kRmChunk + kRmThreads - 1) / kRmThreads;

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kRmThreads, 1)
    resconv_mma_kernel(RcArgs<double> a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[kRmThreads / 32];
  __shared__ double part[2];  // both CTAs' sums of x^2
  constexpr int NT = 4, WARPS = kRmThreads / 32;
  const int Lx = a.Lx, Ly = a.Ly, N = a.N, M2 = 2 * N, W = Ly + 2, PS = mma_plane(Lx, Ly);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* act = reinterpret_cast<double*>(smem_raw);
  double* wsm = act + (size_t)kRcC * PS;
  int* simg = reinterpret_cast<int*>(wsm + 2 * kRmChunk);
  int* occl = simg + M2;
  int* wbuf = occl + M2;
  double* act_peer = cluster.map_shared_rank(act, rank ^ 1);
  double* part_peer = cluster.map_shared_rank(part, rank ^ 1);

  const int G = a.cl.G;
  const int n_work = a.slot_item ? *a.slot_count
                                 : (a.cl.n_cfg_dev ? *a.cl.n_cfg_dev : a.cl.n_cfg) * G;
  const size_t conv_floats = (size_t)kRcC * 9 * kRcC;
  const int convs = 2 * a.blocks;
  const double inv_cn = 1.0 / (double)(kRcC * N), out_scale = trsqrt_eps((double)(a.blocks + 1), 0.0);
  const int co0 = 32 * rank + 2 * (lane & 3);  // this lane's channels: co0 + 8 nt, co0 + 8 nt + 1

  // Site tiles warp and warp + WARPS: this lane's row is site 8 tile + lane / 4.
  const int MT = (N + 7) >> 3;
  const int tiles = warp + WARPS < MT ? 2 : (warp < MT ? 1 : 0);
  int pad[2], site[2];
  bool live[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int st = 8 * (warp + i * WARPS) + (lane >> 2);
    live[i] = i < tiles && st < N;
    site[i] = live[i] ? st : 0;
    const int x = site[i] / Ly;
    pad[i] = (x + 1) * W + site[i] - x * Ly + 1;
  }
  int off[9];  // operand offsets of the nine groups of four k in 4 channels x 9 taps
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    const int k = 4 * j + (lane & 3), tap = k % 9;
    off[j] = (k / 9) * PS + (tap / 3) * W + tap % 3;
  }
  float pre[kRmPre];
  auto prefetch = [&](const float* w) {  // w: 36 k rows of 64 channels
#pragma unroll
    for (int q = 0; q < kRmPre; ++q) {
      const int i = tid + q * kRmThreads, ln = i & 31;
      if (i < kRmChunk)
        pre[q] = __ldg(w + (4 * (i >> 7) + (ln & 3)) * kRcC + 32 * rank + ((i >> 5) & 3) * 8 + (ln >> 2));
    }
  };
  // One convolution of the planes in act; acc starts from the bias.  next: the first chunk that
  // follows.
  auto conv = [&](double (&acc)[2][NT][2], const float* w, const float* bias, const float* next) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const double b0 = (double)__ldg(bias + co0 + 8 * nt), b1 = (double)__ldg(bias + co0 + 8 * nt + 1);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        acc[i][nt][0] = b0;
        acc[i][nt][1] = b1;
      }
    }
    const double* a0 = act + pad[0] - W - 1;
    const double* a1 = act + pad[1] - W - 1;
#pragma unroll 1
    for (int ch = 0; ch < kRcC / 4; ++ch) {
      double* buf = wsm + (ch & 1) * kRmChunk;
#pragma unroll
      for (int q = 0; q < kRmPre; ++q) {
        const int i = tid + q * kRmThreads;
        if (i < kRmChunk) buf[i] = (double)pre[q];
      }
      __syncthreads();
      prefetch(ch + 1 < kRcC / 4 ? w + (size_t)(ch + 1) * 36 * kRcC : next);
      const double* ws = buf + lane;
      if (tiles == 2) {
#pragma unroll
        for (int j = 0; j < 9; ++j) {
          const double x0 = a0[off[j]], x1 = a1[off[j]];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const double b = ws[(j * NT + nt) * 32];
            mma_f64(acc[0][nt], x0, b);
            mma_f64(acc[1][nt], x1, b);
          }
        }
      } else if (tiles == 1) {
#pragma unroll
        for (int j = 0; j < 9; ++j) {
          const double x0 = a0[off[j]];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma_f64(acc[0][nt], x0, ws[(j * NT + nt) * 32]);
        }
      }
      a0 += 4 * PS;
      a1 += 4 * PS;
    }
  };
  // This CTA's half of the new planes to both CTAs, then the borders of all planes.  Both CTAs have
  // finished reading the old planes before the call.
  auto publish = [&](auto value) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (live[i]) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int o = (co0 + 8 * nt + h) * PS + pad[i];
            const double v = value(i, nt, h);
            act[o] = v;
            act_peer[o] = v;
          }
      }
    cluster.sync();
    mma_halo<kRmThreads>(act, kRcC, PS, Lx, Ly);
    __syncthreads();
  };

  prefetch(a.wp);
  const int clusters = gridDim.x >> 1;
  for (int slot = blockIdx.x >> 1; slot < n_work; slot += clusters) {
    const int item = a.slot_item ? a.slot_item[slot] : slot;
    const int c = item / G, g = item - c * G;
    const int smp = a.cl.sample ? a.cl.sample[c] : c;
    const int fr = a.cl.from ? a.cl.from[c] : -1;
    const int to = a.cl.from ? a.cl.to[c] : -1;
    const int8_t* base = a.cl.spins + (int64_t)smp * M2;
    __syncthreads();  // the previous item's readers of simg are done
    for (int m = tid; m < M2; m += kRmThreads) {
      const int src = sym_map(m, g, Lx, Ly, N);  // image[m] = s[g(m)] (g is an involution)
      simg[m] = move_value(src, base[src], fr, to) > 0 ? 1 : -1;
    }
    __syncthreads();
    double x[2][NT][2], acc[2][NT][2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {  // occupation embedding
      const int occ = (simg[site[i]] > 0 ? 1 : 0) + (simg[N + site[i]] > 0 ? 2 : 0);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          x[i][nt][h] = live[i] ? (double)__ldg(a.embed + occ * kRcC + co0 + 8 * nt + h) : 0.0;
    }
    for (int blk = 0; blk < a.blocks; ++blk) {
      double ss = 0.0;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int h = 0; h < 2; ++h) ss = fma(x[i][nt][h], x[i][nt][h], ss);
#pragma unroll
      for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) red[warp] = ss;
      __syncthreads();
      if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < WARPS; ++w) t += red[w];
        part[rank] = t;
        part_peer[rank] = t;
      }
      cluster.sync();  // both sums known; both CTAs are done with the old planes
      const double r = trsqrt_eps((part[0] + part[1]) * inv_cn, kRmsEps);
      const float* w1 = a.wp + (size_t)(2 * blk) * conv_floats;
      const float* w2 = w1 + conv_floats;
      publish([&](int i, int nt, int h) { return gelu_tanh(x[i][nt][h] * r); });
      conv(acc, w1, a.b + (2 * blk) * kRcC, w2);
      cluster.sync();
      publish([&](int i, int nt, int h) { return gelu_tanh(acc[i][nt][h]); });
      conv(acc, w2, a.b + (2 * blk + 1) * kRcC, 2 * blk + 2 < convs ? w2 + conv_floats : a.wp);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int h = 0; h < 2; ++h) x[i][nt][h] = live[i] ? x[i][nt][h] + acc[i][nt][h] : 0.0;
    }
    cluster.sync();
    publish([&](int i, int nt, int h) { return x[i][nt][h] * out_scale; });
    if (rank == 0) {
      constexpr int d = kRcC / 2;
      auto feat = [&](int sg, int aa, int st) {
        const int px = st / Ly;
        return act[(sg * d + aa) * PS + (px + 1) * W + st - px * Ly + 1];
      };
      write_occupied_rows<double, decltype(feat), kRmThreads>(
          simg, occl, wbuf, N, a.n, d, g, Lx, Ly, a.Y + (int64_t)slot * a.n * d,
          a.idx + (int64_t)slot * a.n, a.item_sign + item, feat);
    }
  }
  cluster.sync();  // no CTA leaves while the other may still write to it
}

size_t rm_smem(int Lx, int Ly) {
  return sizeof(double) * ((size_t)kRcC * mma_plane(Lx, Ly) + 2 * kRmChunk) +
         sizeof(int) * (4 * (size_t)Lx * Ly + 4 * Lx + 32);
}

int launch_resconv_mma(const CnnLaunch& q, int N, cudaStream_t st) {
  const nh_backflow_params& p = *q.p;
  const int slots = q.slot_item ? q.max_slots : q.cl->n_cfg * q.cl->G;
  if (slots <= 0) return NH_OK;
  static const cudaError_t attr = cudaFuncSetAttribute(
      resconv_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
  if (attr != cudaSuccess) return check_cuda(attr, "resconv smem attribute");
  int grid = num_sms() & ~1;
  if (grid > 2 * slots) grid = 2 * slots;
  RcArgs<double> a{*q.cl, p.conv_w_packed, p.conv_w_packed + 4 * kRcC, p.conv_b, p.Lx, p.Ly, N,
                   p.layers, p.n_up + p.n_dn, q.mode, q.slot_item, q.slot_count, q.max_slots,
                   nullptr, static_cast<double*>(q.Y), q.idx, q.item_sign, nullptr};
  ProfScope prof_scope(NH_K_RESCONV64, st);
  resconv_mma_kernel<<<grid, kRmThreads, rm_smem(p.Lx, p.Ly), st>>>(a);
  return check_launch("resconv_mma_kernel");
}

// packed = [embed (4, C): [occ][co]] ++ per conv k [ci][tap][co];
// conv_w = [embed (C, 4)] ++ per conv k (C, C, 3, 3).
__global__ void resconv_pack_kernel(const float* __restrict__ w, int C, int convs,
                                    float* packed) {
  const int total = 4 * C + convs * 9 * C * C;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    if (i < 4 * C) {
      const int occ = i / C, co = i - occ * C;
      packed[i] = w[co * 4 + occ];
      continue;
    }
    const int r0 = i - 4 * C;
    const int k = r0 / (9 * C * C);
    const int r = r0 - k * 9 * C * C;  // (ci * 9 + tap) * C + co
    const int co = r % C;
    const int ct = r / C;
    packed[i] = w[4 * C + (size_t)k * 9 * C * C + co * 9 * C + ct];
  }
}

template <typename T, bool GACT>
size_t rc_smem(int N) {
  return sizeof(T) * ((GACT ? 0 : 3 * (size_t)kRcC * (N + 1)) + kRcChunkFloats + 8) +
         sizeof(int) * (4 * (size_t)N + 4 * 32 + 32);
}

constexpr int kRcBigPerSm = 2;  // CTAs per SM of the global-plane kernel (scratch bound)

template <typename T, bool GACT>
int launch_rc_t(const CnnLaunch& q, int N, cudaStream_t st) {
  const nh_backflow_params& p = *q.p;
  const size_t smem = rc_smem<T, GACT>(N);
  if (smem > 227 * 1024)
    return fail(NH_ERR_UNSUPPORTED, "resconv: N=%d needs %zu B of shared memory", N, smem);
  if (GACT && !q.act)
    return fail(NH_ERR_UNSUPPORTED, "resconv: N=%d needs the activation-plane scratch", N);
  const int slots = q.slot_item ? q.max_slots : q.cl->n_cfg * q.cl->G;
  if (slots <= 0) return NH_OK;
  int grid = num_sms() * (GACT ? kRcBigPerSm : 1);
  if (grid > slots) grid = slots;
  static size_t configured = 0;
  if (smem > 48 * 1024 && smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(resconv_kernel<T, GACT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return check_cuda(e, "resconv smem attribute");
    configured = smem;
  }
  RcArgs<T> a{*q.cl, p.conv_w_packed, p.conv_w_packed + 4 * kRcC, p.conv_b, p.Lx, p.Ly, N,
              p.layers, p.n_up + p.n_dn, q.mode, q.slot_item, q.slot_count, q.max_slots,
              q.feat, static_cast<T*>(q.Y), q.idx, q.item_sign, static_cast<T*>(q.act)};
  ProfScope prof_scope(sizeof(T) == 8 ? NH_K_RESCONV64 : NH_K_RESCONV, st);
  resconv_kernel<T, GACT><<<grid, kRcThreads, smem, st>>>(a);
  return check_launch(sizeof(T) == 8 ? "resconv_kernel<double>" : "resconv_kernel<float>");
}

}  // namespace

size_t resconv_packed_floats(int channels, int blocks) {
  return 4 * (size_t)channels + 2 * (size_t)blocks * 9 * channels * channels;
}

int launch_pack_resconv(const float* conv_w, int channels, int blocks, float* packed,
                        cudaStream_t st) {
  const int total = (int)resconv_packed_floats(channels, blocks);
  ProfScope prof_scope(NH_K_PACK, st);
  resconv_pack_kernel<<<(total + 255) / 256, 256, 0, st>>>(conv_w, channels, 2 * blocks,
                                                           packed);
  return check_launch("resconv_pack_kernel");
}

// FP32 keeps its planes in shared memory up to N = 256; FP64 and larger lattices use the
// per-CTA global planes.
size_t resconv_scratch_bytes(int N) {
  return (size_t)num_sms() * kRcBigPerSm * 3 * kRcC * (N + 1) * sizeof(double);
}

int launch_resconv(const CnnLaunch& q, cudaStream_t st) {
  const nh_backflow_params& p = *q.p;
  const int N = p.Lx * p.Ly;
  if (p.channels != kRcC || p.layers < 1 || N % 2 || N > kMaxN)
    return fail(NH_ERR_UNSUPPORTED, "resconv: channels %d (64), blocks %d, N %d", p.channels,
                p.layers, N);
  if (!p.conv_w_packed || !p.conv_b)
    return fail(NH_ERR_INVALID, "resconv: conv_w_packed (nh_pack_resconv_weights) or conv_b "
                "is null");
  if (reinterpret_cast<uintptr_t>(p.conv_w_packed) % 16)
    return fail(NH_ERR_INVALID, "resconv: conv_w_packed must be 16-byte aligned");
  if (q.fp64) {
    // two site tiles per warp of the 512-thread CTAs, planes in shared memory
    if (q.mode == 1 && N <= 16 * (kRmThreads / 32) && rm_smem(p.Lx, p.Ly) <= 226 * 1024)
      return launch_resconv_mma(q, N, st);
    return launch_rc_t<double, true>(q, N, st);
  }
  return rc_smem<float, false>(N) <= 227 * 1024 ? launch_rc_t<float, false>(q, N, st)
                                                 : launch_rc_t<float, true>(q, N, st);
}

}  // namespace nh
