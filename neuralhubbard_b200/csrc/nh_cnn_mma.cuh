// The FP64 backflow CNN of one item on the FP64 tensor-core instruction (mma m8n8k4): the device
// function behind the FP64 cnn_kernel (nh_cnn.cu) and the refinement kernel's in-kernel features
// (nh_refine.cu).
//
// Each layer is an implicit GEMM: M = lattice sites (tiles of 8 consecutive sites), N = output
// channels, K = 9 ci + tap in ascending groups of four.  The instruction chains its four products
// onto the accumulator as FMAs in ascending k (checked against that chain on random operands), so
// the sums are those of the scalar loop, bit for bit.  Activations sit in one set of padded
// planes, (Lx + 2) x (Ly + 2) doubles with the border holding the periodic neighbours, so that a
// lane's nine operand offsets (4 channels x 9 taps = 9 groups of four) are constants; the plane
// stride is 4 mod 16 doubles, which keeps the half-warp's rows of different channels apart.
// Weights are staged in B-fragment order ([k / 4][co / 8][lane]), the next layer's while the
// current one runs.  A warp owns whole site tiles (at most two) times all channels, so every
// output of a layer stays in registers until all inputs have been read and one set of planes is
// enough.
//
// The instruction runs at the DFMA rate (64 FMA per clock and SM, measured), so the gain over
// scalar code is in operand traffic: a warp loads 6 operands per 8 MMAs of 256 FMA where the
// scalar loop loads 6 per 16 FMA and thread.  Measured at 16x16, 19,091 images: 15.0 ms scalar,
// 9.96 ms here (the FMA floor is 8.0 ms).
#pragma once

#include "nh_cnn_item.cuh"
#include "nh_common.cuh"

namespace nh {

// Doubles per padded plane: the smallest stride >= (Lx + 2)(Ly + 2) that is 4 mod 16.
__host__ __device__ __forceinline__ int mma_plane(int Lx, int Ly) {
  const int s = (Lx + 2) * (Ly + 2);
  return s + ((20 - s % 16) % 16);
}

// Shared doubles: planes and one layer's weight fragments.
__host__ __device__ __forceinline__ size_t cnn_mma_doubles(int Lx, int Ly, int C) {
  return (size_t)C * mma_plane(Lx, Ly) + 9 * (size_t)C * C;
}

// Lattice and width the MMA form covers with TH threads: two site tiles per warp, 32 channels.
__host__ __device__ __forceinline__ bool cnn_mma_fits(int Lx, int Ly, int C, int TH) {
  return C == 32 && Lx * Ly <= 16 * (TH / 32);
}

__device__ __forceinline__ void mma_f64(double* c, double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// Border cells of `planes` planes from their periodic interior cells: a lane works out a cell once
// and copies it in the planes of its warp.
template <int TH>
__device__ __forceinline__ void mma_halo(double* act, int planes, int PS, int Lx, int Ly) {
  const int W = Ly + 2, H = 2 * W + 2 * Lx;
  for (int h = threadIdx.x & 31; h < H; h += 32) {
    int x, y;  // padded coordinates of the border cell
    if (h < 2 * W) {
      x = h < W ? 0 : Lx + 1;
      y = h < W ? h : h - W;
    } else {
      x = 1 + ((h - 2 * W) >> 1);
      y = ((h - 2 * W) & 1) ? Ly + 1 : 0;
    }
    const int sx = x == 0 ? Lx : (x == Lx + 1 ? 1 : x);
    const int sy = y == 0 ? Ly : (y == Ly + 1 ? 1 : y);
    double* dst = act + x * W + y;
    const double* src = act + sx * W + sy;
    for (int c = threadIdx.x >> 5; c < planes; c += TH / 32) dst[c * PS] = src[c * PS];
  }
}

// Runs the layers on the item's image configuration (as cnn_layers) and leaves the last layer's
// output in act: channel c at padded site p is act[c * PS + p], PS = mma_plane(Lx, Ly), site
// (x, y) at p = (x + 1)(Ly + 2) + y + 1.  act: C * PS doubles; wsm: 9 C C doubles; simg: 2N ints.
// C = 8 NT.  Block-wide (TH threads); cnn_mma_fits must hold.
template <int NT, int TH>
__device__ void cnn_layers_mma(const float* __restrict__ wp, const float* __restrict__ bias, int Lx,
                               int Ly, int layers, const int8_t* __restrict__ base, int fr, int to,
                               int g, double* act, double* wsm, int* simg) {
  constexpr int C = 8 * NT, KC = C / 4;          // channel groups of a full layer
  constexpr int WARPS = TH / 32;
  constexpr int WREG = (9 * C * C + TH - 1) / TH;  // staged weights per thread
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = Lx * Ly, M2 = 2 * N, W = Ly + 2, PS = mma_plane(Lx, Ly);
  const int MT = (N + 7) >> 3;

  // Weight fragment i of a layer with K rows (packed [k][co]): lane's B[k][co], FP32 in memory.
  auto frag = [&](const float* wl, int K, int i) -> float {
    const int ln = i & 31, nt = (i >> 5) % NT, k = (i >> 5) / NT * 4 + (ln & 3);
    return k < K ? __ldg(wl + k * C + nt * 8 + (ln >> 2)) : 0.0f;
  };

  for (int m = tid; m < M2; m += TH) {
    const int src = sym_map(m, g, Lx, Ly, N);  // image[m] = s[g(m)] (g is an involution)
    const int v = move_value(src, base[src], fr, to) > 0 ? 1 : -1;
    simg[m] = v;
    const int ch = m >= N ? 1 : 0, site = m - ch * N, x = site / Ly;
    act[ch * PS + (x + 1) * W + site - x * Ly + 1] = (double)v;
  }
  for (int i = tid; i < 5 * NT * 32; i += TH) wsm[i] = (double)frag(wp, 18, i);
  __syncthreads();
  mma_halo<TH>(act, 2, PS, Lx, Ly);
  __syncthreads();

  // Site tiles warp and warp + WARPS: this lane's A / C row is site 8 tile + lane / 4 (rows past
  // the lattice read site 0 and are not stored).
  int pad[2];
  bool live[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int s = 8 * (warp + i * WARPS) + (lane >> 2);
    live[i] = s < N;
    const int ss = live[i] ? s : 0, x = ss / Ly;
    pad[i] = (x + 1) * W + ss - x * Ly + 1;
  }
  const int tiles = warp + WARPS < MT ? 2 : (warp < MT ? 1 : 0);
  const int co0 = 2 * (lane & 3);
  // Operand offsets of the nine groups of four k in 4 channels x 9 taps.
  int off[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    const int k = 4 * j + (lane & 3), tap = k % 9;
    off[j] = (k / 9) * PS + (tap / 3) * W + tap % 3;
  }

  const float* wl = wp;
  int cin = 2;
  for (int l = 0; l < layers; ++l) {
    const float* wn = wl + C * cin * 9;  // next layer's weights
    const bool more = l + 1 < layers;
    float wreg[WREG];
    if (more) {
#pragma unroll
      for (int r = 0; r < WREG; ++r) {
        const int i = tid + r * TH;
        wreg[r] = i < 9 * C * C ? frag(wn, 9 * C, i) : 0.0f;
      }
    }
    double acc[2][NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const double b0 = (double)__ldg(bias + l * C + nt * 8 + co0);
      const double b1 = (double)__ldg(bias + l * C + nt * 8 + co0 + 1);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        acc[i][nt][0] = b0;
        acc[i][nt][1] = b1;
      }
    }
    const double* ws = wsm + lane;
    const double* a0 = act + pad[0] - W - 1;
    const double* a1 = act + pad[1] - W - 1;
    auto group = [&](int o, const double* w, bool two) {
      const double x0 = a0[o], x1 = two ? a1[o] : 0.0;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const double b = w[nt * 32];
        mma_f64(acc[0][nt], x0, b);
        if (two) mma_f64(acc[1][nt], x1, b);
      }
    };
    auto layer = [&](bool two) {
      if (l == 0) {  // K = 18: the last group's two extra k have zero weights
#pragma unroll
        for (int j = 0; j < 5; ++j)
          group(j == 4 && (lane & 2) ? 0 : off[j], ws + j * NT * 32, two);
      } else {
#pragma unroll 1
        for (int kc = 0; kc < KC; ++kc) {
#pragma unroll
          for (int j = 0; j < 9; ++j) group(off[j], ws + j * NT * 32, two);
          ws += 9 * NT * 32;
          a0 += 4 * PS;
          a1 += 4 * PS;
        }
      }
    };
    if (tiles == 2)
      layer(true);
    else if (tiles == 1)
      layer(false);
    __syncthreads();  // every input and weight of this layer has been read
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (i < tiles && live[i]) {
        double* dst = act + co0 * PS + pad[i];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          dst[nt * 8 * PS] = more ? gelu_tanh_dev(acc[i][nt][0]) : acc[i][nt][0];
          dst[(nt * 8 + 1) * PS] = more ? gelu_tanh_dev(acc[i][nt][1]) : acc[i][nt][1];
        }
      }
    if (more) {
#pragma unroll
      for (int r = 0; r < WREG; ++r) {
        const int i = tid + r * TH;
        if (i < 9 * C * C) wsm[i] = (double)wreg[r];
      }
    }
    __syncthreads();
    if (more) {
      mma_halo<TH>(act, C, PS, Lx, Ly);
      __syncthreads();
    }
    wl = wn;
    cin = C;
  }
}

}  // namespace nh
