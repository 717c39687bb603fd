// The backflow CNN of one item (configuration x symmetry image) by one block of 128 to 512 threads:
// the device function behind cnn_kernel (nh_cnn.cu) and the fused kernels that compute an item's
// features and consume them in the same block (the amplitude/Pfaffian kernel of the persistent
// local energy, nh_pfaffian.cu, and the FP64 refinement, nh_refine.cu).
//
// Periodic 3x3 convolutions (cross-correlation, code/backflow/models.py:163-167), tanh-GELU
// between layers, on the 2-channel +-1 occupation image of the item's configuration (sample s,
// optional move, image map g: image[m] = s'[g(m)], g an involution).  Activations are
// channel-major with row stride N + 1; each layer's weights are staged in the packed
// [ci][tap][co] layout.
#pragma once

#include "nh_common.cuh"

namespace nh {

__device__ __forceinline__ float gelu_tanh_dev(float x) {
  const float k0 = 0.7978845608028654f;  // sqrt(2 / pi)
  return 0.5f * x * (1.0f + tanhf(k0 * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ double gelu_tanh_dev(double x) {
  const double k0 = 0.7978845608028654;
  return 0.5 * x * (1.0 + tanh(k0 * (x + 0.044715 * x * x * x)));
}

__device__ __forceinline__ void cnn_lds8(const double* p, double* o) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double2 v = reinterpret_cast<const double2*>(p)[k];
    o[2 * k] = v.x;
    o[2 * k + 1] = v.y;
  }
}

// Pairs of FP32 values in one 64-bit register and the packed FMA d = a b + d: the FMA rate of two
// scalar ones (124 against 125 per clock and SM measured) in half the issue slots.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lo2(unsigned long long v) {
  return __uint_as_float((unsigned)v);
}
__device__ __forceinline__ float hi2(unsigned long long v) {
  return __uint_as_float((unsigned)(v >> 32));
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a,
                                     unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// count FP32 values (a multiple of 4) into 16-byte aligned shared memory, as asynchronous 16-byte
// copies where the source is aligned too; visible after the caller's barrier.
template <int TH>
__device__ __forceinline__ void stage_floats(float* dst, const float* src, int count) {
  if (reinterpret_cast<uintptr_t>(src) % 16 == 0) {
    for (int i = 4 * threadIdx.x; i < count; i += 4 * TH)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(dst + i)),
                   "l"(src + i)
                   : "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    for (int i = threadIdx.x; i < count; i += TH) dst[i] = __ldg(src + i);
  }
}

template <int S>
struct Sites {
  static constexpr int value = S;
};

// One task of a periodic 3x3 cross-correlation: S sites x 8 output channels (group grp of cout / 8)
// of cin planes of stride N + 1, weights [ci][tap][co] in shared memory, accumulated in order of
// (ci, tap) onto acc.  With four sites a thread issues 32 FMAs (16 packed) per 4 loads of inputs
// and two broadcast 16-byte weight loads (two cycles of the load port each).
template <typename T, int S>
__device__ __forceinline__ void conv_task(const T* in, int cin, int cout, const T* wsm, int grp,
                                          const int (&site)[S], int Lx, int Ly, T (&acc)[S][8]) {
  const int NS = Lx * Ly + 1;
  int row[S][3], col[S][3];
#pragma unroll
  for (int k = 0; k < S; ++k) {
    const int x = site[k] / Ly, y = site[k] - x * Ly;
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      int xx = x + u - 1, yy = y + u - 1;
      xx = xx < 0 ? xx + Lx : (xx >= Lx ? xx - Lx : xx);
      yy = yy < 0 ? yy + Ly : (yy >= Ly ? yy - Ly : yy);
      row[k][u] = xx * Ly;
      col[k][u] = yy;
    }
  }
  if constexpr (sizeof(T) == 4) {
    // FP32: the eight channels as four pairs (each half of a packed FMA rounds like a scalar one)
    unsigned long long a2[S][4];
#pragma unroll
    for (int k = 0; k < S; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) a2[k][j] = pack2(acc[k][2 * j], acc[k][2 * j + 1]);
#pragma unroll 1
    for (int ci = 0; ci < cin; ++ci) {
      const T* inc = in + ci * NS;
      const T* wc = wsm + ci * 9 * cout + grp * 8;
#pragma unroll
      for (int u = 0; u < 3; ++u) {
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          const ulonglong2* w2 = reinterpret_cast<const ulonglong2*>(wc + (u * 3 + v) * cout);
          const ulonglong2 wa = w2[0], wb = w2[1];
#pragma unroll
          for (int k = 0; k < S; ++k) {
            const float i0 = inc[row[k][u] + col[k][v]];
            const unsigned long long ii = pack2(i0, i0);
            fma2(a2[k][0], ii, wa.x);
            fma2(a2[k][1], ii, wa.y);
            fma2(a2[k][2], ii, wb.x);
            fma2(a2[k][3], ii, wb.y);
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < S; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[k][2 * j] = lo2(a2[k][j]);
        acc[k][2 * j + 1] = hi2(a2[k][j]);
      }
  } else {
#pragma unroll 1
    for (int ci = 0; ci < cin; ++ci) {
      const T* inc = in + ci * NS;
      const T* wc = wsm + ci * 9 * cout + grp * 8;
#pragma unroll
      for (int u = 0; u < 3; ++u) {
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          T w8[8];
          cnn_lds8(wc + (u * 3 + v) * cout, w8);
#pragma unroll
          for (int k = 0; k < S; ++k) {
            const T i0 = inc[row[k][u] + col[k][v]];
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[k][j] = fma(i0, w8[j], acc[k][j]);
          }
        }
      }
    }
  }
}

// Sites per task: four where that still gives every thread of a TH-thread block a task.
__device__ __forceinline__ bool conv_four_sites(int N, int cout, int TH) {
  return N % 4 == 0 && (cout / 8) * (N / 4) >= TH;
}

// Builds the item's image configuration in simg (2N ints, +-1) and runs the layers; returns the
// activation buffer (actA or actB) that holds the last layer's output, C planes of stride N + 1.
// wsm: C * C * 9 values, bsm: C values (shared memory); actA, actB: C (N + 1) values each
// (shared or per-block global memory).  Block-wide: every thread of the TH-thread block calls it.
template <typename T, int TH = kNumThreads>
__device__ T* cnn_layers(const float* __restrict__ wp, const float* __restrict__ bias, int Lx,
                         int Ly, int C, int layers, const int8_t* __restrict__ base, int fr,
                         int to, int g, T* actA, T* actB, T* wsm, T* bsm, int* simg) {
  const int tid = threadIdx.x;
  const int N = Lx * Ly, NS = N + 1, M2 = 2 * N;
  const int ngroups = C / 8;
  for (int m = tid; m < M2; m += TH) {
    const int src = sym_map(m, g, Lx, Ly, N);  // image[m] = s[g(m)] (g is an involution)
    const int v = move_value(src, base[src], fr, to);
    simg[m] = v > 0 ? 1 : -1;
    const int ch = m >= N ? 1 : 0;
    actA[ch * NS + (m - ch * N)] = v > 0 ? T(1) : T(-1);
  }
  T* in = actA;
  T* out = actB;
  int cin = 2;
  const float* wl = wp;
  for (int l = 0; l < layers; ++l) {
    __syncthreads();
    const int cnt = C * cin * 9;
    if constexpr (sizeof(T) == 4)
      stage_floats<TH>(wsm, wl, cnt);
    else
      for (int i = tid; i < cnt; i += TH) wsm[i] = T(__ldg(wl + i));
    for (int i = tid; i < C; i += TH) bsm[i] = T(__ldg(bias + l * C + i));
    __syncthreads();
    const bool act_fn = l < layers - 1;
    auto tasks = [&](auto sites) {
      constexpr int S = decltype(sites)::value;
      const int part = N / S;
      for (int task = tid; task < ngroups * part; task += TH) {
        const int grp = task / part;
        int site[S];
        T acc[S][8];
#pragma unroll
        for (int k = 0; k < S; ++k) {
          site[k] = task - grp * part + k * part;
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[k][j] = bsm[grp * 8 + j];
        }
        conv_task<T, S>(in, cin, C, wsm, grp, site, Lx, Ly, acc);
#pragma unroll
        for (int k = 0; k < S; ++k)
#pragma unroll
          for (int j = 0; j < 8; ++j)
            out[(grp * 8 + j) * NS + site[k]] = act_fn ? gelu_tanh_dev(acc[k][j]) : acc[k][j];
      }
    };
    if constexpr (sizeof(T) == 4) {
      if (conv_four_sites(N, C, TH))
        tasks(Sites<4>{});
      else if (ngroups * N <= TH)  // small lattices: every thread a task
        tasks(Sites<1>{});
      else
        tasks(Sites<2>{});
    } else {
      tasks(Sites<2>{});
    }
    wl += C * cin * 9;
    cin = C;
    T* t = in;
    in = out;
    out = t;
  }
  __syncthreads();
  return in;
}

// Shared-memory footprint of cnn_layers' staging (wsm + bsm) plus simg, occl (2N ints each) and
// the scan scratch of write_occupied_rows (4 Lx + 32 ints), without the activation planes.
template <typename T>
__host__ __device__ constexpr size_t cnn_item_scratch_bytes(int N, int C, int Lx) {
  return sizeof(T) * ((size_t)C * C * 9 + C) + sizeof(int) * (4 * (size_t)N + 4 * Lx + 32);
}

}  // namespace nh
