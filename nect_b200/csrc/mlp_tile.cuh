// fp32 tile products of the plain path's MLP: a block of NTH threads works on a
// tile of NT samples whose vectors are columns of [features][LD] arrays in
// shared memory (LD = NT + 4).
//
// A layer is a product out[o][t] = sum_k M[k][o] * in[k][t] with M [K][N]
// row-major.  A thread owns four consecutive samples and TO outputs: per k one
// 16-byte load of samples and TO weights feed 4 * TO multiply-adds (one sample a
// thread, with a 16-byte weight load for every four multiply-adds, was bound by
// the shared-memory pipe).  8 x 8 products a thread with half the threads
// measured the same: fewer loads a product, fewer warps for the gathers.  Every
// output sums over k in ascending order, one fused multiply-add at a time: the
// bits do not depend on the tiling.  Results stay in registers until the block
// has read the input, so a layer may overwrite it.
#pragma once
#include "hashgrid.cuh"
#include "mlp_simt.cuh"

namespace nectb {

template <int K, int N, int NT, int NTH>
struct TileProduct {
  static constexpr int LD = NT + 4;
  static constexpr int SG = NT / 4;                 // groups of four samples
  static constexpr int SW = SG / 8;                 // warps along the samples
  static constexpr int G = NTH / SG;                // output groups
  static_assert(SG % 8 == 0 && (NTH / 32) % SW == 0, "a warp holds 8 sample groups by 4 output groups");
  static constexpr int kPer = (N + G - 1) / G;
  static constexpr int TO = kPer <= 2 ? 2 : (kPer <= 4 ? 4 : 8);   // outputs of a thread
  static_assert(kPer <= 8 && N % TO == 0 && N % 4 == 0, "output tile");
  float acc[TO][4];

  __device__ __forceinline__ int sample() const {
    return (int)((threadIdx.x / 32) % SW * 8 + threadIdx.x % 8) * 4;
  }
  __device__ __forceinline__ int output() const {
    return (int)((threadIdx.x / 32) / SW * 4 + threadIdx.x / 8 % 4) * TO;
  }
  __device__ __forceinline__ bool active() const { return G * TO == N || output() < N; }

  __device__ __forceinline__ void run(const float* __restrict__ M, const float* __restrict__ in) {
#pragma unroll
    for (int o = 0; o < TO; ++o)
#pragma unroll
      for (int s = 0; s < 4; ++s) acc[o][s] = 0.f;
    if (!active()) return;
    const float* x = in + sample();
    const float* m = M + output();
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
      const float4 v = *reinterpret_cast<const float4*>(x + k * LD);
      float w[TO];
      if constexpr (TO == 2) {
        const float2 q = *reinterpret_cast<const float2*>(m + k * N);
        w[0] = q.x, w[1] = q.y;
      } else {
#pragma unroll
        for (int o = 0; o < TO; o += 4) {
          const float4 q = *reinterpret_cast<const float4*>(m + k * N + o);
          w[o] = q.x, w[o + 1] = q.y, w[o + 2] = q.z, w[o + 3] = q.w;
        }
      }
#pragma unroll
      for (int o = 0; o < TO; ++o) {
        acc[o][0] = fmaf(w[o], v.x, acc[o][0]);
        acc[o][1] = fmaf(w[o], v.y, acc[o][1]);
        acc[o][2] = fmaf(w[o], v.z, acc[o][2]);
        acc[o][3] = fmaf(w[o], v.w, acc[o][3]);
      }
    }
  }

  // out[o][t] = f(acc, o, t) for the thread's outputs and samples (f takes the
  // value, the output and the offset o * LD + t).
  template <typename Fn>
  __device__ __forceinline__ void store(float* __restrict__ out, Fn&& f) const {
    if (!active()) return;
#pragma unroll
    for (int o = 0; o < TO; ++o) {
      const int at = (output() + o) * LD + sample();
      *reinterpret_cast<float4*>(out + at) =
          make_float4(f(acc[o][0], at), f(acc[o][1], at + 1), f(acc[o][2], at + 2), f(acc[o][3], at + 3));
    }
  }
};

// Encodes the tile's points (coordinates px[k * NT + t], `valid[t]` non-zero
// where there is a point) into sX [L * F][LD]; the levels of a sample are dealt
// to NTH / NT threads.  Other columns are zero.
template <int D, int F, int L, int NT, int NTH, typename T>
__device__ __forceinline__ void encode_tile(const GridDev& g, const T* __restrict__ table, const float* sP,
                                            const int* sValid, float tval, float* __restrict__ sX) {
  constexpr int LD = NT + 4, P = NTH / NT;
  const int t = threadIdx.x % NT;
  const bool valid = sValid[t] != 0;
  const float x[4] = {sP[t], sP[NT + t], sP[2 * NT + t], tval};
#pragma unroll 2   // two levels' gathers in flight
  for (int l = threadIdx.x / NT; l < L; l += P) {
    float acc[F];
#pragma unroll
    for (int f = 0; f < F; ++f) acc[f] = 0.f;
    if (valid) encode_level<D, F, T>(g, table, l, x, acc);
#pragma unroll
    for (int f = 0; f < F; ++f) sX[(l * F + f) * LD + t] = acc[f];
  }
}

// The hidden layers of a tile: sX [IN][LD] -> out, the last layer's activations
// (the layers between overwrite each other in out).  Ends without a barrier.
template <int IN, int H, int NT, int NTH>
__device__ __forceinline__ void tile_hidden(const SimtWeights& sw, const float* sX, float* out, int act) {
  {
    TileProduct<IN, kWidth, NT, NTH> p;
    p.run(sw.WT[0], sX);
    __syncthreads();   // out may be sX
    p.store(out, [&](float v, int) { return act_fwd(v, act); });
  }
#pragma unroll 1
  for (int k = 1; k < H; ++k) {
    __syncthreads();
    TileProduct<kWidth, kWidth, NT, NTH> p;
    p.run(sw.WT[0] + IN * kWidth + (k - 1) * kWidth * kWidth, out);
    __syncthreads();
    p.store(out, [&](float v, int) { return act_fwd(v, act); });
  }
}

// dW[j][i] += sum_t G[j][t] * A[i][t] over the tile's samples, G [64][LD], A
// [K][LD].  Thread (jb, ib) owns rows jb + 16 a and columns ib + CB b (CB = NTH /
// 16), so that neighbouring lanes read neighbouring rows, four banks apart.
template <int K, int NT, int NTH>
struct TileWGrad {
  static constexpr int LD = NT + 4;
  static constexpr int CB = NTH / 16;
  static constexpr int IB = (K + CB - 1) / CB;
  float acc[4][IB];
  static __device__ __forceinline__ bool has(int b) { return K % CB == 0 || (int)(threadIdx.x % CB) + CB * b < K; }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < IB; ++b) acc[a][b] = 0.f;
  }
  __device__ __forceinline__ void add(const float* __restrict__ G, const float* __restrict__ A) {
    const float* g0 = G + (threadIdx.x / CB) * LD;
    const float* a0 = A + (threadIdx.x % CB) * LD;
#pragma unroll 1
    for (int t = 0; t < NT; t += 4) {
      float4 g[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) g[a] = *reinterpret_cast<const float4*>(g0 + 16 * a * LD + t);
#pragma unroll
      for (int b = 0; b < IB; ++b) {
        const float4 v = has(b) ? *reinterpret_cast<const float4*>(a0 + CB * b * LD + t) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          acc[a][b] = fmaf(g[a].x, v.x, acc[a][b]);
          acc[a][b] = fmaf(g[a].y, v.y, acc[a][b]);
          acc[a][b] = fmaf(g[a].z, v.z, acc[a][b]);
          acc[a][b] = fmaf(g[a].w, v.w, acc[a][b]);
        }
      }
    }
  }
  __device__ __forceinline__ void flush(float* __restrict__ dst) const {  // dst [64][K]
    const int jb = threadIdx.x / CB, ib = threadIdx.x % CB;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < IB; ++b)
        if (has(b)) atomicAdd(dst + (jb + 16 * a) * K + ib + CB * b, acc[a][b]);
  }
};

// A tile of NT samples: coordinates, validity, dL/dsigma (then dL/dz), in front
// of the columns.
template <int NT>
struct TilePoints {
  float p[3 * NT];
  float d[NT];
  int valid[NT];
};

// Threads of the forward kernels, on tiles of 128 samples.
constexpr int kTileThreads = 256;

// Shared memory of the forward kernels: WT copies and w_out, the points, one
// column buffer that the layers overwrite.
template <int IN, int H, int NT>
__host__ __device__ constexpr size_t tile_forward_smem() {
  return (size_t)simt_weight_floats<IN, H, false>() * 4 + sizeof(TilePoints<NT>) +
         (size_t)(IN > kWidth ? IN : kWidth) * (NT + 4) * 4;
}

}  // namespace nectb
