// Pieces shared by the tensor-core (tcgen05) kernels of training and
// queries: the swizzled operand tiles, the staging of the weights as bf16
// tiles, the encoder's row writer and the hidden activations.
//
// The MLP input row of L levels x F features holds IN = L * F values padded
// with zeros to INP (a multiple of the MMA's K step of 16), split over KT
// tiles of 64 columns (InShape in common.cuh).  Weight tiles: W0 as KT tiles
// [64 outputs][64 inputs], then one [64][64] tile per further hidden layer;
// w_out stays fp32.
#pragma once
#include <cuda_fp16.h>
#include <type_traits>

#include "common.cuh"
#include "hashgrid.cuh"
#include "mlp_simt.cuh"
#include "tcgen05.cuh"

namespace nectb {

constexpr uint32_t kTile = 128 * 128;  // bytes of a [128][64 bf16] tile
constexpr uint32_t kWTile = 64 * 128;  // bytes of a [64][64 bf16] tile

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

// TMEM columns of a block of n_wg warpgroups: 64 each, allocated as a power of two.
__host__ __device__ constexpr uint32_t wg_tmem_cols(int n_wg) {
  return n_wg <= 1 ? 64u : (n_wg == 2 ? 128u : (n_wg <= 4 ? 256u : 512u));
}

// Barrier over the 128 threads of warpgroup wg (named barrier wg + 1; 0 is
// __syncthreads'), and its OR-reduction form.
__device__ __forceinline__ void wg_sync(int wg) { asm volatile("bar.sync %0, 128;" ::"r"(wg + 1) : "memory"); }
__device__ __forceinline__ bool wg_or(int wg, bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred pi, po;\n\t"
      "setp.ne.u32 pi, %1, 0;\n\t"
      "bar.red.or.pred po, %2, 128, pi;\n\t"
      "selp.u32 %0, 1, 0, po;\n\t}\n"
      : "=r"(r)
      : "r"((uint32_t)p), "r"(wg + 1)
      : "memory");
  return r != 0;
}

// fp32 weights (PyTorch layout) -> bf16 swizzled tiles: W0 rows o over KT
// tiles (input columns beyond IN are zero), W1..W_{H-1} rows o in the tiles
// after them; w_out fp32.
template <int L, int F, int H>
__device__ __forceinline__ void stage_mixed_weights(const float* __restrict__ W, uint8_t* sW, float* sWout) {
  using S = InShape<L, F>;
  constexpr int IN = S::IN;
  for (int e = threadIdx.x; e < 64 * S::KT * 8; e += blockDim.x) {
    const int o = e / (S::KT * 8), j = e % (S::KT * 8);
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = (8 * j + q < IN) ? W[o * IN + 8 * j + q] : 0.f;
    tc::st_chunk_bf16(sW + (j / 8) * kWTile, o, j % 8, v);
  }
#pragma unroll 1
  for (int k = 1; k < H; ++k) {
    const float* Wk = W + 64 * IN + (k - 1) * 64 * 64;
    for (int e = threadIdx.x; e < 64 * 8; e += blockDim.x) {
      const int o = e / 8, j = e % 8;
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = Wk[o * 64 + 8 * j + q];
      tc::st_chunk_bf16(sW + (S::KT + k - 1) * kWTile, o, j, v);
    }
  }
  for (int e = threadIdx.x; e < 64; e += blockDim.x) sWout[e] = W[64 * IN + (H - 1) * 64 * 64 + e];
}

// Hidden activation of the tensor-core paths (ReLU, LeakyReLU or none; the
// shapes validate_mlp accepts) and its derivative from the sign of the
// pre-activation.
__device__ __forceinline__ float hidden_act(float x, int act) {
  return act == NECTB_ACT_RELU ? fmaxf(x, 0.f) : (act == NECTB_ACT_LEAKY_RELU ? (x > 0.f ? x : 0.01f * x) : x);
}
// g times the activation's slope at a pre-activation of the given sign.
__device__ __forceinline__ float hidden_grad(float g, bool positive, int act) {
  return act == NECTB_ACT_RELU ? (positive ? g : 0.f) : (act == NECTB_ACT_LEAKY_RELU ? (positive ? g : 0.01f * g) : g);
}

// Activation of 64 accumulator values into row r of a bf16 tile; bit j of m = (x_j > 0).
__device__ __forceinline__ void act_row(const float* h, uint8_t* tile, int r, int act, uint32_t& mlo, uint32_t& mhi) {
  mlo = 0;
  mhi = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float x = h[8 * j + q];
      v[q] = hidden_act(x, act);
      const uint32_t bit = x > 0.f ? 1u : 0u;
      if (8 * j + q < 32) mlo |= bit << (8 * j + q); else mhi |= bit << (8 * j + q - 32);
    }
    tc::st_chunk_bf16(tile, r, j, v);
  }
}

// The raw corner entries of one level at p and the
// fractions along the axes: the integers and fractions of level_corners, with the
// index rule of the level (hash or strides) taken by one uniform branch instead of
// a select per corner, and 32-bit entry offsets from the level's base.
template <int D, int F>
struct LevelFetch {
  using Raw = std::conditional_t<F == 2, unsigned int, uint2>;   // an entry: F fp16 features
  Raw raw[1 << D];
  float f[D];

  __device__ __forceinline__ void load(const GridDev& g, const __half* __restrict__ table, int l, const float* p) {
    uint32_t c[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      const uint32_t res = (uint32_t)g.res[l][k];
      const float q = __fmul_rn(p[k], (float)res);   // as level_corners
      // clamp(floor(q), 0, res - 1): the conversion truncates and takes what is below 0
      // (a t the caller passed as it was) to 0, so the lower end costs nothing
      c[k] = min(__float2uint_rz(q), res - 1u);
      f[k] = q - (float)c[k];
    }
    uint32_t idx[1 << D];
    const bool hashed = (g.hashed_bits >> l) & 1u;
    if (hashed) {
      const uint32_t m = g.hash_mask;
      const uint32_t t1[2] = {c[1] * kPrime1, c[1] * kPrime1 + kPrime1};
      const uint32_t t2[2] = {c[2] * kPrime2, c[2] * kPrime2 + kPrime2};
      uint32_t row[1 << (D - 1)];
#pragma unroll
      for (int r = 0; r < 4; ++r) row[r] = t1[r & 1] ^ t2[r >> 1];
      if constexpr (D == 4) {
        const uint32_t t3[2] = {c[3] * kPrime3, c[3] * kPrime3 + kPrime3};
#pragma unroll
        for (int r = 4; r < 8; ++r) row[r] = row[r - 4] ^ t3[1];
#pragma unroll
        for (int r = 0; r < 4; ++r) row[r] ^= t3[0];
      }
#pragma unroll
      for (int i = 0; i < (1 << D); ++i) idx[i] = ((c[0] + (i & 1)) ^ row[i >> 1]) & m;
    } else {
      uint32_t row[1 << (D - 1)];
      const uint32_t base = c[0] + c[1] * g.stride[l][1] + c[2] * g.stride[l][2] +
                            (D == 4 ? c[D - 1] * g.stride[l][3] : 0u);
#pragma unroll
      for (int r = 0; r < (1 << (D - 1)); ++r) {
        row[r] = base;
#pragma unroll
        for (int k = 1; k < D; ++k)
          if ((r >> (k - 1)) & 1) row[r] += g.stride[l][k];
      }
#pragma unroll
      for (int i = 0; i < (1 << D); ++i) idx[i] = row[i >> 1] + (i & 1);
    }
    // the odd hashed levels' corners through the texture path (a second L1 data
    // pipe beside the load/store unit's), the others as loads
    if (g.tex && hashed && (l & 1)) {
      const int off = (int)g.offset[l];
#pragma unroll
      for (int i = 0; i < (1 << D); ++i) raw[i] = tex1Dfetch<Raw>((cudaTextureObject_t)g.tex, off + (int)idx[i]);
    } else {
      const Raw* at = reinterpret_cast<const Raw*>(table) + g.offset[l];
#pragma unroll
      for (int i = 0; i < (1 << D); ++i) raw[i] = __ldg(at + idx[i]);
    }
  }

  // The level's F features (fused multiply-adds over the corners in order).
  __device__ __forceinline__ void blend(float* out) const {
    float w01[4], wt[D][2];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      wt[k][0] = 1.f - f[k];
      wt[k][1] = f[k];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) w01[q] = wt[0][q & 1] * wt[1][q >> 1];
    float acc[F];
#pragma unroll
    for (int k = 0; k < F; ++k) acc[k] = 0.f;
#pragma unroll
    for (int i = 0; i < (1 << D); ++i) {
      float w = w01[i & 3];
#pragma unroll
      for (int k = 2; k < D; ++k) w = w * wt[k][(i >> k) & 1];
      if constexpr (F == 2) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&raw[i]));
        acc[0] = fmaf(w, v.x, acc[0]);
        acc[1] = fmaf(w, v.y, acc[1]);
      } else {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw[i].x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&raw[i].y));
        acc[0] = fmaf(w, a.x, acc[0]);
        acc[1] = fmaf(w, a.y, acc[1]);
        acc[2] = fmaf(w, b.x, acc[2]);
        acc[3] = fmaf(w, b.y, acc[3]);
      }
    }
#pragma unroll
    for (int k = 0; k < F; ++k) out[k] = acc[k];
  }
};

// Encodes one sample into row r of the swizzled X tiles (bf16), 8 features
// (one 16-byte chunk) at a time, the padding after the last level zero;
// invalid samples write zeros.  The
// corners of two levels of 2 features are fetched before the first is blended (four
// spill at 80 registers: 512 x 512 rays x 512 samples 38.1 ms a step, two 37.7, one
// 38.4), one level of 4 features (two spill in the deep model).
template <int D, int F, int L>
__device__ __forceinline__ void encode_row(const GridDev& g, const __half* __restrict__ table, const float* p,
                                           bool valid, uint8_t* sX, int r) {
  using S = InShape<L, F>;
  constexpr int LPC = 8 / F;  // levels per 16-byte chunk
  constexpr int kGroup = F == 2 ? 2 : 1;   // levels in flight
#pragma unroll 1
  for (int j = 0; j < S::NCH; ++j) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = 0.f;
    if (valid) {
#pragma unroll
      for (int q = 0; q < LPC; q += kGroup) {
        LevelFetch<D, F> lv[kGroup];
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
          const int l = j * LPC + q + k;
          if (L % LPC == 0 || l < L) lv[k].load(g, table, l, p);
        }
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
          const int l = j * LPC + q + k;   // (an odd last level leaves a chunk's second half zero)
          if (L % LPC == 0 || l < L) lv[k].blend(v + (q + k) * F);
        }
      }
    }
    tc::st_chunk_bf16(sX + (j / 8) * kTile, r, j % 8, v);
  }
}

// Copies the warp's 32 encoded rows (rows row0.. of the X tiles) to the encoding
// store, lane r's to row `to` of it (none: kNoRow), evict-first: the store streams
// past the L2 that holds the tables.  Consecutive lanes write consecutive chunks
// of a row: whole sectors, where a lane writing its own row fills half a sector
// at a time.
constexpr uint32_t kNoRow = 0xffffffffu;
template <int L, int F>
__device__ __forceinline__ void store_rows(const uint8_t* sX, int row0, uint32_t to, uint4* __restrict__ xstore) {
  constexpr int NCH = InShape<L, F>::NCH;
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int k = 0; k < NCH; ++k) {
    const int e = 32 * k + lane, row = e / NCH, j = e % NCH;
    const uint32_t dst = __shfl_sync(0xffffffffu, to, row);
    if (dst != kNoRow)
      __stcs(xstore + (size_t)dst * NCH + j,
             *reinterpret_cast<const uint4*>(sX + (j / 8) * kTile + tc::sw128(row0 + row, j % 8)));
  }
  __syncwarp();
}

// Loads 64 fp32 TMEM columns [col, col+64) of this thread's lane.
__device__ __forceinline__ void ld64(uint32_t taddr, float* v) {
#pragma unroll
  for (int c = 0; c < 4; ++c) tc::tmem_ld16(taddr + 16 * c, v + 16 * c);
  tc::tmem_wait_ld();
}

}  // namespace nectb
