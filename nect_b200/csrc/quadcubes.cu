// QuadCubes' composite encoding (nect/network/networks.py:392-449): four 3D
// grids of one configuration over (z, y, x), (y, x, t), (x, z, t) and
// (z, y, t) of each point, with one t for every point of a call, written as
// rows of the MLP's input matrix, and its backward.
//
// Planes.  Three of the grids have t as their last coordinate.  With t fixed,
// a level's trilinear interpolation over (a, b, t) is a bilinear
// interpolation over (a, b) of the blend w0 * v(a, b, t0) + w1 * v(a, b, t0+1)
// (weights and t0 as level_corners computes them for axis 2).  Per call and
// grid the blend is built once into a plane: a dense 2D array of the level's
// (res+1)^2 vertices where that fits in T entries, else (hashed levels) the
// T entries keyed by the (a, b) part of the hash, which is an XOR of per-axis
// terms, so v(a, b, t_v) sits at (key ^ (t_v * pi_2)) & mask.  The grids then
// gather 4 corners from a plane a few tens of MB in size (L2-resident)
// instead of 8 corners spread over a table of up to 2^23 entries per level.
// In the backward the points reduce into a plane-shaped fp32 gradient
// (L2-resident), which is spread to the two time vertices of each of its
// non-zero entries.  Results equal the 3D grid's up to fp32 reassociation
// (fp32 planes) or one fp16 rounding of the blended values (fp16 planes, the
// mixed path, whose MLP then rounds to bf16).
#include <algorithm>
#include <cmath>
#include <cuda_bf16.h>
#include <type_traits>

#include "common.cuh"
#include "hashgrid.cuh"

namespace nectb {
namespace {

struct Plane {
  int n_levels;
  uint32_t hash_mask;
  uint32_t hashed3;   // bit l: the 3D level is hashed
  uint32_t hashed2;   // bit l: the plane level keeps the T hashed entries
  int res[NECTB_MAX_LEVELS];
  int64_t stride2[NECTB_MAX_LEVELS];   // dense 3D stride of the t axis, (res+1)^2
  int64_t off3[NECTB_MAX_LEVELS];      // 3D level offsets (entries)
  int64_t off2[NECTB_MAX_LEVELS];      // plane level offsets (entries)
  int64_t n2[NECTB_MAX_LEVELS];        // plane entries that hold a value
  int64_t total2;
};

bool make_plane(const GridDev& g, Plane* p) {
  if (g.n_dims != 3) return false;
  p->n_levels = g.n_levels;
  p->hash_mask = g.hash_mask;
  p->hashed3 = g.hashed_bits;
  p->hashed2 = 0;
  const int64_t T = (int64_t)g.hash_mask + 1;
  int64_t off = 0;
  for (int l = 0; l < g.n_levels; ++l) {
    const int r = g.res[l][0];
    if (g.res[l][1] != r || g.res[l][2] != r) return false;
    const int64_t v2 = (int64_t)(r + 1) * (r + 1);
    p->res[l] = r;
    p->stride2[l] = v2;
    p->off3[l] = g.offset[l];
    p->off2[l] = off;
    if (v2 <= T) {
      p->n2[l] = v2;
    } else {
      p->n2[l] = T;
      p->hashed2 |= 1u << l;
    }
    off += (p->n2[l] + 7) / 8 * 8;
  }
  p->total2 = off;
  return true;
}

// t -> lower time vertex and its weights, as level_corners computes them.
struct TimeVertex {
  int c;
  float w0, w1;
};
__device__ __forceinline__ TimeVertex time_vertex(float t, int r) {
  const float p = __fmul_rn(t, (float)r);   // rounded product, as level_corners
  int ci = (int)floorf(p);
  ci = ci < 0 ? 0 : (ci > r - 1 ? r - 1 : ci);
  const float f = p - (float)ci;
  return {ci, 1.f - f, f};
}

// The two 3D entries (within the level) of plane entry k at time vertices
// c and c + 1.
__device__ __forceinline__ void plane_sources(const Plane& s, int l, int64_t k, int c, int64_t* e0, int64_t* e1) {
  const uint32_t tt = (uint32_t)c * kPrime2;
  if ((s.hashed2 >> l) & 1u) {
    *e0 = (int64_t)((uint64_t)k ^ (uint64_t)(tt & s.hash_mask));
    *e1 = (int64_t)((uint64_t)k ^ (uint64_t)((tt + kPrime2) & s.hash_mask));
  } else if ((s.hashed3 >> l) & 1u) {
    const uint32_t r1 = (uint32_t)s.res[l] + 1u;
    const uint32_t a = (uint32_t)(k % r1), b = (uint32_t)(k / r1);
    const uint32_t h = a ^ (b * kPrime1);
    *e0 = (int64_t)((h ^ tt) & s.hash_mask);
    *e1 = (int64_t)((h ^ (tt + kPrime2)) & s.hash_mask);
  } else {
    *e0 = k + (int64_t)c * s.stride2[l];
    *e1 = *e0 + s.stride2[l];
  }
}

template <typename T>
__device__ __forceinline__ T from_float(float v);
template <>
__device__ __forceinline__ float from_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Stores F features (F * sizeof(O) bytes, aligned to that size) as O.
template <int F, typename O>
__device__ __forceinline__ void store_features(O* dst, const float* v) {
  if constexpr (sizeof(O) == 4 && F == 4) {
    *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
  } else if constexpr (sizeof(O) == 4 && F == 2) {
    *reinterpret_cast<float2*>(dst) = make_float2(v[0], v[1]);
  } else if constexpr (F == 4) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    uint2 raw;
    raw.x = *reinterpret_cast<unsigned int*>(&lo);
    raw.y = *reinterpret_cast<unsigned int*>(&hi);
    *reinterpret_cast<uint2*>(dst) = raw;
  } else {
    *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(v[0], v[1]);
  }
}

// Builds the plane of every level (grid y = level) from the fp32 table;
// padding entries are zero.
template <int F, typename P>
__global__ void plane_build_kernel(Plane s, const float* __restrict__ table, const float* __restrict__ t,
                                   P* __restrict__ plane) {
  const int l = blockIdx.y;
  const int64_t n = (l + 1 < s.n_levels ? s.off2[l + 1] : s.total2) - s.off2[l];
  const TimeVertex tv = time_vertex(__ldg(t), s.res[l]);
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    P* dst = plane + (s.off2[l] + k) * F;
    if (k >= s.n2[l]) {
#pragma unroll
      for (int f = 0; f < F; ++f) dst[f] = from_float<P>(0.f);
      continue;
    }
    int64_t e0, e1;
    plane_sources(s, l, k, tv.c, &e0, &e1);
    float a[F], b[F];
    Feat<F, float>::load(table, s.off3[l] + e0, a);
    Feat<F, float>::load(table, s.off3[l] + e1, b);
#pragma unroll
    for (int f = 0; f < F; ++f) dst[f] = from_float<P>(fmaf(tv.w0, a[f], tv.w1 * b[f]));
  }
}

// Corners of (a, b) on a plane level: entry indices (within the level) and
// bilinear weights, corner q taking the upper vertex along a when bit 0 is
// set and along b when bit 1 is set; the cell key identifies (a, b)'s cell.
struct PlaneCorners {
  uint32_t idx[4];
  float w[4];
  uint64_t cell;
};
__device__ __forceinline__ void plane_corners(const Plane& s, int l, float a, float b, PlaneCorners& pc) {
  const int r = s.res[l];
  const float pa = __fmul_rn(a, (float)r), pb = __fmul_rn(b, (float)r);   // rounded products, as level_corners
  int ia = (int)floorf(pa), ib = (int)floorf(pb);
  ia = ia < 0 ? 0 : (ia > r - 1 ? r - 1 : ia);
  ib = ib < 0 ? 0 : (ib > r - 1 ? r - 1 : ib);
  const float fa = pa - (float)ia, fb = pb - (float)ib;
  pc.cell = (uint64_t)(uint32_t)ia | ((uint64_t)(uint32_t)ib << 32);
  const bool hashed = (s.hashed2 >> l) & 1u;
  const uint32_t mb = hashed ? kPrime1 : (uint32_t)r + 1u;
  const uint32_t ta[2] = {(uint32_t)ia, (uint32_t)ia + 1u};
  const uint32_t tb[2] = {(uint32_t)ib * mb, (uint32_t)ib * mb + mb};
  const float wa[2] = {1.f - fa, fa}, wb[2] = {1.f - fb, fb};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    pc.idx[q] = hashed ? ((ta[q & 1] ^ tb[q >> 1]) & s.hash_mask) : (ta[q & 1] + tb[q >> 1]);
    pc.w[q] = wa[q & 1] * wb[q >> 1];
  }
}

// Levels a warp collects in shared memory before it writes them: a row's part of
// kEncodeLevels levels goes out as whole consecutive units, where a lane storing its
// own row's levels one by one touches a sector for every 8 bytes (4,882 rays x 512
// samples, 23 levels x 4 features, bf16 rows: the planes 1.67 -> 1.04 ms, the volume
// 1.06 -> 0.74).
constexpr int kEncodeLevels = 8;
constexpr int kEncodeThreads = 256;

// F features of the output type as one unit.
template <int F, typename O>
using Unit = std::conditional_t<F * sizeof(O) == 16, uint4, std::conditional_t<F * sizeof(O) == 8, uint2, unsigned int>>;

template <int F, typename O>
struct EncodeRows {
  Unit<F, O> unit[kEncodeThreads / 32][32][kEncodeLevels + 1];   // a column more than used: no bank conflicts
};

// Encodes the block's points level by level (level(l, acc) gives this thread's
// features) and writes rows [col0, col0 + L * F) of its warp's points.  kFew: the blocks
// along grid y take kEncodeLevels levels each (encode_few).
template <bool kFew, int F, typename O, typename Level>
__device__ __forceinline__ void encode_rows(EncodeRows<F, O>& rows, int n_levels, int64_t n, O* __restrict__ out,
                                            int64_t ld, int col0, Level&& level) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + 32 * warp;   // the warp's first point
  if (i0 >= n) return;   // warp-uniform
  const int here = (int)min((int64_t)32, n - i0);
  auto& mine = rows.unit[warp];
  for (int l0 = kFew ? kEncodeLevels * blockIdx.y : 0; l0 < n_levels; l0 += kEncodeLevels * (kFew ? gridDim.y : 1)) {
    const int nl = min(kEncodeLevels, n_levels - l0);
    if (lane < here) {
#pragma unroll 2   // two levels' gathers in flight
      for (int q = 0; q < nl; ++q) {
        float acc[F];
        level(l0 + q, acc);
        store_features<F, O>(reinterpret_cast<O*>(&mine[lane][q]), acc);
      }
    }
    __syncwarp();
    O* to = out + i0 * ld + col0 + l0 * F;
    if (nl == kEncodeLevels) {
#pragma unroll
      for (int k = 0; k < kEncodeLevels; ++k) {
        const int e = 32 * k + lane, row = e / kEncodeLevels, q = e % kEncodeLevels;
        if (row < here) *reinterpret_cast<Unit<F, O>*>(to + row * ld + q * F) = mine[row][q];
      }
    } else {
      for (int e = lane; e < here * nl; e += 32) {
        const int row = e / nl, q = e - row * nl;
        *reinterpret_cast<Unit<F, O>*>(to + row * ld + q * F) = mine[row][q];
      }
    }
    __syncwarp();
  }
}

// The plane grid's features of (zyx[ca], zyx[cb]) into out[i * ld + col0 + l * F + f].
template <int F, typename P, typename O, bool kFew>
__global__ void __launch_bounds__(kEncodeThreads)
plane_encode_kernel(Plane s, const P* __restrict__ plane, const float* __restrict__ zyx, int64_t n,
                    int ca, int cb, O* __restrict__ out, int64_t ld, int col0) {
  __shared__ EncodeRows<F, O> rows;
  const int64_t i = min(blockIdx.x * (int64_t)blockDim.x + threadIdx.x, n - 1);
  const float a = zyx[i * 3 + ca], b = zyx[i * 3 + cb];
  encode_rows<kFew, F, O>(rows, s.n_levels, n, out, ld, col0, [&](int l, float* acc) {
    PlaneCorners pc;
    plane_corners(s, l, a, b, pc);
    float v[4][F];
#pragma unroll
    for (int q = 0; q < 4; ++q) Feat<F, P>::load(plane, s.off2[l] + pc.idx[q], v[q]);
#pragma unroll
    for (int f = 0; f < F; ++f) {
      acc[f] = 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[f] = fmaf(pc.w[q], v[q][f], acc[f]);
    }
  });
}

// The (z, y, x) grid's features into columns [0, L * F) of the rows, the raw inputs
// (z, y, x, t) after the four grids when `identity`, and zeros from column `pad` to
// the end of the row.
template <int F, typename O, bool kFew>
__global__ void __launch_bounds__(kEncodeThreads)
volume_encode_kernel(GridDev g, const float* __restrict__ table, const float* __restrict__ zyx,
                     const float* __restrict__ t, int64_t n, int identity, O* __restrict__ out, int64_t ld, int pad) {
  __shared__ EncodeRows<F, O> rows;
  const int64_t i = min(blockIdx.x * (int64_t)blockDim.x + threadIdx.x, n - 1);
  const float x[3] = {zyx[i * 3], zyx[i * 3 + 1], zyx[i * 3 + 2]};
  encode_rows<kFew, F, O>(rows, g.n_levels, n, out, ld, 0, [&](int l, float* acc) {
    LevelCorners<3> lc;
    level_corners<3>(g, l, x, lc);
    float v[8][F];
#pragma unroll
    for (int c = 0; c < 8; ++c) Feat<F, float>::load(table, g.offset[l] + lc.idx[c], v[c]);
#pragma unroll
    for (int f = 0; f < F; ++f) {
      acc[f] = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[f] = fmaf(lc.w[c], v[c][f], acc[f]);
    }
  });
  if ((kFew && blockIdx.y > 0) || blockIdx.x * (int64_t)blockDim.x + threadIdx.x >= n) return;
  // the rest of the row, 16 bytes at a time where it starts on such a boundary
  constexpr int kPer = 16 / sizeof(O);
  const int col = 4 * g.n_levels * F;
  const float in[4] = {x[0], x[1], x[2], identity ? __ldg(t) : 0.f};
  O* row = out + i * ld;
  auto value = [&](int c) { return from_float<O>(identity && c < col + 4 ? in[c - col] : 0.f); };
  int c = col;
  if (pad == col + (identity ? 4 : 0) && col % kPer == 0) {
    for (; c + kPer <= ld; c += kPer) {
      uint4 raw;
      O* v = reinterpret_cast<O*>(&raw);
#pragma unroll
      for (int k = 0; k < kPer; ++k) v[k] = k < 4 && c == col ? value(c + k) : from_float<O>(0.f);
      *reinterpret_cast<uint4*>(row + c) = raw;
    }
  }
  for (; c < ld; ++c)
    if (c < pad ? identity : true) row[c] = value(c);
}

// The scatters take 32 * kWalkSegment consecutive points a block, each of its warps some
// levels of all of them.  Where most points lie next to their predecessor (a ray's
// samples, as the module loop passes them) a lane marches over kWalkSegment
// consecutive points with its cell's vertex sums in registers (CellMarch,
// PlaneMarch); otherwise the lanes take consecutive points and a warp merges runs of
// points in one cell.  4,882 rays x 512 samples, 23 levels x 4 features, 2^19 entries,
// against the merging form alone: the volume 1.25 -> 0.98 ms, the planes 1.68 -> 1.41
// (bound by the L1's lines: every lane reads its own row and reduces its own entries).
constexpr int kWalkSegment = 16, kWalkSegmentFew = 4;   // (few points: walk_few)
constexpr float kWalkStep = 1.f / 64.f;   // largest |dz| + |dy| + |dx| to a neighbour
constexpr int kWalkWarps = 12;
constexpr int kPlaneWarps = 6;   // of two levels each

// The block's points: point k of lane l's segment at [c][33 k + l], so that a warp
// reads them without bank conflicts (the lanes' points are kWalkSegment apart in
// memory, and the L1's lines are what bounds the walk).
template <int kSegment>
struct WalkPoints {
  float c[3][kSegment * 33];
};

// Loads the block's points; whether they are walked through (block-uniform).
template <int kSegment>
__device__ __forceinline__ bool walks(WalkPoints<kSegment>& pts, const float* __restrict__ zyx, int64_t p0,
                                      int64_t n) {
  const int values = 3 * (int)min((int64_t)32 * kSegment, n - p0);
  for (int e = threadIdx.x; e < values; e += blockDim.x) {
    const int point = e / 3;
    pts.c[e - 3 * point][point % kSegment * 33 + point / kSegment] = zyx[p0 * 3 + e];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  bool next = false;
  if (p0 + lane * kSegment + 1 < n) {
    float d = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) d += fabsf(pts.c[k][33 + lane] - pts.c[k][lane]);
    next = d <= kWalkStep;
  }
  return __popc(__ballot_sync(0xffffffffu, next)) >= 16;
}

// Gradient of levels [l0, l1) of the (z, y, x) grid: dL/d(features) in
// columns [0, L * F) of the rows.
template <int F, typename S, int kSegment>
__global__ void __launch_bounds__(kWalkWarps * 32, 2)
volume_scatter_kernel(GridDev g, const float* __restrict__ zyx, int64_t n,
                      const S* __restrict__ dout, int64_t ld, float* __restrict__ grad, int l0, int l1) {
  const int64_t p0 = blockIdx.x * (int64_t)(32 * kSegment);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  __shared__ WalkPoints<kSegment> pts;
  if (walks(pts, zyx, p0, n)) {
    const int64_t first = p0 + (int64_t)lane * kSegment;
    const int count = (int)max((int64_t)0, min((int64_t)kSegment, n - first));
    for (int l = l0 + warp; l < l1; l += warps) {
      auto march = [&](auto hashed) {
        CellMarch<3, F, hashed()> m(g, l, grad, 0.f);
        const S* src = dout + first * ld + l * F;
        float d[F], dn[F];   // this point's, and the next one's on its way
        if (count > 0) load_grad_row<F, S>(src, dn);
#pragma unroll 1
        for (int k = 0; k < count; ++k) {
#pragma unroll
          for (int f = 0; f < F; ++f) d[f] = dn[f];
          src += ld;
          if (k + 1 < count) load_grad_row<F, S>(src, dn);
          const float x[3] = {pts.c[0][33 * k + lane], pts.c[1][33 * k + lane], pts.c[2][33 * k + lane]};
          m.add(x, d);
        }
        m.finish();
      };
      if ((g.hashed_bits >> l) & 1u)
        march(std::true_type{});
      else
        march(std::false_type{});
    }
    return;
  }
  for (int l = l0 + warp; l < l1; l += warps)
    for (int k = 0; k < kSegment && p0 + 32 * k < n; ++k) {   // every lane takes part in the warp's shuffles
      const int64_t i = p0 + 32 * k + lane;
      const bool valid = i < n;
      float p[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) p[c] = valid ? zyx[i * 3 + c] : 0.f;
      scatter_warp<3, F, true, S, true>(g, grad, p, valid, dout + (valid ? i : 0) * ld, F, 1, 0u, l, l + 1);
    }
}

// Gradient of one hashed level of the (z, y, x) grid, restricted to the
// corners whose entry lies in half `half` of the level (entry >> shift ==
// half): two such passes keep each pass's reductions within 67 MB of a 2^23 x 4
// fp32 level, which L2 holds, where the whole level (134 MB) does not.  No run
// merging (hashed levels' samples rarely share cells).
template <int F, typename S>
__global__ void volume_scatter_half_kernel(GridDev g, const float* __restrict__ zyx, int64_t n,
                                           const S* __restrict__ dout, int64_t ld, float* __restrict__ grad, int l,
                                           int shift, uint32_t half) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float x[3] = {zyx[i * 3], zyx[i * 3 + 1], zyx[i * 3 + 2]};
  LevelCorners<3> lc;
  level_corners<3>(g, l, x, lc);
  float d[F];
  load_grad_row<F, S>(dout + i * ld + l * F, d);
  float* base = grad + g.offset[l] * F;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    if ((lc.idx[c] >> shift) != half) continue;
    float v[F];
#pragma unroll
    for (int f = 0; f < F; ++f) v[f] = lc.w[c] * d[f];
    red_entry<F>(base + (int64_t)lc.idx[c] * F, v);
  }
}

// CellMarch on a plane level: the four vertices of the current cell by the parities
// of their coordinates.
template <int F>
struct PlaneMarch {
  uint32_t mb, mask;
  bool hashed, any = false;
  int res;
  float* base;
  int v[2][2];
  float acc[4][F];

  __device__ __forceinline__ void init(const Plane& s, int l, float* grad) {
    hashed = (s.hashed2 >> l) & 1u;
    res = s.res[l];
    mb = hashed ? kPrime1 : (uint32_t)res + 1u;
    mask = hashed ? s.hash_mask : 0xffffffffu;
    base = grad + s.off2[l] * F;
#pragma unroll
    for (int k = 0; k < 2; ++k) v[k][0] = v[k][1] = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int f = 0; f < F; ++f) acc[c][f] = 0.f;
  }

  // Reduces and clears the slots whose vertex changes.
  __device__ __forceinline__ void leave(const uint32_t (*x)[2]) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint32_t h = (uint32_t)v[1][r] * mb, e = (uint32_t)v[0][0], o = (uint32_t)v[0][1];
      reduce_row<F>(base, hashed ? (e ^ h) & mask : e + h, hashed ? (o ^ h) & mask : o + h, x[0][0] | x[1][r],
                    x[0][1] | x[1][r], acc[2 * r], acc[2 * r + 1]);
    }
  }

  __device__ __forceinline__ void add(float a, float b, const float* d) {
    const float x[2] = {a, b};
    uint32_t ch[2][2], moved = 0;
    int c[2][2];
    float w[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float p = __fmul_rn(x[k], (float)res);   // as plane_corners
      int ci = (int)floorf(p);
      ci = ci < 0 ? 0 : (ci > res - 1 ? res - 1 : ci);
      const float f = p - (float)ci, u = 1.f - f;
      w[k][0] = (ci & 1) ? f : u;
      w[k][1] = (ci & 1) ? u : f;
      c[k][0] = (ci + 1) & ~1;
      c[k][1] = ci | 1;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        ch[k][q] = (uint32_t)(c[k][q] ^ v[k][q]);
        moved |= ch[k][q];
      }
    }
    if (moved != 0u || !any) {
      if (any) leave(ch);
      any = true;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        v[k][0] = c[k][0];
        v[k][1] = c[k][1];
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float wc = w[0][q] * w[1][r];
#pragma unroll
        for (int f = 0; f < F; ++f) acc[2 * r + q][f] = fmaf(wc, d[f], acc[2 * r + q][f]);
      }
  }

  __device__ __forceinline__ void finish() {
    const uint32_t all[2][2] = {{1u, 1u}, {1u, 1u}};
    if (any) leave(all);
    any = false;
  }
};

// Gradient of a plane grid into the plane-shaped fp32 gradient, 4 corners a level;
// a warp takes two levels.  Points that do not walk: on levels where a warp's 32
// points form at most 24 runs of equal cells, each run's sums are reduced once by
// its first lane.
template <int F, typename S, int kSegment>
__global__ void __launch_bounds__(kPlaneWarps * 32)
plane_scatter_kernel(Plane s, const float* __restrict__ zyx, int64_t n, int ca, int cb,
                     const S* __restrict__ dout, int64_t ld, int col0, float* __restrict__ pgrad) {
  const int64_t p0 = blockIdx.x * (int64_t)(32 * kSegment);
  const int lane = threadIdx.x & 31, l0 = 2 * (int)(blockIdx.y * kPlaneWarps + (threadIdx.x >> 5));
  const int nl = min(2, s.n_levels - l0);
  __shared__ WalkPoints<kSegment> pts;
  const bool walk = walks(pts, zyx, p0, n);
  if (nl <= 0) return;
  if (walk) {
    const int64_t first = p0 + (int64_t)lane * kSegment;
    const int count = (int)max((int64_t)0, min((int64_t)kSegment, n - first));
    PlaneMarch<F> m[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) m[q].init(s, min(l0 + q, s.n_levels - 1), pgrad);
    const S* src = dout + first * ld + col0 + l0 * F;
    float d[2][F], dn[2][F];   // this point's, and the next one's on their way
    auto fetch = [&]() {
      load_grad_row<F, S>(src, dn[0]);
      if (nl > 1) load_grad_row<F, S>(src + F, dn[1]);
      src += ld;
    };
    if (count > 0) fetch();
#pragma unroll 1
    for (int k = 0; k < count; ++k) {
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int f = 0; f < F; ++f) d[q][f] = dn[q][f];
      if (k + 1 < count) fetch();
      const float a = pts.c[ca][33 * k + lane], b = pts.c[cb][33 * k + lane];
      m[0].add(a, b, d[0]);
      if (nl > 1) m[1].add(a, b, d[1]);
    }
    m[0].finish();
    m[1].finish();
    return;
  }
  for (int k = 0; k < kSegment && p0 + 32 * k < n; ++k) {
    const int64_t i = p0 + 32 * k + lane;
    const bool valid = i < n;
    const float a = valid ? zyx[i * 3 + ca] : 0.f, b = valid ? zyx[i * 3 + cb] : 0.f;
    const S* src = dout + (valid ? i : 0) * ld + col0;
#pragma unroll 1
    for (int l = l0; l < l0 + nl; ++l) {
      PlaneCorners pc;
      plane_corners(s, l, a, b, pc);
      float d[F];
      if (valid) {
        load_grad_row<F, S>(src + l * F, d);
      } else {
#pragma unroll
        for (int f = 0; f < F; ++f) d[f] = 0.f;
      }
      float* base = pgrad + s.off2[l] * F;
      const uint64_t key = valid ? pc.cell : ~uint64_t(0);
      const uint64_t prev = __shfl_up_sync(0xffffffffu, key, 1);
      const bool head = (lane == 0) || (prev != key);
      const uint32_t heads = __ballot_sync(0xffffffffu, head);
      if (__popc(heads) <= 24) {
        const uint32_t later = heads & ~((2u << lane) - 1u);
        const int end = later ? (__ffs(later) - 2) : 31;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float v[F];
#pragma unroll
          for (int f = 0; f < F; ++f) v[f] = run_sum(pc.w[q] * d[f], lane, end);
          if (head && valid) red_entry<F>(base + (int64_t)pc.idx[q] * F, v);
        }
      } else if (valid) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float v[F];
#pragma unroll
          for (int f = 0; f < F; ++f) v[f] = pc.w[q] * d[f];
          red_entry<F>(base + (int64_t)pc.idx[q] * F, v);
        }
      }
    }
  }
}

// Adds the plane-shaped gradient to the 3D gradient table at the two time
// vertices (grid y = level).  Plane levels keyed by the hash: one thread per
// 3D entry e gathers plane entries e ^ c0 and e ^ c1 (an XOR is its own
// inverse, so every 3D entry has one writer).  Dense plane levels: one thread
// per non-zero plane entry; on dense 3D levels its two vertices are its own
// (different t slabs), on hashed ones they may collide and are reduced
// atomically.
template <int F>
__global__ void plane_spread_kernel(Plane s, const float* __restrict__ t, const float* __restrict__ pgrad,
                                    float* __restrict__ grad) {
  const int l = blockIdx.y;
  const TimeVertex tv = time_vertex(__ldg(t), s.res[l]);
  const float* src = pgrad + s.off2[l] * F;
  float* dst = grad + s.off3[l] * F;
  const bool hashed2 = (s.hashed2 >> l) & 1u, hashed3 = (s.hashed3 >> l) & 1u;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < s.n2[l];
       k += (int64_t)gridDim.x * blockDim.x) {
    if (hashed2) {
      int64_t j0, j1;   // the plane entries whose vertices are 3D entry k
      plane_sources(s, l, k, tv.c, &j0, &j1);
      float g0[F], g1[F];
      Feat<F, float>::load(src, j0, g0);
      Feat<F, float>::load(src, j1, g1);
      bool any = false;
#pragma unroll
      for (int f = 0; f < F; ++f) any |= (g0[f] != 0.f) | (g1[f] != 0.f);
      if (!any) continue;
#pragma unroll
      for (int f = 0; f < F; ++f) dst[k * F + f] += fmaf(tv.w0, g0[f], tv.w1 * g1[f]);
      continue;
    }
    float g[F];
    Feat<F, float>::load(src, k, g);
    bool any = false;
#pragma unroll
    for (int f = 0; f < F; ++f) any |= g[f] != 0.f;
    if (!any) continue;
    int64_t e0, e1;
    plane_sources(s, l, k, tv.c, &e0, &e1);
    float v0[F], v1[F];
#pragma unroll
    for (int f = 0; f < F; ++f) {
      v0[f] = tv.w0 * g[f];
      v1[f] = tv.w1 * g[f];
    }
    if (hashed3) {
      red_entry<F>(dst + e0 * F, v0);
      red_entry<F>(dst + e1 * F, v1);
    } else {
#pragma unroll
      for (int f = 0; f < F; ++f) {
        dst[e0 * F + f] += v0[f];
        dst[e1 * F + f] += v1[f];
      }
    }
  }
}

// The plane grids in the reference's input order (networks.py:438-446):
// (y, x, t), (x, z, t), (z, y, t); the (a, b) columns of zyx.
constexpr int kPlaneCols[3][2] = {{1, 2}, {2, 0}, {0, 1}};

dim3 plane_grid(const Plane& s) {
  int64_t widest = 0;
  for (int l = 0; l < s.n_levels; ++l) widest = std::max(widest, s.n2[l]);
  return dim3((unsigned)std::min<int64_t>(ceil_div(widest, 256), 4096), (unsigned)s.n_levels);
}

size_t plane_bytes(const Plane& s, int F) { return ((size_t)s.total2 * F * 4 + 255) & ~size_t(255); }

int check_grid(const NectbHashGrid* grid, GridDev* g, Plane* s) {
  if (!make_grid_dev(grid, g)) return set_error(NECTB_ERR_INVALID, "invalid hash grid description");
  NECTB_REQUIRE(grid->n_dims == 3 && grid->feature_dtype == NECTB_F32,
                "QuadCubes grids are 3D with fp32 tables");
  NECTB_REQUIRE(grid->n_features == 2 || grid->n_features == 4, "n_features must be 2 or 4");
  NECTB_REQUIRE(make_plane(*g, s), "QuadCubes grids need the same resolution on every axis");
  return NECTB_OK;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// Whether the encoders' blocks take kEncodeLevels levels of their points in place of all:
// where one of all would not give every SM a block (23 levels x 4 features, 2^17 entries,
// the whole call: 10,240 points 147 -> 82 us, 30,720 142 -> 94; 37,888 at the line).
bool encode_few(int64_t n) { return ceil_div(n, kEncodeThreads) < 148; }

template <int F, typename P, typename O, bool kFew>
int encode_all(const GridDev& g, const Plane& s, const float* const* tables, const float* zyx, int64_t n,
               const float* t, int identity, O* out, int64_t ld, P* plane, cudaStream_t st) {
  const dim3 blocks((unsigned)ceil_div(n, kEncodeThreads), kFew ? (unsigned)ceil_div(g.n_levels, kEncodeLevels) : 1u);
  const int LF = g.n_levels * F;
  volume_encode_kernel<F, O, kFew><<<blocks, kEncodeThreads, 0, st>>>(g, tables[0], zyx, t, n, identity, out, ld,
                                                                      4 * LF + (identity ? 4 : 0));
  if (int rc = launch_status("volume_encode_kernel")) return rc;
  for (int k = 0; k < 3; ++k) {
    plane_build_kernel<F, P><<<plane_grid(s), 256, 0, st>>>(s, tables[k + 1], t, plane);
    if (int rc = launch_status("plane_build_kernel")) return rc;
    plane_encode_kernel<F, P, O, kFew><<<blocks, kEncodeThreads, 0, st>>>(
        s, plane, zyx, n, kPlaneCols[k][0], kPlaneCols[k][1], out, ld, (k + 1) * LF);
    if (int rc = launch_status("plane_encode_kernel")) return rc;
  }
  return NECTB_OK;
}

constexpr int64_t kScatterGroupBytes = int64_t(64) << 20;

// Whether the scatters' blocks take segments of kWalkSegmentFew points: where those of
// kWalkSegment would give fewer than three blocks to two SMs (23 levels x 4 features, 2^17
// entries, encode and backward: 10,240 points along rays 376 -> 232 us, loose 385 -> 247;
// 76,800 421 -> 416 and 651 -> 583; 148,480 along rays 589 with 16 points, 596 with four).
bool walk_few(int64_t n) { return 2 * ceil_div(n, 32 * kWalkSegment) < 3 * 148; }

template <int F, typename S, int kSegment>
int backward_all(const GridDev& g, const Plane& s, const float* zyx, int64_t n, const float* t, const S* dout,
                 int64_t ld, float* const* grads, float* pgrad, cudaStream_t st) {
  const unsigned blocks = (unsigned)ceil_div(n, 256), walk_blocks = (unsigned)ceil_div(n, 32 * kSegment);
  const dim3 plane_blocks(walk_blocks, (unsigned)ceil_div(s.n_levels, 2 * kPlaneWarps));
  const int LF = g.n_levels * F;
  // One pass per group of consecutive levels whose gradient slice is at most
  // kScatterGroupBytes (a hashed level of 2^23 entries is a group of its own),
  // so that a pass's reductions find their lines in L2 and each line is
  // written back about once; the passes re-read the points and their rows.
  for (int l0 = 0; l0 < g.n_levels;) {
    int l1 = l0 + 1;
    auto level_bytes = [&](int l) {
      const int64_t end = l + 1 < g.n_levels ? g.offset[l + 1] : g.total_entries;
      return (end - g.offset[l]) * F * 4;
    };
    int64_t bytes = level_bytes(l0);
    while (l1 < g.n_levels && bytes + level_bytes(l1) <= kScatterGroupBytes) bytes += level_bytes(l1++);
    if (l1 == l0 + 1 && ((g.hashed_bits >> l0) & 1u) && bytes > kScatterGroupBytes) {
      // a hashed level above the group size: one pass per half of its entries
      int log2T = 0;
      while ((1u << log2T) < g.hash_mask + 1u) ++log2T;
      for (uint32_t h = 0; h < 2; ++h) {
        volume_scatter_half_kernel<F, S><<<blocks, 256, 0, st>>>(g, zyx, n, dout, ld, grads[0], l0, log2T - 1, h);
        if (int rc = launch_status("volume_scatter_half_kernel")) return rc;
      }
    } else {
      volume_scatter_kernel<F, S, kSegment><<<walk_blocks, 32 * std::min(l1 - l0, kWalkWarps), 0, st>>>(
          g, zyx, n, dout, ld, grads[0], l0, l1);
      if (int rc = launch_status("volume_scatter_kernel")) return rc;
    }
    l0 = l1;
  }
  for (int k = 0; k < 3; ++k) {
    if (int rc = cuda_status(cudaMemsetAsync(pgrad, 0, (size_t)s.total2 * F * 4, st), "cudaMemsetAsync")) return rc;
    plane_scatter_kernel<F, S, kSegment><<<plane_blocks, 32 * kPlaneWarps, 0, st>>>(
        s, zyx, n, kPlaneCols[k][0], kPlaneCols[k][1], dout, ld, (k + 1) * LF, pgrad);
    if (int rc = launch_status("plane_scatter_kernel")) return rc;
    plane_spread_kernel<F><<<plane_grid(s), 256, 0, st>>>(s, t, pgrad, grads[k + 1]);
    if (int rc = launch_status("plane_spread_kernel")) return rc;
  }
  return NECTB_OK;
}

}  // namespace
}  // namespace nectb

using namespace nectb;

extern "C" size_t nectb_quadcubes_workspace_bytes(const NectbHashGrid* grid) {
  GridDev g;
  Plane s;
  if (!grid || !make_grid_dev(grid, &g) || !make_plane(g, &s)) return 0;
  return plane_bytes(s, grid->n_features);
}

extern "C" int nectb_quadcubes_encode(const NectbHashGrid* grid, const float* const* tables, const float* zyx,
                                      int64_t n, const float* t, int identity, void* out, int64_t out_ld,
                                      int out_dtype, void* workspace, size_t workspace_bytes, void* stream) {
  clear_error();
  GridDev g;
  Plane s;
  if (int rc = check_grid(grid, &g, &s)) return rc;
  NECTB_REQUIRE(n >= 0, "negative size");
  if (n == 0) return NECTB_OK;
  NECTB_REQUIRE(tables && zyx && t && out && workspace, "null pointer");
  for (int k = 0; k < 4; ++k) NECTB_REQUIRE(tables[k] && aligned16(tables[k]), "tables must be 16-byte aligned");
  NECTB_REQUIRE(out_dtype == NECTB_F32 || out_dtype == NECTB_BF16, "out_dtype must be NECTB_F32 or NECTB_BF16");
  const int F = grid->n_features;
  const size_t esz = out_dtype == NECTB_F32 ? 4 : 2;
  NECTB_REQUIRE(out_ld >= 4 * (int64_t)g.n_levels * F + (identity ? 4 : 0), "out_ld narrower than a row");
  NECTB_REQUIRE(aligned16(out) && (out_ld * esz) % 16 == 0, "out and its rows must be 16-byte aligned");
  NECTB_REQUIRE(aligned16(workspace), "workspace must be 16-byte aligned");
  if (workspace_bytes < plane_bytes(s, F))
    return set_error(NECTB_ERR_WORKSPACE, "workspace %zu bytes < %zu", workspace_bytes, plane_bytes(s, F));
  cudaStream_t st = (cudaStream_t)stream;
  ProfScope ps(kProfModel, st);
  const int id = identity ? 1 : 0;
  auto run = [&](auto f, auto* o, auto* pl) {
    using P = std::decay_t<decltype(*pl)>;
    using O = std::decay_t<decltype(*o)>;
    return encode_few(n) ? encode_all<f(), P, O, true>(g, s, tables, zyx, n, t, id, o, out_ld, pl, st)
                         : encode_all<f(), P, O, false>(g, s, tables, zyx, n, t, id, o, out_ld, pl, st);
  };
  auto rows = [&](auto* o, auto* pl) {
    return F == 2 ? run(std::integral_constant<int, 2>{}, o, pl) : run(std::integral_constant<int, 4>{}, o, pl);
  };
  return out_dtype == NECTB_F32 ? rows((float*)out, (float*)workspace) : rows((__nv_bfloat16*)out, (__half*)workspace);
}

extern "C" int nectb_quadcubes_encode_backward(const NectbHashGrid* grid, const float* zyx, int64_t n,
                                               const float* t, const void* dout, int64_t dout_ld, int dout_dtype,
                                               float* const* grads, void* workspace, size_t workspace_bytes,
                                               void* stream) {
  clear_error();
  GridDev g;
  Plane s;
  if (int rc = check_grid(grid, &g, &s)) return rc;
  NECTB_REQUIRE(n >= 0, "negative size");
  if (n == 0) return NECTB_OK;
  NECTB_REQUIRE(zyx && t && dout && grads && workspace, "null pointer");
  for (int k = 0; k < 4; ++k) NECTB_REQUIRE(grads[k] && aligned16(grads[k]), "grads must be 16-byte aligned");
  NECTB_REQUIRE(dout_dtype == NECTB_F32 || dout_dtype == NECTB_BF16, "dout_dtype must be NECTB_F32 or NECTB_BF16");
  const int F = grid->n_features;
  NECTB_REQUIRE(dout_ld >= 4 * (int64_t)g.n_levels * F, "dout_ld narrower than the four grids' columns");
  NECTB_REQUIRE(aligned16(dout) && (dout_ld * (dout_dtype == NECTB_F32 ? 4 : 2)) % 16 == 0,
                "dout and its rows must be 16-byte aligned");
  NECTB_REQUIRE(aligned16(workspace), "workspace must be 16-byte aligned");
  if (workspace_bytes < plane_bytes(s, F))
    return set_error(NECTB_ERR_WORKSPACE, "workspace %zu bytes < %zu", workspace_bytes, plane_bytes(s, F));
  cudaStream_t st = (cudaStream_t)stream;
  ProfScope ps(kProfModel, st);
  float* pg = (float*)workspace;
  auto run = [&](auto f, const auto* d) {
    return walk_few(n) ? backward_all<f(), std::decay_t<decltype(*d)>, kWalkSegmentFew>(g, s, zyx, n, t, d, dout_ld,
                                                                                        grads, pg, st)
                       : backward_all<f(), std::decay_t<decltype(*d)>, kWalkSegment>(g, s, zyx, n, t, d, dout_ld,
                                                                                     grads, pg, st);
  };
  auto rows = [&](const auto* d) {
    return F == 2 ? run(std::integral_constant<int, 2>{}, d) : run(std::integral_constant<int, 4>{}, d);
  };
  return dout_dtype == NECTB_F32 ? rows((const float*)dout) : rows((const __nv_bfloat16*)dout);
}
