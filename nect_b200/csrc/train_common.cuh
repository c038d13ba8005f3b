// Pieces shared by the plain (fp32 SIMT) and mixed (bf16 tcgen05) fused
// training kernels: per-ray records, the ray-preparation kernel, the ray
// scheduler and sample regeneration.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "common.cuh"
#include "geometry.cuh"
#include "hashgrid.cuh"
#include "ray_plan.cuh"

namespace nectb {

// Everything a fused kernel needs to regenerate the samples of one ray
// without touching positions in memory.  64 bytes.
struct RayRec {
  double sx, sy, sz;   // first sample (normalised, clamped), fp64 as in the reference
  double dx, dy, dz;   // spacing
  int32_t count;       // samples written by the reference loop
  float scale;         // distances[r] / max_distance_traveled (base_trainer.py:552-554)
  float y;             // measured value proj[perm[start + r]]
  float gsig;          // dL/dsigma for every sample of the ray (set by the forward)
};
static_assert(sizeof(RayRec) == 64, "RayRec must be 64 bytes");

enum { kPhaseForward = 1, kPhaseBackward = 2 };

// Continuous-scan steps: at most this many sub-angles per batch.
constexpr int kMaxSubAngles = 32;

struct TrainArgs {
  const int64_t* perm;
  int64_t perm_len;
  int64_t start;
  int num_rays;
  int n_pixels;  // nDetector[0] * nDetector[1]
  int n_cols = 1;  // nDetector[1]
  // a re-projection (a whole view or any range of its pixels): no backward follows, so
  // no ray order is made and no rows are stored, whatever the workspace holds
  bool query = false;
  int claim = 1;   // slots a warp claims at a time (slots_per_claim)
  int S;
  float angle;
  float t;
  float maxd;
  int uniform;
  float max_dist;
  const float* jitter;
  const float* det_off;
  const float* projection;
  int loss_type;
  float loss_scale;
  int max_blocks;  // > 0: cap on the persistent grids (queries); 0: default
  // > 0: the forward runs one block of this many warpgroups per SM under the
  // shared-SM carveout (re-projection pieces beside serving kernels); 0: the tuning's
  int fwd_warpgroups = 0;
  // Re-projections: room for the column form's sigmas, of col_rays rays (groups of
  // 32) at a time; null: none.
  float* col_sigma = nullptr;
  int col_rays = 0;
  // the encoders may fetch corners through a texture object over the table
  // (false: loads only, no texture object created)
  bool texture = true;
  int phase = kPhaseForward | kPhaseBackward;  // which half of the step to run
  float run_threshold = 0.75f;                 // run merging of the scatter (set from the tuning)
  // Continuous scan (sub > 1): num_rays = sub * (pixels of the batch) virtual
  // rays, sub-angle-major (ray v = j * pixels + r is pixel r at sub_angle[j],
  // with jitter[v] and det_off[2v..2v+1]); n_pixels = sub * detector pixels,
  // slot index = pixel * sub + j.
  int sub = 1;
  float sub_angle[kMaxSubAngles];
};

enum : unsigned int { kFlagDuplicatePixels = 1u };

// Workspace (ray_plan.cuh) of R rays over P slots, without staging.
inline size_t workspace_bytes(int R, int P) { return (size_t)R * sizeof(RayRec) + (size_t)P * 4 + 256; }

inline Workspace carve_workspace(void* ws, int R, int P, size_t size = 0) {
  Workspace w;
  w.rays = (RayRec*)ws;
  w.slot = (int32_t*)((char*)ws + (size_t)R * sizeof(RayRec));
  w.counters = (unsigned int*)((char*)w.slot + (((size_t)P * 4 + 63) & ~size_t(63)));
  const size_t base = (workspace_bytes(R, P) + 255) & ~size_t(255);
  if (size > base) {
    w.stage = (float*)((char*)ws + base);
    w.stage_bytes = size - base;
  }
  return w;
}

// Time slice of a 4D grid at the batch's t (mixed training).  Along t a
// level's 16-corner interpolation is a blend of two time vertices with the
// same weights for every sample of the batch, and the vertices' entries are
// the 3D vertex's entry XOR a per-level constant (hashed levels: the hash is
// an XOR of per-axis terms, masked) or plus a per-level offset (dense levels:
// t is the outermost stride).  So per level
//   slice[k] = w0 * table[k ^ c0] + w1 * table[k ^ c1]   (hashed)
//   slice[k] = w0 * table[k + c0] + w1 * table[k + c1]   (dense, k < x*y*z vertices)
// and the 3D view g3 of the grid (same resolutions, strides and hash, slice
// offsets) indexes it: the 3D kernels then gather 8 corners instead of 16.
// Gradients reduced into a slice-shaped table g are spread back by
//   dtable[e] += w0 * g[e ^ c0] + w1 * g[e ^ c1]          (hashed; conflict-free)
//   dtable[k + c0] += w0 * g[k], dtable[k + c1] += w1 * g[k]  (dense)
struct TimeSlice {
  GridDev g3;
  int64_t off4[NECTB_MAX_LEVELS];    // the 4D level offsets
  int64_t n_real[NECTB_MAX_LEVELS];  // slice entries that exist (T, or the dense x*y*z vertices)
  int64_t c0[NECTB_MAX_LEVELS], c1[NECTB_MAX_LEVELS];
  float w0[NECTB_MAX_LEVELS], w1[NECTB_MAX_LEVELS];
};

// t -> vertex and weights exactly as level_corners computes them for axis 3.
inline TimeSlice make_time_slice(const GridDev& g, float t) {
  TimeSlice s;
  s.g3 = g;
  s.g3.n_dims = 3;
  int64_t off = 0;
  for (int l = 0; l < g.n_levels; ++l) {
    s.off4[l] = g.offset[l];
    const int r = g.res[l][3];
    const float p = t * (float)r;
    int ci = (int)std::floor(p);
    ci = ci < 0 ? 0 : (ci > r - 1 ? r - 1 : ci);
    const float f = p - (float)ci;
    s.w0[l] = 1.f - f;
    s.w1[l] = f;
    const bool hashed = (g.hashed_bits >> l) & 1u;
    if (hashed) {
      const uint32_t term = (uint32_t)ci * kPrime3;
      s.c0[l] = (int64_t)(term & g.hash_mask);
      s.c1[l] = (int64_t)((term + kPrime3) & g.hash_mask);
      s.n_real[l] = (int64_t)g.hash_mask + 1;
    } else {
      const int64_t s3 = g.stride[l][3];
      s.c0[l] = (int64_t)ci * s3;
      s.c1[l] = (int64_t)(ci + 1) * s3;
      s.n_real[l] = s3;
    }
    s.g3.offset[l] = off;
    off += hashed ? s.n_real[l] : (s.n_real[l] + 7) / 8 * 8;
  }
  s.g3.total_entries = off;
  return s;
}

// Bytes of a 4D grid's time slice (fp16) and its fp32 gradient, for one step.
inline size_t slice_bytes(const GridDev& g) {
  const int64_t n3 = make_time_slice(g, 0.f).g3.total_entries;
  return align256((size_t)n3 * g.n_features * 2) + align256((size_t)n3 * g.n_features * 4);
}

// A texture object over an fp16 table (entry_bytes 4 or 8), cached per
// buffer, or 0 where none can be made; the encoders fetch the odd hashed
// levels' corners through it.
cudaTextureObject_t table_texture(const void* ptr, size_t bytes, int entry_bytes);

// Bytes of the fp16 time slice alone (forward-only queries).
inline size_t slice_half_bytes(const GridDev& g) {
  return align256((size_t)make_time_slice(g, 0.f).g3.total_entries * g.n_features * 2);
}

// Warp per ray: set-up, sample count (warp ballot), measured value, scale;
// claims the ray's detector pixel in slot[]; finalises rays without samples
// (y_pred = 0, their loss term and gradient).
constexpr int kRayPrepThreads = 256;
__global__ void ray_prep_kernel(NectbGeometry g, TrainArgs a, RayRec* __restrict__ recs, int32_t* __restrict__ slot,
                                unsigned int* __restrict__ ctrl, float* __restrict__ y_pred, float* __restrict__ loss);

// Position of sample i of a prepared ray, after the Projector clamp
// (projector.py:127); returns false for the zero points the trainer drops
// (base_trainer.py:523).
__device__ __forceinline__ bool sample_point(const RayRec& r, int i, float* p) {
  const float px = r.sx + i * r.dx;
  const float py = r.sy + i * r.dy;
  const float pz = r.sz + i * r.dz;
  p[0] = clamp01f(pz);
  p[1] = clamp01f(py);
  p[2] = clamp01f(px);
  return !(p[0] == 0.f && p[1] == 0.f && p[2] == 0.f);
}

__device__ __forceinline__ RayRec load_ray(const RayRec* recs, int r) { return recs[r]; }

// Warp-uniform scheduler: hands out the rays of the batch that have samples,
// in detector-pixel order (neighbouring rays run together, so the blocks in
// flight touch a compact part of the tables and the L2 keeps it), or in batch
// order when the batch repeats a pixel.  Returns -1 when none are left.
// A claim of one slot costs an atomic on one address, which bound batches of very few
// rays; in pixel order a warp then claims several neighbouring slots at a time
// (slots_per_claim) and is handed their rays one after the other.
struct SlotClaim {
  int ray = -1;            // of this lane's slot of the claim
  unsigned int left = 0;   // lanes whose rays have not been handed out
};
__device__ __forceinline__ int next_ray(SlotClaim& claim, unsigned int* cursor, const int32_t* __restrict__ slot,
                                        const RayRec* __restrict__ recs, const TrainArgs& a, bool by_pixel,
                                        int lane) {
  while (by_pixel && claim.left == 0) {
    unsigned int at = 0;
    if (lane == 0) at = atomicAdd(cursor, (unsigned)a.claim);
    at = __shfl_sync(0xffffffffu, at, 0);
    if (at >= (unsigned)a.n_pixels) return -1;
    claim.ray = lane < a.claim && at + lane < (unsigned)a.n_pixels ? slot[at + lane] : -1;
    claim.left = __ballot_sync(0xffffffffu, claim.ray >= 0);
  }
  if (by_pixel) {
    const int from = __ffs(claim.left) - 1;
    claim.left &= claim.left - 1;
    return __shfl_sync(0xffffffffu, claim.ray, from);
  }
  while (true) {
    unsigned int idx = 0;
    if (lane == 0) idx = atomicAdd(cursor, 1u);
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (idx >= (unsigned)a.num_rays) return -1;
    if (recs[idx].count > 0) return (int)idx;
  }
}

// The rays with samples in scheduling order, for the two-pass backward's
// rounds of equal ray counts: order[rank] = ray, ranks 0..ctrl[6]-1, and
// offs[rank] = samples of the rays ranked before it (the ray's first row in
// the encoding store).  Three launches over the scheduling indices (strips of
// the detector, strip_slot, or batch positions when the batch repeats a pixel):
// per-block counts, one block scanning them, and the per-block compaction, so
// that order is kept.
__global__ void order_count_kernel(const int32_t* __restrict__ slot, const RayRec* __restrict__ recs,
                                   const unsigned int* __restrict__ ctrl, int R, int P, int cols, int sub,
                                   unsigned int* __restrict__ block_sums,
                                   unsigned long long* __restrict__ block_samples);
__global__ void order_scan_kernel(unsigned int* __restrict__ block_sums, unsigned long long* __restrict__ block_samples,
                                  int n_blocks, unsigned int* __restrict__ ctrl);
__global__ void order_compact_kernel(const int32_t* __restrict__ slot, const RayRec* __restrict__ recs,
                                     const unsigned int* __restrict__ ctrl, int R, int P, int cols, int sub,
                                     const unsigned int* __restrict__ block_sums,
                                     const unsigned long long* __restrict__ block_samples,
                                     int32_t* __restrict__ order, uint64_t* __restrict__ offs);

// Scheduler over ranks [lo, hi) of the ordered rays (one round); the rank of
// the returned ray is written to *sched.  Returns -1 when none are left.
__device__ __forceinline__ int next_ray_ranked(unsigned int* cursor, const int32_t* __restrict__ order,
                                               unsigned int n_valid, int lo, int hi, int lane, int* sched) {
  unsigned int idx = 0;
  if (lane == 0) idx = (unsigned)lo + atomicAdd(cursor, 1u);
  idx = __shfl_sync(0xffffffffu, idx, 0);
  if (idx >= min((unsigned)hi, n_valid)) return -1;
  *sched = (int)idx;
  return order[idx];
}

// Loss gradient dL/dy_pred for one ray (mean over rays, nect/config.py:481-497),
// times the ray's scale (dy_pred/dsigma).
__device__ __forceinline__ float loss_grad(float y_pred, float y, int loss_type, int R, float scale) {
  const float d = y_pred - y;
  float g;
  if (loss_type == 1)
    g = (d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f)) / (float)R;
  else
    g = 2.f * d / (float)R;
  return g * scale;
}

__device__ __forceinline__ float loss_term(float y_pred, float y, int loss_type) {
  const float d = y_pred - y;
  return loss_type == 1 ? fabsf(d) : d * d;
}

}  // namespace nectb
