// Ray sampling kernel: the drop-in for the reference's sample_points<T>
// (nect/sampling/ct_sampling.cu:578-602) and host sample<T> (:606-648).
//
// One warp per ray instead of one thread per ray: lanes evaluate 32
// consecutive samples at a time, turn them in shared memory and write the
// [R,S,3] output in whole 128-byte runs; the zero fill of unwritten samples
// happens in the same pass (the reference first memsets the whole tensor).  The
// break index (= per-ray sample count) is found with a warp ballot.
// 9,765 rays x 512 samples (60 MB written): 25.5 -> 16.6 us (9.2 at the copy rate); the
// fp64 set-up, on eight lanes of a block instead of every lane, took 3.6 of them.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "geometry.cuh"

namespace nectb {

namespace {

constexpr int kWarpsPerBlock = 8;

__global__ void __launch_bounds__(kWarpsPerBlock * 32)
sample_kernel(NectbGeometry g, const int64_t* __restrict__ perm, int64_t perm_len, int64_t start, int num_rays,
              int S, int part, float angle, float maxd, int uniform, const float* __restrict__ jitter,
              const float* __restrict__ det_off, float* __restrict__ points, float* __restrict__ distances,
              int32_t* __restrict__ counts) {
  const int lane = threadIdx.x & 31;
  // the block's eight rays are set up by eight lanes: the fp64 divisions once per
  // ray instead of on every lane of its warp
  __shared__ RaySetup setups[kWarpsPerBlock];
  if (threadIdx.x < kWarpsPerBlock) {
    const int mine = blockIdx.x * kWarpsPerBlock + threadIdx.x;
    int ray_index = 0;
    RaySetup s;
    s.valid = 0;
    s.distance = 0.f;
    if (mine < num_rays && ray_lookup(perm, perm_len, start, mine, num_rays, g, ray_index))
      ray_setup(g, ray_index, det_off[2 * (int64_t)mine], det_off[2 * (int64_t)mine + 1], jitter[mine], angle, S, maxd,
                uniform != 0, s);
    setups[threadIdx.x] = s;
  }
  __syncthreads();
  const int tid = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (tid >= num_rays) return;
  const RaySetup r = setups[threadIdx.x >> 5];
  int count = 0;
  if (r.valid) count = warp_sample_count(g, r, S, lane);
  if (lane == 0 && blockIdx.y == 0) {
    distances[tid] = r.distance;
    if (counts) counts[tid] = count;
  }
  if (!points) return;
  constexpr int kRuns = 4;
  __shared__ float turn[kWarpsPerBlock][96 * kRuns];
  float* mine = turn[threadIdx.x >> 5];
  float* out = points + (int64_t)tid * S * 3;
  // Writes runs() runs of 32 samples from sample `base` on, the values of valid ones turned
  // in shared memory.
  auto write = [&](int base, auto runs) {
    constexpr int Q = runs();
    const int n = 3 * min(32 * Q, S - base);   // values of these runs
    float v[3 * Q];
#pragma unroll
    for (int k = 0; k < 3 * Q; ++k) v[k] = 0.f;
    if (base < count) {   // warp-uniform
      __syncwarp();
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int i = base + 32 * q + lane;
        float pz = 0.f, py = 0.f, px = 0.f;
        if (i < count) sample_at(g, r, i, pz, py, px);
        mine[96 * q + 3 * lane + 0] = pz;
        mine[96 * q + 3 * lane + 1] = py;
        mine[96 * q + 3 * lane + 2] = px;
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 3 * Q; ++k) v[k] = mine[32 * k + lane];
    }
#pragma unroll
    for (int k = 0; k < 3 * Q; ++k)
      if (32 * k + lane < n) out[3 * (int64_t)base + 32 * k + lane] = v[k];
  };
  // four runs at a time, with one a warp of a long ray waits for each
  const int end = (int)min((int64_t)S, (int64_t)(blockIdx.y + 1) * part);
  if (S > 64)
    for (int base = blockIdx.y * part; base < end; base += 32 * kRuns)
      write(base, std::integral_constant<int, kRuns>{});
  else
    for (int base = 0; base < S; base += 32) write(base, std::integral_constant<int, 1>{});
}

// Samples of a ray that a warp writes: all of them, or parts of at least 512 where the
// launch has fewer blocks than every second SM (200 rays x 4096 samples, cylinder: 30.8
// us with a warp a ray and one run at a time, 26.7 with four, 20.6 in parts; cone 18.5 ->
// 13.2).
int samples_per_warp(int num_rays, int S) {
  const int blocks = (int)ceil_div(num_rays, kWarpsPerBlock);
  const int parts = std::max(1, std::min(S / 512, 148 / blocks));
  return (int)ceil_div(ceil_div(S, parts), 128) * 128;
}

}  // namespace

int validate_geometry(const NectbGeometry* g) {
  NECTB_REQUIRE(g != nullptr, "geometry is null");
  NECTB_REQUIRE(g->kind >= NECTB_CONE_VOXEL && g->kind <= NECTB_PARALLEL_CYLINDRICAL, "unknown geometry kind %d",
                g->kind);
  NECTB_REQUIRE(g->nDetector[0] > 0 && g->nDetector[1] > 0, "nDetector must be positive");
  NECTB_REQUIRE((int64_t)g->nDetector[0] * g->nDetector[1] <= INT32_MAX, "nDetector has more than 2^31 - 1 pixels");
  return NECTB_OK;
}

}  // namespace nectb

extern "C" int nectb_sample(const NectbGeometry* geometry, const int64_t* random_ray_index,
                            int64_t random_ray_index_len, int64_t starting_ray_index, int32_t num_rays,
                            int32_t num_points_per_ray, float angle_rad, float max_ray_distance_per_point,
                            int32_t uniform_ray_spacing, const float* jitter, const float* detector_offset,
                            float* points, float* distances, int32_t* counts, void* stream) {
  using namespace nectb;
  clear_error();
  if (int rc = validate_geometry(geometry)) return rc;
  NECTB_REQUIRE(num_rays >= 0 && num_points_per_ray >= 0, "negative sizes");
  if (num_rays == 0) return NECTB_OK;
  NECTB_REQUIRE(random_ray_index && jitter && detector_offset && distances, "null input/output pointer");
  NECTB_REQUIRE((int64_t)num_rays * num_points_per_ray * 3 < (int64_t(1) << 40), "points tensor too large");
  const int part = samples_per_warp(num_rays, std::max(num_points_per_ray, 1));
  const dim3 blocks((unsigned)ceil_div(num_rays, kWarpsPerBlock),
                    points ? (unsigned)std::max<int64_t>(1, ceil_div(num_points_per_ray, part)) : 1u);
  ProfScope ps(kProfSample, (cudaStream_t)stream);
  sample_kernel<<<blocks, kWarpsPerBlock * 32, 0, (cudaStream_t)stream>>>(
      *geometry, random_ray_index, random_ray_index_len, starting_ray_index, num_rays, num_points_per_ray, part,
      angle_rad, max_ray_distance_per_point, uniform_ray_spacing, jitter, detector_offset, points, distances, counts);
  return launch_status("sample_kernel");
}
