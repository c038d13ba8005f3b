// Plain fp32 fused training step (SIMT MLP), the path the mixed-precision
// tensor-core kernels are measured against.
//
// Three launches per batch:
//   1. ray_prep_kernel   warp per ray: entry/exit, count, measured value.
//   2. fwd_plain_kernel  blocks step through tiles of 128 samples (32
//                        consecutive samples of each of four rays): encode,
//                        MLP, warp-shuffle sum along the ray -> y_pred, loss,
//                        dL/dsigma for the ray.
//   3. bwd_plain_kernel  the same tiles: re-encode, forward, backward through
//                        the MLP, fp32 weight-gradient tile products
//                        accumulated in registers, table gradients by vector
//                        atomics.
// Sample positions and encodings live only in registers and shared memory.
#include <algorithm>
#include <type_traits>

#include "mlp_tile.cuh"
#include "train_common.cuh"

namespace nectb {

__global__ void ray_prep_kernel(NectbGeometry g, TrainArgs a, RayRec* __restrict__ recs, int32_t* __restrict__ slot,
                                unsigned int* __restrict__ ctrl, float* __restrict__ y_pred, float* __restrict__ loss) {
  const int lane = threadIdx.x & 31;
  // The block's eight rays are set up by eight lanes: the fp64 divisions once per
  // ray instead of on every lane of its warp (512 x 512 rays: 422 -> 229 us, 138 of
  // that from the windowed count).
  constexpr int kRays = kRayPrepThreads / 32;
  __shared__ RaySetup setups[kRays];
  __shared__ int indices[kRays], slots[kRays];   // detector pixel (-1: outside the batch), scheduling slot
  const int n_batch = a.num_rays / a.sub;
  if (threadIdx.x < kRays) {
    const int v = blockIdx.x * kRays + threadIdx.x;
    RaySetup s;
    s.valid = 0;
    s.distance = 0.f;
    int ray_index = 0, sidx = 0;
    bool ok = false;
    if (v < a.num_rays) {
      // continuous scan: virtual ray v is pixel rb of the batch at sub-angle j
      const int j = v / n_batch, rb = v - j * n_batch;
      const float angle = a.sub > 1 ? a.sub_angle[j] : a.angle;
      // perm == nullptr: the detector pixels start, start + 1, ... in order
      // (re-projection queries, whole views or pieces of them; the slots are
      // indexed from the first pixel); jitter / detector offsets default to 0
      // when absent.
      if (a.perm) {
        ok = ray_lookup(a.perm, a.perm_len, a.start, rb, n_batch, g, ray_index);
        sidx = ray_index;
      } else {
        ray_index = (int)a.start + v;
        ok = v < a.n_pixels;
        sidx = v;
      }
      if (ok)
        ray_setup(g, ray_index, a.det_off ? a.det_off[2 * (int64_t)v] : 0.f,
                  a.det_off ? a.det_off[2 * (int64_t)v + 1] : 0.f, a.jitter ? a.jitter[v] : 0.f, angle, a.S, a.maxd,
                  a.uniform != 0, s);
    }
    setups[threadIdx.x] = s;
    indices[threadIdx.x] = ok && ray_index >= 0 ? ray_index : -1;
    slots[threadIdx.x] = sidx;
  }
  __syncthreads();
  const int tid = blockIdx.x * kRays + (threadIdx.x >> 5);
  if (tid >= a.num_rays) return;
  const RaySetup r = setups[threadIdx.x >> 5];
  const int ray_index = indices[threadIdx.x >> 5], sidx = slots[threadIdx.x >> 5], j = tid / n_batch;
  int count = 0;
  if (r.valid) count = warp_sample_count(g, r, a.S, lane);
  if (lane == 0) {
    RayRec rec;
    rec.sx = r.start.x;
    rec.sy = r.start.y;
    rec.sz = r.start.z;
    rec.dx = r.step.x;
    rec.dy = r.step.y;
    rec.dz = r.step.z;
    rec.count = count;
    rec.scale = r.distance / a.max_dist;
    // proj[perm[start:start+R]] (projector.py:130); rays past the end of the
    // permutation are not part of the reference batch and get y = 0 here.
    rec.y = (ray_index >= 0 && a.projection) ? a.projection[ray_index] : 0.f;
    rec.gsig = 0.f;
    if (count > 0) {
      if (atomicCAS(slot + (int64_t)sidx * a.sub + j, -1, tid) != -1) atomicOr(ctrl + 3, kFlagDuplicatePixels);
    } else {
      // no samples: y_pred = 0 (the reference's zero attenuation sum)
      y_pred[tid] = 0.f;
      rec.gsig = loss_grad(0.f, rec.y, a.loss_type, a.num_rays, rec.scale) * a.loss_scale;
      atomicAdd(loss, loss_term(0.f, rec.y, a.loss_type) / (float)a.num_rays);
    }
    recs[tid] = rec;
  }
}

__device__ __forceinline__ bool ordered_valid(const int32_t* __restrict__ slot, const RayRec* __restrict__ recs,
                                              bool by_pixel, int idx, int n, int cols, int sub, int* ray) {
  if (idx >= n) return false;
  const int r = by_pixel ? slot[strip_slot(idx, n, cols, sub)] : idx;
  *ray = r;
  return r >= 0 && recs[r].count > 0;
}

// Exclusive scan of one value per thread over a block of kOrderBlock threads
// (32 warps); returns the thread's prefix, *total the block's sum.  Callers
// that scan again into the same warp_sums synchronise first.
template <typename T>
__device__ __forceinline__ T block_scan(T v, T* warp_sums, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const T w = warp_sums[lane];
    T z = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T y = __shfl_up_sync(0xffffffffu, z, o);
      if (lane >= o) z += y;
    }
    warp_sums[lane] = z - w;  // exclusive over warps
    if (lane == 31) warp_sums[32] = z;
  }
  __syncthreads();
  *total = warp_sums[32];
  return warp_sums[warp] + x - v;
}

__global__ void __launch_bounds__(kOrderBlock)
order_count_kernel(const int32_t* __restrict__ slot, const RayRec* __restrict__ recs,
                   const unsigned int* __restrict__ ctrl, int R, int P, int cols, int sub,
                   unsigned int* __restrict__ block_sums,
                   unsigned long long* __restrict__ block_samples) {
  __shared__ unsigned int ws[33];
  __shared__ unsigned long long ws64[33];
  const bool by_pixel = !(ctrl[3] & kFlagDuplicatePixels);
  int ray = -1;
  const bool v = ordered_valid(slot, recs, by_pixel, blockIdx.x * kOrderBlock + threadIdx.x, by_pixel ? P : R, cols, sub,
                               &ray);
  unsigned int total;
  unsigned long long samples;
  block_scan<unsigned int>(v ? 1u : 0u, ws, &total);
  block_scan<unsigned long long>(v ? (unsigned long long)recs[ray].count : 0ull, ws64, &samples);
  if (threadIdx.x == 0) {
    block_sums[blockIdx.x] = total;
    block_samples[blockIdx.x] = samples;
  }
}

__global__ void __launch_bounds__(kOrderBlock)
order_scan_kernel(unsigned int* __restrict__ block_sums, unsigned long long* __restrict__ block_samples, int n_blocks,
                  unsigned int* __restrict__ ctrl) {
  __shared__ unsigned int ws[33];
  __shared__ unsigned long long ws64[33];
  unsigned int carry = 0;
  unsigned long long carry64 = 0;
  for (int b0 = 0; b0 < n_blocks; b0 += kOrderBlock) {  // block-uniform loop
    const int b = b0 + threadIdx.x;
    unsigned int total;
    unsigned long long total64;
    const unsigned int x = block_scan<unsigned int>(b < n_blocks ? block_sums[b] : 0u, ws, &total);
    const unsigned long long x64 = block_scan<unsigned long long>(b < n_blocks ? block_samples[b] : 0ull, ws64,
                                                                  &total64);
    if (b < n_blocks) {
      block_sums[b] = carry + x;
      block_samples[b] = carry64 + x64;
    }
    carry += total;
    carry64 += total64;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    ctrl[6] = carry;                        // rays with samples
    ctrl[9] = (unsigned)(carry64 / 32 + carry / 2);   // about their chunks of 32 samples
  }
}

__global__ void __launch_bounds__(kOrderBlock)
order_compact_kernel(const int32_t* __restrict__ slot, const RayRec* __restrict__ recs,
                     const unsigned int* __restrict__ ctrl, int R, int P, int cols, int sub,
                     const unsigned int* __restrict__ block_sums,
                     const unsigned long long* __restrict__ block_samples, int32_t* __restrict__ order,
                     uint64_t* __restrict__ offs) {
  __shared__ unsigned int ws[33];
  __shared__ unsigned long long ws64[33];
  const bool by_pixel = !(ctrl[3] & kFlagDuplicatePixels);
  int ray = -1;
  const bool v = ordered_valid(slot, recs, by_pixel, blockIdx.x * kOrderBlock + threadIdx.x, by_pixel ? P : R, cols, sub,
                               &ray);
  unsigned int total;
  unsigned long long samples;
  const unsigned int rank = block_scan<unsigned int>(v ? 1u : 0u, ws, &total);
  const unsigned long long off =
      block_scan<unsigned long long>(v ? (unsigned long long)recs[ray].count : 0ull, ws64, &samples);
  if (v) {
    order[block_sums[blockIdx.x] + rank] = ray;
    offs[block_sums[blockIdx.x] + rank] = block_samples[blockIdx.x] + off;
  }
}

namespace {

constexpr int kPlainFwdSamples = 128;

// Bound by shared-memory wavefronts (78 % of their rate) in the products and by
// the gathers' latency between them.  16,384 rays x 256 samples, 16 x 2 levels,
// 2 x 64: 2.49 -> 1.45 ms against one sample a thread, 0.91 ms of it the MLP (its
// multiply-adds take 0.49 ms).
// Three blocks an SM in 3D: 80 registers a thread; at 100 the same step 1.49 ms.  In 4D,
// 80 registers spill: 262,144 rays x 512 samples 65.0 ms with three blocks, 54.0 with two.
template <int D, int F, int L, int H>
__global__ void __launch_bounds__(kTileThreads, D == 4 ? 2 : 3)
fwd_plain_kernel(GridDev grid, const float* __restrict__ table, const float* __restrict__ W, TrainArgs a,
                 RayRec* __restrict__ recs, const int32_t* __restrict__ slot, unsigned int* __restrict__ ctrl,
                 int act, int out_act, float* __restrict__ y_pred, float* __restrict__ loss) {
  constexpr int IN = L * F, NT = kPlainFwdSamples, LD = NT + 4;
  const bool by_pixel = !(ctrl[3] & kFlagDuplicatePixels);
  extern __shared__ float4 smem4[];
  float* smem = reinterpret_cast<float*>(smem4);
  const SimtWeights sw = stage_weights<IN, H, false>(W, smem);
  TilePoints<NT>* pts = reinterpret_cast<TilePoints<NT>*>(smem + simt_weight_floats<IN, H, false>());
  float* buf = reinterpret_cast<float*>(pts + 1);   // every layer's columns in turn
  const int t = threadIdx.x, lane = t & 31;
  const bool owner = t < NT;   // the first NT threads hold the tile's samples, a warp 32 of one ray
  float loss_acc = 0.f, sum = 0.f;
  int ray = -1, base = 0;
  SlotClaim claim;
  RayRec rec;
  rec.count = 0;
  while (true) {
    bool valid = false;
    if (owner) {
      if (ray < a.num_rays && (ray < 0 || base >= rec.count)) {
        const int r = next_ray(claim, ctrl, slot, recs, a, by_pixel, lane);
        if (r < 0) {
          ray = a.num_rays;
          rec.count = 0;
        } else {
          rec = load_ray(recs, r);
          ray = r;
          base = 0;
          sum = 0.f;
        }
      }
      float p[4] = {0.f, 0.f, 0.f, 0.f};
      if (ray < a.num_rays && base + lane < rec.count) valid = sample_point(rec, base + lane, p);
#pragma unroll
      for (int k = 0; k < 3; ++k) pts->p[k * NT + t] = p[k];
      pts->valid[t] = valid ? 1 : 0;
    }
    if (!__syncthreads_or(owner && ray < a.num_rays)) break;
    encode_tile<D, F, L, NT, kTileThreads, float>(grid, table, pts->p, pts->valid, a.t, buf);
    __syncthreads();
    tile_hidden<IN, H, NT, kTileThreads>(sw, buf, buf, act);
    __syncthreads();
    if (owner && ray < a.num_rays) {
      if (valid) sum += act_fwd(dot_col<kWidth, LD>(sw.wout, buf + t), out_act);
      base += 32;
      if (base >= rec.count) {
        const float s = warp_sum(sum);
        if (lane == 0) {
          const float yp = s * rec.scale;
          y_pred[ray] = yp;
          recs[ray].gsig = loss_grad(yp, rec.y, a.loss_type, a.num_rays, rec.scale) * a.loss_scale;
          loss_acc += loss_term(yp, rec.y, a.loss_type);
        }
      }
    }
  }
  __shared__ float red[NT / 32];
  if (owner && lane == 0) red[t >> 5] = loss_acc;
  __syncthreads();
  if (t == 0) {
    float s = 0.f;
    for (int w = 0; w < NT / 32; ++w) s += red[w];
    atomicAdd(loss, s / (float)a.num_rays);
  }
}

// Shared-memory plan of the fp32 backward for IN inputs and H hidden layers:
// both weight copies and tiles of 64 samples where two such blocks share an SM
// (one block's gathers run beside the other's products), else 128, 64 or 32
// samples in one block, the last with the PyTorch-layout weights read from the
// global buffer through L1 (the deep models).
template <int IN, int H>
struct PlainBwdPlan {
  static constexpr size_t kBudget = 227 * 1024;
  static constexpr int kRows = IN > kWidth ? IN : kWidth;   // rows of a_H, then of the gradients
  static constexpr size_t bytes(int nt, bool both) {
    return (size_t)(both ? simt_weight_floats<IN, H, true>() : simt_weight_floats<IN, H, false>()) * 4 +
           (size_t)nt * 20 + (size_t)(IN + (H - 1) * kWidth + kRows) * (nt + 4) * 4;
  }
  static constexpr bool kTwo = bytes(64, true) <= 113 * 1024;
  static constexpr bool kBoth = bytes(32, true) <= kBudget;
  // rows of 76 inputs split into groups of 4 outputs only, which 32 samples need
  static constexpr int NT =
      IN % 8 != 0 ? 32 : (kTwo ? 64 : (bytes(128, kBoth) <= kBudget ? 128 : (bytes(64, kBoth) <= kBudget ? 64 : 32)));
  // 4 x 8 products a thread; the deep models' tiles of 32 samples take 4 x 2 and 4 x 4
  static constexpr int NTH = NT == 64 ? 128 : 256;
  static constexpr size_t smem = bytes(NT, kBoth);
  static_assert(smem <= kBudget, "fp32 backward does not fit shared memory");
  static_assert(sizeof(TilePoints<32>) == 32 * 20, "tile points");
};

// The fp32 backward over tiles of NT samples.  next(pts) has the block's
// threads write the next tile's points with their dL/dsigma and returns, after
// a barrier, whether there is one.
// Bound by shared-memory wavefronts (68 %) in the products, with the gathers and
// the table reductions beside them.  16,384 rays x 256 samples, 16 x 2 levels, 2 x
// 64: 10.96 -> 4.58 ms against one sample a thread (multiply-adds 1.96 ms;
// without the gathers 3.95, without the scatter 3.9, without the weight gradients
// 3.8 ms).  The gradients in a_H's place leave the L1 92 KB with two blocks an SM:
// 4.77 -> 4.58 ms.
template <int D, int F, int L, int H, typename T, typename Next>
__device__ __forceinline__ void plain_backward(const GridDev& grid, const T* __restrict__ table,
                                               const float* __restrict__ W, float tval, int act, int out_act,
                                               float* __restrict__ table_grad, float* __restrict__ W_grad,
                                               float* smem, Next&& next) {
  constexpr int IN = L * F;
  using Plan = PlainBwdPlan<IN, H>;
  constexpr int NT = Plan::NT, NTH = Plan::NTH, LD = NT + 4;
  constexpr int kSegment = 8;   // samples of a thread in the 4D scatter
  const SimtWeights sw = stage_weights<IN, H, Plan::kBoth>(W, smem);
  TilePoints<NT>& pts =
      *reinterpret_cast<TilePoints<NT>*>(smem + simt_weight_floats<IN, H, Plan::kBoth>());
  float* sX = reinterpret_cast<float*>(&pts + 1);   // [IN][LD]
  float* sA = sX + IN * LD;                         // [H][64][LD]  a_1..a_H
  float* sG = sA + (H - 1) * kWidth * LD;           // [max(64, IN)][LD]  the gradients, in a_H's place
  const int t = threadIdx.x;
  TileWGrad<IN, NT, NTH> g0;
  g0.zero();
  TileWGrad<kWidth, NT, NTH> gh[H - 1];
#pragma unroll
  for (int k = 0; k < H - 1; ++k) gh[k].zero();
  constexpr int RT = NTH / kWidth;   // threads of a row
  float dwout = 0.f;                 // of w_out[t / RT], over the thread's samples
  while (next(pts)) {
    encode_tile<D, F, L, NT, NTH, T>(grid, table, pts.p, pts.valid, tval, sX);
    __syncthreads();
    // forward: a_1..a_H into sA
    {
      TileProduct<IN, kWidth, NT, NTH> p;
      p.run(sw.WT[0], sX);
      p.store(sA, [&](float v, int) { return act_fwd(v, act); });
    }
#pragma unroll
    for (int k = 1; k < H; ++k) {
      __syncthreads();
      TileProduct<kWidth, kWidth, NT, NTH> p;
      p.run(sw.WT[k], sA + (k - 1) * kWidth * LD);
      p.store(sA + k * kWidth * LD, [&](float v, int) { return act_fwd(v, act); });
    }
    __syncthreads();
    const float* aH = sG;
    if (t < NT) {
      const float z = dot_col<kWidth, LD>(sw.wout, aH + t);
      pts.d[t] = pts.valid[t] ? pts.d[t] * act_grad_z(z, out_act) : 0.f;
    }
    __syncthreads();
    // w_out gradient, and G_H = dz * w_out * act'(a_H)
    {
      const int j = t / RT;
      const float wj = sw.wout[j];
#pragma unroll 4
      for (int s = 4 * (t % RT); s < NT; s += 4 * RT) {
        const float4 v = *reinterpret_cast<const float4*>(aH + j * LD + s);
        const float4 dz = *reinterpret_cast<const float4*>(pts.d + s);
        dwout = fmaf(dz.x, v.x, dwout);
        dwout = fmaf(dz.y, v.y, dwout);
        dwout = fmaf(dz.z, v.z, dwout);
        dwout = fmaf(dz.w, v.w, dwout);
        *reinterpret_cast<float4*>(sG + j * LD + s) =
            make_float4(dz.x * wj * act_grad_a(v.x, act), dz.y * wj * act_grad_a(v.y, act),
                        dz.z * wj * act_grad_a(v.z, act), dz.w * wj * act_grad_a(v.w, act));
      }
    }
#pragma unroll
    for (int k = H - 1; k >= 1; --k) {
      __syncthreads();
      const float* ak = sA + (k - 1) * kWidth * LD;
      gh[k - 1].add(sG, ak);
      // G_k = (W_k^T G_{k+1}) * act'(a_k); W_k is [64 out][64 in] = M[j][i]
      TileProduct<kWidth, kWidth, NT, NTH> p;
      p.run(sw.W[k], sG);
      __syncthreads();
      p.store(sG, [&](float v, int at) { return v * act_grad_a(ak[at], act); });
    }
    __syncthreads();
    g0.add(sG, sX);
    // dX = W_0^T G_1 (W_0 is [64][IN] = M[j][i]), then the scatter
    {
      TileProduct<kWidth, IN, NT, NTH> p;
      p.run(sw.W[0], sG);
      __syncthreads();
      p.store(sG, [&](float v, int) { return v; });
    }
    __syncthreads();
    if constexpr (D == 4) {
      // A thread takes one level of kSegment consecutive samples and marches over
      // them: 16 reductions a sample and level otherwise (300,007 points along rays, 16 x
      // 2 levels: 0.91 -> 0.81 ms; 16 x 4: 1.43 -> 1.34).  Points in no order, which a
      // training loop does not pass, lose 3 to 6 % by it (300,007: 1.46 -> 1.52, 16 x 4
      // 2.24 -> 2.30 ms), 10,000 of either kind nothing.  With the 8 of 3D, sample by
      // sample is the faster (16,384 rays x 256: 4.58 against 5.31 ms).
      for (int e = t; e < L * (NT / kSegment); e += NTH) {
        const int l = e / (NT / kSegment), first = e % (NT / kSegment) * kSegment;
        auto march = [&](auto hashed) {
          CellMarch<D, F, hashed()> m(grid, l, table_grad, tval);
#pragma unroll 1
          for (int s = first; s < first + kSegment; ++s) {
            if (!pts.valid[s]) continue;
            const float x[3] = {pts.p[s], pts.p[NT + s], pts.p[2 * NT + s]};
            float d[F];
#pragma unroll
            for (int f = 0; f < F; ++f) d[f] = sG[(l * F + f) * LD + s];
            m.add(x, d);
          }
          m.finish();
        };
        if ((grid.hashed_bits >> l) & 1u)
          march(std::true_type{});
        else
          march(std::false_type{});
      }
    } else {
      const int s = t % NT;
      if (pts.valid[s]) {
        const float x[3] = {pts.p[s], pts.p[NT + s], pts.p[2 * NT + s]};
#pragma unroll 1
        for (int l = t / NT; l < L; l += NTH / NT) {
          float d[F];
#pragma unroll
          for (int f = 0; f < F; ++f) d[f] = sG[(l * F + f) * LD + s];
          scatter_level<D, F>(grid, table_grad, l, x, d);
        }
      }
    }
    __syncthreads();
  }
  g0.flush(W_grad);
#pragma unroll
  for (int k = 0; k < H - 1; ++k) gh[k].flush(W_grad + kWidth * IN + k * kWidth * kWidth);
#pragma unroll
  for (int o = 1; o < RT; o <<= 1) dwout += __shfl_xor_sync(0xffffffffu, dwout, o);
  if (t % RT == 0) atomicAdd(W_grad + kWidth * IN + (H - 1) * kWidth * kWidth + t / RT, dwout);
}

// Blocks of the fp32 backward: two to an SM where the plan fits twice.
template <int IN, int H>
__host__ __device__ constexpr int plain_bwd_per_sm() {
  return PlainBwdPlan<IN, H>::kTwo ? 2 : 1;
}

// The training backward: tiles of 32 consecutive samples of each of NT / 32 rays.
template <int D, int F, int L, int H>
__global__ void __launch_bounds__(PlainBwdPlan<L * F, H>::NTH, plain_bwd_per_sm<L * F, H>())
bwd_plain_kernel(GridDev grid, const float* __restrict__ table, const float* __restrict__ W, TrainArgs a,
                 const RayRec* __restrict__ recs, const int32_t* __restrict__ slot, unsigned int* __restrict__ ctrl,
                 int act, int out_act, float* __restrict__ table_grad, float* __restrict__ W_grad) {
  constexpr int NT = PlainBwdPlan<L * F, H>::NT;
  const bool by_pixel = !(ctrl[3] & kFlagDuplicatePixels);
  extern __shared__ float4 smem4[];
  const int t = threadIdx.x, lane = t & 31;
  int ray = -1, base = 0;
  SlotClaim claim;
  RayRec rec;
  rec.count = 0;
  rec.gsig = 0.f;
  plain_backward<D, F, L, H>(
      grid, table, W, a.t, act, out_act, table_grad, W_grad, reinterpret_cast<float*>(smem4),
      [&](TilePoints<NT>& pts) -> bool {
        bool active = false;
        if (t < NT) {
          if (ray < a.num_rays && (ray < 0 || base >= rec.count)) {
            const int r = next_ray(claim, ctrl + 1, slot, recs, a, by_pixel, lane);
            if (r < 0) {
              ray = a.num_rays;
              rec.count = 0;
            } else {
              rec = load_ray(recs, r);
              ray = r;
              base = 0;
            }
          }
          active = ray < a.num_rays;
          float p[4] = {0.f, 0.f, 0.f, 0.f};
          const bool valid = active && base + lane < rec.count && sample_point(rec, base + lane, p);
#pragma unroll
          for (int k = 0; k < 3; ++k) pts.p[k * NT + t] = p[k];
          pts.valid[t] = valid ? 1 : 0;
          pts.d[t] = rec.gsig;
          base += 32;
        }
        return __syncthreads_or(active) != 0;
      });
}

// Backward of the model at n independent points (nectb_model_backward):
// gradients of sum_i dsigma[i] * sigma(x_i) added to the table and weight
// gradients, the points read from x (n x 3, (z, y, x); t broadcast in 4D).
// Tables of either precision are gathered.
template <int D, int F, int L, int H, typename T>
__global__ void __launch_bounds__(PlainBwdPlan<L * F, H>::NTH, plain_bwd_per_sm<L * F, H>())
model_bwd_kernel(GridDev grid, const T* __restrict__ table, const float* __restrict__ W, const float* __restrict__ x,
                 int64_t n, float tval, const float* __restrict__ t_dev, const float* __restrict__ dsigma, int act,
                 int out_act, float* __restrict__ table_grad, float* __restrict__ W_grad) {
  constexpr int NT = PlainBwdPlan<L * F, H>::NT;
  extern __shared__ float4 smem4[];
  const int t = threadIdx.x;
  if (D == 4 && t_dev) tval = *t_dev;   // the broadcast timestep, read on the device
  int64_t c0 = (int64_t)blockIdx.x * NT;
  plain_backward<D, F, L, H>(
      grid, table, W, tval, act, out_act, table_grad, W_grad, reinterpret_cast<float*>(smem4),
      [&](TilePoints<NT>& pts) -> bool {
        if (c0 >= n) return false;
        if (t < NT) {
          const int64_t i = c0 + t;
          const bool valid = i < n;
#pragma unroll
          for (int k = 0; k < 3; ++k) pts.p[k * NT + t] = valid ? x[i * 3 + k] : 0.f;
          pts.valid[t] = valid ? 1 : 0;
          pts.d[t] = valid ? dsigma[i] : 0.f;
        }
        c0 += (int64_t)gridDim.x * NT;
        __syncthreads();
        return true;
      });
}

template <int D, int F, int L, int H, typename T>
int launch_model_bwd(const GridDev& grid, const void* table, const float* W, const float* x, int64_t n, float tval,
                     const float* t_dev, const float* dsigma, int act, int out_act, float* table_grad, float* W_grad,
                     cudaStream_t s) {
  constexpr int IN = L * F;
  using Plan = PlainBwdPlan<IN, H>;
  auto k = model_bwd_kernel<D, F, L, H, T>;
  const size_t smem = Plan::smem;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int blocks =
      (int)std::max<int64_t>(1, std::min<int64_t>(plain_bwd_per_sm<IN, H>() * sms, ceil_div(n, Plan::NT)));
  ProfScope ps(kProfModel, s);
  k<<<blocks, Plan::NTH, smem, s>>>(grid, (const T*)table, W, x, n, tval, t_dev, dsigma, act, out_act, table_grad, W_grad);
  return launch_status("model_bwd_kernel");
}

template <int D, int F, int L, int H>
int run_plain(const NectbGeometry& geo, const GridDev& grid, const float* table, const float* W, const TrainArgs& a,
              Workspace ws, int act, int out_act, float* table_grad, float* W_grad, float* y_pred, float* loss,
              cudaStream_t s) {
  constexpr int IN = L * F;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  (void)geo;

  auto fk = fwd_plain_kernel<D, F, L, H>;
  const size_t fsmem = tile_forward_smem<IN, H, kPlainFwdSamples>();
  set_smem(fk, fsmem, a.max_blocks > 0);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fk, kTileThreads, fsmem);
  int fblocks = std::max(1, std::min<int>(sms * std::max(per_sm, 1), (int)ceil_div(a.num_rays, kPlainFwdSamples / 32)));
  if (a.max_blocks > 0) fblocks = std::min(fblocks, a.max_blocks);
  if (a.phase & kPhaseForward) {
    {
      ProfScope ps(kProfForward, s);
      fk<<<fblocks, kTileThreads, fsmem, s>>>(grid, table, W, a, ws.rays, ws.slot, ws.counters, act, out_act, y_pred, loss);
    }
    if (int rc = launch_status("fwd_plain_kernel")) return rc;
  }
  if (!table_grad || !(a.phase & kPhaseBackward)) return NECTB_OK;  // forward only (queries, split step)

  using Plan = PlainBwdPlan<IN, H>;
  auto bk = bwd_plain_kernel<D, F, L, H>;
  const size_t bsmem = Plan::smem;
  cudaFuncSetAttribute(bk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsmem);
  const int bblocks =
      std::max(1, std::min<int>(plain_bwd_per_sm<IN, H>() * sms, (int)ceil_div(a.num_rays, Plan::NT / 32)));
  {
    ProfScope ps(kProfBackward, s);
    bk<<<bblocks, Plan::NTH, bsmem, s>>>(grid, table, W, a, ws.rays, ws.slot, ws.counters, act, out_act,
                                            table_grad, W_grad);
  }
  return launch_status("bwd_plain_kernel");
}

}  // namespace

int model_backward(const GridDev& g, const NectbMLP& mlp, int dtype, const void* table, const float* W,
                   const float* x, int64_t n, float tval, const float* t_dev, const float* dsigma, float* table_grad,
                   float* W_grad, cudaStream_t s) {
  const bool h = dtype == NECTB_F16;
  const int D = g.n_dims, F = g.n_features, L = g.n_levels, H = mlp.n_hidden_layers;
  const int act = mlp.activation, oact = mlp.output_activation;
  const int rc = dispatch_shape(D, F, L, H, [&](auto d, auto f, auto l, auto hl) {
    return h ? launch_model_bwd<d(), f(), l(), hl(), __half>(g, table, W, x, n, tval, t_dev, dsigma, act, oact,
                                                             table_grad, W_grad, s)
             : launch_model_bwd<d(), f(), l(), hl(), float>(g, table, W, x, n, tval, t_dev, dsigma, act, oact,
                                                            table_grad, W_grad, s);
  });
  if (rc != kUnsupportedShape) return rc;
  return set_error(NECTB_ERR_INVALID, "model backward: unsupported configuration (n_dims %d, n_features %d, "
                   "n_levels %d, hidden %d)", D, F, L, H);
}

int train_plain(const NectbGeometry& geo, const GridDev& grid, const NectbMLP& mlp, const float* table,
                const float* W, int nW, const TrainArgs& a, Workspace ws, float* table_grad, float* W_grad,
                float* y_pred, float* loss, cudaStream_t s) {
  (void)nW;
  const int D = grid.n_dims, F = grid.n_features, L = grid.n_levels, H = mlp.n_hidden_layers;
  const int act = mlp.activation, oact = mlp.output_activation;
  const int rc = dispatch_shape(D, F, L, H, [&](auto d, auto f, auto l, auto h) {
    return run_plain<d(), f(), l(), h()>(geo, grid, table, W, a, ws, act, oact, table_grad, W_grad, y_pred, loss,
                                         s);
  });
  if (rc != kUnsupportedShape) return rc;
  return set_error(NECTB_ERR_INVALID, "plain path: unsupported model shape (n_dims %d, n_features %d, n_levels %d, "
                   "hidden %d)", D, F, L, H);
}

}  // namespace nectb
