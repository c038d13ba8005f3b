// Query kernels: slice / volume points and detector re-projections of a
// trained model.
//
// nectb_query_points runs one persistent launch over the 128-point chunks of
// any number of work items (slices, volume slabs) of any number of requests:
// each block takes chunks from an atomic cursor, finds the chunk's item by
// binary search over the items' chunk offsets, generates the points from the
// item's origin and step vectors (no coordinate arrays in memory), evaluates
// the model and writes de-normalised values.  The mixed model runs its MLP on
// tcgen05 (the forward tile of the training kernel); the plain model the fp32
// SIMT MLP.  nectb_query_reproject reuses the fused training forward over all
// detector pixels of a view.
#include <algorithm>

#include "mixed_common.cuh"
#include "mlp_tile.cuh"
#include "train_common.cuh"

namespace nectb {

int validate_geometry(const NectbGeometry* g);
int validate_mlp(const NectbMLP* m, const GridDev& g);
int64_t mlp_param_count(const NectbMLP* m);
int train_forward_only(const NectbGeometry& geo, const GridDev& grid, const NectbMLP& mlp, const void* table,
                       const float* W, const TrainArgs& a, Workspace ws, float* y_pred, float* loss, cudaStream_t s);
int launch_time_slice(const GridDev& grid, const __half* table, float t, __half* slice, cudaStream_t s);

namespace {

constexpr int kQThreads = 128;
__device__ __forceinline__ int find_item(const NectbQueryItem* __restrict__ items, int n, int64_t chunk) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (items[mid].chunk_begin <= chunk)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

struct QPoint {
  float p[4];
  bool valid;
  float* dst;
  float scale, offset;
};

__device__ __forceinline__ QPoint query_point(const NectbQueryItem& it, int64_t chunk, int t) {
  QPoint q;
  const int64_t k = (chunk - it.chunk_begin) * 128 + t;
  const int64_t n = (int64_t)it.nu * it.nv;
  q.valid = k < n;
  q.p[0] = q.p[1] = q.p[2] = 0.f;
  q.p[3] = it.t;
  q.dst = nullptr;
  q.scale = it.out_scale;
  q.offset = it.out_offset;
  if (q.valid) {
    const int i = (int)(k % it.nu), j = (int)(k / it.nu);
#pragma unroll
    for (int a = 0; a < 3; ++a) q.p[a] = clamp01f(it.origin[a] + (float)i * it.du[a] + (float)j * it.dv[a]);
    q.dst = it.out + (int64_t)j * it.out_stride + i;
  }
  return q;
}

// A stack: items that differ only in their place along axis 0 and their output (the
// z-slices of a volume).  Neighbours along axis 0 follow each other in a level's
// entries (hash prime and stride 1), so a warp's lanes take 2^lanes_log2 items at
// the same point of their planes, where 32 points of one item would touch up to 32
// lines per corner (256^3 points of the 19 x 4 model: 12.6 -> 3.6 ms, the L2's random
// sectors before, instruction issue, 64 %, now; 129^3 fp32 1.06 -> 0.92): a tile is 2^lanes_log2 items by 128 / 2^lanes_log2 points.
struct Stack {
  int lanes_log2;   // < 0: not a stack
  int64_t tiles;    // of the whole stack
};
constexpr int kStackItems = 4096;   // most items looked through

// Whether the items are a stack; all threads of the block call.
__device__ __forceinline__ Stack find_stack(const NectbQueryItem* __restrict__ items, int n, int64_t total_chunks) {
  const NectbQueryItem a = items[0];
  const int64_t points = (int64_t)a.nu * a.nv, m = (points + 127) / 128;
  bool ok = n >= 8 && n <= kStackItems && points > 0 && a.du[0] == 0.f && a.dv[0] == 0.f && m * n == total_chunks &&
            total_chunks < (int64_t(1) << 28);
  if (ok) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const NectbQueryItem& b = items[i];
      ok = ok && b.nu == a.nu && b.nv == a.nv && b.origin[1] == a.origin[1] && b.origin[2] == a.origin[2] &&
           b.t == a.t && b.out_scale == a.out_scale && b.out_offset == a.out_offset && b.out_stride == a.out_stride &&
           b.chunk_begin == i * m;
#pragma unroll
      for (int k = 0; k < 3; ++k) ok = ok && b.du[k] == a.du[k] && b.dv[k] == a.dv[k];
    }
  }
  Stack s;
  s.lanes_log2 = -1;
  s.tiles = total_chunks;
  if (__syncthreads_and(ok)) {
    // 32 items a warp unless that leaves more than a sixteenth of the lanes without one
    s.lanes_log2 = 5;
    while (s.lanes_log2 > 3 && (((n - 1) >> s.lanes_log2) + 1 << s.lanes_log2) - n > n / 16) --s.lanes_log2;
    s.tiles = (((int64_t)n - 1 >> s.lanes_log2) + 1) * ((points + (128 >> s.lanes_log2) - 1) >> (7 - s.lanes_log2));
  }
  return s;
}

// Point of thread t of a stack's tile.
__device__ __forceinline__ QPoint stack_point(const NectbQueryItem* __restrict__ items, int n, const Stack& s,
                                              int64_t tile, int t) {
  const NectbQueryItem& a = items[0];
  const int64_t points = (int64_t)a.nu * a.nv;
  const int per = 128 >> s.lanes_log2;   // points of an item in a tile
  const int64_t per_group = (points + per - 1) / per;
  const int64_t group = tile / per_group;
  const int64_t item = (group << s.lanes_log2) + (t & ((1 << s.lanes_log2) - 1));
  const int64_t k = (tile - group * per_group) * per + (t >> s.lanes_log2);
  QPoint q;
  q.valid = item < n && k < points;
  q.p[0] = q.p[1] = q.p[2] = 0.f;
  q.p[3] = a.t;
  q.dst = nullptr;
  q.scale = a.out_scale;
  q.offset = a.out_offset;
  if (q.valid) {
    const int i = (int)(k % a.nu), j = (int)(k / a.nu);
    q.p[0] = clamp01f(items[item].origin[0] + (float)i * a.du[0] + (float)j * a.dv[0]);
#pragma unroll
    for (int c = 1; c < 3; ++c) q.p[c] = clamp01f(a.origin[c] + (float)i * a.du[c] + (float)j * a.dv[c]);
    q.dst = items[item].out + (int64_t)j * a.out_stride + i;
  }
  return q;
}

// A block is n_wg = blockDim / 128 independent warpgroups sharing one copy of
// the weight tiles; each takes chunks of 128 points on its own, with its own X
// tiles (which the layers' activations overwrite), 64 TMEM columns, mbarrier and
// named barrier.  kMaxWg = 1: one warpgroup a block, at most 128 registers, so
// that three blocks share an SM with other kernels (capped grids: a server's
// lanes).  kMaxWg > 1: one block an SM for a launch that has the GPU to itself.
// Waits on the gathers and on the layers' chain of products, so the more
// warpgroups an SM holds the better: 256^3 points of the 19 x 4 model with 6
// layers (one 107 KB block an SM before) 17.8 -> 12.5 ms, a 256^2 slice of the 4D
// 16 x 2 model 49.5 -> 35.7 us.
template <int D, int F, int L, int H, int ACT, int kMaxWg>
__global__ void __launch_bounds__(kQThreads * kMaxWg, kMaxWg == 1 ? 4 : 1)
query_mixed_kernel(GridDev grid, const __half* __restrict__ table, const float* __restrict__ W,
                   const NectbQueryItem* __restrict__ items, int n_items, int64_t total_chunks,
                   unsigned int* __restrict__ counter, int out_act) {
  using S = InShape<L, F>;
  constexpr int KT = S::KT;
  constexpr int act = ACT;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = align1024(smem_raw);
  const int n_wg = blockDim.x / kQThreads;
  uint8_t* sW = base;                   // KT + H - 1 weight tiles
  float* sWout = reinterpret_cast<float*>(sW + (KT + H - 1) * kWTile + n_wg * KT * kTile);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sWout + 64);              // [kMaxWg]
  long long* chunks = reinterpret_cast<long long*>(bars + kMaxWg);       // [kMaxWg]
  int* item = reinterpret_cast<int*>(chunks + kMaxWg);                   // [kMaxWg]
  uint32_t* tslot = reinterpret_cast<uint32_t*>(item + kMaxWg);

  const int t = threadIdx.x, warp = t >> 5;
  const int wg = t / kQThreads, r = t % kQThreads;
  uint8_t* sX = sW + (KT + H - 1) * kWTile + wg * KT * kTile;
  uint64_t* bar = bars + wg;
  // fp32 weights -> bf16 swizzled tiles (same layout as the training kernels)
  stage_mixed_weights<L, F, H>(W, sW, sWout);
  const uint32_t ncols = wg_tmem_cols(n_wg);
  if (warp == 0) {
    tc::tmem_alloc(tslot, ncols);
    tc::tmem_relinquish();
  }
  if (r == 0) tc::mbar_init(bar, 1);
  tc::fence_async_smem();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const Stack stack = find_stack(items, n_items, total_chunks);
  const uint32_t tm = *tslot + 64u * wg;   // this warpgroup's columns
  const uint32_t my_lanes = tm + ((uint32_t)(32 * (warp & 3)) << 16);
  const uint32_t sX_a = tc::smem_u32(sX), sW_a = tc::smem_u32(sW);
  constexpr uint32_t idesc = tc::idesc_bf16(128, 64, false, false);
  uint32_t phase = 0;
  bool timed_out = false;
  while (true) {
    if (r == 0) {
      const long long c = (long long)atomicAdd(counter, 1u);
      chunks[wg] = c;
      item[wg] = c < stack.tiles && stack.lanes_log2 < 0 ? find_item(items, n_items, c) : 0;
    }
    wg_sync(wg);
    const long long chunk = chunks[wg];
    if (chunk >= stack.tiles) break;
    const QPoint q = stack.lanes_log2 < 0 ? query_point(items[item[wg]], chunk, r)
                                          : stack_point(items, n_items, stack, chunk, r);
    encode_row<D, F, L>(grid, table, q.p, q.valid, sX, r);   // the encoder's row writer (fp16 gathers, bf16 row)
    // every layer writes the warpgroup's 64 TMEM columns; its input is X for
    // k = 0, else the previous layer's activations, which overwrite X's first
    // tile once layer 0's product has completed
    float z = 0.f;
#pragma unroll
    for (int k = 0; k < H; ++k) {
      tc::fence_async_smem();
      tc::fence_before();
      wg_sync(wg);
      if (r == 0) {
        tc::fence_after();
        if (k == 0) {
#pragma unroll
          for (int c = 0; c < S::INP / 16; ++c)
            tc::mma(tm, tc::desc_k(sX_a + (c / 4) * kTile, c % 4), tc::desc_k(sW_a + (c / 4) * kWTile, c % 4), idesc,
                    c > 0);
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            tc::mma(tm, tc::desc_k(sX_a, c), tc::desc_k(sW_a + (KT + k - 1) * kWTile, c), idesc, c > 0);
        }
        tc::commit(bar);
      }
      timed_out = !tc::mbar_wait(bar, phase);
      phase ^= 1;
      if (wg_or(wg, timed_out)) {
        timed_out = true;
        break;
      }
      tc::fence_after();
#pragma unroll
      for (int half = 0; half < 2; ++half) {   // 32 columns at a time
        float v[32];
        tc::tmem_ld16(my_lanes + 32 * half, v);
        tc::tmem_ld16(my_lanes + 32 * half + 16, v + 16);
        tc::tmem_wait_ld();
        if (k + 1 < H) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float a8[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) a8[j] = hidden_act(v[8 * c + j], act);
            tc::st_chunk_bf16(sX, r, 4 * half + c, a8);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) z = fmaf(sWout[32 * half + j], hidden_act(v[j], act), z);
        }
      }
    }
    if (timed_out) break;
    if (q.valid) *q.dst = fmaf(act_fwd(z, out_act), q.scale, q.offset);
    tc::fence_before();
  }
  if (timed_out) {
    tc::mbar_wait(bar, phase);  // let the MMA in flight finish before TMEM is freed
    if (r == 0) atomicOr(counter + 1, 1u);
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after();
    tc::tmem_dealloc(*tslot, ncols);
  }
}

// Warpgroups of the wide form: as many as the registers of the shape allow (80 a
// thread for 3D grids of 16 levels and two layers, 102 for the deep model, 128
// otherwise; the training forward's numbers) and the shared memory holds.
template <int D, int L, int F, int H>
struct QueryShape {
  using S = InShape<L, F>;
  static constexpr size_t bytes(int n_wg) {
    return 1024 + (S::KT + H - 1) * kWTile + (size_t)n_wg * S::KT * kTile + 64 * 4 + 6 * 20 + 16;
  }
  static constexpr int kRegWg = D == 3 ? (H == 2 ? 6 : (L == 16 ? 4 : 5)) : 4;
  static constexpr int kMaxWg = bytes(kRegWg) <= 227 * 1024 ? kRegWg : 4;
  static_assert(bytes(kMaxWg) <= 227 * 1024 && kMaxWg * 64 <= 512, "query block");
};

// fp32: a chunk is a tile of 128 points (mlp_tile.cuh).
template <int D, int F, typename T, int L, int H>
__global__ void __launch_bounds__(kTileThreads)
query_plain_kernel(GridDev grid, const T* __restrict__ table, const float* __restrict__ W,
                   const NectbQueryItem* __restrict__ items, int n_items, int64_t total_chunks,
                   unsigned int* __restrict__ counter, int act, int out_act) {
  constexpr int IN = L * F, NT = 128, LD = NT + 4;
  extern __shared__ float4 smem4[];
  float* smem = reinterpret_cast<float*>(smem4);
  const SimtWeights sw = stage_weights<IN, H, false>(W, smem);
  TilePoints<NT>* pts = reinterpret_cast<TilePoints<NT>*>(smem + simt_weight_floats<IN, H, false>());
  float* buf = reinterpret_cast<float*>(pts + 1);
  __shared__ long long s_chunk;
  __shared__ int s_item;
  const int t = threadIdx.x;
  const Stack stack = find_stack(items, n_items, total_chunks);
  while (true) {
    if (t == 0) {
      const long long c = (long long)atomicAdd(counter, 1u);
      s_chunk = c;
      s_item = c < stack.tiles && stack.lanes_log2 < 0 ? find_item(items, n_items, c) : 0;
    }
    __syncthreads();
    const long long chunk = s_chunk;
    if (chunk >= stack.tiles) break;
    const NectbQueryItem& it = items[s_item];
    QPoint q;
    q.valid = false;
    if (t < NT) {
      q = stack.lanes_log2 < 0 ? query_point(it, chunk, t) : stack_point(items, n_items, stack, chunk, t);
#pragma unroll
      for (int k = 0; k < 3; ++k) pts->p[k * NT + t] = q.p[k];
      pts->valid[t] = q.valid ? 1 : 0;
    }
    const float tval = it.t;
    __syncthreads();
    encode_tile<D, F, L, NT, kTileThreads, T>(grid, table, pts->p, pts->valid, tval, buf);
    __syncthreads();
    tile_hidden<IN, H, NT, kTileThreads>(sw, buf, buf, act);
    __syncthreads();
    if (q.valid) *q.dst = fmaf(act_fwd(dot_col<kWidth, LD>(sw.wout, buf + t), out_act), q.scale, q.offset);
  }
}

int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int D, int F, int L, int H, int ACT>
int launch_query_mixed(const GridDev& g, const void* table, const float* W, const NectbQueryItem* items, int n,
                       int64_t chunks, unsigned int* counter, int oact, int max_blocks, cudaStream_t s) {
  using Q = QueryShape<D, L, F, H>;
  GridDev gt = g;  // with a texture over the table for the gathers
  gt.tex = table_texture(table, (size_t)g.total_entries * F * sizeof(__half), F * (int)sizeof(__half));
  ProfScope ps(kProfModel, s);
  if (max_blocks > 0) {
    auto k = query_mixed_kernel<D, F, L, H, ACT, 1>;
    set_smem(k, Q::bytes(1), true);
    const int blocks =
        (int)std::max<int64_t>(1, std::min<int64_t>({chunks, 3 * (int64_t)sm_count(), (int64_t)max_blocks}));
    k<<<blocks, kQThreads, Q::bytes(1), s>>>(gt, (const __half*)table, W, items, n, chunks, counter, oact);
  } else {
    // a launch below one chunk a warpgroup spreads over the SMs first
    auto k = query_mixed_kernel<D, F, L, H, ACT, Q::kMaxWg>;
    const int sms = sm_count();
    const int wgs = (int)std::max<int64_t>(1, std::min<int64_t>(Q::kMaxWg, ceil_div(chunks, sms)));
    set_smem(k, Q::bytes(Q::kMaxWg), false);
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(chunks, wgs), sms));
    k<<<blocks, kQThreads * wgs, Q::bytes(wgs), s>>>(gt, (const __half*)table, W, items, n, chunks, counter, oact);
  }
  return launch_status("query_mixed_kernel");
}

template <int D, int F, typename T, int L, int H>
int launch_query_plain(const GridDev& g, const void* table, const float* W, const NectbQueryItem* items, int n,
                       int64_t chunks, unsigned int* counter, int act, int oact, int max_blocks, cudaStream_t s) {
  constexpr int IN = L * F;
  auto k = query_plain_kernel<D, F, T, L, H>;
  const size_t smem = tile_forward_smem<IN, H, 128>();
  set_smem(k, smem, true);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kTileThreads, smem);
  int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(chunks, (int64_t)sm_count() * std::max(per_sm, 1)));
  if (max_blocks > 0) blocks = std::min(blocks, max_blocks);
  ProfScope ps(kProfModel, s);
  k<<<blocks, kTileThreads, smem, s>>>(g, (const T*)table, W, items, n, chunks, counter, act, oact);
  return launch_status("query_plain_kernel");
}

}  // namespace
}  // namespace nectb

using namespace nectb;

namespace {

// Items of one launch on grid g (a 3D or 4D table, or the 3D view of a 4D
// table's time slice).
int query_points_impl(const GridDev& g, bool f16_table, const NectbMLP* mlp, const void* grid_params,
                      const float* mlp_params, const NectbQueryItem* items, int32_t n_items, int64_t total_chunks,
                      unsigned int* counter, int32_t max_blocks, cudaStream_t s) {
  if (int rc = validate_mlp(mlp, g)) return rc;
  if (n_items == 0 || total_chunks == 0) return NECTB_OK;
  NECTB_REQUIRE(grid_params && mlp_params && items && counter && n_items > 0 && total_chunks > 0,
                "null pointer or empty query");
  NECTB_REQUIRE(total_chunks < (int64_t(1) << 31), "too many chunks in one launch");
  NECTB_REQUIRE(((uintptr_t)grid_params & 15u) == 0, "grid_params must be 16-byte aligned");
  if (int rc = cuda_status(cudaMemsetAsync(counter, 0, sizeof(unsigned int), s), "memset query counter")) return rc;
  const int D = g.n_dims, F = g.n_features, L = g.n_levels, H = mlp->n_hidden_layers;
  const int act = mlp->activation, oact = mlp->output_activation;
  const bool mixed = mlp->compute_dtype != NECTB_F32;
  if (mixed) {
    NECTB_REQUIRE(f16_table, "mixed queries need an fp16 table");
    NECTB_REQUIRE(H >= 2, "mixed queries need at least 2 hidden layers");
    const int rc = dispatch_shape(D, F, L, H, [&](auto d, auto f, auto l, auto h) {
      if (act == NECTB_ACT_RELU)
        return launch_query_mixed<d(), f(), l(), h(), NECTB_ACT_RELU>(g, grid_params, mlp_params, items, n_items,
                                                                       total_chunks, counter, oact, max_blocks, s);
      if constexpr (l() != 16) {
        if (act == NECTB_ACT_LEAKY_RELU)
          return launch_query_mixed<d(), f(), l(), h(), NECTB_ACT_LEAKY_RELU>(
              g, grid_params, mlp_params, items, n_items, total_chunks, counter, oact, max_blocks, s);
      }
      return set_error(NECTB_ERR_INVALID, "mixed queries: hidden activation %d is not instantiated for this shape",
                       act);
    });
    if (rc != kUnsupportedShape) return rc;
  } else {
    const int rc = dispatch_shape(D, F, L, H, [&](auto d, auto f, auto l, auto hl) {
      return f16_table ? launch_query_plain<d(), f(), __half, l(), hl()>(g, grid_params, mlp_params, items, n_items,
                                                                         total_chunks, counter, act, oact,
                                                                         max_blocks, s)
                       : launch_query_plain<d(), f(), float, l(), hl()>(g, grid_params, mlp_params, items, n_items,
                                                                        total_chunks, counter, act, oact,
                                                                        max_blocks, s);
    });
    if (rc != kUnsupportedShape) return rc;
  }
  return set_error(NECTB_ERR_INVALID, "queries: unsupported configuration (n_dims %d, n_features %d, n_levels %d, "
                   "hidden %d)", D, F, L, H);
}

// A 4D fp16 grid's slice layout, or false.
bool slice_grid(const NectbHashGrid* grid, GridDev* g3) {
  GridDev g;
  if (!grid || grid->n_dims != 4 || grid->feature_dtype != NECTB_F16 || !make_grid_dev(grid, &g)) return false;
  *g3 = make_time_slice(g, 0.f).g3;
  return true;
}

}  // namespace

extern "C" int nectb_query_points(const NectbHashGrid* grid, const NectbMLP* mlp, const void* grid_params,
                                  const float* mlp_params, const NectbQueryItem* items, int32_t n_items,
                                  int64_t total_chunks, unsigned int* counter, int32_t max_blocks, void* stream) {
  clear_error();
  GridDev g;
  if (!make_grid_dev(grid, &g)) return set_error(NECTB_ERR_INVALID, "invalid hash grid description");
  return query_points_impl(g, grid->feature_dtype == NECTB_F16, mlp, grid_params, mlp_params, items, n_items,
                           total_chunks, counter, max_blocks, (cudaStream_t)stream);
}

extern "C" size_t nectb_time_slice_bytes(const NectbHashGrid* grid) {
  GridDev g3;
  if (!slice_grid(grid, &g3)) return 0;
  return (size_t)g3.total_entries * g3.n_features * 2;
}

extern "C" int nectb_time_slice(const NectbHashGrid* grid, const void* grid_params, float t, void* slice,
                                size_t slice_bytes, void* stream) {
  clear_error();
  GridDev g, g3;
  if (!slice_grid(grid, &g3) || !make_grid_dev(grid, &g))
    return set_error(NECTB_ERR_INVALID, "time slice: needs a valid 4D grid with an fp16 table");
  NECTB_REQUIRE(grid_params && slice, "null pointer");
  NECTB_REQUIRE(((uintptr_t)grid_params & 15u) == 0 && ((uintptr_t)slice & 15u) == 0,
                "grid_params and slice must be 16-byte aligned");
  NECTB_REQUIRE(t >= 0.f && t <= 1.f, "t must lie in [0, 1]");
  const size_t need = (size_t)g3.total_entries * g3.n_features * 2;
  if (slice_bytes < need) return set_error(NECTB_ERR_WORKSPACE, "slice of %zu bytes < required %zu", slice_bytes, need);
  return launch_time_slice(g, (const __half*)grid_params, t, (__half*)slice, (cudaStream_t)stream);
}

extern "C" int nectb_query_points_slice(const NectbHashGrid* grid, const NectbMLP* mlp, const void* slice,
                                        const float* mlp_params, const NectbQueryItem* items, int32_t n_items,
                                        int64_t total_chunks, unsigned int* counter, int32_t max_blocks,
                                        void* stream) {
  clear_error();
  GridDev g3;
  if (!slice_grid(grid, &g3))
    return set_error(NECTB_ERR_INVALID, "slice queries: needs a valid 4D grid with an fp16 table");
  return query_points_impl(g3, true, mlp, slice, mlp_params, items, n_items, total_chunks, counter, max_blocks,
                           (cudaStream_t)stream);
}

namespace {

// Pixels [begin, begin + count) of a re-projection at (angle, t), written to
// out[begin ...].  stage: use the workspace past the base size (a 4D mixed
// model's time slice).
int reproject_range(const NectbGeometry* geometry, const NectbHashGrid* grid, const NectbMLP* mlp,
                    const void* grid_params, const float* mlp_params, float angle_rad, float t,
                    int32_t num_points_per_ray, float max_ray_distance_per_point, float max_distance_traveled,
                    float* out, int32_t begin, int32_t count, void* workspace, size_t workspace_size,
                    int32_t max_blocks, int32_t warpgroups, bool stage, cudaStream_t s) {
  clear_error();
  if (int rc = validate_geometry(geometry)) return rc;
  GridDev g;
  if (!make_grid_dev(grid, &g)) return set_error(NECTB_ERR_INVALID, "invalid hash grid description");
  if (int rc = validate_mlp(mlp, g)) return rc;
  NECTB_REQUIRE(grid_params && mlp_params && out, "null pointer");
  NECTB_REQUIRE(((uintptr_t)grid_params & 15u) == 0, "grid_params must be 16-byte aligned");
  NECTB_REQUIRE(num_points_per_ray >= 1 && max_distance_traveled > 0.f, "bad sampling parameters");
  const int P = geometry->nDetector[0] * geometry->nDetector[1];
  NECTB_REQUIRE(begin >= 0 && count >= 1 && (int64_t)begin + count <= P, "pixel range outside the detector");
  NECTB_REQUIRE(warpgroups >= 0 && warpgroups <= kFwdMaxWarpgroups, "warpgroups_per_sm must be 0..%d",
                kFwdMaxWarpgroups);
  if (!workspace || workspace_size < workspace_bytes(count, count))
    return set_error(NECTB_ERR_WORKSPACE, "workspace of %zu bytes < required %zu", workspace_size,
                     workspace_bytes(count, count));
  TrainArgs a;
  a.perm = nullptr;  // the pixels begin, begin + 1, ... in pixel order
  a.perm_len = count;
  a.start = begin;
  a.num_rays = count;
  a.n_pixels = count;
  a.S = num_points_per_ray;
  a.angle = angle_rad;
  a.t = t;
  a.maxd = max_ray_distance_per_point;
  a.uniform = 1;
  a.max_dist = max_distance_traveled;
  a.jitter = nullptr;
  a.det_off = nullptr;
  a.projection = nullptr;
  a.loss_type = 2;
  a.loss_scale = 0.f;
  a.max_blocks = max_blocks;
  a.fwd_warpgroups = max_blocks > 0 ? 0 : warpgroups;
  a.n_cols = geometry->nDetector[1];
  a.query = true;
  // a whole view with room past the base size: the column form's sigmas, groups of 32 rays at a time
  const size_t base = align256(workspace_bytes(count, count));
  if (!stage && max_blocks <= 0 && workspace_size > base) {
    const int64_t fit = (int64_t)((workspace_size - base) / ((size_t)num_points_per_ray * sizeof(float)));
    a.col_rays = (int)(std::min<int64_t>(fit, count + (int64_t)31) / 32 * 32);
    if (a.col_rays > 0) a.col_sigma = reinterpret_cast<float*>(static_cast<char*>(workspace) + base);
  }
  Workspace ws = carve_workspace(workspace, count, count, stage ? workspace_size : 0);
  float* y = out + begin;
  float* loss = reinterpret_cast<float*>(ws.counters + 8);
  if (int rc = cuda_status(cudaMemsetAsync(ws.counters, 0, 64, s), "memset counters")) return rc;
  if (int rc = cuda_status(cudaMemsetAsync(ws.slot, 0xFF, (size_t)count * 4, s), "memset slots")) return rc;
  {
    ProfScope ps(kProfRayPrep, s);
    ray_prep_kernel<<<(unsigned)ceil_div(count, kRayPrepThreads / 32), kRayPrepThreads, 0, s>>>(*geometry, a, ws.rays, ws.slot, ws.counters, y,
                                                                  loss);
  }
  if (int rc = launch_status("ray_prep_kernel")) return rc;
  return train_forward_only(*geometry, g, *mlp, grid_params, mlp_params, a, ws, y, loss, s);
}

}  // namespace

extern "C" int nectb_query_reproject(const NectbGeometry* geometry, const NectbHashGrid* grid, const NectbMLP* mlp,
                                     const void* grid_params, const float* mlp_params, float angle_rad, float t,
                                     int32_t num_points_per_ray, float max_ray_distance_per_point,
                                     float max_distance_traveled, float* out, void* workspace,
                                     size_t workspace_size, int32_t max_blocks, void* stream) {
  const int P = geometry ? geometry->nDetector[0] * geometry->nDetector[1] : 0;
  return reproject_range(geometry, grid, mlp, grid_params, mlp_params, angle_rad, t, num_points_per_ray,
                         max_ray_distance_per_point, max_distance_traveled, out, 0, P, workspace, workspace_size,
                         max_blocks, 0, false, (cudaStream_t)stream);
}

extern "C" int nectb_query_reproject_range(const NectbGeometry* geometry, const NectbHashGrid* grid,
                                           const NectbMLP* mlp, const void* grid_params, const float* mlp_params,
                                           float angle_rad, float t, int32_t num_points_per_ray,
                                           float max_ray_distance_per_point, float max_distance_traveled,
                                           float* out, int32_t pixel_begin, int32_t pixel_count, void* workspace,
                                           size_t workspace_size, int32_t max_blocks, int32_t warpgroups_per_sm,
                                           void* stream) {
  return reproject_range(geometry, grid, mlp, grid_params, mlp_params, angle_rad, t, num_points_per_ray,
                         max_ray_distance_per_point, max_distance_traveled, out, pixel_begin, pixel_count, workspace,
                         workspace_size, max_blocks, warpgroups_per_sm, true, (cudaStream_t)stream);
}

extern "C" size_t nectb_query_reproject_slice_bytes(const NectbHashGrid* grid, const NectbMLP* mlp,
                                                    int32_t pixel_count) {
  GridDev g;
  if (!grid || !mlp || pixel_count < 1 || !make_grid_dev(grid, &g)) return 0;
  if (g.n_dims != 4 || mlp->compute_dtype == NECTB_F32 || grid->feature_dtype != NECTB_F16) return 0;
  return slice_half_bytes(g) + 512;
}
