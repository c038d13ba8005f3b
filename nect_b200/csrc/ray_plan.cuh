// The order in which a batch's rays are scheduled and the split of the workspace that
// holds it.  Host and device code without CUDA calls, so that it can be checked on the
// CPU.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define NECTB_HD __host__ __device__ __forceinline__
#else
#define NECTB_HD inline
struct uint4;
#endif

namespace nectb {

struct RayRec;

// Slot of scheduling index idx: the detector in strips of 32 rows, a strip
// column by column, so that 32 consecutive rays are vertical neighbours.
// Their paths differ along axis 0 only (the rotation axis), whose vertices
// share sectors of the tables.  A permutation of [0, P) for whole rows of
// pixels; the pixels of a part of a row (a piece of a view) keep their order.
NECTB_HD int strip_slot(int idx, int P, int cols, int sub) {
  const int line = cols * sub;   // 32 of them may exceed an int, strip * 32 of them do not
  if (P % line != 0) return idx;
  const int rows = P / line, strip = idx / line / 32;
  const int left = rows - 32 * strip, h = left < 32 ? left : 32, rem = idx - strip * 32 * line;
  const int cj = rem / h, row = 32 * strip + rem - cj * h;   // cj = column * sub + sub-angle
  return row * line + cj;
}

// Slots a warp claims at a time where no ray order is made: one for every 64 slots a ray
// has, up to 32.  More, and a claim of a random batch holds several rays for one warp
// too often (2,000 rays x 100 samples on 65,536 pixels, mixed without staging: 0.36 ms a
// step with one, 0.40 with eight); fewer, and a batch of very few rays waits for the
// claims (fp32, 65,536 pixels: one ray 37.1 -> 1.14 ms a step, 32 rays 3.0 -> 0.23).
NECTB_HD int slots_per_claim(int R, int P) {
  const int n = P / (R > 1 ? R : 1) / 64;
  return n < 1 ? 1 : (n > 32 ? 32 : n);
}

// The two-pass mixed backward: the most rounds a staging buffer may need
// before the fused single-pass backward is used instead (the recommended
// staging is sized for NectbTuning::staged_rounds, 4 by default).
constexpr int kMaxStagedRounds = 64;
constexpr size_t kStagingCap = size_t(16) << 30;  // largest staging buffer recommended
// A round staging less than this leaves part of the GPU idle in the scatter:
// batches below it take one round (24,999 rays x 100 samples: the scatter of a
// step 1.12 ms in four rounds of four level passes, 0.58 ms in one launch).
constexpr size_t kStagedRoundMin = size_t(1) << 30;
constexpr int kOrderBlock = 1024;                  // threads of the ray-order kernels

// Stored encodings: the forward writes each sample's bf16 MLP input row, which
// the backward reads back instead of gathering the tables again.  Largest
// store the recommended staging size includes.
constexpr size_t kEncodingStoreCap = size_t(80) << 30;

// Staged samples per ray: S rounded up so that each run of four samples of a
// ray's features is 16-byte aligned.
NECTB_HD int ray_slots(int S) { return (S + 3) & ~3; }

inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }
inline int order_blocks(int R, int P) { return (std::max(R, P) + kOrderBlock - 1) / kOrderBlock; }

// Bytes at the front of the staging region: the ray order, its block sums,
// the sample offset of every ranked ray and their block sums.
inline size_t order_bytes(int R, int P) {
  const size_t nb = (size_t)order_blocks(R, P) + 1;
  return align256((size_t)R * 4) + align256(nb * 4) + align256((size_t)R * 8) + align256(nb * 8);
}

// Workspace: RayRec[R] | slot[P] (int32: batch index of the ray through each
// detector pixel, -1 if none) | 64-byte control block (scheduling cursors of
// the forward and backward, error word, flags).
// Any workspace bytes beyond workspace_bytes() (from a 256-byte boundary) are
// the staging buffer of the two-pass mixed backward.
struct Workspace {
  RayRec* rays;
  int32_t* slot;
  unsigned int* counters;  // [0] forward cursor, [1] backward cursor, [2] error word, [3] flags,
                           // [6] rays with samples, [7] encoding-store rows the forward
                           // filled, [8] forward loss sum (split step),
                           // [9] chunks of 32 samples (about)
  float* stage = nullptr;
  size_t stage_bytes = 0;
};

// Split of the staging region of the two-pass mixed backward:
//   order[R] int32 | block sums | offs[R] uint64 (first stored row of each
//   ranked ray) | block sums | encoding store [xcap rows of row_bytes] |
//   staged dL/d(encoding) of one round of per_round rays (per_ray bytes each).
// The staged rounds take the recommended size for `rounds` rounds (capped at
// kStagingCap) and the encoding store the rest, up to R * S rows; where the
// store would lose rows to rounds of kStagedRoundMin, the rounds are as small as
// `rounds` allows instead; when that leaves less than one ray's rows there is no
// store and the rounds take the whole region.  per_round == 0: no staging (the
// fused single-pass backward).
// The store starts at the same address whatever the split, so a backward half
// reading rows [0, min(its xcap, the forward's)) never reads its own staging.
struct StageLayout {
  int32_t* order = nullptr;
  unsigned int* block_sums = nullptr;
  uint64_t* offs = nullptr;
  unsigned long long* block_samples = nullptr;
  uint4* xstore = nullptr;
  uint32_t xcap = 0;  // rows of the encoding store
  float* stage = nullptr;
  int64_t per_round = 0;
};

// Bytes of a round when a batch takes `rounds` of them.
inline size_t round_bytes(int R, int rounds, size_t per_ray) {
  const int64_t per_round = ((int64_t)R + rounds - 1) / rounds;
  return std::min((size_t)per_round * per_ray, kStagingCap / per_ray * per_ray);
}

// The recommended bytes of a round: of `rounds` rounds, or of fewer where those
// would stage less than kStagedRoundMin.
inline size_t staged_round_bytes(int R, int rounds, size_t per_ray) {
  const int64_t most = (int64_t)((size_t)R * per_ray / kStagedRoundMin);
  return round_bytes(R, (int)std::max<int64_t>(1, std::min<int64_t>(rounds, most)), per_ray);
}

// store == false: no encoding store whatever the buffer size (the backward
// recomputes every sample's encoding from the tables).
inline StageLayout stage_layout(const Workspace& ws, int R, int P, int S, size_t row_bytes, size_t per_ray,
                                int rounds, bool store = true) {
  StageLayout L;
  const size_t ob = order_bytes(R, P);
  // 16-byte aligned rows, stored and staged, whatever the caller's workspace pointer
  const uintptr_t start = reinterpret_cast<uintptr_t>(ws.stage), skip = ((start + 15) & ~uintptr_t(15)) - start;
  if (!ws.stage || ws.stage_bytes <= ob + skip || R <= 0) return L;
  char* p = reinterpret_cast<char*>(ws.stage) + skip;
  const size_t nb = (size_t)order_blocks(R, P) + 1;
  L.order = reinterpret_cast<int32_t*>(p);
  L.block_sums = reinterpret_cast<unsigned int*>(p + align256((size_t)R * 4));
  L.offs = reinterpret_cast<uint64_t*>(p + align256((size_t)R * 4) + align256(nb * 4));
  L.block_samples = reinterpret_cast<unsigned long long*>(p + align256((size_t)R * 4) + align256(nb * 4) +
                                                          align256((size_t)R * 8));
  const size_t avail = ws.stage_bytes - ob - skip;
  size_t want = staged_round_bytes(R, rounds, per_ray);
  // rows before large rounds: 65,536 rays x 256 samples on a 4D grid of 16 x 2 levels, in half of
  // the recommended size, 8.67 ms a step with rounds of kStagedRoundMin and no rows, 6.26 with them
  const size_t all = std::min<size_t>((size_t)R * S, 0xffffffffu) * row_bytes;
  if (store && avail < want + all + 256) want = round_bytes(R, rounds, per_ray);
  size_t xbytes = 0;
  if (store && avail >= want + (size_t)S * row_bytes + 256) {
    const size_t rows = std::min<size_t>({(avail - want - 256) / row_bytes, (size_t)R * S, 0xffffffffu});
    if (rows >= (size_t)S) {
      L.xcap = (uint32_t)rows;
      xbytes = align256(rows * row_bytes);
      L.xstore = reinterpret_cast<uint4*>(p + ob);
    }
  }
  L.stage = reinterpret_cast<float*>(p + ob + xbytes);
  L.per_round = avail < xbytes ? 0 : std::min<int64_t>((int64_t)((avail - xbytes) / per_ray), R);
  if (L.per_round <= 0 || (R + L.per_round - 1) / L.per_round > kMaxStagedRounds) {
    L.per_round = 0;
    L.xstore = nullptr;
    L.xcap = 0;
  }
  return L;
}

// The staged backward's weight gradients gather in the tensor cores' accumulators,
// which lose about 2e-8 of the sum per product (three times the length measured 3e-5 of
// the gradient), so they are added to fp32 memory at least once per R / rounds rays,
// however many rays a launch has: at its end where it has no more than that, else inside
// it too.  The stretches of the batch (1: at the ends alone).
NECTB_HD int accumulator_stretches(int64_t R, int64_t per_round, int rounds) {
  return per_round <= (R + rounds - 1) / rounds ? 1 : rounds;
}

// Tiles (of four 32-sample chunks) of a stretch for each of the launch's blocks.
NECTB_HD int stretch_tiles(unsigned int chunks, int stretches, int blocks) {
  if (stretches <= 1) return 0x7fffffff;
  const uint64_t per = ((uint64_t)chunks + 4 * (uint64_t)stretches * blocks - 1) / (4 * (uint64_t)stretches * blocks);
  return per < 1 ? 1 : (int)per;
}

}  // namespace nectb
