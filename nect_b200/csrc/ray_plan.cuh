// The order in which a batch's rays are scheduled.  Host and device code without CUDA
// types, so that it can be checked on the CPU.
#pragma once

#ifdef __CUDACC__
#define NECTB_HD __host__ __device__ __forceinline__
#else
#define NECTB_HD inline
#endif

namespace nectb {

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

}  // namespace nectb
