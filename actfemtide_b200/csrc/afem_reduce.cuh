// Sums over the blocks of a launch, finished inside the launch.
//
// Every block leaves one complex partial sum per system; the block that finishes last adds them and
// can act on the result, so a dot product needs no launch of its own.  The sum runs in two steps:
// the last block of each group of 32 adds the group's sums with one load per lane, the last of those
// adds the groups' (one block adding all 1,184 rows of a full grid took 10 to 20 us at 16 systems).
// The order of the additions is fixed by the block numbers, so results do not depend on timing.
#pragma once

#include <cuda_runtime.h>

namespace afem {

constexpr int RED_SYS = 32;     // systems of a set
constexpr int RED_GROUPS = 64;  // groups of 32 blocks: at most 2,048 blocks

// One set of sums: part[system * rows + block], group[system * RED_GROUPS + group] and
// RED_GROUPS + 1 counters that are zero between launches.
struct RedSet {
  double2* part;
  double2* group;
  unsigned* cnt;
  int rows;
};

// After the block (number bid of nblk) wrote its part: true in the one block that gets the sums of
// all, out[s] (shared memory) for s < nsys, visible to the whole block.
__device__ __forceinline__ bool reduce_blocks(const RedSet& R, int bid, int nblk, int nsys, double2* out) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  const int grp = bid >> 5, gs = min(32, nblk - (grp << 5)), ng = (nblk + 31) >> 5;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (threadIdx.x == 0) last = atomicAdd(R.cnt + 1 + grp, 1u) == (unsigned)gs - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  for (int s = w; s < nsys; s += nw) {
    double2 v = lane < gs ? __ldcg(R.part + (long)s * R.rows + (grp << 5) + lane) : make_double2(0.0, 0.0);
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, m);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, m);
    }
    if (lane == 0) {
      if (ng == 1) out[s] = v;
      else R.group[s * RED_GROUPS + grp] = v;
    }
  }
  if (threadIdx.x == 0) R.cnt[1 + grp] = 0;
  __threadfence();
  __syncthreads();
  if (ng == 1) return true;
  if (threadIdx.x == 0) last = atomicAdd(R.cnt, 1u) == (unsigned)ng - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  if (threadIdx.x == 0) R.cnt[0] = 0;
  for (int s = w; s < nsys; s += nw) {
    double2 v = lane < ng ? __ldcg(R.group + s * RED_GROUPS + lane) : make_double2(0.0, 0.0);
    if (lane + 32 < ng) {
      const double2 u = __ldcg(R.group + s * RED_GROUPS + lane + 32);
      v.x += u.x;
      v.y += u.y;
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, m);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, m);
    }
    if (lane == 0) out[s] = v;
  }
  __syncthreads();
  return true;
}

// The same sums by every block for itself, after a grid barrier: out[s] for s < nsys in shared memory.
// (For grids of a few hundred blocks at most: each block reads all parts.)
__device__ __forceinline__ void sum_blocks(const RedSet& R, int nblk, int nsys, double2* out) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int s = threadIdx.x >> 5; s < nsys; s += nw) {
    double2 v = make_double2(0.0, 0.0);
#pragma unroll 8
    for (int b = lane; b < nblk; b += 32) {
      const double2 u = __ldcg(R.part + (long)s * R.rows + b);
      v.x += u.x;
      v.y += u.y;
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, m);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, m);
    }
    if (lane == 0) out[s] = v;
  }
  __syncthreads();
}

// The block's part from lanes that carry systems s0 .. s0 + SPL - 1 of a row of LPR lanes (values
// zero on lanes that do not count): rows of a warp are folded by shuffles, warps in order.
// buf: shared memory, NS values per warp of the block.
template <int NS, int SPL, int LPR>
__device__ __forceinline__ void block_pair(double (&v)[SPL][2], int s0, bool lead, const RedSet& R, int bid,
                                           double2* buf) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
  for (int m = LPR; m < 32; m <<= 1)
#pragma unroll
    for (int i = 0; i < SPL; ++i) {
      v[i][0] += __shfl_xor_sync(0xffffffffu, v[i][0], m);
      v[i][1] += __shfl_xor_sync(0xffffffffu, v[i][1], m);
    }
  if (lane < LPR && lead)
#pragma unroll
    for (int i = 0; i < SPL; ++i) buf[w * NS + s0 + i] = make_double2(v[i][0], v[i][1]);
  __syncthreads();
  if (threadIdx.x < NS) {
    double2 a = make_double2(0.0, 0.0);
    for (int k = 0; k < nw; ++k) {
      a.x += buf[k * NS + threadIdx.x].x;
      a.y += buf[k * NS + threadIdx.x].y;
    }
    R.part[(long)threadIdx.x * R.rows + bid] = a;
  }
}

}  // namespace afem
