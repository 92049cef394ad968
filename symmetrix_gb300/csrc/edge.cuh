// What the edge kernels of both layers share: a lane's edge, and sums over the lanes.
#pragma once

#include "device.cuh"

namespace smx {

// This lane's edge of a chunk, loaded ahead of its staging.
struct LaneEdge {
  float vx, vy, vz, r, x;  // x: offset inside spline interval iv
  int tj, j, iv;
  __device__ __forceinline__ void load(const DevModel& m, const EdgeIn& in, long e) {
    vx = static_cast<float>(in.xyz[3 * e]);
    vy = static_cast<float>(in.xyz[3 * e + 1]);
    vz = static_cast<float>(in.xyz[3 * e + 2]);
    const double rd = in.r[e];
    r = static_cast<float>(rd);
    iv = spline_at(m, rd, x);
    tj = in.ntype_e[e];
    j = in.nidx[e];
  }
};

constexpr int kSumEdges = 4;  // edges summed over the lanes at a time
constexpr int kSumRow = 33;   // row pitch of their terms: 32 rows read at one column hit all banks

// Sums over the lanes of the terms of n edges (n <= kSumEdges): lane 8 e + v adds component
// pair v of edge e, four partial sums in a fixed order, into the 16 floats at out + e PITCH, or
// with HALVES the sums of lanes 0-15 and 16-31 into the 32 there.
template <bool HALVES, int PITCH>
__device__ __forceinline__ void sum_lanes(const float2* buf, float* out, int n) {
  const int lane = threadIdx.x & 31, e = lane >> 3, v = lane & 7;
  __syncwarp();
  if (e < n) {
    const float2* row = buf + lane * kSumRow;
    float2 p0 = make_float2(0.0f, 0.0f), p1 = p0, p2 = p0, p3 = p0;
    constexpr int step = HALVES ? 2 : 4, third = HALVES ? 16 : 2;
#pragma unroll
    for (int i = 0; i < 8 * step; i += step) {
      p0 = __fadd2_rn(p0, row[i]);
      p1 = __fadd2_rn(p1, row[i + 1]);
      p2 = __fadd2_rn(p2, row[i + third]);
      p3 = __fadd2_rn(p3, row[i + third + 1]);
    }
    float2* o = reinterpret_cast<float2*>(out + PITCH * e + 2 * v);
    p0 = __fadd2_rn(p0, p1);
    p2 = __fadd2_rn(p2, p3);
    *o = HALVES ? p0 : __fadd2_rn(p0, p2);
    if (HALVES) o[8] = p2;
  }
  __syncwarp();
}

// Warps the chip holds at once, 12 per SM: a node's edges are split over `split` warps, in
// chunks of edge_chunk(split), while all parts still fit at once.
constexpr long kSlots = 12 * 152;
inline int edge_split(long items) {
  return items > 2 * kSlots ? 1 : (items > kSlots ? 2 : static_cast<int>(items * 16 < kSlots ? 16 : kSlots / items));
}
inline int edge_chunk(int split) { return split == 1 ? kEdgeChunk : (split <= 2 ? 16 : (split <= 8 ? 8 : 4)); }

}  // namespace smx
