// What the layer-1 forward and its adjoint share: instruction groups, staged edges and the
// async copies into shared memory.
#pragma once

#include "cg_canon.h"
#include "edge.cuh"

namespace smx {

// Instruction groups, ordered by l1 inside a group.  L_max = 1: all ten.  L_max = 2 (17
// instructions): by the l of H1, {0, 1} (the ten instructions of L_max = 1) and two halves of
// l = 2, so that a group's paths fit the registers of a lane.
__host__ __device__ constexpr int l1_groups(int LMAX) { return LMAX == 1 ? 1 : 3; }
__host__ __device__ constexpr int grp_count(int G) { return G == 0 ? 10 : (G == 1 ? 4 : 3); }
__host__ __device__ constexpr int grp_ins(int LMAX, int G, int i) {
  constexpr int a[10] = {0, 3, 2, 1, 6, 5, 4, 9, 8, 7};
  constexpr int b[10] = {0, 4, 3, 1, 9, 8, 5, 14, 13, 10}, b1[4] = {11, 15, 2, 16}, b2[3] = {6, 12, 7};
  return LMAX == 1 ? a[i] : (G == 0 ? b[i] : (G == 1 ? b1[i] : b2[i]));
}
// first slot of group G in a spline row (DevModel::spl1)
__host__ __device__ constexpr int grp_slot(int G) {
  int s = 0;
  for (int w = 0; w < G; ++w) s += grp_count(w);
  return s;
}
// the H1 rows [row0, row0 + rows) that group G reads
__host__ __device__ constexpr int grp_row0(int G) { return G == 0 ? 0 : 4; }
__host__ __device__ constexpr int grp_rows(int G) { return G == 0 ? 4 : 5; }
__host__ __device__ constexpr int ins_paths(int LMAX, int q) {
  return (2 * ins_l1(LMAX, q) + 1) * (2 * ins_l2(LMAX, q) + 1);
}
// output l of instruction q, its place among the instructions with that l and their number
__host__ __device__ constexpr int ins_l(int LMAX, int q) {
  constexpr int a[10] = {0, 0, 1, 1, 1, 2, 2, 2, 3, 3};
  constexpr int b[17] = {0, 0, 0, 1, 1, 1, 1, 1, 2, 2, 2, 2, 2, 3, 3, 3, 3};
  return LMAX == 1 ? a[q] : b[q];
}
__host__ __device__ constexpr int ins_e(int LMAX, int q) {
  int e = 0;
  for (int w = 0; w < q; ++w) e += ins_l(LMAX, w) == ins_l(LMAX, q);
  return e;
}
__host__ __device__ constexpr int ins_ne(int LMAX, int l) {
  int e = 0;
  for (int w = 0; w < ins_count(LMAX); ++w) e += ins_l(LMAX, w) == l;
  return e;
}
// row lme of component 0 of instruction q; component m is m * ins_ne rows on
__host__ __device__ constexpr int ins_row(int LMAX, int q) {
  int o = 0;
  for (int l = 0; l < ins_l(LMAX, q); ++l) o += (2 * l + 1) * ins_ne(LMAX, l);
  return o + ins_e(LMAX, q);
}
__host__ __device__ constexpr int l1_rows(int LMAX) {
  int o = 0;
  for (int l = 0; l < 4; ++l) o += (2 * l + 1) * ins_ne(LMAX, l);
  return o;
}

// Paths.  CANON (DevModel::cg_val): the zero pattern of the real Clebsch-Gordan coefficients
// is compiled in (cg_canon.h) and paths that reach no output are left out, 12 of 88 at
// L_max = 1 and 56 of 243 at L_max = 2; otherwise every path, the table read at run time.
template <int LMAX, bool CANON>
__host__ __device__ constexpr bool path_used(int q, int a, int b) {
  return !CANON || cg_m(LMAX, ins_poff(LMAX, q) + a * (2 * ins_l2(LMAX, q) + 1) + b, 0) >= 0;
}
// place of path (q, a, b) among the used paths of its instruction
template <int LMAX, bool CANON>
__host__ __device__ constexpr int path_at(int q, int a, int b) {
  int n = 0;
  for (int v = 0; v <= a; ++v)
    for (int w = 0; w < (v < a ? 2 * ins_l2(LMAX, q) + 1 : b); ++w) n += path_used<LMAX, CANON>(q, v, w);
  return n;
}
// offset of the group's i-th instruction in its path list (i = grp_count: the list's length)
template <int LMAX, int G, bool CANON>
__host__ __device__ constexpr int grp_off(int i) {
  int s = 0;
  for (int w = 0; w < i; ++w) {
    const int q = grp_ins(LMAX, G, w);
    s += path_at<LMAX, CANON>(q, 2 * ins_l1(LMAX, q), 2 * ins_l2(LMAX, q) + 1);
  }
  return s;
}
// f(q, a, b, path index) as integral constants over the used paths of instruction i of a group
template <int LMAX, int G, bool CANON, int I, typename F>
__device__ __forceinline__ void for_paths(F&& f) {
  constexpr int q = grp_ins(LMAX, G, I), nb = 2 * ins_l2(LMAX, q) + 1, g0 = grp_off<LMAX, G, CANON>(I);
  static_for<ins_paths(LMAX, q)>([&](auto pc) {
    constexpr int p = decltype(pc)::value, a = p / nb, b = p % nb;
    if constexpr (path_used<LMAX, CANON>(q, a, b))
      f(std::integral_constant<int, a>{}, std::integral_constant<int, b>{},
        std::integral_constant<int, g0 + path_at<LMAX, CANON>(q, a, b)>{});
  });
}

// Up to 32 edges of a node staged by one warp, those inside the cut-off packed to the front.
struct EdgeStage {
  float Y[kEdgeChunk][16];  // Y_lm
  int4 meta[kEdgeChunk];    // offset inside the spline interval (float bits), spline row, neighbour
};

// Stage the warp's edges (lanes with `active`): first where their spline rows and neighbours
// are (the slot of this lane's edge, and the count), so that the first edge's loads can go
// out, then their Y_lm.
__device__ __forceinline__ int stage_rows(const DevModel& m, EdgeStage& st, const LaneEdge& ed, int ti, bool active,
                                           int& count) {
  const unsigned ball = __ballot_sync(0xffffffffu, active);
  const int pos = __popc(ball & ((1u << (threadIdx.x & 31)) - 1u));
  count = __popc(ball);
  __syncwarp();  // the last chunk has been read
  if (active) {
    const int a = ti < ed.tj ? ti : ed.tj, b = ti < ed.tj ? ed.tj : ti;
    st.meta[pos] = make_int4(__float_as_int(ed.x), (a * (2 * m.S - a - 1) / 2 + b) * m.nint + ed.iv, ed.j, 0);
  }
  __syncwarp();
  return pos;
}
__device__ __forceinline__ void stage_Y(EdgeStage& st, const LaneEdge& ed, bool active, int pos) {
  if (active) {
    float Y[16];
    sph_harm16<false>(ed.vx, ed.vy, ed.vz, Y, nullptr);
#pragma unroll
    for (int v = 0; v < 4; ++v)
      *reinterpret_cast<float4*>(&st.Y[pos][4 * v]) = make_float4(Y[4 * v], Y[4 * v + 1], Y[4 * v + 2], Y[4 * v + 3]);
  }
  __syncwarp();
}

__device__ __forceinline__ void read_Y(const float* Y, float* y) {
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const float4 f = *reinterpret_cast<const float4*>(Y + 4 * v);
    y[4 * v] = f.x;
    y[4 * v + 1] = f.y;
    y[4 * v + 2] = f.z;
    y[4 * v + 3] = f.w;
  }
}

__device__ __forceinline__ void async_copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// (LMAX, C, CANON): the common channel counts compiled in for the canonical tables (addresses
// fold to immediates; 0: any)
template <typename F>
void dispatch_layer1(const DevModel& m, F&& f) {
  auto by_c = [&](auto lc) {
    if (!m.cg_val) {
      f(lc, std::integral_constant<int, 0>{}, std::false_type{});
      return;
    }
    switch (m.C) {
      case 32: f(lc, std::integral_constant<int, 32>{}, std::true_type{}); break;
      case 64: f(lc, std::integral_constant<int, 64>{}, std::true_type{}); break;
      case 128: f(lc, std::integral_constant<int, 128>{}, std::true_type{}); break;
      default: f(lc, std::integral_constant<int, 0>{}, std::true_type{}); break;
    }
  };
  if (m.L_max == 2)
    by_c(std::integral_constant<int, 2>{});
  else
    by_c(std::integral_constant<int, 1>{});
}

}  // namespace smx
