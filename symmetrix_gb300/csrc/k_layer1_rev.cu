// Layer-1 adjoint (reverse_Phi1, libsymmetrix/source/mace.cpp:504-605).
//
// With g_p = sum_lme CG[lme,p] dPhi1[i,lme,k], p = (q, a, b) and h_b = H1[j, b, k]:
//   u_qb = sum_a g_qab Y_a,   H1_adj[j, b, k] += sum_q R1_q u_qb
//   dE/dY_a = sum_k sum_q sum_b g_qab (R1_q h_b)
//   dE/dx_ij = (sum_k sum_q R1'_q sum_b u_qb h_b) u + sum_a dE/dY_a dY_a/dx
// so two FMAs per path and edge (u and dE/dY).
//
// One warp per (centre node, 32 channels), a warp being a whole block: the lane holds the
// g of its channel in registers for all of the node's edges, nothing couples two warps, and
// there is no block barrier.  An edge's terms depend on no other edge, so a node's edges may
// also be split over several warps (small systems).  The next edge's cubics are loaded into
// the registers that this edge's have just left, instruction by instruction.  dE/dY_a and
// the radial term are summed over the lanes four edges at a time through shared memory, and
// only these sums meet dY_a/dx.
//
// What bounds it: issue slots (63% of the cycles issue, at 12 warps per SM and 168
// registers; 255 registers, 8 warps: 0.55 -> 0.58 ms).  Against one block per node with two
// instruction halves of channel pairs, which met at a barrier for every edge (8 warps per SM,
// 47% of the cycles issuing, four FMAs on each of the 88 paths): 4096 atoms, 128 channels,
// 213k edges 0.733 -> 0.533 ms; L_max = 2, 2197 atoms, 178k edges 2.12 -> 1.15 ms.  Without the
// paths that reach no output 0.475 and 0.975 ms; with the cubics of two instructions side by
// side in the table, so that a packed FMA takes both, 0.444 and 0.960 ms.
//
// L_max = 2 (17 instructions): three instruction groups in turn (layer1.cuh), so that a
// group's g fits the registers; the H1_adj rows of l = 0, 1 are added once, those of l = 2
// twice.  (One launch per group, 16 warps per SM for the two of l = 2: the same time.)
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "layer1.cuh"

namespace smx {

namespace {

// has an earlier instruction of the group, or an earlier used path of this one, touched
// dE/dY_a of its l1 (component b and on of instruction i come next)?
template <int LMAX, int G, bool CANON>
__host__ __device__ constexpr bool dY_started(int i, int a, int b) {
  const int q = grp_ins(LMAX, G, i);
  for (int w = 0; w <= i; ++w) {
    const int qw = grp_ins(LMAX, G, w);
    if (ins_l1(LMAX, qw) != ins_l1(LMAX, q)) continue;
    for (int v = 0; v < (w < i ? 2 * ins_l2(LMAX, qw) + 1 : b); ++v)
      if (path_used<LMAX, CANON>(qw, a, v)) return true;
  }
  return false;
}
// is dE/dY_c touched by the group at all?
template <int LMAX, int G, bool CANON>
__host__ __device__ constexpr bool dY_used(int c) {
  for (int w = 0; w < grp_count(G); ++w) {
    const int q = grp_ins(LMAX, G, w), l1 = ins_l1(LMAX, q);
    if (l1 == 0 || c < l1 * l1 || c >= (l1 + 1) * (l1 + 1)) continue;
    for (int b = 0; b < 2 * ins_l2(LMAX, q) + 1; ++b)
      if (path_used<LMAX, CANON>(q, c - l1 * l1, b)) return true;
  }
  return false;
}
// is there a used path (q, a' < a, b)?
template <int LMAX, bool CANON>
__host__ __device__ constexpr bool u_started(int q, int a, int b) {
  for (int v = 0; v < a; ++v)
    if (path_used<LMAX, CANON>(q, v, b)) return true;
  return false;
}
// has an earlier instruction of the group added to H1_adj row l2^2 + b of instruction i?
template <int LMAX, int G, bool CANON>
__host__ __device__ constexpr bool row_started(int i, int b) {
  const int q = grp_ins(LMAX, G, i);
  for (int w = 0; w < i; ++w) {
    const int qw = grp_ins(LMAX, G, w);
    if (ins_l2(LMAX, qw) == ins_l2(LMAX, q) && u_started<LMAX, CANON>(qw, 2 * ins_l1(LMAX, qw) + 1, b)) return true;
  }
  return false;
}

// shared memory of one warp
struct RevSmem {
  EdgeStage st;   // Y rows: once an edge is done, (dE/dr term, dE/dY_1 .. dE/dY_15) in their place
  float2 buf[1];             // [kSumEdges * 8][kSumRow] per-lane terms; before the edges: dPhi1 rows
};

// One edge, group G, this lane's channel; c: the edge's cubics, replaced by those of the
// next edge (cn); t: this lane's slot of the edge in RevSmem::buf.
template <int LMAX, int G, bool CANON>
__device__ __forceinline__ void rev_edge(const float* g, float4* c, const float4* __restrict__ cn, int C, float x,
                                         const float* Y, const float* h, float* hadj, float2* t) {
  float y[16];
  read_Y(Y, y);
  constexpr int r0 = grp_row0(G);
  float dY[16], dr = 0.0f;
  float2 R2 = make_float2(0.0f, 0.0f), Rd2 = R2;
  static_for<grp_count(G)>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr int q = grp_ins(LMAX, G, i);
    constexpr int l1 = ins_l1(LMAX, q), l2 = ins_l2(LMAX, q), nb = 2 * l2 + 1;
    float R, Rd;
    if constexpr (i % 2 == 0 && i + 1 < grp_count(G)) {  // the pair's values and derivatives at once
      spline2(c[i], c[i + 1], make_float2(x, x), R2, Rd2);
      c[i] = __ldg(cn + i * C);
      c[i + 1] = __ldg(cn + (i + 1) * C);
      R = R2.x;
      Rd = Rd2.x;
    } else if constexpr (i % 2 == 1) {
      R = R2.y;
      Rd = Rd2.y;
    } else {  // by the two-row Horner scheme
      R = fmaf(c[i].w, x, c[i].z);
      Rd = fmaf(c[i].w, x, R);
      R = fmaf(R, x, c[i].y);
      Rd = fmaf(Rd, x, R);
      R = fmaf(R, x, c[i].x);
      c[i] = __ldg(cn + i * C);
    }
    float us[nb], rh[nb];
#pragma unroll
    for (int b = 0; b < nb; ++b) rh[b] = R * h[l2 * l2 - r0 + b];
    for_paths<LMAX, G, CANON, i>([&](auto ac, auto bc, auto pc) {
      constexpr int a = decltype(ac)::value, b = decltype(bc)::value;
      const float gp = g[decltype(pc)::value];
      if constexpr (l1 == 0) {
        us[b] = gp;
      } else {
        us[b] = u_started<LMAX, CANON>(q, a, b) ? fmaf(gp, y[l1 * l1 + a], us[b]) : gp * y[l1 * l1 + a];
        float& d = dY[l1 * l1 + a];
        d = dY_started<LMAX, G, CANON>(i, a, b) ? fmaf(gp, rh[b], d) : gp * rh[b];
      }
    });
    float w = 0.0f;
    static_for<nb>([&](auto bc) {
      constexpr int b = decltype(bc)::value;
      if constexpr (u_started<LMAX, CANON>(q, 2 * l1 + 1, b)) {
        w = fmaf(us[b], h[l2 * l2 - r0 + b], w);
        float& o = hadj[l2 * l2 - r0 + b];
        o = row_started<LMAX, G, CANON>(i, b) ? fmaf(R, us[b], o) : R * us[b];
      }
    });
    dr = i == 0 ? w * Rd : fmaf(w, Rd, dr);
  });
  static_for<16>([&](auto cc) {
    if constexpr (decltype(cc)::value > 0 && !dY_used<LMAX, G, CANON>(decltype(cc)::value)) dY[decltype(cc)::value] = 0.0f;
  });
  t[0] = make_float2(dr, dY[1]);
#pragma unroll
  for (int v = 1; v < 8; ++v) t[kSumRow * v] = make_float2(dY[2 * v], dY[2 * v + 1]);
}

// a + b as its rounding and what that drops (Knuth, The Art of Computer Programming 2, 4.2.2)
__device__ __forceinline__ float2 two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return make_float2(s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t)));
}

// Group G over the edges of chunks `split` apart; the edge forces of the earlier groups
// of the same warp are in f1 already (DevModel::f1_stride).
template <int LMAX, int G, int CT, bool CANON>
__device__ __forceinline__ void rev_group(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                          const float* __restrict__ dPhi1, fix64* __restrict__ H1_adj,
                                          float* __restrict__ f1, RevSmem& s, int i, int k, int part, int split,
                                          int cs) {
  constexpr int NI = ins_count(LMAX), NL2 = (LMAX + 1) * (LMAX + 1);
  constexpr int NQ = grp_count(G), NP = grp_off<LMAX, G, CANON>(NQ), NR = grp_rows(G), r0 = grp_row0(G);
  const int C = CT > 0 ? CT : m.C;
  const int lane = threadIdx.x & 31;
  const int ti = in.node_type[i];
  const int e0 = in.first[i], e1 = in.end(i);
  float g[NP];  // of this lane's channel, from the node's dPhi1 rows
  LaneEdge ed;
  ed.load(m, in, min(e0 + part * cs + lane, e1 - 1));
  if constexpr (CANON) {  // one or two terms per path, from the instruction's rows
    static_for<NQ>([&](auto ic) {
      constexpr int w = decltype(ic)::value;
      constexpr int q = grp_ins(LMAX, G, w), l = ins_l(LMAX, q), p0 = ins_poff(LMAX, q), nb = 2 * ins_l2(LMAX, q) + 1;
      float D[2 * l + 1];
#pragma unroll
      for (int v = 0; v < 2 * l + 1; ++v)
        D[v] = __ldg(dPhi1 + (static_cast<size_t>(i) * l1_rows(LMAX) + ins_row(LMAX, q) + v * ins_ne(LMAX, l)) * C + k);
      for_paths<LMAX, G, CANON, w>([&](auto ac, auto bc, auto pc) {
        constexpr int p = p0 + decltype(ac)::value * nb + decltype(bc)::value;
        const float2 cg = __ldg(m.cg_val + p);
        float v = cg.x * D[cg_m(LMAX, p, 0)];
        if constexpr (cg_m(LMAX, p, 1) >= 0) v = fmaf(cg.y, D[cg_m(LMAX, p, 1)], v);
        g[decltype(pc)::value] = v;
      });
    });
  } else {  // any table: all paths first, through the compressed rows
    float* sD = reinterpret_cast<float*>(s.buf);  // [n_lme][32]; a lane reads only its own column
    float* sP = sD + m.n_lme * 32;                // [n_p][32]
    __syncwarp();
    for (int lme = 0; lme < m.n_lme; ++lme)
      async_copy4(sD + lme * 32 + lane, dPhi1 + (static_cast<size_t>(i) * m.n_lme + lme) * C + k);
    async_wait();
    for (int p = 0; p < m.n_p; ++p) {
      float v = 0.0f;
      for (int t = __ldg(m.cg_rev_off + p), t1 = __ldg(m.cg_rev_off + p + 1); t < t1; ++t)
        v = fmaf(__ldg(m.cg_rev_v + t), sD[__ldg(m.cg_rev_lme + t) * 32 + lane], v);
      sP[p * 32 + lane] = v;
    }
    static_for<NQ>([&](auto ic) {
      constexpr int w = decltype(ic)::value;
      constexpr int q = grp_ins(LMAX, G, w), p0 = ins_poff(LMAX, q), g0 = grp_off<LMAX, G, CANON>(w);
#pragma unroll
      for (int p = 0; p < ins_paths(LMAX, q); ++p) g[g0 + p] = sP[(p0 + p) * 32 + lane];
    });
    __syncwarp();
  }
  for (int eb = e0 + part * cs; eb < e1; eb += split * cs) {
    const int ne = min(cs, e1 - eb);
    const long e = static_cast<long>(eb) + lane;
    if (eb > e0 + part * cs) ed.load(m, in, min(eb + lane, e1 - 1));
    const bool active = lane < ne && ed.r < m.r_cut;
    int na;
    const int pos = stage_rows(m, s.st, ed, ti, active, na);
    if (na > 0) {
      float4 c[NQ];
      float h[NR];
      int4 mt = s.st.meta[0];
      {
        const float4* cp = m.spl1 + (static_cast<size_t>(mt.y) * NI + grp_slot(G)) * C + k;
#pragma unroll
        for (int w = 0; w < NQ; ++w) c[w] = __ldg(cp + w * C);
        const float* hp = H1 + (static_cast<size_t>(mt.z) * NL2 + r0) * C + k;
#pragma unroll
        for (int b = 0; b < NR; ++b) h[b] = __ldg(hp + b * C);
      }
      stage_Y(s.st, ed, active, pos);
      for (int a = 0; a < na; ++a) {
        const int4 mn = s.st.meta[min(a + 1, na - 1)];
        const float4* cn = m.spl1 + (static_cast<size_t>(mn.y) * NI + grp_slot(G)) * C + k;
        float hv[NR], hadj[NR];
        const float* hp = H1 + (static_cast<size_t>(mn.z) * NL2 + r0) * C + k;
#pragma unroll
        for (int b = 0; b < NR; ++b) {
          hv[b] = h[b];
          h[b] = __ldg(hp + b * C);
        }
        rev_edge<LMAX, G, CANON>(g, c, cn, C, __int_as_float(mt.x), s.st.Y[a], hv, hadj,
                          s.buf + (a % kSumEdges) * 8 * kSumRow + lane);
        fix64* dst = H1_adj + (static_cast<size_t>(mt.z) * NL2 + r0) * C + k;
#pragma unroll
        for (int b = 0; b + 1 < NR; b += 2) add_fixed2(dst + b * C, dst + (b + 1) * C, make_float2(hadj[b], hadj[b + 1]));
        if constexpr (NR % 2) add_fixed(dst + (NR - 1) * C, hadj[NR - 1]);
        mt = mn;
        if (a % kSumEdges == kSumEdges - 1 || a == na - 1)
          sum_lanes<false, 16>(s.buf, &s.st.Y[a - a % kSumEdges][0], a % kSumEdges + 1);
      }
    }
    if (lane < ne) {  // this lane's edge: the sums against u and dY/dx
      float fx = 0.0f, fy = 0.0f, fz = 0.0f;
      if (active) {
        float Y[16], D[48];
        sph_harm16<true>(ed.vx, ed.vy, ed.vz, Y, D);
        const float* S = s.st.Y[pos];
        const float d = __fdiv_rn(S[0], ed.r);
        fx = __fmul_rn(d, ed.vx);
        fy = __fmul_rn(d, ed.vy);
        fz = __fmul_rn(d, ed.vz);
#pragma unroll
        for (int q = 1; q < 16; ++q) {
          fx = fmaf(S[q], D[q], fx);
          fy = fmaf(S[q], D[16 + q], fy);
          fz = fmaf(S[q], D[32 + q], fz);
        }
      }
      const float f[3] = {fx, fy, fz};
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        if constexpr (LMAX == 1) {
          f1[3 * e + v] = f[v];
        } else {
          float2* o = reinterpret_cast<float2*>(f1) + 3 * e + v;
          if constexpr (G == 0) {
            *o = make_float2(f[v], 0.0f);
          } else {
            const float2 a = *o, s = two_sum(a.x, f[v]);
            const float low = a.y + s.y;  // (undefined beside an infinity)
            *o = make_float2(s.x, low == low ? low : 0.0f);
          }
        }
      }
    }
  }
}

// item: (node, 32-channel slice, part of the node's edges), parts fastest
template <int LMAX, int CT, bool CANON>
__device__ __forceinline__ void rev_item(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                         const float* __restrict__ dPhi1, fix64* __restrict__ H1_adj,
                                         float* __restrict__ f1, RevSmem& s, int item, int split, int cs) {
  const int ns = (CT > 0 ? CT : m.C) >> 5;
  const int part = item % split, w = item / split;
  const int i = in.atom_at(w / ns), slice = w % ns;
  if (in.first[i] + part * cs >= in.end(i)) return;
  const int k = slice * 32 + (threadIdx.x & 31);
  float* f1s = f1 + slice * m.f1_stride * (LMAX == 2 ? 2 : 1);
  rev_group<LMAX, 0, CT, CANON>(m, in, H1, dPhi1, H1_adj, f1s, s, i, k, part, split, cs);
  if constexpr (LMAX == 2) {
    rev_group<LMAX, 1, CT, CANON>(m, in, H1, dPhi1, H1_adj, f1s, s, i, k, part, split, cs);
    rev_group<LMAX, 2, CT, CANON>(m, in, H1, dPhi1, H1_adj, f1s, s, i, k, part, split, cs);
  }
}

}  // namespace

// 12 warps per SM either way (168 registers, three warps per scheduler); asked for 11, the
// compiler orders the L_max = 1 kernel's loads better (ms, 11 : 12, 213k edges of 128 channels
// 0.444 : 0.453; L_max = 2, 178k edges 0.962 : 0.959).
template <int LMAX, int CT, bool CANON, bool P>
__global__ void __launch_bounds__(32, LMAX == 1 ? 11 : 12) k_layer1_rev(DevModel m, EdgeIn in, const float* __restrict__ H1,
                                                      const float* __restrict__ dPhi1, fix64* __restrict__ H1_adj,
                                                      float* __restrict__ f1, int split, int cs) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char dyn[];
  RevSmem& s = *reinterpret_cast<RevSmem*>(dyn);
  const int n = in.N * split * ((CT > 0 ? CT : m.C) >> 5);
  AtomCursor cur{P ? m.sched : nullptr, n, 0};
  for (int b = cur.first(); b < n; b = cur.next())
    rev_item<LMAX, CT, CANON>(m, in, H1, dPhi1, H1_adj, f1, s, b, split, cs);
  cur.done();
}

namespace {

size_t rev_smem(const DevModel& m) {
  const size_t rows = m.cg_val ? 0 : m.n_lme + m.n_p;
  return offsetof(RevSmem, buf) + std::max<size_t>(sizeof(float2) * kSumEdges * 8 * kSumRow, sizeof(float) * 32 * rows);
}

}  // namespace

void launch_layer1_rev(const DevModel& m, const EdgeIn& in, const float* H1, const float* dPhi1, fix64* H1_adj,
                       float* f1, cudaStream_t s) {
  if (in.N <= 0) return;
  const long items = static_cast<long>(in.N) * (m.C >> 5);
  // parts pay the g prologue again (us, whole : split: 64 items 24.6 : 12.3 (16 parts), 1000
  // items 55.3 : 59.4 (3), 1998 items, one full wave and a nearly empty one, 105.5 : 98.3 (2))
  const int split = edge_split(items), cs = edge_chunk(split);
  DevModel mk;
  const int grid = atom_grid(m, kAkLayer1Rev, static_cast<int>(items * split), mk);
  dispatch_layer1(m, [&](auto lc, auto cc, auto nc) {
    constexpr int LM = decltype(lc)::value, CT = decltype(cc)::value;
    constexpr bool CANON = decltype(nc)::value;
    if (mk.sched)
      launch_pdl(k_layer1_rev<LM, CT, CANON, true>, grid, 32, rev_smem(m), s, mk, in, H1, dPhi1, H1_adj, f1, split, cs);
    else
      launch_pdl(k_layer1_rev<LM, CT, CANON, false>, grid, 32, rev_smem(m), s, mk, in, H1, dPhi1, H1_adj, f1, split, cs);
  });
}

int layer1_rev_residency(const DevModel& m) {
  int r = 0;
  dispatch_layer1(m, [&](auto lc, auto cc, auto nc) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &r, k_layer1_rev<decltype(lc)::value, decltype(cc)::value, decltype(nc)::value, true>, 32, rev_smem(m));
  });
  return r;
}

}  // namespace smx
