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
// What bounds it: issue slots and the packed dependencies between them (64% of the cycles
// issue, at 12 warps per SM and 168 registers; 255 registers without the spills of 50 bytes,
// 8 warps: 0.55 -> 0.58 ms).  Against one block per node with two instruction halves of
// channel pairs, which met at a barrier for every edge (8 warps per SM, 47% of the cycles
// issuing, four FMAs per path): 4096 atoms, 128 channels, 213k edges 0.733 -> 0.533 ms;
// L_max = 2, 2197 atoms, 178k edges 2.12 -> 1.15 ms.
//
// L_max = 2 (17 instructions, 243 paths): three instruction groups in turn, by the l of
// H1: {0, 1} (the ten instructions of L_max = 1) and two halves of l = 2, so that a group's
// g fits the registers and the H1_adj rows of l = 0, 1 are added once, those of l = 2 twice.
#include <cuda_runtime.h>

#include <algorithm>

#include "device.cuh"
#include "kernels.h"

namespace smx {

namespace {

// instruction groups, ordered by l1 (Y_00 = 1: an l1 = 0 instruction has u = g and no dE/dY)
__host__ __device__ constexpr int rev_groups(int LMAX) { return LMAX == 1 ? 1 : 3; }
__host__ __device__ constexpr int rev_count(int LMAX, int G) { return G == 0 ? 10 : (G == 1 ? 3 : 4); }
__host__ __device__ constexpr int rev_ins(int LMAX, int G, int i) {
  constexpr int a[10] = {0, 3, 2, 1, 6, 5, 4, 9, 8, 7};
  constexpr int b[10] = {0, 4, 3, 1, 9, 8, 5, 14, 13, 10}, b1[3] = {6, 2, 7}, b2[4] = {11, 15, 12, 16};
  return LMAX == 1 ? a[i] : (G == 0 ? b[i] : (G == 1 ? b1[i] : b2[i]));
}
// the H1 rows [row0, row0 + rows) that group G reads and adds to
__host__ __device__ constexpr int rev_row0(int G) { return G == 0 ? 0 : 4; }
__host__ __device__ constexpr int rev_rows(int G) { return G == 0 ? 4 : 5; }
__host__ __device__ constexpr int ins_paths(int LMAX, int q) {
  return (2 * ins_l1(LMAX, q) + 1) * (2 * ins_l2(LMAX, q) + 1);
}
// offset of the group's i-th instruction in its path list
template <int LMAX, int G>
__host__ __device__ constexpr int rev_goff(int i) {
  int s = 0;
  for (int w = 0; w < i; ++w) s += ins_paths(LMAX, rev_ins(LMAX, G, w));
  return s;
}
// is the i-th instruction the first of its group with its l1 (l2)?
template <int LMAX, int G>
__host__ __device__ constexpr bool rev_first_l1(int i) {
  for (int w = 0; w < i; ++w)
    if (ins_l1(LMAX, rev_ins(LMAX, G, w)) == ins_l1(LMAX, rev_ins(LMAX, G, i))) return false;
  return true;
}
template <int LMAX, int G>
__host__ __device__ constexpr bool rev_first_l2(int i) {
  for (int w = 0; w < i; ++w)
    if (ins_l2(LMAX, rev_ins(LMAX, G, w)) == ins_l2(LMAX, rev_ins(LMAX, G, i))) return false;
  return true;
}

constexpr int kSumEdges = 4;  // edges summed over the lanes at a time
constexpr int kSumRow = 33;   // row pitch of their terms: 32 rows read at one column hit all banks

// shared memory of one warp
struct RevSmem {
  float Y[kEdgeChunk][16];   // Y_lm of the staged edges; then (dE/dR term, dE/dY_1 .. dE/dY_15)
  int4 meta[kEdgeChunk];     // offset inside the spline interval (float bits), spline row, j
  float2 buf[1];             // [kSumEdges * 8][kSumRow] per-lane terms; before the edges: dPhi1 rows
};

__device__ __forceinline__ void async_copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One edge, group G, this lane's channel; c: the edge's cubics, replaced by those of the
// next edge (cn); t: this lane's slot of the edge in RevSmem::buf.
template <int LMAX, int G>
__device__ __forceinline__ void rev_edge(const float* g, float4* c, const float4* __restrict__ cn, int C, float x,
                                         const float* Y, const float* h, float* hadj, float2* t) {
  float y[16];
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const float4 f = *reinterpret_cast<const float4*>(Y + 4 * v);
    y[4 * v] = f.x;
    y[4 * v + 1] = f.y;
    y[4 * v + 2] = f.z;
    y[4 * v + 3] = f.w;
  }
  constexpr int r0 = rev_row0(G);
  float dY[16], dr = 0.0f;
  static_for<rev_count(LMAX, G)>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr int q = rev_ins(LMAX, G, i);
    constexpr int l1 = ins_l1(LMAX, q), l2 = ins_l2(LMAX, q), g0 = rev_goff<LMAX, G>(i), nb = 2 * l2 + 1;
    constexpr bool first1 = rev_first_l1<LMAX, G>(i), first2 = rev_first_l2<LMAX, G>(i);
    // value and derivative by the two-row Horner scheme
    float R = fmaf(c[i].w, x, c[i].z);
    float Rd = fmaf(c[i].w, x, R);
    R = fmaf(R, x, c[i].y);
    Rd = fmaf(Rd, x, R);
    R = fmaf(R, x, c[i].x);
    c[i] = __ldg(cn + q * C);
    float us[nb], rh[nb];
#pragma unroll
    for (int b = 0; b < nb; ++b) rh[b] = R * h[l2 * l2 - r0 + b];
#pragma unroll
    for (int a = 0; a < 2 * l1 + 1; ++a) {
#pragma unroll
      for (int b = 0; b < nb; ++b) {
        const float gp = g[g0 + a * nb + b];
        if constexpr (l1 == 0) {
          us[b] = gp;
        } else {
          us[b] = a == 0 ? gp * y[l1 * l1] : fmaf(gp, y[l1 * l1 + a], us[b]);
          dY[l1 * l1 + a] = (first1 && b == 0) ? gp * rh[b] : fmaf(gp, rh[b], dY[l1 * l1 + a]);
        }
      }
    }
    float w = us[0] * h[l2 * l2 - r0];
#pragma unroll
    for (int b = 1; b < nb; ++b) w = fmaf(us[b], h[l2 * l2 - r0 + b], w);
    dr = i == 0 ? w * Rd : fmaf(w, Rd, dr);
#pragma unroll
    for (int b = 0; b < nb; ++b) {
      float& o = hadj[l2 * l2 - r0 + b];
      o = first2 ? R * us[b] : fmaf(R, us[b], o);
    }
  });
  t[0] = make_float2(dr, dY[1]);
#pragma unroll
  for (int v = 1; v < 8; ++v) t[kSumRow * v] = make_float2(dY[2 * v], dY[2 * v + 1]);
}

// The sums over the lanes of edges [a0, a0 + n) (n <= kSumEdges) into their Y rows: lane
// 8 e + v adds component pair v of edge e, four partial sums in a fixed order.
__device__ __forceinline__ void rev_sums(RevSmem& s, int a0, int n) {
  const int lane = threadIdx.x & 31, e = lane >> 3, v = lane & 7;
  __syncwarp();
  if (e < n) {
    const float2* row = s.buf + lane * kSumRow;
    float2 p0 = make_float2(0.0f, 0.0f), p1 = p0, p2 = p0, p3 = p0;
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      p0 = __fadd2_rn(p0, row[i]);
      p1 = __fadd2_rn(p1, row[i + 1]);
      p2 = __fadd2_rn(p2, row[i + 2]);
      p3 = __fadd2_rn(p3, row[i + 3]);
    }
    *reinterpret_cast<float2*>(&s.Y[a0 + e][2 * v]) = __fadd2_rn(__fadd2_rn(p0, p1), __fadd2_rn(p2, p3));
  }
  __syncwarp();
}

// Group G over the edges of chunks `split` apart; `add`: the edge forces of an earlier group
// of the same warp are in f1 already.
template <int LMAX, int G, int CT>
__device__ __forceinline__ void rev_group(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                          const float* __restrict__ dPhi1, fix64* __restrict__ H1_adj,
                                          float* __restrict__ f1, RevSmem& s, int i, int k, int part, int split,
                                          int cs) {
  constexpr int NI = ins_count(LMAX), NL2 = (LMAX + 1) * (LMAX + 1);
  constexpr int NQ = rev_count(LMAX, G), NP = rev_goff<LMAX, G>(NQ), NR = rev_rows(G), r0 = rev_row0(G);
  const int C = CT > 0 ? CT : m.C;
  const int lane = threadIdx.x & 31;
  const int ti = in.node_type[i];
  const int e0 = in.first[i], e1 = in.end(i);
  // g of this lane's channel from the node's dPhi1 rows
  float g[NP];
  float* sD = reinterpret_cast<float*>(s.buf);  // [n_lme][32]
  __syncwarp();
  for (int lme = 0; lme < m.n_lme; ++lme)  // (a lane reads only its own column back)
    async_copy4(sD + lme * 32 + lane, dPhi1 + (static_cast<size_t>(i) * m.n_lme + lme) * C + k);
  // this lane's edge of a chunk; the first chunk's loads overlap the copies
  float vx, vy, vz, rr;
  int tj, nj;
  auto load = [&](int eb) {
    const long e = min(eb + lane, e1 - 1);
    vx = static_cast<float>(in.xyz[3 * e]);
    vy = static_cast<float>(in.xyz[3 * e + 1]);
    vz = static_cast<float>(in.xyz[3 * e + 2]);
    rr = static_cast<float>(in.r[e]);
    tj = in.ntype_e[e];
    nj = in.nidx[e];
  };
  load(e0 + part * cs);
  async_wait();
  if (m.cg_rev_pad) {  // two terms per path, all loads independent
    static_for<NQ>([&](auto ic) {
      constexpr int w = decltype(ic)::value;
      constexpr int q = rev_ins(LMAX, G, w), p0 = ins_poff(LMAX, q), g0 = rev_goff<LMAX, G>(w);
#pragma unroll
      for (int p = 0; p < ins_paths(LMAX, q); ++p) {
        const int4 tt = __ldg(reinterpret_cast<const int4*>(m.cg_rev_pad) + p0 + p);
        g[g0 + p] = fmaf(__int_as_float(tt.w), sD[tt.z * 32 + lane], __int_as_float(tt.y) * sD[tt.x * 32 + lane]);
      }
    });
  } else {  // any number of terms: all paths first, through the compressed rows
    float* sP = sD + m.n_lme * 32;  // [NP][32]
    for (int p = 0; p < m.n_p; ++p) {
      float v = 0.0f;
      for (int t = __ldg(m.cg_rev_off + p), t1 = __ldg(m.cg_rev_off + p + 1); t < t1; ++t)
        v = fmaf(__ldg(m.cg_rev_v + t), sD[__ldg(m.cg_rev_lme + t) * 32 + lane], v);
      sP[p * 32 + lane] = v;
    }
    static_for<NQ>([&](auto ic) {
      constexpr int w = decltype(ic)::value;
      constexpr int q = rev_ins(LMAX, G, w), p0 = ins_poff(LMAX, q), g0 = rev_goff<LMAX, G>(w);
#pragma unroll
      for (int p = 0; p < ins_paths(LMAX, q); ++p) g[g0 + p] = sP[(p0 + p) * 32 + lane];
    });
  }
  for (int eb = e0 + part * cs; eb < e1; eb += split * cs) {
    const int ne = min(cs, e1 - eb);
    const long e = static_cast<long>(eb) + lane;
    if (eb > e0 + part * cs) load(eb);
    const bool active = lane < ne && rr < m.r_cut;
    const unsigned ball = __ballot_sync(0xffffffffu, active);
    const int na = __popc(ball), pos = __popc(ball & ((1u << lane) - 1u));
    __syncwarp();  // the last chunk's sums have been read
    if (active) {  // (inactive edges are left out of the staged list)
      float Y[16];
      sph_harm16<false>(vx, vy, vz, Y, nullptr);
#pragma unroll
      for (int v = 0; v < 4; ++v)
        *reinterpret_cast<float4*>(&s.Y[pos][4 * v]) = make_float4(Y[4 * v], Y[4 * v + 1], Y[4 * v + 2], Y[4 * v + 3]);
      int iv = static_cast<int>(rr * m.inv_h);
      iv = iv < 0 ? 0 : (iv >= m.nint ? m.nint - 1 : iv);
      const int a = ti < tj ? ti : tj, b = ti < tj ? tj : ti;
      s.meta[pos] = make_int4(__float_as_int(rr - static_cast<float>(iv) * m.h),
                              (a * (2 * m.S - a - 1) / 2 + b) * m.nint + iv, nj, 0);
    }
    __syncwarp();
    if (na > 0) {
      float4 c[NQ];
      float h[NR];
      int4 mt = s.meta[0];
      {
        const float4* cp = m.spl1_fwd + static_cast<size_t>(mt.y) * NI * C + k;
        static_for<NQ>([&](auto ic) {
          constexpr int w = decltype(ic)::value;
          c[w] = __ldg(cp + rev_ins(LMAX, G, w) * C);
        });
        const float* hp = H1 + (static_cast<size_t>(mt.z) * NL2 + r0) * C + k;
#pragma unroll
        for (int b = 0; b < NR; ++b) h[b] = __ldg(hp + b * C);
      }
      for (int a = 0; a < na; ++a) {
        const int4 mn = s.meta[min(a + 1, na - 1)];
        const float4* cn = m.spl1_fwd + static_cast<size_t>(mn.y) * NI * C + k;
        float hv[NR], hadj[NR];
        const float* hp = H1 + (static_cast<size_t>(mn.z) * NL2 + r0) * C + k;
#pragma unroll
        for (int b = 0; b < NR; ++b) {
          hv[b] = h[b];
          h[b] = __ldg(hp + b * C);
        }
        rev_edge<LMAX, G>(g, c, cn, C, __int_as_float(mt.x), s.Y[a], hv, hadj,
                          s.buf + (a % kSumEdges) * 8 * kSumRow + lane);
        fix64* dst = H1_adj + (static_cast<size_t>(mt.z) * NL2 + r0) * C + k;
#pragma unroll
        for (int b = 0; b < NR; ++b) add_fixed(dst + b * C, hadj[b]);
        mt = mn;
        if (a % kSumEdges == kSumEdges - 1 || a == na - 1)
          rev_sums(s, a - a % kSumEdges, a % kSumEdges + 1);
      }
    }
    if (lane < ne) {  // this lane's edge: the sums against u and dY/dx
      float fx = 0.0f, fy = 0.0f, fz = 0.0f;
      if (active) {
        float Y[16], D[48];
        sph_harm16<true>(vx, vy, vz, Y, D);
        const float* S = s.Y[pos];
        const float d = S[0] / rr;
        fx = d * vx;
        fy = d * vy;
        fz = d * vz;
#pragma unroll
        for (int q = 1; q < 16; ++q) {
          fx = fmaf(S[q], D[q], fx);
          fy = fmaf(S[q], D[16 + q], fy);
          fz = fmaf(S[q], D[32 + q], fz);
        }
      }
      float* o = f1 + 3 * e;
      o[0] = G > 0 ? o[0] + fx : fx;
      o[1] = G > 0 ? o[1] + fy : fy;
      o[2] = G > 0 ? o[2] + fz : fz;
    }
  }
}

// item: (node, 32-channel slice, part of the node's edges), parts fastest
template <int LMAX, int CT>
__device__ __forceinline__ void rev_item(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                         const float* __restrict__ dPhi1, fix64* __restrict__ H1_adj,
                                         float* __restrict__ f1, RevSmem& s, int item, int split, int cs) {
  const int ns = (CT > 0 ? CT : m.C) >> 5;
  const int part = item % split, w = item / split;
  const int i = in.atom_at(w / ns), slice = w % ns;
  if (in.first[i] + part * cs >= in.end(i)) return;
  const int k = slice * 32 + (threadIdx.x & 31);
  float* f1s = f1 + slice * m.f1_stride;
  rev_group<LMAX, 0, CT>(m, in, H1, dPhi1, H1_adj, f1s, s, i, k, part, split, cs);
  if constexpr (LMAX == 2) {
    rev_group<LMAX, 1, CT>(m, in, H1, dPhi1, H1_adj, f1s, s, i, k, part, split, cs);
    rev_group<LMAX, 2, CT>(m, in, H1, dPhi1, H1_adj, f1s, s, i, k, part, split, cs);
  }
}

}  // namespace

template <int LMAX, int CT, bool P>
__global__ void __launch_bounds__(32, 12) k_layer1_rev(DevModel m, EdgeIn in, const float* __restrict__ H1,
                                                      const float* __restrict__ dPhi1, fix64* __restrict__ H1_adj,
                                                      float* __restrict__ f1, int split, int cs) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char dyn[];
  RevSmem& s = *reinterpret_cast<RevSmem*>(dyn);
  const int n = in.N * split * ((CT > 0 ? CT : m.C) >> 5);
  AtomCursor cur{P ? m.sched : nullptr, n, 0};
  for (int b = cur.first(); b < n; b = cur.next())
    rev_item<LMAX, CT>(m, in, H1, dPhi1, H1_adj, f1, s, b, split, cs);
  cur.done();
}

namespace {

// channel counts with a compile-time specialisation (addresses fold to immediates)
template <typename F>
void dispatch_rev(const DevModel& m, F&& f) {
  auto by_c = [&](auto lc) {
    switch (m.C) {
      case 32: f(lc, std::integral_constant<int, 32>{}); break;
      case 64: f(lc, std::integral_constant<int, 64>{}); break;
      case 128: f(lc, std::integral_constant<int, 128>{}); break;
      default: f(lc, std::integral_constant<int, 0>{}); break;
    }
  };
  if (m.L_max == 2)
    by_c(std::integral_constant<int, 2>{});
  else
    by_c(std::integral_constant<int, 1>{});
}

// Warps the chip holds at once (12 per SM).  A node's edges are split over `split` warps
// while all parts still fit at once, each part paying the g prologue again, and over two
// when the items would run as one full and one nearly empty wave (us, whole : split:
// 64 items 24.6 : 12.3 (16 parts), 1000 items 55.3 : 59.4 (3), 1998 items 105.5 : 98.3 (2)).
constexpr long kSlots = 12 * 152;

size_t rev_smem(const DevModel& m) {
  const size_t rows = m.n_lme + (m.cg_rev_pad ? 0 : m.n_p);
  return offsetof(RevSmem, buf) + std::max<size_t>(sizeof(float2) * kSumEdges * 8 * kSumRow, sizeof(float) * 32 * rows);
}

}  // namespace

void launch_layer1_rev(const DevModel& m, const EdgeIn& in, const float* H1, const float* dPhi1, fix64* H1_adj,
                       float* f1, cudaStream_t s) {
  if (in.N <= 0) return;
  const long items = static_cast<long>(in.N) * (m.C >> 5);
  const int split =
      items > 2 * kSlots ? 1 : (items > kSlots ? 2 : static_cast<int>(std::min<long>(16, kSlots / items)));
  const int cs = split == 1 ? kEdgeChunk : (split <= 2 ? 16 : (split <= 8 ? 8 : 4));
  DevModel mk;
  const int grid = atom_grid(m, kAkLayer1Rev, static_cast<int>(items * split), mk);
  dispatch_rev(m, [&](auto lc, auto cc) {
    constexpr int LM = decltype(lc)::value, CT = decltype(cc)::value;
    if (mk.sched)
      launch_pdl(k_layer1_rev<LM, CT, true>, grid, 32, rev_smem(m), s, mk, in, H1, dPhi1, H1_adj, f1, split, cs);
    else
      launch_pdl(k_layer1_rev<LM, CT, false>, grid, 32, rev_smem(m), s, mk, in, H1, dPhi1, H1_adj, f1, split, cs);
  });
}

int layer1_rev_residency(const DevModel& m) {
  int r = 0;
  dispatch_rev(m, [&](auto lc, auto cc) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k_layer1_rev<decltype(lc)::value, decltype(cc)::value, true>, 32,
                                                  rev_smem(m));
  });
  return r;
}

}  // namespace smx
