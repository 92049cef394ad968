// Layer-0 kernels: the neighbour sum A0 with its symmetric contraction M0, and their adjoints.
//
// Reference stages restated here (libsymmetrix/source/mace.cpp):
//   k_layer0_fwd    : compute_Y + compute_R0 + compute_A0 (:66-201) + compute_M0 (:348-370)
//   k_contract0_rev : reverse_M0 (:372-395)
//   k_layer0_rev    : reverse_A0 (:203-271)
//
// The edge kernels run one warp per node (and 64 channels in the forward), a warp being a
// block: no block barriers, all per-channel arithmetic on channel pairs with the packed FMA,
// and the next edge's cubics loaded into the registers that this edge's have left.  What
// bounds them is the L2 gather of the folded spline rows, 8 KB per edge at 128 channels
// (0.08 ms for 213k edges at the 21.9 TB/s of a plain gather), and of the contraction's
// coefficients, 0.2 MB per node.  Against a block of two warp groups per node whose sums met
// in shared memory, five-and-forty scalar FMAs per edge and channel for the force and
// polynomials with the products of pairs in registers (255 of them): 4096 atoms, 128
// channels, forward 0.165 -> 0.130 ms, adjoints together 0.262 -> 0.181 ms; L_max = 2, 2197
// atoms 0.225 -> 0.122 and 0.260 -> 0.188 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "edge.cuh"
#include "kernels.h"
#include "poly_canon.h"

namespace smx {

namespace {

constexpr int kRow0 = 18;

// Up to 32 edges of a node staged by one warp, those inside the cut-off packed to the front.
struct L0Stage {
  // (Y_lm, Y_lm): operands of the packed FMAs.  In the adjoint, once an edge is done: its sums in
  // their place (the row pitch: 16-byte reads of the lanes' own rows hit all banks)
  alignas(16) float2 Y2[kEdgeChunk][kRow0];
  int2 meta[kEdgeChunk];      // offset inside the spline interval (float bits), ordered-pair spline row
};

// rows first, so that the first edge's loads can go out (as stage_rows in layer1.cuh)
__device__ __forceinline__ int stage_rows0(const DevModel& m, L0Stage& st, const LaneEdge& ed, int ti, bool active,
                                           int& count) {
  const unsigned ball = __ballot_sync(0xffffffffu, active);
  const int pos = __popc(ball & ((1u << (threadIdx.x & 31)) - 1u));
  count = __popc(ball);
  __syncwarp();  // the last chunk has been read
  if (active) st.meta[pos] = make_int2(__float_as_int(ed.x), (ti * m.S + ed.tj) * m.nint + ed.iv);
  __syncwarp();
  return pos;
}
__device__ __forceinline__ void stage_Y0(L0Stage& st, const LaneEdge& ed, bool active, int pos) {
  if (active) {
    float Y[16];
    sph_harm16<false>(ed.vx, ed.vy, ed.vz, Y, nullptr);
#pragma unroll
    for (int v = 0; v < 8; ++v)
      *reinterpret_cast<float4*>(&st.Y2[pos][2 * v]) = make_float4(Y[2 * v], Y[2 * v], Y[2 * v + 1], Y[2 * v + 1]);
  }
  __syncwarp();
}
__device__ __forceinline__ void read_Y2(const float2* Y2, float2* y) {
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const float4 f = *reinterpret_cast<const float4*>(Y2 + 2 * v);
    y[2 * v] = make_float2(f.x, f.y);
    y[2 * v + 1] = make_float2(f.z, f.w);
  }
}

// split terms of a channel pair (write_split)
__device__ __forceinline__ void write_split2(__nv_bfloat16* row, int K, int T, int col, float2 v) {
  const __nv_bfloat162 hi = __float22bfloat162_rn(v);
  *reinterpret_cast<__nv_bfloat162*>(row + col) = hi;
  if (T == 3) {
    const float2 h = __bfloat1622float2(hi);
    *reinterpret_cast<__nv_bfloat162*>(row + K + col) = __float22bfloat162_rn(make_float2(v.x - h.x, v.y - h.y));
  }
}

// P_LM and its weighted gradient for the generated polynomials, by a compile-time LM
template <int LM>
__device__ __forceinline__ float2 contract_value(const float2* x, const float2* cf, int S) {
  if constexpr (LM == 0) return poly::value_LM0(x, cf, S);
  if constexpr (LM == 1) return poly::value_LM1(x, cf, S);
  if constexpr (LM == 2) return poly::value_LM2(x, cf, S);
  if constexpr (LM == 3) return poly::value_LM3(x, cf, S);
  if constexpr (LM == 4) return poly::value_LM4(x, cf, S);
  if constexpr (LM == 5) return poly::value_LM5(x, cf, S);
  if constexpr (LM == 6) return poly::value_LM6(x, cf, S);
  if constexpr (LM == 7) return poly::value_LM7(x, cf, S);
  if constexpr (LM == 8) return poly::value_LM8(x, cf, S);
}
template <int LM>
__device__ __forceinline__ void contract_grad(const float2* x, float2 w, const float2* cf, int S, float2* g) {
  if constexpr (LM == 0) poly::grad_LM0(x, w, cf, S, g);
  if constexpr (LM == 1) poly::grad_LM1(x, w, cf, S, g);
  if constexpr (LM == 2) poly::grad_LM2(x, w, cf, S, g);
  if constexpr (LM == 3) poly::grad_LM3(x, w, cf, S, g);
  if constexpr (LM == 4) poly::grad_LM4(x, w, cf, S, g);
  if constexpr (LM == 5) poly::grad_LM5(x, w, cf, S, g);
  if constexpr (LM == 6) poly::grad_LM6(x, w, cf, S, g);
  if constexpr (LM == 7) poly::grad_LM7(x, w, cf, S, g);
  if constexpr (LM == 8) poly::grad_LM8(x, w, cf, S, g);
}

constexpr int kDepth0 = 2;  // edges in flight per warp of the forward

}  // namespace

// ---------------------------------------------------------------------------
// Layer 0 forward: A0[i,lm,k] = sum_j Y_lm(x_ij) R0'_{ti,tj,l}(r_ij)[k] with the
// folded ordered-pair splines, then M0[i,LM,k] = P_{ti,LM,k}(A0[i,:,k]) for the lane's two
// channels.  (The contraction as a kernel of its own, a warp per output LM: 0.108 + 0.039 ms
// against 0.137 ms together, before the row pitch of the staged Y.)
// ---------------------------------------------------------------------------
template <int NLM, int CT>
__device__ __forceinline__ void layer0_fwd_item(const DevModel& m, const EdgeIn& in, float* __restrict__ A0,
                                                float* __restrict__ M0, float* __restrict__ zbl_e, L0Stage& st,
                                                float* sA, int i, int slice) {
  const int C = CT > 0 ? CT : m.C, C2 = C >> 1;
  const int lane = threadIdx.x & 31;
  const bool live = slice * 32 + lane < C2;
  const int cp = live ? slice * 32 + lane : slice * 32, kc = 2 * cp;
  const int ti = in.node_type[i];
  const int e0 = in.first[i], e1 = in.end(i);
  float2 acc[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) acc[q] = make_float2(0.0f, 0.0f);
  for (int eb = e0; eb < e1; eb += kEdgeChunk) {
    LaneEdge ed;
    ed.load(m, in, min(eb + lane, e1 - 1));
    int na;
    const bool active = eb + lane < e1 && ed.r < m.r_cut;
    const int pos = stage_rows0(m, st, ed, ti, active, na);
    if (na == 0) continue;
    float4 c[kDepth0][8];
    static_for<kDepth0>([&](auto dc) {
      constexpr int d = decltype(dc)::value;
      const float4* p = m.spl0 + static_cast<size_t>(st.meta[min(d, na - 1)].y) * 4 * C + cp;
#pragma unroll
      for (int q = 0; q < 8; ++q) c[d][q] = __ldg(p + q * C2);
    });
    stage_Y0(st, ed, active, pos);
    for (int a0 = 0; a0 < na; a0 += kDepth0) {
      static_for<kDepth0>([&](auto dc) {
        constexpr int d = decltype(dc)::value;
        const int a = a0 + d;
        if (a >= na) return;
        const float4* p = m.spl0 + static_cast<size_t>(st.meta[min(a + kDepth0, na - 1)].y) * 4 * C + cp;
        const float x = __int_as_float(st.meta[a].x);
        const float2 x2 = make_float2(x, x);
        float2 y[16];
        read_Y2(st.Y2[a], y);
        static_for<4>([&](auto lc) {
          constexpr int l = decltype(lc)::value;
          const float2 R = spline2_val(c[d][2 * l], c[d][2 * l + 1], x2);
          c[d][2 * l] = __ldg(p + 2 * l * C2);
          c[d][2 * l + 1] = __ldg(p + (2 * l + 1) * C2);
          if constexpr (l == 0) {
            acc[0] = __fadd2_rn(R, acc[0]);  // Y_00 = 1 (sph_harm16)
          } else {
#pragma unroll
            for (int q = l * l; q < (l + 1) * (l + 1); ++q) acc[q] = fma2(R, y[q], acc[q]);
          }
        });
      });
    }
  }
  if (m.has_zbl && slice == 0) {  // ZBL energy of node i: sum over its directed edges (zbl.cpp:96-125)
    float z = 0.0f;
    for (int e = e0 + lane; e < e1; e += 32) {
      float V, dV;
      zbl_edge(m, m.zbl_pair[ti * m.S + in.ntype_e[e]], static_cast<float>(in.r[e]), V, dV);
      z += V;
    }
    z = warp_sum(z);
    if (lane == 0) zbl_e[i] = z;
  }
  if (m.dens_spl[0]) {  // density-normalised A0: A0 /= 1 + sum_j s(r_ij)  (mace.cpp:273-297)
    const float S = dens_factor(m, 0, in, i, ti);
    if (lane == 0 && slice == 0) m.dens_s[0][i] = S;
#pragma unroll
    for (int q = 0; q < 16; ++q) acc[q] = make_float2(acc[q].x / S, acc[q].y / S);
  }
  if (live)
#pragma unroll
    for (int q = 0; q < 16; ++q)
      *reinterpret_cast<float2*>(A0 + (static_cast<size_t>(i) * 16 + q) * C + kc) = acc[q];
  auto put = [&](int LM, float2 v) {  // M0 nullptr: only the split rows are consumed
    if (!live) return;
    if (M0) *reinterpret_cast<float2*>(M0 + (static_cast<size_t>(i) * m.nLM + LM) * C + kc) = v;
    if (m.op_m0)  // BF16 form: the H1 GEMM's split operand
      write_split2(m.op_m0 + (static_cast<size_t>(i) * m.nLM + LM) * split_xterms(m.tc_terms) * C, C, m.tc_terms, kc, v);
  };
  if (m.poly_canon) {  // generated straight-line polynomials, A0 columns in registers
    const float2* cf = reinterpret_cast<const float2*>(m.coef0 + static_cast<size_t>(ti * m.nLM) * m.T0 * C) + cp;
    const size_t sst = static_cast<size_t>(m.T0) * C2;
    static_for<NLM>([&](auto lc) {
      constexpr int LM = decltype(lc)::value;
      put(LM, contract_value<LM>(acc, cf + LM * sst, C2));
    });
    return;
  }
  float2* x = reinterpret_cast<float2*>(sA) + lane;  // [17][32]: this lane's columns (+ constant one)
#pragma unroll
  for (int q = 0; q < 16; ++q) x[q * 32] = acc[q];
  x[16 * 32] = make_float2(1.0f, 1.0f);
  for (int LM = 0; LM < m.nLM; ++LM) {
    const int t0 = m.mono0_off[LM], t1 = m.mono0_off[LM + 1];
    const float2* cf = reinterpret_cast<const float2*>(m.coef0 + (static_cast<size_t>(ti * m.nLM + LM) * m.T0) * C) + cp;
    float2 f = make_float2(0.0f, 0.0f);
    for (int t = t0; t < t1; ++t) {
      const int pk = __ldg(m.mono0 + t);
      const float2 p = mul2(mul2(x[(pk & 255) * 32], x[((pk >> 8) & 255) * 32]), x[(pk >> 16) * 32]);
      f = fma2(__ldg(cf + static_cast<size_t>(t - t0) * C2), p, f);
    }
    put(LM, f);
  }
}

__host__ __device__ inline int layer0_slices(int C) { return (C + 63) / 64; }

// (this kernel and k_contract0_rev hold the generated polynomials and have no persistent form:
// their blocks are single warps, which gain nothing from one, and the code would double)
template <int NLM, int CT>
__global__ void __launch_bounds__(32, 12) k_layer0_fwd(DevModel m, EdgeIn in, float* __restrict__ A0,
                                                       float* __restrict__ M0, float* __restrict__ zbl_e) {
  pdl_begin();
  __shared__ L0Stage st;
  extern __shared__ __align__(16) float dyn[];
  const int ns = layer0_slices(CT > 0 ? CT : m.C), b = blockIdx.x;
  layer0_fwd_item<NLM, CT>(m, in, A0, M0, zbl_e, st, dyn, in.atom_at(b / ns), b % ns);
}

// ---------------------------------------------------------------------------
// Layer-0 contraction adjoint (mace.cpp:372-395):
//   A0_adj[i,:,k] = sum_LM M0_adj[i,LM,k] grad P_{ti,LM,k}(A0[i,:,k]).
// A block per node, a lane per channel pair: one warp per 64 channels, or (SPLIT, small
// systems) a warp per output LM and 64 channels, whose gradients meet in shared memory and
// are added in the order of LM.  The one warp adds whole gradients of the outputs in that order
// too: a node's bits do not depend on the form, which follows from the number of nodes, so a
// molecule gives the same forces alone and in a batch.
// ---------------------------------------------------------------------------
constexpr int contract0_max_warps(int NLM, int CT, bool SPLIT) {
  return (SPLIT ? NLM : 1) * (CT > 0 ? (CT + 63) / 64 : (NLM == 9 ? 2 : 4));
}
// (SPLIT: 20 warps per SM)
template <int NLM, int CT, bool SPLIT>
__global__ void __launch_bounds__(32 * contract0_max_warps(NLM, CT, SPLIT),
                                  !SPLIT || contract0_max_warps(NLM, CT, SPLIT) > 10
                                      ? 1
                                      : 20 / contract0_max_warps(NLM, CT, SPLIT))
    k_contract0_rev(DevModel m, const int* __restrict__ node_type, const int* __restrict__ order, const float* __restrict__ A0,
                    const float* __restrict__ M0_adj, float* __restrict__ A0_adj) {
  pdl_begin();
  extern __shared__ __align__(16) float dyn[];
  const int C = CT > 0 ? CT : m.C, C2 = C >> 1, ns = layer0_slices(C);
  const int i = order ? order[blockIdx.x] : blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int slice = SPLIT ? warp % ns : warp, part = SPLIT ? warp / ns : 0, parts = SPLIT ? m.nLM : 1;
  const bool live = slice * 32 + lane < C2;
  const int cp = live ? slice * 32 + lane : slice * 32;
  const int ti = node_type[i];
  const float2* xr = reinterpret_cast<const float2*>(A0 + static_cast<size_t>(i) * 16 * C) + cp;
  const float2* w = reinterpret_cast<const float2*>(M0_adj + static_cast<size_t>(i) * m.nLM * C) + cp;
  const size_t sst = static_cast<size_t>(m.T0) * C2;
  const float2* cf = reinterpret_cast<const float2*>(m.coef0 + static_cast<size_t>(ti * m.nLM) * m.T0 * C) + cp;
  float2 x[16], dA[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    x[q] = __ldg(xr + q * C2);
    dA[q] = make_float2(0.0f, 0.0f);
  }
  if (m.poly_canon) {  // generated code, registers only
    static_for<NLM>([&](auto lc) {
      constexpr int LM = decltype(lc)::value;
      if constexpr (SPLIT) {
        if (LM == part) contract_grad<LM>(x, __ldg(w + LM * C2), cf + LM * sst, C2, dA);
      } else {
        float2 g[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) g[q] = make_float2(0.0f, 0.0f);
        contract_grad<LM>(x, __ldg(w + LM * C2), cf + LM * sst, C2, g);
#pragma unroll
        for (int q = 0; q < 16; ++q) dA[q] = LM == 0 ? g[q] : __fadd2_rn(dA[q], g[q]);
      }
    });
  } else {  // data-driven monomial lists, this lane's columns in shared memory
    float2* sA = reinterpret_cast<float2*>(dyn) + warp * 17 * 32 * 2 + lane;  // [17][32]
    float2* sG = sA + 17 * 32;                                               // (row 16 absorbs the constant slot)
#pragma unroll
    for (int q = 0; q < 17; ++q) sA[q * 32] = q < 16 ? x[q < 16 ? q : 0] : make_float2(1.0f, 1.0f);
    for (int LM = part; LM < m.nLM; LM += parts) {
#pragma unroll
      for (int q = 0; q < 17; ++q) sG[q * 32] = make_float2(0.0f, 0.0f);
      const float2 wl = __ldg(w + LM * C2);
      const int t0 = m.mono0_off[LM], t1 = m.mono0_off[LM + 1];
      for (int t = t0; t < t1; ++t) {
        const int pk = __ldg(m.mono0 + t);
        const int a = (pk & 255) * 32, b = ((pk >> 8) & 255) * 32, c = (pk >> 16) * 32;
        const float2 cw = mul2(__ldg(cf + LM * sst + static_cast<size_t>(t - t0) * C2), wl);
        const float2 xa = sA[a], xb = sA[b], xc = sA[c];
        sG[a] = fma2(mul2(cw, xb), xc, sG[a]);
        sG[b] = fma2(mul2(cw, xa), xc, sG[b]);
        sG[c] = fma2(mul2(cw, xa), xb, sG[c]);
      }
#pragma unroll
      for (int q = 0; q < 16; ++q) dA[q] = LM == part ? sG[q * 32] : __fadd2_rn(dA[q], sG[q * 32]);
    }
  }
  float2* out = reinterpret_cast<float2*>(A0_adj + static_cast<size_t>(i) * 16 * C) + cp;
  float S = 1.0f;  // reverse_A0_scaled (mace.cpp:299-346): c_i = dA . A0 / s_i, dA /= s_i
  auto density = [&](float2 d2) {
    const float dot = block_sum(live ? d2.x + d2.y : 0.0f);
    S = m.dens_s[0][i];
    if (threadIdx.x == 0) m.dens_c[0][i] = dot / S;
  };
  auto store = [&](int q, float2 v) {
    if (m.dens_spl[0]) v = make_float2(v.x / S, v.y / S);
    if (live) out[q * C2] = v;
  };
  float2 d2 = make_float2(0.0f, 0.0f);
  if constexpr (!SPLIT) {
    if (m.dens_spl[0]) {
#pragma unroll
      for (int q = 0; q < 16; ++q) d2 = fma2(dA[q], x[q], d2);
      density(d2);
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) store(q, dA[q]);
  } else {
    // [nwarp][16][32], behind the data-driven columns
    float2* sum = reinterpret_cast<float2*>(dyn) + (m.poly_canon ? 0 : nwarp * 17 * 32 * 2) + lane;
#pragma unroll
    for (int q = 0; q < 16; ++q) sum[(warp * 16 + q) * 32] = dA[q];
    __syncthreads();
    auto row = [&](int q) {  // warp (LM, slice) takes the rows q = LM (mod nLM) of its slice
      float2 s = sum[(slice * 16 + q) * 32];
      for (int u = 1; u < parts; ++u) s = __fadd2_rn(s, sum[((u * ns + slice) * 16 + q) * 32]);
      return s;
    };
    if (m.dens_spl[0]) {  // by the warps of output 0, in the order of the other form
      if (part == 0)
#pragma unroll
        for (int q = 0; q < 16; ++q) d2 = fma2(row(q), x[q], d2);
      density(d2);
    }
    for (int q = part; q < 16; q += parts) store(q, row(q));
  }
}

// ---------------------------------------------------------------------------
// Layer-0 edge adjoint (mace.cpp:203-271): dE/dx_ij from A0_adj through the folded
// radial splines and Y_lm; ZBL and the density factors add their terms; forces =
// -(layer 0 + layer 1).  A warp sums all channels of its node's edges, up to two channel
// pairs per lane at a time: dE/dY_lm and the radial term over the lanes four edges at a
// time, and only these sums meet dY_lm/dx.  Lanes sum in float32 up to 64 channels (with two
// pairs per lane, each half of the warp has 64), whose forces are added in float64.
// ---------------------------------------------------------------------------
namespace {

struct Rev0Smem {
  L0Stage st;
  float2 buf[kSumEdges * 8 * kSumRow];
};

}  // namespace

template <int CT>
__device__ __forceinline__ void layer0_rev_item(const DevModel& m, const EdgeIn& in, const float* __restrict__ A0_adj,
                                                const float* __restrict__ f1, double* __restrict__ forces,
                                                Rev0Smem& s, int i, int part, int split, int cs) {
  constexpr int NP = CT > 0 && CT <= 64 ? 1 : 2;  // channel pairs per lane
  const int C = CT > 0 ? CT : m.C, C2 = C >> 1;
  const int lane = threadIdx.x & 31;
  const int ti = in.node_type[i];
  const int e0 = in.first[i], e1 = in.end(i);
  if (e0 + part * cs >= e1) return;
  const bool local = i < in.n_local;  // a halo centre: layer 0 only
  LaneEdge ed;
  ed.load(m, in, min(e0 + part * cs + lane, e1 - 1));
  // the lane's pairs of a channel block: cb + lane, or cb + l, cb + l + 16 (l = lane in the first half
  // of the warp, lane + 16 in the second); zero adjoints past the last
  float2 dA[NP][16];
  int cp[NP];
  auto load_dA = [&](int cb) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const int c = cb + lane + (NP == 2 ? (lane & 16) + 16 * p : 0);
      cp[p] = c < C2 ? c : 0;
      const float2* a = reinterpret_cast<const float2*>(A0_adj + static_cast<size_t>(i) * 16 * C) + cp[p];
#pragma unroll
      for (int q = 0; q < 16; ++q) dA[p][q] = c < C2 ? __ldg(a + q * C2) : make_float2(0.0f, 0.0f);
    }
  };
  load_dA(0);
  for (int eb = e0 + part * cs; eb < e1; eb += split * cs) {
    const int ne = min(cs, e1 - eb);
    const long e = static_cast<long>(eb) + lane;
    if (eb > e0 + part * cs) ed.load(m, in, min(eb + lane, e1 - 1));
    const bool active = lane < ne && ed.r < m.r_cut;
    int na;
    const int pos = stage_rows0(m, s.st, ed, ti, active, na);
    double f[3] = {0.0, 0.0, 0.0};  // of this lane's edge
    for (int cb = 0; cb < C2 && na > 0; cb += 32 * NP) {
      if (C2 > 32 * NP) load_dA(cb);
      float4 c[NP][8];
      {
        const float4* r = m.spl0 + static_cast<size_t>(s.st.meta[0].y) * 4 * C;
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
          for (int q = 0; q < 8; ++q) c[p][q] = __ldg(r + q * C2 + cp[p]);
      }
      if (cb > 0) __syncwarp();  // (the last block's sums have been read)
      stage_Y0(s.st, ed, active, pos);
      for (int a = 0; a < na; ++a) {
        const float4* r = m.spl0 + static_cast<size_t>(s.st.meta[min(a + 1, na - 1)].y) * 4 * C;
        const float x = __int_as_float(s.st.meta[a].x);
        const float2 x2 = make_float2(x, x);
        float2 y[16], dY[16], dr = make_float2(0.0f, 0.0f);
        read_Y2(s.st.Y2[a], y);
        static_for<4>([&](auto lc) {
          constexpr int l = decltype(lc)::value;
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            float2 R, Rd;
            spline2(c[p][2 * l], c[p][2 * l + 1], x2, R, Rd);
            c[p][2 * l] = __ldg(r + 2 * l * C2 + cp[p]);
            c[p][2 * l + 1] = __ldg(r + (2 * l + 1) * C2 + cp[p]);
            float2 dR;
            if constexpr (l == 0) {  // Y_00 = 1 with a zero gradient (sph_harm16): the R_0' term alone
              dR = dA[p][0];
            } else {
#pragma unroll
              for (int q = l * l; q < (l + 1) * (l + 1); ++q) {
                dR = q == l * l ? mul2(dA[p][q], y[q]) : fma2(dA[p][q], y[q], dR);
                dY[q] = p == 0 ? mul2(dA[p][q], R) : fma2(dA[p][q], R, dY[q]);
              }
            }
            dr = l == 0 && p == 0 ? mul2(dR, Rd) : fma2(dR, Rd, dr);
          }
        });
        float2* t = s.buf + (a % kSumEdges) * 8 * kSumRow + lane;
        t[0] = make_float2(dr.x + dr.y, dY[1].x + dY[1].y);
#pragma unroll
        for (int v = 1; v < 8; ++v)
          t[kSumRow * v] = make_float2(dY[2 * v].x + dY[2 * v].y, dY[2 * v + 1].x + dY[2 * v + 1].y);
        if (a % kSumEdges == kSumEdges - 1 || a == na - 1)
          sum_lanes<NP == 2, 2 * kRow0>(s.buf, &s.st.Y2[a - a % kSumEdges][0].x, a % kSumEdges + 1);
      }
      if (active) {
        float Y[16], D[48];
        sph_harm16<true>(ed.vx, ed.vy, ed.vz, Y, D);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          float S[16];  // (dE/dr term, dE/dY_1 .. dE/dY_15)
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const float4 w = *reinterpret_cast<const float4*>(&s.st.Y2[pos][8 * p + 2 * v]);
            S[4 * v] = w.x;
            S[4 * v + 1] = w.y;
            S[4 * v + 2] = w.z;
            S[4 * v + 3] = w.w;
          }
          const float d = __fdiv_rn(S[0], ed.r);
          float fx = __fmul_rn(d, ed.vx), fy = __fmul_rn(d, ed.vy), fz = __fmul_rn(d, ed.vz);
#pragma unroll
          for (int q = 1; q < 16; ++q) {
            fx = fmaf(S[q], D[q], fx);
            fy = fmaf(S[q], D[16 + q], fy);
            fz = fmaf(S[q], D[32 + q], fz);
          }
          f[0] += fx;
          f[1] += fy;
          f[2] += fz;
        }
      }
    }
    if (lane < ne) {  // this lane's edge
      if (m.has_zbl && local) {  // node_forces -= xyz / r * dV_ZBL/dr (zbl.cpp:118-121)
        float V, dV;
        const double r = in.r[e];
        zbl_edge(m, m.zbl_pair[ti * m.S + ed.tj], static_cast<float>(r), V, dV);
        for (int a = 0; a < 3; ++a) f[a] = fma(in.xyz[3 * e + a] / r, static_cast<double>(dV), f[a]);
      }
      for (int layer = 0; layer < 2; ++layer) {  // through the density factors (mace.cpp:334-339, :744-749)
        if (!m.dens_spl[layer] || (layer == 1 && !local)) continue;
        float v, d;
        const double r = in.r[e];
        dens_eval(m, layer, ti, ed.tj, static_cast<float>(r), v, d);
        const double g = static_cast<double>(m.dens_c[layer][i]) * static_cast<double>(d) / r;
        for (int a = 0; a < 3; ++a) f[a] = fma(-g, in.xyz[3 * e + a], f[a]);
      }
      for (int a = 0; a < 3; ++a) {
        const double w = local ? f1_sum(f1, m.f1_stride, C >> 5, m.f1_width, 3 * e + a) : 0.0;
        forces[3 * e + a] = -(f[a] + w);
      }
    }
  }
}

template <int CT, bool P>
__global__ void __launch_bounds__(32, 12) k_layer0_rev(DevModel m, EdgeIn in, const float* __restrict__ A0_adj,
                                                       const float* __restrict__ f1, double* __restrict__ forces,
                                                       int split, int cs) {
  pdl_begin();
  __shared__ Rev0Smem s;
  const int n = in.N * split;
  AtomCursor cur{P ? m.sched : nullptr, n, 0};
  for (int b = cur.first(); b < n; b = cur.next())
    layer0_rev_item<CT>(m, in, A0_adj, f1, forces, s, in.atom_at(b / split), b % split, split, cs);
  cur.done();
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
namespace {

// warps of the contraction adjoint's block
int contract0_warps(const DevModel& m, bool split) { return (split ? m.nLM : 1) * layer0_slices(m.C); }
// A warp per output while the (node, 64 channels) warps are fewer than this (us, one : a warp
// per output: 300 nodes of L_max = 2 and 128 channels 77 : 21, 999 of 64 channels 34 : 16,
// 2197 of L_max = 2 and 128 channels 65 : 103, 4096 of 128 channels 71 : 76)
constexpr long kContractWarps = 3000;
bool contract0_split(const DevModel& m, long n) { return n * layer0_slices(m.C) < kContractWarps; }

// f(outputs, C): the kernels with generated polynomials, 9 (L_max = 2) or 4 (L_max = 1) outputs
// and the channel counts compiled in (0: any)
template <typename F>
void dispatch_poly(const DevModel& m, F&& f) {
  if (m.nLM == 9) {
    constexpr std::integral_constant<int, 9> n{};
    m.C == 128 ? f(n, std::integral_constant<int, 128>{}) : f(n, std::integral_constant<int, 0>{});
    return;
  }
  constexpr std::integral_constant<int, 4> n{};
  switch (m.C) {
    case 64: f(n, std::integral_constant<int, 64>{}); break;
    case 128: f(n, std::integral_constant<int, 128>{}); break;
    default: f(n, std::integral_constant<int, 0>{}); break;
  }
}
template <typename F>
void dispatch_c0(int C, F&& f) {
  switch (C) {
    case 32: f(std::integral_constant<int, 32>{}); break;
    case 64: f(std::integral_constant<int, 64>{}); break;
    case 128: f(std::integral_constant<int, 128>{}); break;
    default: f(std::integral_constant<int, 0>{}); break;
  }
}

size_t fwd0_smem(const DevModel& m) { return m.poly_canon ? 0 : 17 * 32 * sizeof(float2); }
size_t contract0_smem(int warps, bool split, bool canon) {
  return warps * ((split ? 16 : 0) + (canon ? 0 : 2 * 17)) * 32 * sizeof(float2);
}
size_t contract0_smem(const DevModel& m, bool split) {
  return contract0_smem(contract0_warps(m, split), split, m.poly_canon != 0);
}

}  // namespace

// Dynamic shared memory above 48 KB must be opted into once per kernel (outside any stream
// capture).  The limit belongs to the function, which serves every engine of the process, so
// it is the most that any model of the instantiation needs (data-driven polynomials of its
// widest block: 204,800 bytes for 4 outputs of 256 channels, 230,400 for 9 of 128): set by
// each engine's own need, a later engine's would narrow an earlier one's.
cudaError_t init_edge_kernels(const DevModel& m) {
  cudaError_t e = init_layer1_kernels(m);
  dispatch_poly(m, [&](auto nc, auto cc) {
    constexpr int NLM = decltype(nc)::value, CT = decltype(cc)::value;
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_contract0_rev<NLM, CT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(contract0_smem(contract0_max_warps(NLM, CT, true), true, false)));
  });
  return e;
}

void launch_layer0_fwd(const DevModel& m, const EdgeIn& in, float* A0, float* M0, float* zbl_e, cudaStream_t s) {
  if (in.N <= 0) return;
  dispatch_poly(m, [&](auto nc, auto cc) {
    launch_pdl(k_layer0_fwd<decltype(nc)::value, decltype(cc)::value>, in.N * layer0_slices(m.C), 32, fwd0_smem(m), s, m,
               in, A0, M0, zbl_e);
  });
}

void launch_layer0_rev(const DevModel& m, const EdgeIn& in, const float* A0, const float* M0_adj, const float* f1,
                       float* A0_adj, double* forces, cudaStream_t s) {
  if (in.N <= 0) return;
  const bool by_lm = contract0_split(m, in.N);
  dispatch_poly(m, [&](auto nc, auto cc) {
    auto go = [&](auto sc) {
      launch_pdl(k_contract0_rev<decltype(nc)::value, decltype(cc)::value, decltype(sc)::value>, in.N,
                 32 * contract0_warps(m, by_lm), contract0_smem(m, by_lm), s, m, in.node_type, in.order, A0, M0_adj, A0_adj);
    };
    by_lm ? go(std::true_type{}) : go(std::false_type{});
  });
  const int split = edge_split(in.N), cs = edge_chunk(split);
  DevModel mk;
  const int grid = atom_grid(m, kAkLayer0Rev, in.N * split, mk);
  dispatch_c0(m.C, [&](auto cc) {
    constexpr int CT = decltype(cc)::value;
    if (mk.sched)
      launch_pdl(k_layer0_rev<CT, true>, grid, 32, 0, s, mk, in, A0_adj, f1, forces, split, cs);
    else
      launch_pdl(k_layer0_rev<CT, false>, grid, 32, 0, s, mk, in, A0_adj, f1, forces, split, cs);
  });
}

// resident blocks per SM of the layer-0 kernels at this model's launch shapes
void layer0_residency(const DevModel& m, int* per_sm) {
  dispatch_poly(m, [&](auto nc, auto cc) {
    constexpr int NLM = decltype(nc)::value, CT = decltype(cc)::value;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[kAkLayer0Fwd], k_layer0_fwd<NLM, CT>, 32, fwd0_smem(m));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[kAkContract0Rev], k_contract0_rev<NLM, CT, false>,
                                                  32 * contract0_warps(m, false), contract0_smem(m, false));
  });
  dispatch_c0(m.C, [&](auto cc) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[kAkLayer0Rev], k_layer0_rev<decltype(cc)::value, true>, 32, 0);
  });
}

}  // namespace smx
