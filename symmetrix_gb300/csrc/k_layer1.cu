// Layer-1 forward: the tensor-product neighbour sum, compute_R1 + compute_Phi1
// (libsymmetrix/source/mace.cpp:92-116, :453-502).  Its adjoint is in k_layer1_rev.cu.
//
// Every kernel works on one centre node at a time: one block per node, or a persistent
// grid claiming nodes (AtomCursor), in the order EdgeIn::atom_at gives.
//
// L_max = 2 (17 instructions, 243 paths): four instruction groups, one channel per
// thread, scalar FMAs; from 64 channels each node's channels are split over two blocks
// (DevModel::l2_split) so that two blocks share an SM.
#include <cuda_runtime.h>

#include <algorithm>

#include "device.cuh"
#include "kernels.h"

namespace smx {

namespace {

// number of CG paths (l1 m1, l2 m2) of instruction q
__host__ __device__ constexpr int ins_paths(int LMAX, int q) {
  return (2 * ins_l1(LMAX, q) + 1) * (2 * ins_l2(LMAX, q) + 1);
}

// sum_p CG[lme,p] sP[p][k] over row lme of the padded forward table, KF terms, all loads
// independent
template <int KF>
__device__ __forceinline__ float cg_row(const int2* __restrict__ row, const float* sP, int stride, int k) {
  int2 t[KF];
#pragma unroll
  for (int u = 0; u < KF; ++u) t[u] = __ldg(row + u);
  float s = 0.0f;
#pragma unroll
  for (int u = 0; u < KF; ++u) s = fmaf(__int_as_float(t[u].y), sP[t[u].x * stride + k], s);
  return s;
}

// f(std::integral_constant<int, KF>) for the padded forward table's row length, KF = 0
// for the compressed-row walk (no padded table)
template <typename F>
__device__ __forceinline__ void dispatch_kf(int kp, F&& f) {
  switch (kp) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 7: f(std::integral_constant<int, 7>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    default: f(std::integral_constant<int, 0>{}); break;
  }
}

// Phi1[i,lme,k] = sum_p CG[lme,p] sP[p][k] for the rows lme with (lme mod nrow_groups) ==
// row_group (the BF16 form also writes them as the A1 GEMM's split operand, regrouped per
// l); sP holds this block's channels with row stride `stride`, k is the global channel
template <int KF>
__device__ __forceinline__ void l1_fwd_epilogue(const DevModel& m, int N, int i, const float* sP, int stride, int kk,
                                                int k, int row_group, int nrow_groups, float* __restrict__ Phi1) {
  const int C = m.C, T = m.tc_terms, XT = split_xterms(T);
  for (int l = 0; l < 4; ++l) {
    const int ne = m.num_e[l], Kl = ne * C;
    for (int mm = 0; mm < 2 * l + 1; ++mm)
      for (int e = 0; e < ne; ++e) {
        const int lme = m.lme_off[l] + mm * ne + e;
        if (lme % nrow_groups != row_group) continue;
        float s = 0.0f;
        if constexpr (KF > 0) {
          s = cg_row<KF>(m.cg_fwd_pad + static_cast<size_t>(lme) * KF, sP, stride, kk);
        } else {
          const int p1 = __ldg(m.cg_fwd_off + lme + 1);
          for (int p = __ldg(m.cg_fwd_off + lme); p < p1; ++p)
            s = fmaf(__ldg(m.cg_fwd_v + p), sP[__ldg(m.cg_fwd_p + p) * stride + kk], s);
        }
        if (Phi1) Phi1[(static_cast<size_t>(i) * m.n_lme + lme) * C + k] = s;  // nullptr: split rows only
        if (m.op_phi1) {
          __nv_bfloat16* row = m.op_phi1 + static_cast<size_t>(XT) * N * m.lme_off[l] * C +
                               (static_cast<size_t>(i) * (2 * l + 1) + mm) * XT * Kl;
          write_split(row, Kl, T, e * C + k, s);
        }
      }
  }
}

// Edge chunk staged for the forward kernels.
struct L1Stage {
  float2 Y2[kEdgeChunk][16];            // (Y_lm, Y_lm): operand of the packed FMAs
  float x[kEdgeChunk];                  // offset inside the spline interval
  int row[kEdgeChunk];                  // spline row (pair * nint + interval), or -1
  int j[kEdgeChunk];
  int act[kEdgeChunk];                  // compacted list of active edges (r < r_cut)
  int nact;
};

// Stage edges [eb, eb+ne) (ne <= 32; warp 0) with the unordered species-pair rows.
__device__ __forceinline__ void stage_l1(const DevModel& m, const EdgeIn& in, int ti, int eb, int ne,
                                         L1Stage& st) {
  if (threadIdx.x >= 32) return;
  const int t = threadIdx.x;
  bool active = false;
  if (t < ne) {
    const long e = static_cast<long>(eb) + t;
    const float vx = static_cast<float>(in.xyz[3 * e]);
    const float vy = static_cast<float>(in.xyz[3 * e + 1]);
    const float vz = static_cast<float>(in.xyz[3 * e + 2]);
    const float rr = static_cast<float>(in.r[e]);
    float Y[16];
    sph_harm16<false>(vx, vy, vz, Y, nullptr);
#pragma unroll
    for (int c = 0; c < 16; ++c) st.Y2[t][c] = make_float2(Y[c], Y[c]);
    int iv = static_cast<int>(rr * m.inv_h);
    iv = iv < 0 ? 0 : (iv >= m.nint ? m.nint - 1 : iv);
    st.x[t] = rr - static_cast<float>(iv) * m.h;
    const int tj = in.ntype_e[e];
    const int a = ti < tj ? ti : tj, b = ti < tj ? tj : ti;
    const int pr = a * (2 * m.S - a - 1) / 2 + b;
    active = rr < m.r_cut;
    st.row[t] = active ? pr * m.nint + iv : -1;
    st.j[t] = in.nidx[e];
  }
  const unsigned ball = __ballot_sync(0xffffffffu, active);
  if (active) st.act[__popc(ball & ((1u << t) - 1u))] = t;
  if (t == 0) st.nact = __popc(ball);
}

}  // namespace

// ---------------------------------------------------------------------------
// Layer 1 forward: Phi1r[i,p,k] = sum_j R1_q(r_ij)[k] Y_{l1 m1}(x_ij) H1[j, l2 m2, k]
// accumulated in registers, then Phi1[i,lme,k] = sum_p CG[lme,p] Phi1r[i,p,k].
//
// One thread per channel with scalar FMAs over all instructions, on the per-channel
// spline table spl1_fwd ([npairs][nint][n_instr][C] float4).  The forward pass moves
// the same 20 KB spline row per edge as the adjoint but does a third of its
// arithmetic, so it is bound by the L2 gathers: it is laid out for residency (128
// registers, four blocks of 128 threads per SM) rather than for the packed FMAs.
// ---------------------------------------------------------------------------
template <int LMAX, int CT>
__device__ __forceinline__ void layer1_fwd_atom(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                                float* __restrict__ Phi1, int i) {
  constexpr int NL2 = (LMAX + 1) * (LMAX + 1);
  constexpr int NI = ins_count(LMAX);
  constexpr int NP = ins_np(LMAX);
  extern __shared__ float dyn[];
  __shared__ L1Stage st;
  const int C = CT > 0 ? CT : m.C;
  const int k = threadIdx.x;
  const int ti = in.node_type[i];
  const int e0 = in.first[i], e1 = in.end(i);
  float acc[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) acc[p] = 0.0f;
  for (int eb = e0; eb < e1; eb += kEdgeChunk) {
    const int ne = min(kEdgeChunk, e1 - eb);
    __syncthreads();
    stage_l1(m, in, ti, eb, ne, st);
    __syncthreads();
    const int na = st.nact;
    for (int a = 0; a < na; ++a) {
      const int t = st.act[a];
      const float x = st.x[t];
      float hv[NL2];
      const float* hj = H1 + static_cast<size_t>(st.j[t]) * NL2 * C + k;
#pragma unroll
      for (int b = 0; b < NL2; ++b) hv[b] = __ldg(hj + b * C);
      const float4* cp = m.spl1_fwd + static_cast<size_t>(st.row[t]) * NI * C + k;
      const float2* Y2 = st.Y2[t];
      for_each_ins<LMAX>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        constexpr int l1 = ins_l1(LMAX, q), l2 = ins_l2(LMAX, q), p0 = ins_poff(LMAX, q);
        const float R = spline_val(__ldg(cp + q * C), x);
#pragma unroll
        for (int a1 = 0; a1 < 2 * l1 + 1; ++a1) {
          const float ry = R * Y2[l1 * l1 + a1].x;
#pragma unroll
          for (int b = 0; b < 2 * l2 + 1; ++b)
            acc[p0 + a1 * (2 * l2 + 1) + b] = fmaf(ry, hv[l2 * l2 + b], acc[p0 + a1 * (2 * l2 + 1) + b]);
        }
      });
    }
  }
  if (m.dens_spl[1]) {  // layer-1 density factor for node_tail (mace.cpp:681-705)
    const float S = dens_factor(m, 1, in, i, ti);
    if (threadIdx.x == 0) m.dens_s[1][i] = S;
  }
  float* sP = dyn;  // [NP][C]: this thread's Phi1r column
#pragma unroll
  for (int p = 0; p < NP; ++p) sP[p * C + k] = acc[p];
  // Phi1 rows are [l][m][e] (lme = lme_off[l] + m n_e + e); each thread reads back only its
  // own column of sP
  dispatch_kf(m.cg_fwd_kp, [&](auto kc) {
    l1_fwd_epilogue<decltype(kc)::value>(m, in.N, i, sP, C, k, k, 0, 1, Phi1);
  });
}

template <int LMAX, int CT, bool P>
__global__ void __launch_bounds__(256) k_layer1_fwd(DevModel m, EdgeIn in, const float* __restrict__ H1,
                                                    float* __restrict__ Phi1) {
  pdl_begin();
  AtomCursor cur{P ? m.sched : nullptr, in.N, 0};
  for (int b = cur.first(); b < in.N; b = cur.next())
    layer1_fwd_atom<LMAX, CT>(m, in, H1, Phi1, in.atom_at(b));
  cur.done();
}

// ===========================================================================
// L_max = 2 (hidden irreps up to 2e: 17 instructions, 243 CG paths).  The paths do not
// fit one thread's registers, so the instructions are split over four thread groups
// per channel ({11,13,15,16}, {1,4,5,8,12}, {0,2,6,10}, {3,7,9,14}: exhaustive local
// search for equal scalar work, 202/201/196/202 FMAs per edge, and 62/57/62/62 paths);
// one channel per thread, scalar FMAs.  Block = 4 groups x C threads.
// ===========================================================================
namespace {

constexpr int kL2Groups = 4;
// channels per block of the L_max = 2 layer-1 kernels (a warp multiple)
__host__ __device__ inline int l2_slice_width(const DevModel& m) {
  return ((m.C + m.l2_split - 1) / m.l2_split + 31) & ~31;
}
__host__ __device__ constexpr int l2_count(int g) { return g == 1 ? 5 : 4; }
__host__ __device__ constexpr int l2_ins(int g, int i) {
  constexpr int t0[4] = {11, 13, 15, 16}, t1[5] = {1, 4, 5, 8, 12}, t2[4] = {0, 2, 6, 10}, t3[4] = {3, 7, 9, 14};
  return g == 0 ? t0[i] : (g == 1 ? t1[i] : (g == 2 ? t2[i] : t3[i]));
}
template <int G>
__host__ __device__ constexpr int l2_goff(int i) {
  int s = 0;
  for (int w = 0; w < i; ++w) s += ins_paths(2, l2_ins(G, w));
  return s;
}
template <int G>
__host__ __device__ constexpr int l2_np() {
  return l2_goff<G>(l2_count(G));
}
constexpr int kL2MaxNp = 62;

// Forward, group G, one staged chunk: acc[local path] += R_q Y_{l1 m1} H1[j, l2 m2, k].
template <int G>
__device__ __forceinline__ void l2_fwd_chunk(const DevModel& m, const float* __restrict__ H1,
                                             const L1Stage& st, int C, int k, float* acc) {
  constexpr int NL2 = 9, NI = 17;
  const int na = st.nact;
  for (int a = 0; a < na; ++a) {
    const int t = st.act[a];
    const float x = st.x[t];
    float hv[NL2];
    const float* hj = H1 + static_cast<size_t>(st.j[t]) * NL2 * C + k;
#pragma unroll
    for (int b = 0; b < NL2; ++b) hv[b] = __ldg(hj + b * C);
    const float4* cp = m.spl1_fwd + static_cast<size_t>(st.row[t]) * NI * C + k;
    static_for<l2_count(G)>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      constexpr int q = l2_ins(G, i);
      constexpr int l1 = ins_l1(2, q), l2 = ins_l2(2, q), g0 = l2_goff<G>(i);
      const float R = spline_val(__ldg(cp + q * C), x);
#pragma unroll
      for (int a1 = 0; a1 < 2 * l1 + 1; ++a1) {
        const float ry = R * st.Y2[t][l1 * l1 + a1].x;
#pragma unroll
        for (int b = 0; b < 2 * l2 + 1; ++b)
          acc[g0 + a1 * (2 * l2 + 1) + b] = fmaf(ry, hv[l2 * l2 + b], acc[g0 + a1 * (2 * l2 + 1) + b]);
      }
    });
  }
}

template <int G>
__device__ __forceinline__ void l2_store(float* sP, int C, int k, const float* acc) {
  static_for<l2_count(G)>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr int q = l2_ins(G, i);
    constexpr int np = ins_paths(2, q), p0 = ins_poff(2, q), g0 = l2_goff<G>(i);
#pragma unroll
    for (int p = 0; p < np; ++p) sP[(p0 + p) * C + k] = acc[g0 + p];
  });
}

}  // namespace

// Layer-1 forward, L_max = 2: slice h of the channels of node i (channels h*CH ..
// h*CH + CH - 1, CH = l2_slice_width(m)); four groups of CH threads, group G running the
// instructions of group G.
__device__ __forceinline__ void layer1_fwd_l2_atom(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                                   float* __restrict__ Phi1, int i, int h) {
  extern __shared__ float dyn[];
  __shared__ L1Stage st;
  const int C = m.C, CH = l2_slice_width(m);
  const int grp = threadIdx.x / CH, kk = threadIdx.x - grp * CH;
  const bool live = kk < CH && h * CH + kk < C;
  const int k = live ? h * CH + kk : 0;
  const int ti = in.node_type[i];
  const int e0 = in.first[i], e1 = in.end(i);
  float acc[kL2MaxNp];
#pragma unroll
  for (int p = 0; p < kL2MaxNp; ++p) acc[p] = 0.0f;
  for (int eb = e0; eb < e1; eb += kEdgeChunk) {
    const int ne = min(kEdgeChunk, e1 - eb);
    __syncthreads();
    stage_l1(m, in, ti, eb, ne, st);
    __syncthreads();
    switch (grp) {
      case 0: l2_fwd_chunk<0>(m, H1, st, C, k, acc); break;
      case 1: l2_fwd_chunk<1>(m, H1, st, C, k, acc); break;
      case 2: l2_fwd_chunk<2>(m, H1, st, C, k, acc); break;
      default: l2_fwd_chunk<3>(m, H1, st, C, k, acc); break;
    }
  }
  if (m.dens_spl[1]) {
    const float S = dens_factor(m, 1, in, i, ti);
    if (threadIdx.x == 0 && h == 0) m.dens_s[1][i] = S;
  }
  float* sP = dyn;  // [NP][CH]: Phi1r of the slice
  if (live) {
    switch (grp) {
      case 0: l2_store<0>(sP, CH, kk, acc); break;
      case 1: l2_store<1>(sP, CH, kk, acc); break;
      case 2: l2_store<2>(sP, CH, kk, acc); break;
      default: l2_store<3>(sP, CH, kk, acc); break;
    }
  }
  __syncthreads();
  // Phi1 rows of the slice, group G taking the rows lme = G (mod 4)
  if (!live) return;
  dispatch_kf(m.cg_fwd_kp, [&](auto kc) {
    l1_fwd_epilogue<decltype(kc)::value>(m, in.N, i, sP, CH, kk, k, grp, kL2Groups, Phi1);
  });
}

// work item b = (atom, channel slice); the return in the atom body above happens after
// its last barrier
template <bool P>
__global__ void __launch_bounds__(512, 1) k_layer1_fwd_l2(DevModel m, EdgeIn in, const float* __restrict__ H1,
                                                          float* __restrict__ Phi1) {
  pdl_begin();
  const int ns = m.l2_split, n = in.N * ns;
  AtomCursor cur{P ? m.sched : nullptr, n, 0};
  for (int b = cur.first(); b < n; b = cur.next()) layer1_fwd_l2_atom(m, in, H1, Phi1, in.atom_at(b / ns), b % ns);
  cur.done();
}

namespace {

template <int CT, bool P>
cudaError_t set_smem(const DevModel& m) {
  return cudaFuncSetAttribute(k_layer1_fwd<1, CT, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(sizeof(float) * ins_np(1) * m.C));
}

template <bool P>
cudaError_t set_smem_l2(const DevModel& m) {
  return cudaFuncSetAttribute(k_layer1_fwd_l2<P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(sizeof(float) * ins_np(2) * m.C));
}

// Channel counts with a compile-time specialisation (addresses fold to immediates).
template <typename F>
void dispatch_c(int C, F&& f) {
  switch (C) {
    case 32: f(std::integral_constant<int, 32>{}); break;
    case 64: f(std::integral_constant<int, 64>{}); break;
    case 128: f(std::integral_constant<int, 128>{}); break;
    case 256: f(std::integral_constant<int, 256>{}); break;
    default: f(std::integral_constant<int, 0>{}); break;
  }
}

// the one-block-per-atom (false) or persistent (true) instantiation
template <typename F>
void dispatch_p(bool persistent, F&& f) {
  if (persistent)
    f(std::true_type{});
  else
    f(std::false_type{});
}

}  // namespace

cudaError_t init_layer1_kernels(const DevModel& m) {
  cudaError_t e = cudaSuccess;
  for (bool p : {false, true}) {
    if (m.L_max == 2)
      dispatch_p(p, [&](auto pc) { e = set_smem_l2<decltype(pc)::value>(m); });
    else
      dispatch_c(m.C, [&](auto ct) {
        dispatch_p(p, [&](auto pc) { e = set_smem<decltype(ct)::value, decltype(pc)::value>(m); });
      });
    if (e != cudaSuccess) return e;
  }
  return e;
}

void launch_layer1_fwd(const DevModel& m, const EdgeIn& in, const float* H1, float* Phi1, cudaStream_t s) {
  if (in.N <= 0) return;
  DevModel mk;
  const int grid = atom_grid(m, kAkLayer1Fwd, m.L_max == 2 ? in.N * m.l2_split : in.N, mk);
  dispatch_p(mk.sched != nullptr, [&](auto pc) {
    constexpr bool P = decltype(pc)::value;
    if (m.L_max == 2) {
      launch_pdl(k_layer1_fwd_l2<P>, grid, kL2Groups * l2_slice_width(m),
                 sizeof(float) * ins_np(2) * l2_slice_width(m), s, mk, in, H1, Phi1);
      return;
    }
    const size_t smem = sizeof(float) * ins_np(1) * m.C;
    dispatch_c(m.C, [&](auto ct) {
      launch_pdl(k_layer1_fwd<1, decltype(ct)::value, P>, grid, m.C, smem, s, mk, in, H1, Phi1);
    });
  });
}

// resident blocks per SM of the persistent layer-1 kernels at this model's launch shapes
void layer1_residency(const DevModel& m, int* per_sm) {
  int f = 0;
  if (m.L_max == 2)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f, k_layer1_fwd_l2<true>, kL2Groups * l2_slice_width(m),
                                                  sizeof(float) * ins_np(2) * l2_slice_width(m));
  else
    dispatch_c(m.C, [&](auto ct) {
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f, k_layer1_fwd<1, decltype(ct)::value, true>, m.C,
                                                    sizeof(float) * ins_np(1) * m.C);
    });
  per_sm[kAkLayer1Fwd] = f;
  per_sm[kAkLayer1Rev] = layer1_rev_residency(m);
}

}  // namespace smx
