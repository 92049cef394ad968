// Layer-1 forward: the tensor-product neighbour sum, compute_R1 + compute_Phi1
// (libsymmetrix/source/mace.cpp:92-116, :453-502):
//   Phi1r[i,p,k] = sum_j Y_{l1 m1}(x_ij) (R1_q(r_ij)[k] H1[j, l2 m2, k]),  p = (q, m1, m2)
//   Phi1[i,lme,k] = sum_p CG[lme,p] Phi1r[i,p,k]
// Its adjoint is in k_layer1_rev.cu.
//
// One warp per (centre node, 32 channels, instruction group): the lane sums the group's paths
// of its channel in registers, the next edge's cubics replacing this edge's instruction by
// instruction, so that DEPTH whole edges (5 KB each per warp at L_max = 1) are always in
// flight.  The sums run over a node's edges in list order whatever the system around it: a
// molecule in a batch gives the bits that it gives alone.
//
// What bounds it: the L2 gather of the spline rows, 20 KB per edge at L_max = 1 and 128
// channels, which a plain gather kernel of as many rows runs at 21.9 TB/s (0.20 ms for 213k
// edges).  One block of C threads per node, no prefetch, all paths and a table walk for the
// Clebsch-Gordan rows took 0.373 ms on the 4096-atom box (213k edges), this form 0.250 ms;
// L_max = 2, 2197 atoms, 178k edges 0.816 -> 0.435 ms; 64 atoms of 32 channels 37 -> 14.5 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "layer1.cuh"

namespace smx {

namespace {

// sum_p CG[lme,p] sP[p][lane] over row lme of the padded table, KF terms, all loads independent
template <int KF>
__device__ __forceinline__ float cg_row(const int2* __restrict__ row, const float* sP, int lane) {
  int2 t[KF];
#pragma unroll
  for (int u = 0; u < KF; ++u) t[u] = __ldg(row + u);
  float s = 0.0f;
#pragma unroll
  for (int u = 0; u < KF; ++u) s = fmaf(__int_as_float(t[u].y), sP[t[u].x * 32 + lane], s);
  return s;
}

// f(std::integral_constant<int, KF>) for the padded table's row length, KF = 0 for the
// compressed-row walk (no padded table)
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

constexpr int kRowsAhead = 4;  // rows whose table and column loads are in flight together

// Phi1[i,lme,k] for the rows lme = warp (mod nwarp) (the BF16 form also writes them as the A1
// GEMM's split operand, regrouped per l); sP [NP][32] holds this block's channels
template <int KF>
__device__ __forceinline__ void fwd_rows(const DevModel& m, int C, int N, int i, const float* sP, int lane, int k,
                                         int warp, int nwarp, float* __restrict__ Phi1) {
  const int T = m.tc_terms, XT = split_xterms(T);
  for (int l = 0; l < 4; ++l) {
    const int ne = m.num_e[l], Kl = ne * C;
    const int rows = (2 * l + 1) * ne;
    const unsigned inv = ne > 0 ? 65536u / ne + 1 : 0;  // q / ne = q inv >> 16 for q < 64
    for (int q0 = warp; q0 < rows; q0 += kRowsAhead * nwarp) {
      float s[kRowsAhead];
#pragma unroll
      for (int u = 0; u < kRowsAhead; ++u) {  // (rows past the end: the last one again)
        const int lme = m.lme_off[l] + min(q0 + u * nwarp, rows - 1);
        s[u] = 0.0f;
        if constexpr (KF > 0) {
          s[u] = cg_row<KF>(m.cg_fwd_pad + static_cast<size_t>(lme) * KF, sP, lane);
        } else {
          const int p1 = __ldg(m.cg_fwd_off + lme + 1);
          for (int p = __ldg(m.cg_fwd_off + lme); p < p1; ++p)
            s[u] = fmaf(__ldg(m.cg_fwd_v + p), sP[__ldg(m.cg_fwd_p + p) * 32 + lane], s[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < kRowsAhead; ++u) {
        const int q = q0 + u * nwarp;
        if (q >= rows) break;
        if (Phi1)  // nullptr: split rows only
          Phi1[(static_cast<size_t>(i) * m.n_lme + m.lme_off[l] + q) * C + k] = s[u];
        if (m.op_phi1) {
          const int mm = static_cast<int>(q * inv >> 16), e = q - mm * ne;
          __nv_bfloat16* row = m.op_phi1 + static_cast<size_t>(XT) * N * m.lme_off[l] * C +
                               (static_cast<size_t>(i) * (2 * l + 1) + mm) * XT * Kl;
          write_split(row, Kl, T, e * C + k, s[u]);
        }
      }
    }
  }
}

// Group G of node i: its path sums
template <int LMAX, int G, int CT, bool CANON, int DEPTH>
__device__ __forceinline__ void fwd_sums(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                         EdgeStage& st, float* acc, int i, int k) {
  constexpr int NI = ins_count(LMAX), NL2 = (LMAX + 1) * (LMAX + 1);
  constexpr int NQ = grp_count(G), NP = grp_off<LMAX, G, CANON>(NQ), NR = grp_rows(G), r0 = grp_row0(G);
  const int C = CT > 0 ? CT : m.C;
  const int lane = threadIdx.x & 31;
  const int ti = in.node_type[i];
  const int e0 = in.first[i], e1 = in.end(i);
#pragma unroll
  for (int p = 0; p < NP; ++p) acc[p] = 0.0f;
  for (int eb = e0; eb < e1; eb += kEdgeChunk) {
    LaneEdge ed;
    ed.load(m, in, min(eb + lane, e1 - 1));
    int na;
    const bool active = eb + lane < e1 && ed.r < m.r_cut;
    const int pos = stage_rows(m, st, ed, ti, active, na);
    if (na == 0) continue;
    float4 c[DEPTH][NQ];
    float h[DEPTH][NR];
    static_for<DEPTH>([&](auto dc) {
      constexpr int d = decltype(dc)::value;
      const int4 mt = st.meta[min(d, na - 1)];
      const float4* cp = m.spl1 + (static_cast<size_t>(mt.y) * NI + grp_slot(G)) * C + k;
#pragma unroll
      for (int w = 0; w < NQ; ++w) c[d][w] = __ldg(cp + w * C);
      const float* hp = H1 + (static_cast<size_t>(mt.z) * NL2 + r0) * C + k;
#pragma unroll
      for (int b = 0; b < NR; ++b) h[d][b] = __ldg(hp + b * C);
    });
    stage_Y(st, ed, active, pos);
    for (int a0 = 0; a0 < na; a0 += DEPTH) {
      static_for<DEPTH>([&](auto dc) {
        constexpr int d = decltype(dc)::value;
        const int a = a0 + d;
        if (a >= na) return;
        const int4 mn = st.meta[min(a + DEPTH, na - 1)];
        const float4* cn = m.spl1 + (static_cast<size_t>(mn.y) * NI + grp_slot(G)) * C + k;
        const float* hp = H1 + (static_cast<size_t>(mn.z) * NL2 + r0) * C + k;
        const float x = __int_as_float(st.meta[a].x);
        float hv[NR], y[16];
#pragma unroll
        for (int b = 0; b < NR; ++b) {
          hv[b] = h[d][b];
          h[d][b] = __ldg(hp + b * C);
        }
        read_Y(st.Y[a], y);
        float2 R2 = make_float2(0.0f, 0.0f);
        static_for<NQ>([&](auto ic) {
          constexpr int w = decltype(ic)::value;
          constexpr int q = grp_ins(LMAX, G, w);
          constexpr int l1 = ins_l1(LMAX, q), l2 = ins_l2(LMAX, q), nb = 2 * l2 + 1;
          float R;
          if constexpr (w % 2 == 0 && w + 1 < NQ) {  // the pair's values at once
            R2 = spline2_val(c[d][w], c[d][w + 1], make_float2(x, x));
            c[d][w] = __ldg(cn + w * C);
            c[d][w + 1] = __ldg(cn + (w + 1) * C);
            R = R2.x;
          } else if constexpr (w % 2 == 1) {
            R = R2.y;
          } else {
            R = spline_val(c[d][w], x);
            c[d][w] = __ldg(cn + w * C);
          }
          float rh[nb];
#pragma unroll
          for (int b = 0; b < nb; ++b) rh[b] = R * hv[l2 * l2 - r0 + b];
          for_paths<LMAX, G, CANON, w>([&](auto ac, auto bc, auto pc) {
            constexpr int v = decltype(ac)::value, b = decltype(bc)::value, p = decltype(pc)::value;
            if constexpr (l1 == 0)  // Y_00 = 1
              acc[p] = fmaf(R, hv[l2 * l2 - r0 + b], acc[p]);
            else
              acc[p] = fmaf(rh[b], y[l1 * l1 + v], acc[p]);
          });
        });
      });
    }
  }
}

// General tables: the path sums of group G into sP ([NP of all groups][32])
template <int LMAX, int G, int CT>
__device__ __forceinline__ void fwd_group(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                          EdgeStage& st, float* sP, int i, int k) {
  float acc[grp_off<LMAX, G, false>(grp_count(G))];
  fwd_sums<LMAX, G, CT, false, 1>(m, in, H1, st, acc, i, k);
  static_for<grp_count(G)>([&](auto ic) {
    constexpr int w = decltype(ic)::value;
    constexpr int q = grp_ins(LMAX, G, w), p0 = ins_poff(LMAX, q), g0 = grp_off<LMAX, G, false>(w);
#pragma unroll
    for (int p = 0; p < ins_paths(LMAX, q); ++p) sP[(p0 + p) * 32 + (threadIdx.x & 31)] = acc[g0 + p];
  });
}

__device__ __forceinline__ void fwd_density(const DevModel& m, const EdgeIn& in, int i) {
  const float S = dens_factor(m, 1, in, i, in.node_type[i]);  // for node_tail (mace.cpp:681-705)
  if (threadIdx.x == 0) m.dens_s[1][i] = S;
}

// Canonical tables: the rows of the group's instructions straight from its path sums
template <int LMAX, int G, int CT, int DEPTH>
__device__ __forceinline__ void fwd_canon(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                          float* __restrict__ Phi1, int i, int slice, EdgeStage& st) {
  constexpr int NQ = grp_count(G), NP = grp_off<LMAX, G, true>(NQ);
  const int C = CT > 0 ? CT : m.C;
  const int k = slice * 32 + (threadIdx.x & 31);
  float acc[NP];
  fwd_sums<LMAX, G, CT, true, DEPTH>(m, in, H1, st, acc, i, k);
  if (m.dens_spl[1] && G == 0 && slice == 0) fwd_density(m, in, i);
  const int T = m.tc_terms, XT = split_xterms(T);
  static_for<NQ>([&](auto ic) {
    constexpr int w = decltype(ic)::value;
    constexpr int q = grp_ins(LMAX, G, w), l = ins_l(LMAX, q), ne = ins_ne(LMAX, l), e = ins_e(LMAX, q);
    constexpr int p0 = ins_poff(LMAX, q), nb = 2 * ins_l2(LMAX, q) + 1;
    float out[2 * l + 1];
#pragma unroll
    for (int v = 0; v < 2 * l + 1; ++v) out[v] = 0.0f;
    for_paths<LMAX, G, true, w>([&](auto ac, auto bc, auto pc) {
      constexpr int p = p0 + decltype(ac)::value * nb + decltype(bc)::value, m0 = cg_m(LMAX, p, 0), m1 = cg_m(LMAX, p, 1);
      const float2 cg = __ldg(m.cg_val + p);
      out[m0] = fmaf(cg.x, acc[decltype(pc)::value], out[m0]);
      if constexpr (m1 >= 0) out[m1] = fmaf(cg.y, acc[decltype(pc)::value], out[m1]);
    });
    if (Phi1) {  // nullptr: split rows only
      float* o = Phi1 + (static_cast<size_t>(i) * l1_rows(LMAX) + ins_row(LMAX, q)) * C + k;
#pragma unroll
      for (int v = 0; v < 2 * l + 1; ++v) o[v * ne * C] = out[v];
    }
    if (m.op_phi1) {  // BF16 form: the A1 GEMM's split operand, rows (node, m) per l
      constexpr int off = ins_row(LMAX, q) - e;
      const int Kl = ne * C;
      __nv_bfloat16* row = m.op_phi1 + static_cast<size_t>(XT) * in.N * off * C +
                           static_cast<size_t>(i) * (2 * l + 1) * XT * Kl;
#pragma unroll
      for (int v = 0; v < 2 * l + 1; ++v) write_split(row + v * XT * Kl, Kl, T, e * C + k, out[v]);
    }
  });
}

// General tables, item (node, 32-channel slice); the block: one warp per group, whose path
// sums meet in shared memory before the Clebsch-Gordan rows
template <int LMAX, int CT>
__device__ __forceinline__ void fwd_general(const DevModel& m, const EdgeIn& in, const float* __restrict__ H1,
                                            float* __restrict__ Phi1, int item, unsigned char* dyn) {
  constexpr int NG = l1_groups(LMAX);
  const int C = CT > 0 ? CT : m.C, ns = C >> 5;
  const int i = in.atom_at(item / ns), slice = item % ns;
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int k = slice * 32 + lane;
  EdgeStage& st = reinterpret_cast<EdgeStage*>(dyn)[grp];
  float* sP = reinterpret_cast<float*>(dyn + NG * sizeof(EdgeStage));  // [NP][32]
  if (grp == 0) fwd_group<LMAX, 0, CT>(m, in, H1, st, sP, i, k);
  if constexpr (LMAX == 2) {
    if (grp == 1) fwd_group<LMAX, 1, CT>(m, in, H1, st, sP, i, k);
    if (grp == 2) fwd_group<LMAX, 2, CT>(m, in, H1, st, sP, i, k);
  }
  if (m.dens_spl[1] && slice == 0) fwd_density(m, in, i);
  __syncthreads();
  dispatch_kf(m.cg_fwd_kp, [&](auto kc) {
    fwd_rows<decltype(kc)::value>(m, C, in.N, i, sP, lane, k, grp, NG, Phi1);
  });
}

}  // namespace

// Blocks: general tables, one per (node, slice) with the groups' warps in it; canonical ones,
// one warp per (node, slice, group).  DEPTH 1: 168 registers, 12 warps per SM; DEPTH 2: 8.
// (Asked for 11, DEPTH 1 keeps the 12 and its loads are ordered better, ms, 11 : 12: 213k edges
// 0.250 : 0.252, L_max 2, 178k edges 0.435 : 0.440; for 13, 0.352 and 0.497.)
__host__ __device__ constexpr int fwd_groups_in_block(int LMAX, bool CANON) { return CANON ? 1 : l1_groups(LMAX); }

template <int LMAX, int CT, bool CANON, int DEPTH, bool P>
__global__ void __launch_bounds__(32 * fwd_groups_in_block(LMAX, CANON),
                                  (DEPTH == 1 ? (CANON ? 11 : 12) : 8) / fwd_groups_in_block(LMAX, CANON))
    k_layer1_fwd(DevModel m, EdgeIn in, const float* __restrict__ H1, float* __restrict__ Phi1) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char dyn[];
  constexpr int NG = l1_groups(LMAX) / fwd_groups_in_block(LMAX, CANON);
  const int ns = (CT > 0 ? CT : m.C) >> 5, n = in.N * ns * NG;
  AtomCursor cur{P ? m.sched : nullptr, n, 0};
  for (int b = cur.first(); b < n; b = cur.next()) {
    if constexpr (!CANON) {
      fwd_general<LMAX, CT>(m, in, H1, Phi1, b, dyn);
    } else {
      EdgeStage& st = *reinterpret_cast<EdgeStage*>(dyn);
      const int grp = b % NG, item = b / NG, i = in.atom_at(item / ns), slice = item % ns;
      if (grp == 0) fwd_canon<LMAX, 0, CT, DEPTH>(m, in, H1, Phi1, i, slice, st);
      if constexpr (LMAX == 2) {
        if (grp == 1) fwd_canon<LMAX, 1, CT, DEPTH>(m, in, H1, Phi1, i, slice, st);
        if (grp == 2) fwd_canon<LMAX, 2, CT, DEPTH>(m, in, H1, Phi1, i, slice, st);
      }
    }
  }
  cur.done();
}

namespace {

size_t fwd_smem(int lmax, bool canon) {
  return canon ? sizeof(EdgeStage) : l1_groups(lmax) * sizeof(EdgeStage) + sizeof(float) * ins_np(lmax) * 32;
}

// Canonical items up to which two edges are kept in flight: DEPTH 2 has 8 warps per SM, so past
// two rounds of them (one, for the longer edges of L_max 2) the warps hide the loads themselves
// (us, one : two edges: 64 items 16.5 : 14.4, 2000 items 57.4 : 47.1, 16400 items 252 : 266;
// 3600 items of L_max 2 73 : 82).
constexpr long deep_items(int lmax) { return (lmax == 1 ? 16 : 8) * 152; }

}  // namespace

// Once per model, after its upload.  One thread per (row, channel): its cubics gathered, then
// written back in pairs
template <int LMAX>
__global__ void k_pair_splines(float4* __restrict__ spl, long rows, int C) {
  constexpr int NI = ins_count(LMAX);
  const long n = rows * C;
  for (long t = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; t < n;
       t += static_cast<long>(gridDim.x) * blockDim.x) {
    float4* p = spl + t / C * NI * C + t % C;
    float4 c[NI];
#pragma unroll
    for (int q = 0; q < NI; ++q) c[q] = p[q * C];
    static_for<l1_groups(LMAX)>([&](auto gc) {
      constexpr int G = decltype(gc)::value;
      static_for<grp_count(G)>([&](auto ic) {
        constexpr int w = decltype(ic)::value, slot = grp_slot(G) + w, q = grp_ins(LMAX, G, w);
        if constexpr (w % 2 == 0 && w + 1 < grp_count(G)) {
          constexpr int q2 = grp_ins(LMAX, G, w + 1 < grp_count(G) ? w + 1 : w);
          p[slot * C] = make_float4(c[q].x, c[q2].x, c[q].y, c[q2].y);
          p[(slot + 1) * C] = make_float4(c[q].z, c[q2].z, c[q].w, c[q2].w);
        } else if constexpr (w % 2 == 0) {
          p[slot * C] = c[q];
        }
      });
    });
  }
}

void launch_pair_splines(float4* spl, long rows, int C, int L_max) {
  if (rows <= 0) return;
  const int blocks = static_cast<int>(std::min<long>((rows * C + 127) / 128, 152L * 32));
  if (L_max == 2)
    k_pair_splines<2><<<blocks, 128>>>(spl, rows, C);
  else
    k_pair_splines<1><<<blocks, 128>>>(spl, rows, C);
}

bool canonical_cg(int L_max, const std::vector<int>& off, const std::vector<int>& lme, const std::vector<float>& v,
                  const int* lme_off, const int* num_e, std::vector<float>& val) {
  const int np = ins_np(L_max);
  if (static_cast<int>(off.size()) != np + 1) return false;
  for (int l = 0, o = 0; l < 4; o += (2 * l + 1) * num_e[l], ++l)
    if (num_e[l] != ins_ne(L_max, l) || lme_off[l] != o) return false;
  val.assign(2 * np, 0.0f);
  for (int q = 0; q < ins_count(L_max); ++q)
    for (int p = ins_poff(L_max, q); p < ins_poff(L_max, q) + ins_paths(L_max, q); ++p)
      for (int t = off[p]; t < off[p + 1]; ++t) {
        const int ne = ins_ne(L_max, ins_l(L_max, q)), d = lme[t] - ins_row(L_max, q);
        const int mm = d >= 0 && d % ne == 0 ? d / ne : -1;
        const int w = mm < 0 ? -1 : (cg_m(L_max, p, 0) == mm ? 0 : (cg_m(L_max, p, 1) == mm ? 1 : -1));
        if (w < 0 || val[2 * p + w] != 0.0f) return false;  // outside the pattern, or given twice
        val[2 * p + w] = v[t];
      }
  return true;
}

// (every block's shared memory is below 48 KB: no opt-in)
cudaError_t init_layer1_kernels(const DevModel&) { return cudaSuccess; }

void launch_layer1_fwd(const DevModel& m, const EdgeIn& in, const float* H1, float* Phi1, cudaStream_t s) {
  if (in.N <= 0) return;
  const bool canon = m.cg_val != nullptr;
  const int nb = fwd_groups_in_block(m.L_max, canon);
  const long items = static_cast<long>(in.N) * (m.C >> 5) * (l1_groups(m.L_max) / nb);
  const bool deep = canon && items <= deep_items(m.L_max);
  DevModel mk;
  const int grid = atom_grid(m, kAkLayer1Fwd, static_cast<int>(items), mk);
  const size_t smem = fwd_smem(m.L_max, canon);
  dispatch_layer1(m, [&](auto lc, auto cc, auto nc) {
    constexpr int LM = decltype(lc)::value, CT = decltype(cc)::value;
    constexpr bool CANON = decltype(nc)::value;
    auto go = [&](auto dc, auto pc) {
      launch_pdl(k_layer1_fwd<LM, CT, CANON, decltype(dc)::value, decltype(pc)::value>, grid, 32 * nb, smem, s, mk, in,
                 H1, Phi1);
    };
    constexpr std::integral_constant<int, 1> one{};
    constexpr std::integral_constant<int, CANON ? 2 : 1> two{};
    if (mk.sched)
      deep ? go(two, std::true_type{}) : go(one, std::true_type{});
    else
      deep ? go(two, std::false_type{}) : go(one, std::false_type{});
  });
}

// resident blocks per SM of the persistent layer-1 kernels at this model's launch shapes
// (the forward's at DEPTH 1; at DEPTH 2, up to deep_items items, 8 of the blocks are resident and
// the others of the grid find few items left)
void layer1_residency(const DevModel& m, int* per_sm) {
  dispatch_layer1(m, [&](auto lc, auto cc, auto nc) {
    constexpr int LM = decltype(lc)::value, CT = decltype(cc)::value;
    constexpr bool CANON = decltype(nc)::value;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[kAkLayer1Fwd], k_layer1_fwd<LM, CT, CANON, 1, true>,
                                                  32 * fwd_groups_in_block(LM, CANON), fwd_smem(LM, CANON));
  });
  per_sm[kAkLayer1Rev] = layer1_rev_residency(m);
}

}  // namespace smx
