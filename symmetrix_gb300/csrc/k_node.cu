// Node-level kernels: channel-mixing GEMMs, the layer-1 node tail (symmetric
// contraction M1, H2, readouts, energy and the adjoint seeds), and small utilities.
//
// Reference stages restated here (libsymmetrix/source/mace.cpp):
//   k_gemm       : compute_H1 / reverse_H1 (:397-451), compute_A1 / reverse_A1 (:607-679)
//   k_node_tail  : compute_M1 (:759-777), compute_H2 (:796-832), compute_readouts (:876-903)
//                  with MultilayerPerceptron::evaluate_gradient (multilayer_perceptron.cpp:76-150),
//                  reverse_H2 (:834-874), reverse_M1 (:779-794)
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>

#include "device.cuh"
#include "kernels.h"
#include "poly_canon.h"

namespace smx {

// ---------------------------------------------------------------------------
// FP32 SIMT GEMM, 64x64 tile, 16-deep k slices, 256 threads with a 4x4 register
// tile each.  blockIdx.z selects the segment.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_gemm(GemmBatch gb) {
  pdl_begin();
  const GemmSeg g = gb.s[blockIdx.z];
  const int row0 = blockIdx.x * 64, col0 = blockIdx.y * 64;
  if (row0 >= g.rows || col0 >= g.ncols) return;
  __shared__ __align__(16) float As[16][64 + 4];
  __shared__ __align__(16) float Bs[16][64];
  const int tid = threadIdx.x;
  const int tr = tid >> 4, tc = tid & 15;
  // A loader: row tid/4, k offset (tid%4)*4
  const int a_row = row0 + (tid >> 2);
  const int a_k = (tid & 3) * 4;
  const float* a_ptr = nullptr;
  if (a_row < g.rows) {
    const int node = a_row / g.rpn, sub = a_row - node * g.rpn;
    a_ptr = g.X + node * g.x_ns + g.x_off + static_cast<long>(sub) * g.x_rs;
  }
  // B loader: k row tid/16, cols (tid%16)*4
  const int b_k = tid >> 4;
  const int b_col = col0 + (tid & 15) * 4;
  float acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0f;
  for (int k0 = 0; k0 < g.K; k0 += 16) {
    float4 av = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a_ptr) av = __ldg(reinterpret_cast<const float4*>(a_ptr + k0 + a_k));
    float4 bv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (b_col < g.ncols) bv = __ldg(reinterpret_cast<const float4*>(g.B + static_cast<long>(k0 + b_k) * g.ncols + b_col));
    __syncthreads();
    As[a_k + 0][tid >> 2] = av.x;
    As[a_k + 1][tid >> 2] = av.y;
    As[a_k + 2][tid >> 2] = av.z;
    As[a_k + 3][tid >> 2] = av.w;
    *reinterpret_cast<float4*>(&Bs[b_k][(tid & 15) * 4]) = bv;
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      const float4 a4 = *reinterpret_cast<const float4*>(&As[kk][tr * 4]);
      const float4 b4 = *reinterpret_cast<const float4*>(&Bs[kk][tc * 4]);
      const float ar[4] = {a4.x, a4.y, a4.z, a4.w};
      const float br[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(ar[a], br[b], acc[a][b]);
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = row0 + tr * 4 + a;
    if (r >= g.rows) continue;
    const int node = r / g.rpn, sub = r - node * g.rpn;
    float* y = g.Y + node * g.y_ns + g.y_off + static_cast<long>(sub) * g.y_rs + col0 + tc * 4;
    if (col0 + tc * 4 < g.ncols) *reinterpret_cast<float4*>(y) = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
  }
}

void launch_gemm(const GemmBatch& b, cudaStream_t s) {
  int maxr = 0, maxc = 0;
  for (int q = 0; q < b.n; ++q) {
    maxr = b.s[q].rows > maxr ? b.s[q].rows : maxr;
    maxc = b.s[q].ncols > maxc ? b.s[q].ncols : maxc;
  }
  if (maxr == 0 || b.n == 0) return;
  dim3 grid(ceil_div(maxr, 64), ceil_div(maxc, 64), b.n);
  launch_pdl(k_gemm, grid, 256, 0, s, b);
}

// ---------------------------------------------------------------------------
// Layer-1 node tail, one block per node, one thread per channel.
//   M1[k] = P1_{ti,k}(A1[i,:,k]) and its gradient,
//   H2 = W_H1[ti]^T H1[i,0,:] + W_M1^T M1,
//   E_i = e0[ti] + w1 . H1[i,0,:] + w2 . s*silu(W1 H2)           (float64 output),
//   dE/dH2 (MLP gradient), H1_adj[i,0,:] = w1 + W_H1[ti] dE/dH2 (other rows 0; fixed point),
//   M1_adj = W_M1 dE/dH2, A1_adj[i,lm,k] = dM1/dA1[lm] * M1_adj[k].
// ---------------------------------------------------------------------------
__device__ __forceinline__ void axpy4(float4& y, float a, float4 x) {
  y.x = fmaf(a, x.x, y.x);
  y.y = fmaf(a, x.y, y.y);
  y.z = fmaf(a, x.z, y.z);
  y.w = fmaf(a, x.w, y.w);
}

__device__ __forceinline__ void node_tail_atom(const DevModel& m, const int* __restrict__ ntype, float* __restrict__ A1,
                                               const float* __restrict__ H1, float* __restrict__ M1o,
                                               float* __restrict__ H2o, float* __restrict__ A1_adj,
                                               fix64* __restrict__ H1_adj, float* __restrict__ M1_adj_o,
                                               float* __restrict__ H2_adj_o, const float* __restrict__ zbl_e,
                                               double* __restrict__ energies, int N, int i) {
  extern __shared__ __align__(16) float dyn[];
  const int C = m.C, k = threadIdx.x;
  const int nwarp = C >> 5, lane = k & 31, warp = k >> 5;
  const int ti = ntype[i];
  const int nh = m.n_hidden;
  float* sX = dyn;              // [17][C]
  float* sG = sX + 17 * C;      // [17][C]
  float* sM1 = sG + 17 * C;     // [C]
  float* sH10 = sM1 + C;        // [C]
  float* sH2 = sH10 + C;        // [C]
  float* sdH2 = sH2 + C;        // [C]
  float* sRed = sdH2 + C;       // [33][8]
  float* sS = sRed + 33 * 8;    // [33] readout-MLP gradient factors
  float* sE = sS + 33;          // [33] energy terms
  float f = 0.0f;
  const float* cf = m.coef1 + static_cast<size_t>(ti) * m.T1 * C + k;
  const bool dens = m.dens_spl[1] != nullptr;
  const float S1 = dens ? m.dens_s[1][i] : 1.0f;
  if (dens) {  // density-normalised A1, kept scaled (compute_A1_scaled, mace.cpp:681-705)
#pragma unroll
    for (int q = 0; q < 16; ++q) A1[(static_cast<size_t>(i) * 16 + q) * C + k] /= S1;
  }
  if (m.poly_canon) {  // generated straight-line M1 polynomial and gradient
    float x[16], g[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      x[q] = A1[(static_cast<size_t>(i) * 16 + q) * C + k];
      g[q] = 0.0f;
    }
    f = poly::value_grad_M1(x, cf, C, g);
#pragma unroll
    for (int q = 0; q < 16; ++q) sG[q * C + k] = g[q];
  } else {
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    sX[q * C + k] = A1[(static_cast<size_t>(i) * 16 + q) * C + k];
    sG[q * C + k] = 0.0f;
  }
  sX[16 * C + k] = 1.0f;
  sG[16 * C + k] = 0.0f;
  for (int t = 0; t < m.T1; ++t) {
    const int pk = __ldg(m.mono1 + t);
    const int a = pk & 255, b = (pk >> 8) & 255, c = pk >> 16;
    const float w = __ldg(cf + static_cast<size_t>(t) * C);
    const float xa = sX[a * C + k], xb = sX[b * C + k], xc = sX[c * C + k];
    f = fmaf(w, xa * xb * xc, f);
    sG[a * C + k] += w * xb * xc;
    sG[b * C + k] += w * xa * xc;
    sG[c * C + k] += w * xa * xb;
  }
  }
  sM1[k] = f;
  const float h10 = H1[static_cast<size_t>(i) * m.nLM * C + k];
  sH10[k] = h10;
  __syncthreads();
  // H2 = W_H1[ti]^T H1[i,0,:] + W_M1^T M1.  A thread has four output channels and a quarter
  // of the rows, so that a weight row is read in 16-byte loads, C / 2 of them in all and
  // independent; the quarters meet in shared memory (sX is free: the polynomial is done)
  const int C4 = C >> 2, quarter = k / C4, c4 = k - quarter * C4, r0 = quarter * C4;
  float4* sP = reinterpret_cast<float4*>(sX);  // [2][4 quarters][C / 4]
  {
    const float4* W = reinterpret_cast<const float4*>(m.H2W_H1 + static_cast<size_t>(ti) * C * C) + r0 * C4 + c4;
    const float4* WM = reinterpret_cast<const float4*>(m.H2W_M1) + r0 * C4 + c4;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
#pragma unroll 8
    for (int r = r0; r < r0 + C4; ++r, W += C4, WM += C4) {
      axpy4(p, sH10[r], __ldg(W));
      axpy4(q, sM1[r], __ldg(WM));
    }
    sP[k] = make_float4(p.x + q.x, p.y + q.y, p.z + q.z, p.w + q.w);
  }
  __syncthreads();
  const float h2 = (sX[k] + sX[C + k]) + (sX[2 * C + k] + sX[3 * C + k]);
  sH2[k] = h2;
  // hidden pre-activations s_u = W1[u,:] . H2 and the linear readout w1 . H1[i,0,:] (slot nh)
#pragma unroll 4
  for (int u = 0; u <= nh; ++u) {
    float v = (u < nh) ? __ldg(m.ro2_w1 + static_cast<size_t>(u) * C + k) * h2 : __ldg(m.ro1 + k) * h10;
    v = warp_sum(v);
    if (lane == 0) sRed[u * 8 + warp] = v;
  }
  __syncthreads();
  for (int u = k; u <= nh; u += C) {  // one thread per hidden unit
    float s = 0.0f;
    for (int w = 0; w < nwarp; ++w) s += sRed[u * 8 + w];
    if (u < nh) {
      const float w2 = __ldg(m.ro2_w2 + u), sg = 1.0f / (1.0f + expf(-s));
      sS[u] = w2 * (m.ro2_scale * sg + m.ro2_scale * s * sg * (1.0f - sg));
      sE[u] = w2 * (m.ro2_scale * s * sg);
    } else {
      sE[u] = s;
    }
  }
  __syncthreads();
  float dh2 = 0.0f;
  for (int u = 0; u < nh; ++u) dh2 = fmaf(sS[u], __ldg(m.ro2_w1 + static_cast<size_t>(u) * C + k), dh2);
  sdH2[k] = dh2;
  if (k == 0) {
    double e = static_cast<double>(__ldg(m.e0 + ti)) + static_cast<double>(sE[nh]);
    for (int u = 0; u < nh; ++u) e += static_cast<double>(sE[u]);
    if (zbl_e) e += static_cast<double>(zbl_e[i]);
    energies[i] = e;
  }
  __syncthreads();
  // H1_adj[i,0,:] = w1 + W_H1[ti] dE/dH2 and M1_adj = W_M1 dE/dH2: as above
  {
    const float4* WT = reinterpret_cast<const float4*>(m.H2W_H1_T + static_cast<size_t>(ti) * C * C) + r0 * C4 + c4;
    const float4* WMT = reinterpret_cast<const float4*>(m.H2W_M1_T) + r0 * C4 + c4;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
#pragma unroll 8
    for (int r = r0; r < r0 + C4; ++r, WT += C4, WMT += C4) {
      const float d = sdH2[r];
      axpy4(p, d, __ldg(WT));
      axpy4(q, d, __ldg(WMT));
    }
    sP[k] = p;
    sP[C + k] = q;
  }
  __syncthreads();
  const float* sQ = sX + 4 * C;
  const float ha = __ldg(m.ro1 + k) + ((sX[k] + sX[C + k]) + (sX[2 * C + k] + sX[3 * C + k]));
  const float m1a = (sQ[k] + sQ[C + k]) + (sQ[2 * C + k] + sQ[3 * C + k]);
  if (dens) {  // reverse_A1_scaled (mace.cpp:707-757): c_i = dA1 . A1 / s_i, dA1 /= s_i
    float dot = 0.0f;
#pragma unroll
    for (int q = 0; q < 16; ++q) dot = fmaf(sG[q * C + k] * m1a, A1[(static_cast<size_t>(i) * 16 + q) * C + k], dot);
    dot = block_sum(dot);
    if (k == 0) m.dens_c[1][i] = dot / S1;
  }
  // A1_adj = dM1/dA1 * M1_adj (/ S1 when density-normalised; no division sequence otherwise)
  auto a1adj = [&](int q) { return dens ? sG[q * C + k] * m1a / S1 : sG[q * C + k] * m1a; };
  if (A1_adj)  // nullptr: only the split rows below are consumed
#pragma unroll
    for (int q = 0; q < 16; ++q) A1_adj[(static_cast<size_t>(i) * 16 + q) * C + k] = a1adj(q);
  if (m.op_a1adj) {  // BF16 form: the Phi1_adj GEMM's split operand, rows (node, m) per l
    const int T = m.tc_terms;
    const size_t pitch = static_cast<size_t>(split_xterms(T)) * C;
    for (int l = 0; l < 4; ++l) {
      if (m.num_e[l] == 0) continue;
      __nv_bfloat16* row = m.op_a1adj + pitch * (static_cast<size_t>(N) * l * l + static_cast<size_t>(i) * (2 * l + 1));
      for (int mm = 0; mm < 2 * l + 1; ++mm, row += pitch) write_split(row, C, T, k, a1adj(l * l + mm));
    }
  }
  // H1_adj in fixed point: the layer-1 adjoint adds its edge terms to these rows
  H1_adj[static_cast<size_t>(i) * m.nLM * C + k] = to_fixed(ha);
  for (int LM = 1; LM < m.nLM; ++LM) H1_adj[(static_cast<size_t>(i) * m.nLM + LM) * C + k] = 0ull;
  M1o[static_cast<size_t>(i) * C + k] = f;
  H2o[static_cast<size_t>(i) * C + k] = h2;
  M1_adj_o[static_cast<size_t>(i) * C + k] = m1a;
  H2_adj_o[static_cast<size_t>(i) * C + k] = dh2;
}

// What bounds it: the chain of dependent phases of a node and the 0.26 MB of weights that each
// node reads through L2 (4 C^2 + the species' polynomial).  One output channel per thread and
// 4-byte loads of the weights, every thread evaluating the readout's activations: 0.115 ms
// (FP32) / 0.119 ms (BF16) for 4096 nodes of 128 channels, now 0.095 / 0.097; 300 nodes 33 ->
// 24 us, 64 of 32 channels 17 -> 13.  80 registers: at 64 the large system gains 0.002 ms and
// the small ones lose 2 to 4 us.
template <bool P>
__global__ void __launch_bounds__(256, 3) k_node_tail(DevModel m, const int* __restrict__ ntype, float* __restrict__ A1,
                                                   const float* __restrict__ H1, float* __restrict__ M1o,
                                                   float* __restrict__ H2o, float* __restrict__ A1_adj,
                                                   fix64* __restrict__ H1_adj, float* __restrict__ M1_adj_o,
                                                   float* __restrict__ H2_adj_o, const float* __restrict__ zbl_e,
                                                   double* __restrict__ energies, int N) {
  pdl_begin();
  AtomCursor cur{P ? m.sched : nullptr, N, 0};
  for (int i = cur.first(); i < N; i = cur.next())
    node_tail_atom(m, ntype, A1, H1, M1o, H2o, A1_adj, H1_adj, M1_adj_o, H2_adj_o, zbl_e, energies, N, i);
  cur.done();
}

size_t node_tail_smem(const DevModel& m) { return sizeof(float) * (34 * m.C + 4 * m.C + 33 * 8 + 2 * 33); }

void launch_node_tail(const DevModel& m, const int* node_type, int N, float* A1, const float* H1, float* M1,
                      float* H2, float* A1_adj, fix64* H1_adj, float* M1_adj, float* H2_adj, const float* zbl_e,
                      double* energies, cudaStream_t s) {
  if (N <= 0) return;
  DevModel mk;
  const int grid = atom_grid(m, kAkNodeTail, N, mk);
  if (mk.sched)
    launch_pdl(k_node_tail<true>, grid, m.C, node_tail_smem(m), s, mk, node_type, A1, H1, M1, H2, A1_adj, H1_adj,
               M1_adj, H2_adj, zbl_e, energies, N);
  else
    launch_pdl(k_node_tail<false>, grid, m.C, node_tail_smem(m), s, mk, node_type, A1, H1, M1, H2, A1_adj, H1_adj,
               M1_adj, H2_adj, zbl_e, energies, N);
}

void node_tail_residency(const DevModel& m, int* per_sm) {
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[kAkNodeTail], k_node_tail<true>, m.C, node_tail_smem(m));
}

// H1_adj from its fixed-point accumulator: float rows for the float32 GEMM and the stage
// reads, and in the BF16 form the M0_adj GEMM's split operand rows (write_split with
// `terms` products: row pitch split_xterms(terms) * C; rows grouped by L, lgroup_row).
__global__ void k_fixed_rows(const fix64* __restrict__ src, float* __restrict__ dst, __nv_bfloat16* __restrict__ bf,
                             long rows, int C, int terms) {
  pdl_begin();
  const long n = rows * C;
  for (long t = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; t < n;
       t += static_cast<long>(gridDim.x) * blockDim.x) {
    const float v = from_fixed(src[t]);
    dst[t] = v;
    if (bf) {  // (L_max 1: nLM = 4)
      const long r = t / C;
      write_split(bf + lgroup_row(rows >> 2, r >> 2, static_cast<int>(r & 3)) * split_xterms(terms) * C, C, terms,
                  static_cast<int>(t - r * C), v);
    }
  }
}

void launch_fixed_rows(const fix64* src, float* dst, __nv_bfloat16* bf, long rows, int C, int terms, int nLM,
                       cudaStream_t s) {
  if (bf && nLM != 4) throw std::invalid_argument("the split H1_adj rows exist for L_max 1 only");
  if (rows <= 0) return;
  const long n = rows * C;
  const int blocks = static_cast<int>(std::min<long>((n + 255) / 256, 152L * 16));
  launch_pdl(k_fixed_rows, blocks, 256, 0, s, src, dst, bf, rows, C, terms);
}

// Single-stage calls (the reference binding's reverse_Phi1): the fixed-point H1_adj
// accumulator from float rows (zero: from nothing), and the per-edge forces of the layer-1
// adjoint, node_forces = (zero ? 0 : node_forces) - sum over channel slices of f1.
__global__ void k_rows_to_fixed(const float* __restrict__ src, fix64* __restrict__ dst, long n, int zero) {
  for (long t = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; t < n;
       t += static_cast<long>(gridDim.x) * blockDim.x)
    dst[t] = zero ? 0ull : to_fixed(src[t]);
}

__global__ void k_forces_from_f1(double* __restrict__ forces, const float* __restrict__ f1, long stride, int planes,
                                 int width, long n, int zero) {
  for (long t = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; t < n;
       t += static_cast<long>(gridDim.x) * blockDim.x) {
    forces[t] = (zero ? 0.0 : forces[t]) - f1_sum(f1, stride, planes, width, t);
  }
}

void launch_rows_to_fixed(const float* src, fix64* dst, long n, bool zero, cudaStream_t s) {
  if (n <= 0) return;
  k_rows_to_fixed<<<static_cast<int>(std::min<long>((n + 255) / 256, 152L * 16)), 256, 0, s>>>(src, dst, n, zero);
}

void launch_forces_from_f1(double* forces, const float* f1, long stride, int planes, int width, long n,
                           bool zero, cudaStream_t s) {
  if (n <= 0) return;
  k_forces_from_f1<<<static_cast<int>(std::min<long>((n + 255) / 256, 152L * 16)), 256, 0, s>>>(forces, f1, stride,
                                                                                               planes, width, n, zero);
}

// Centre atoms sorted by species (a counting sort; the order inside a species is
// arbitrary: every atom's results are computed the same way whichever block takes it).
// One block.
__global__ void __launch_bounds__(1024) k_species_order(const int* __restrict__ ntype, int N, int S,
                                                        int* __restrict__ order) {
  pdl_begin();
  extern __shared__ int cnt[];  // [S]: counts, then scatter cursors
  for (int t = threadIdx.x; t < S; t += blockDim.x) cnt[t] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < N; i += blockDim.x) atomicAdd(&cnt[ntype[i]], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int o = 0;
    for (int t = 0; t < S; ++t) {
      const int c = cnt[t];
      cnt[t] = o;
      o += c;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < N; i += blockDim.x) order[atomicAdd(&cnt[ntype[i]], 1)] = i;
}

void launch_species_order(const int* node_type, int N, int S, int* order, cudaStream_t s) {
  if (N <= 0) return;
  launch_pdl(k_species_order, 1, 1024, sizeof(int) * S, s, node_type, N, S, order);
}

// The host API's input check, on the device: flags (a mapped host word) receive one bit
// per violated condition (kBad* in kernels.h); first[] must already be the scan of
// num_neigh.  Grid-stride over max(N, E).
__global__ void k_validate_inputs(int N, long E, int S, double r_cut, const int* __restrict__ node_types,
                                  const int* __restrict__ num_neigh, const int* __restrict__ first,
                                  const int* __restrict__ nidx, const int* __restrict__ ntype_e,
                                  const double* __restrict__ xyz, const double* __restrict__ r,
                                  unsigned* __restrict__ flags) {
  unsigned bad = 0;
  const long n = E > N ? E : N;
  for (long t = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; t < n;
       t += static_cast<long>(gridDim.x) * blockDim.x) {
    if (t < N) {
      if (node_types[t] < 0 || node_types[t] >= S) bad |= kBadNodeType;
      if (num_neigh[t] < 0) bad |= kBadNumNeigh;
    }
    if (t < E) {
      if (nidx[t] < 0 || nidx[t] >= N) bad |= kBadNeighIndex;
      if (ntype_e[t] < 0 || ntype_e[t] >= S) bad |= kBadNeighType;
      const double re = r[t];
      if (!(re > 0.0 && re < r_cut) || !isfinite(xyz[3 * t]) || !isfinite(xyz[3 * t + 1]) || !isfinite(xyz[3 * t + 2]))
        bad |= kBadEdge;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && static_cast<long>(first[N]) != E) bad |= kBadEdgeCount;
  bad = __reduce_or_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0 && bad) atomicOr(flags, bad);
}

void launch_validate_inputs(int N, long E, int S, double r_cut, const int* node_types, const int* num_neigh,
                            const int* first, const int* nidx, const int* ntype_e, const double* xyz, const double* r,
                            unsigned* flags, cudaStream_t s) {
  const long n = E > N ? E : N;
  const int grid = static_cast<int>(std::min<long>(ceil_div(n > 0 ? n : 1, 256), 152L * 8));
  k_validate_inputs<<<grid, 256, 0, s>>>(N, E, S, r_cut, node_types, num_neigh, first, nidx, ntype_e, xyz, r, flags);
}

// first[0] = 0, first[i+1] = first[i] + num_neigh[i]; one block, sequential tiles of 8192: a
// warp scans eight rows of 32 (coalesced), the next tile's loads in flight meanwhile (32512
// nodes: 30 us with 1024 per tile -> 9.6 us).
__global__ void __launch_bounds__(1024) k_scan_first(const int* __restrict__ num_neigh, int N, int* __restrict__ first) {
  constexpr int kRows = 8, kTile = 1024 * kRows;
  __shared__ int sw[2][32];
  if (threadIdx.x == 0) first[0] = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int v[kRows], carry = 0;  // carry: the same in every thread
  auto load = [&](int base) {
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      const int idx = base + (warp * kRows + q) * 32 + lane;
      v[q] = idx < N ? num_neigh[idx] : 0;
    }
  };
  load(0);
  for (int base = 0, turn = 0; base < N; base += kTile, turn ^= 1) {
    int x[kRows], sum = 0;
#pragma unroll
    for (int q = 0; q < kRows; ++q) x[q] = v[q];
    if (base + kTile < N) load(base + kTile);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int q = 0; q < kRows; ++q) {
        const int y = __shfl_up_sync(0xffffffffu, x[q], o);
        if (lane >= o) x[q] += y;
      }
#pragma unroll
    for (int q = 0; q < kRows; ++q) {  // the warp's rows one after the other
      const int row = __shfl_sync(0xffffffffu, x[q], 31);
      x[q] += sum;
      sum += row;
    }
    if (lane == 0) sw[turn][warp] = sum;
    __syncthreads();
    int w = sw[turn][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    const int below = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
    const int before = carry + (warp > 0 ? below : 0);
    carry += __shfl_sync(0xffffffffu, w, 31);
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      const int idx = base + (warp * kRows + q) * 32 + lane;
      if (idx < N) first[idx + 1] = before + x[q];
    }
  }
}

void launch_scan_first(const int* num_neigh, int N, int* first, cudaStream_t s) {
  k_scan_first<<<1, 1024, 0, s>>>(num_neigh, N, first);
}

}  // namespace smx
