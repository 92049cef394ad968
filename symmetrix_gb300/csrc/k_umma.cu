// Channel-mixing GEMMs on the tcgen05 tensor cores (the BF16 precision form).
//
//   Y[rows, N] = X[rows, K] . B[N, K]^T     X, B bf16 (K contiguous), Y f32
//
// One CTA per 128-row x NT-column tile.  Thread 0 streams 64-wide k-blocks of the X
// tile and the B tile with TMA (128-byte swizzled boxes) through a ring of up to four
// shared-memory stages (full/empty mbarriers); a stage holds the k-block of every stored
// split term (X: hi, lo; B: W_hi, W_lo).  Thread 32 issues, per 16-wide step of the
// k-block, one tcgen05.mma (M=128, N=NT, K=16) per split product (x_hi W_hi, x_hi W_lo,
// x_lo W_hi) into an f32 accumulator in tensor memory, so each term is loaded once and
// used by every product that needs it, and releases each stage with tcgen05.commit;
// after the last commit the four warps read their 32 accumulator lanes back with
// tcgen05.ld and store them through an affine row map straight into the engine's
// feature layouts.
//
// These GEMMs restate compute_H1, compute_A1, reverse_A1 and reverse_H1
// (libsymmetrix/source/mace.cpp:397-451, :607-679) with bf16 operands and f32
// accumulation.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <stdexcept>
#include <string>

#include "kernels.h"
#include "sm100.cuh"

namespace smx {

namespace {

constexpr int kBoxK = 64;      // bf16 elements per TMA box row (128 B: one swizzle atom row)
constexpr int kTileM = 128;

__device__ __forceinline__ void record_timeout(unsigned* status) {
  if (status) atomicOr(status, 1u);
}

constexpr int kStages = 4;     // maximum shared-memory ring depth (k-blocks in flight)

// Up to four independent GEMMs in one launch (blockIdx.z selects the segment; the
// blocks beyond a segment's tile counts return at once).  blockIdx.x runs over the
// segment's tiles N-tile fastest, so the CTAs that read the same 128-row X tile run
// back to back and all but the first find it in L2.
struct UmmaSegDev {
  CUtensorMap ta, tb;
  UmmaOut o;
  int K, NT, tiles_m, tiles_n, stages, terms;
};
struct UmmaGroupDev {
  UmmaSegDev s[4];
  // test of the error path: the producer issues no load and the MMA thread waits
  // wait_ns for one, so its bounded wait runs out with nothing in flight
  int skip_loads;
  uint64_t wait_ns;
};

__global__ void __launch_bounds__(128, 1) k_umma_gemm(const __grid_constant__ UmmaGroupDev grp, unsigned* status) {
  pdl_begin();
  const UmmaSegDev& seg = grp.s[blockIdx.z];
  const int tile_n = static_cast<int>(blockIdx.x % static_cast<unsigned>(seg.tiles_n));
  const int tile_m = static_cast<int>(blockIdx.x / static_cast<unsigned>(seg.tiles_n));
  if (tile_m >= seg.tiles_m) return;
  const CUtensorMap& ta = seg.ta;
  const CUtensorMap& tb = seg.tb;
  const UmmaOut& o = seg.o;
  const int K = seg.K, NT = seg.NT, terms = seg.terms;
  const int XT = split_xterms(terms), WT = split_wterms(terms);
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[kStages], empty[kStages], bar_mma;  // kStages >= seg.stages
  __shared__ uint32_t tmem_base;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int KB = K / kBoxK;
  const int S = KB < seg.stages ? KB : seg.stages;
  const uint32_t a_bytes = kTileM * kBoxK * 2, b_bytes = static_cast<uint32_t>(NT) * kBoxK * 2;
  // stage = the XT X boxes, then the WT B boxes (all 1024-B multiples)
  const uint32_t stage_bytes = XT * a_bytes + WT * b_bytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = tile_m * kTileM, n0 = tile_n * NT;
  const uint32_t ncols = NT <= 32 ? 32u : (NT <= 64 ? 64u : (NT <= 128 ? 128u : 256u));

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      sm100::mbar_init(&full[s], 1);
      sm100::mbar_init(&empty[s], 1);
    }
    sm100::mbar_init(&bar_mma, 1);
    sm100::fence_mbar_init();
  }
  if (warp == 0) {
    sm100::tmem_alloc(&tmem_base, ncols);
    sm100::tmem_relinquish();
  }
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();
  const uint32_t tmem = tmem_base;

  // producer: k-block kb goes to stage kb % S once the MMAs of k-block kb - S released it
  int loads = 0;
  bool prod_ok = true;
  if (threadIdx.x == 0 && !grp.skip_loads) {
    for (int kb = 0; kb < KB; ++kb) {
      const int s = kb % S;
      if (kb >= S && !sm100::mbar_wait(&empty[s], ((kb / S) - 1) & 1)) {
        prod_ok = false;
        break;
      }
      uint8_t* st = smem + static_cast<size_t>(s) * stage_bytes;
      sm100::mbar_arrive_expect_tx(&full[s], stage_bytes);
      for (int t = 0; t < XT; ++t) sm100::tma_load_2d(st + t * a_bytes, &ta, t * K + kb * kBoxK, m0, &full[s]);
      for (int u = 0; u < WT; ++u)
        sm100::tma_load_2d(st + XT * a_bytes + u * b_bytes, &tb, u * K + kb * kBoxK, n0, &full[s]);
      ++loads;
    }
  }
  // MMA issuer
  bool issued = false, mma_ok = true;
  if (threadIdx.x == 32) {
    const uint32_t idesc = sm100::idesc_bf16_f32(kTileM, NT);
    for (int kb = 0; kb < KB; ++kb) {
      const int s = kb % S;
      if (!sm100::mbar_wait(&full[s], (kb / S) & 1, grp.wait_ns)) {
        mma_ok = false;
        break;
      }
      sm100::tc_fence_after();
      const uint32_t x0 = sm100::smem_u32(smem + static_cast<size_t>(s) * stage_bytes), w0 = x0 + XT * a_bytes;
#pragma unroll
      for (int k = 0; k < kBoxK / 16; ++k) {  // 16 elements (32 B) per MMA inside the 128-B swizzled row
        // x_hi W_hi, then x_hi W_lo (terms >= 2), then x_lo W_hi (terms 3)
        sm100::umma_bf16(tmem, sm100::sdesc_sw128(x0 + k * 32), sm100::sdesc_sw128(w0 + k * 32), idesc,
                         (kb | k) != 0 ? 1u : 0u);
        if (terms >= 2)
          sm100::umma_bf16(tmem, sm100::sdesc_sw128(x0 + k * 32), sm100::sdesc_sw128(w0 + b_bytes + k * 32), idesc,
                           1u);
        if (terms == 3)
          sm100::umma_bf16(tmem, sm100::sdesc_sw128(x0 + a_bytes + k * 32), sm100::sdesc_sw128(w0 + k * 32), idesc,
                           1u);
      }
      sm100::umma_commit(&empty[s]);
      issued = true;
    }
    // bar_mma: every MMA issued above has completed (also on the error path)
    if (issued) sm100::umma_commit(&bar_mma);
  }
  const int ok = __syncthreads_and((prod_ok && mma_ok) ? 1 : 0);
  const int any_mma = __syncthreads_or(issued ? 1 : 0);
  bool done = false;
  if (any_mma) done = sm100::mbar_wait(&bar_mma, 0);
  const int all_done = __syncthreads_and((done && ok) ? 1 : 0);
  sm100::tc_fence_after();
  if (all_done) {
    const int r = m0 + warp * 32 + lane;
    const bool row_ok = r < o.rows;
    long base = 0;
    bool write = row_ok;
    if (row_ok) {
      base = static_cast<long>(r / o.rpn) * o.y_ns + o.y_off + static_cast<long>(r % o.rpn) * o.y_rs +
             (o.select ? 0 : n0);
      if (o.select) write = ((r % o.rpn) == 0) == (tile_n == 0);
    }
    // Each 32-column chunk goes through a 4 KB staging tile per warp (the ring's shared
    // memory is free once every MMA has completed): a lane holds one row after tcgen05.ld,
    // while a coalesced store wants eight lanes on 128 contiguous bytes of one row.  The
    // float4 groups of row t sit at slot q ^ (t & 7), so both the row-wise writes and the
    // transposed reads hit all 32 banks.
    float* stg = reinterpret_cast<float*>(smem) + warp * 32 * 32;
    const int sub = lane >> 3, c4 = lane & 7;
    for (int c0 = 0; c0 < NT; c0 += 32) {
      float v[32];
      sm100::tmem_ld32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(c0), v);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        reinterpret_cast<float4*>(stg + lane * 32)[q ^ (lane & 7)] =
            make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int t = 4 * j + sub;  // the warp's row this lane stores now
        const long b = __shfl_sync(0xffffffffu, base, t);
        const int w = __shfl_sync(0xffffffffu, write ? 1 : 0, t);
        const float4 val = reinterpret_cast<const float4*>(stg + t * 32)[c4 ^ (t & 7)];
        if (w) reinterpret_cast<float4*>(o.Y + b + c0)[c4] = val;
      }
      __syncwarp();  // the next chunk overwrites the staging tile
    }
  } else if (threadIdx.x == 0) {
    record_timeout(status);
    // no TMA copy may still be landing in shared memory when the CTA exits: wait for
    // the last load issued into each stage
    for (int kb = loads - S > 0 ? loads - S : 0; kb < loads; ++kb) sm100::mbar_wait(&full[kb % S], (kb / S) & 1);
  }
  sm100::tc_fence_before();
  __syncthreads();
  if (warp == 0) sm100::tmem_dealloc(tmem, ncols);
}

// ---------------------------------------------------------------------------
// Float32 GEMMs:  Y[rows, N] = X[rows, K] . B[N, K]^T with float32 X, split in the kernel.
//
// x = x0 + x1 + x2 and w = w0 + w1 + w2 in bf16, eight products (all but x2 w2, 2^-34).  The tensor
// core's running sum is cut towards zero at every 16-wide step: what it loses has the sum's sign,
// so it stays in sums over many results (total energies), where a chain of FMAs errs either way.
// So the leading terms lie on a grid: x0 is x rounded to 2^-7 of the power of two above the largest
// of its row's k-block, w0 the same over its row of B, both integers of at most 8 bits there.  Their
// products add exactly up to K = 1024 (14 + 10 bits of the accumulator's 24; where a row's k-blocks
// differ, their ratio comes out of the 9 or so bits that sums of either sign leave free), and the
// other seven, 2^-7 and less of them, go into a second accumulator that the epilogue adds: what is
// cut there is 2^-7 of what it was.  x1 and x2 hold what the grid leaves to 2^-26 of the block's
// largest; so that this is 2^-26 of the largest contribution whatever the channels' units, x_k is
// taken times the power of two above B's largest |w_nk| over n, and w_nk divided by it.
// Error against float64, 2-norm, this kernel : the SIMT one, in 1e-8 (random rows; of one sign; with
// one nonzero; with elements over 12 orders of magnitude; sums of integers are exact in both):
//   K =  64, N =  64   3.5 : 14.6   2.6 : 12.2   3.1 : 2.5   3.8 : 11.0
//   K = 128, N = 128   3.7 : 20.2   2.3 : 16.0   3.2 : 2.5   4.0 : 15.9
//   K = 384, N = 128   5.0 : 35.0   2.2 : 28.9   3.4 : 2.6   5.6 : 26.6
//   K = 640, N = 128   7.2 : 45.1   2.8 : 34.6   3.6 : 2.5   8.2 : 34.5
//   K = 768, N = 256   7.6 : 49.9   3.1 : 40.9   3.4 : 2.5   8.9 : 37.3
// and no mean loss (its part along the results is below 0.1 in every random case).  Times, us: 28672 x
// 128 x 384 36.0 : 80.1, 20480 x 384 x 128 37.2 : 69.9.  (Terms of each value's own 8 bits, six
// products, the steps round three accumulators of x0 w0: 45.2 and 36.5 us; mean loss 1.8 at K = 64,
// 9.5 at 384; total energies of 1000 to 3000 atoms of 128 channels 1.6-1.9e-7 off, now 3-5e-8.)
// Rows with values that have no split (infinities, NaN, finite ones from 2^112 on) give what
// chains of FMAs give: see plain_tile.  The weights all have one (checked where they are laid out).
// Eight warps read the float32 rows where the producers left them (the row map of the SIMT
// GEMM) and split them into the swizzled operand layout, a k-block ahead in registers; one
// thread of a ninth brings the weights' terms by TMA and issues the MMAs.
// ---------------------------------------------------------------------------
struct F32SegDev {
  CUtensorMap tb;
  GemmSeg g;
  const float* scale;  // F32Weights::scale
  int NT, tiles_m, tiles_n, stages;
};
struct F32GroupDev {
  F32SegDev s[4];
  int skip_loads;  // test of the error path, as in UmmaGroupDev
  uint64_t wait_ns;
};
constexpr int kF32Split = 256;                // threads that split X and store Y
constexpr int kF32Threads = kF32Split + 32;   // and a warp whose first lane issues TMA and MMAs
constexpr uint32_t kATerm = kTileM * kBoxK * 2;  // bytes of one X term of a k-block

// 1.5 2^23 grid steps of a row's k-block, m the bits of its largest |x| (a NaN from 2^112 on)
__device__ __forceinline__ float grid_magic(uint32_t m) {
  m = min(m & 0x7f800000u, 238u << 23);
  return __uint_as_float((m + (17u << 23)) | 0x400000u);
}
__device__ __forceinline__ float to_grid(float x, float magic) { return __fsub_rn(__fadd_rn(x, magic), magic); }
__device__ __forceinline__ float bf16_lo(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// A tile with a value that has no split (an infinity, a NaN, or a finite value from 2^112 on,
// whose grid has no magic number): its sums as the SIMT kernel forms them, chains of
// FMAs over k on the float32 weights.
__device__ __forceinline__ void plain_tile(const GemmSeg& g, const long* x_row, int m0, int n0, int NT, int tid) {
  for (int t = tid; t < kTileM * NT; t += kF32Split) {
    const int row = t / NT, n = n0 + t - row * NT, r = m0 + row;
    if (x_row[row] < 0) continue;
    const float *x = g.X + x_row[row], *w = g.B + n;
    float s = 0.0f;
    for (int k = 0; k < g.K; ++k) s = fmaf(__ldg(x + k), __ldg(w + static_cast<size_t>(k) * g.ncols), s);
    g.Y[static_cast<long>(r / g.rpn) * g.y_ns + g.y_off + static_cast<long>(r % g.rpn) * g.y_rs + n] = s;
  }
}

// Up to K = 128 two CTAs per SM with one stage each (96 KB, 256 TMEM columns) overlap one's
// splitting and stores with the other's MMAs; above, one CTA with two stages.
__global__ void __launch_bounds__(kF32Threads, 2) k_umma_f32(const __grid_constant__ F32GroupDev grp,
                                                             unsigned* status) {
  pdl_begin();
  const F32SegDev& seg = grp.s[blockIdx.z];
  const GemmSeg& g = seg.g;
  const int tile_n = static_cast<int>(blockIdx.x % static_cast<unsigned>(seg.tiles_n));
  const int tile_m = static_cast<int>(blockIdx.x / static_cast<unsigned>(seg.tiles_n));
  if (tile_m >= seg.tiles_m) return;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[kStages], split[kStages], empty[kStages], bar_mma;
  __shared__ uint32_t tmem_base;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int NT = seg.NT, S = seg.stages;
  const int KB = (g.K + kBoxK - 1) / kBoxK, Kp = KB * kBoxK;
  const uint32_t b_bytes = static_cast<uint32_t>(NT) * kBoxK * 2, stage_bytes = 3 * kATerm + 3 * b_bytes;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = tile_m * kTileM, n0 = tile_n * NT;
  const uint32_t used = static_cast<uint32_t>(2 * NT);
  const uint32_t ncols = used <= 64 ? 64u : (used <= 128 ? 128u : (used <= 256 ? 256u : 512u));
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      sm100::mbar_init(&full[s], 1);
      sm100::mbar_init(&split[s], kF32Split);
      sm100::mbar_init(&empty[s], 1);
    }
    sm100::mbar_init(&bar_mma, 1);
    sm100::fence_mbar_init();
  }
  if (warp == 0) {
    sm100::tmem_alloc(&tmem_base, ncols);
    sm100::tmem_relinquish();
  }
  __shared__ long x_row[kTileM];  // offsets of the tile's rows, -1 past the end
  if (tid < kTileM) {
    const int r = m0 + tid, node = r / g.rpn, sub = r - node * g.rpn;
    x_row[tid] = r < g.rows ? node * g.x_ns + g.x_off + static_cast<long>(sub) * g.x_rs : -1;
  }
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();
  const uint32_t tmem = tmem_base;

  // a k-block row is 16 float4: a warp reads two rows at a time, 16 rows in all; this thread
  // has float4 c of rows warp * 16 + lane / 16 + 2 j
  const int c = lane & 15, row0 = warp * 16 + (lane >> 4);
  float4 v[8], sc;
  auto load = [&](int kb) {
    const int k = kb * kBoxK + 4 * c;
    sc = __ldg(reinterpret_cast<const float4*>(seg.scale + k));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const long o = x_row[row0 + 2 * j];
      v[j] = o >= 0 && k < g.K ? __ldg(reinterpret_cast<const float4*>(g.X + o + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  bool ok = true, issued = false;
  int loads = 0;
  float low = 0.0f;  // sum of this thread's smallest terms
  if (tid < kF32Split) {
    load(0);
    for (int kb = 0; kb < KB; ++kb) {
      const int s = kb % S;
      if (kb >= S && !sm100::mbar_wait(&empty[s], ((kb / S) - 1) & 1, grp.wait_ns)) {  // the stage's last MMAs are done
        ok = false;
        break;
      }
      uint8_t* st = smem + static_cast<size_t>(s) * stage_bytes;
      // 16-byte group q (8 elements) of row r sits at slot q ^ (r & 7) of its 128-byte row
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int row = row0 + 2 * j;
        uint8_t* a = st + row * 128 + ((c >> 1) ^ (row & 7)) * 16 + (c & 1) * 8;
        float4 x = make_float4(v[j].x * sc.x, v[j].y * sc.y, v[j].z * sc.z, v[j].w * sc.w);
        uint32_t big = max(max(__float_as_uint(fabsf(x.x)), __float_as_uint(fabsf(x.y))),
                           max(__float_as_uint(fabsf(x.z)), __float_as_uint(fabsf(x.w))));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) big = max(big, __shfl_xor_sync(0xffffffffu, big, o));
        const float magic = grid_magic(big);
        float4 y = make_float4(to_grid(x.x, magic), to_grid(x.y, magic), to_grid(x.z, magic), to_grid(x.w, magic));
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          const uint2 w = make_uint2(bf16_pair(y.x, y.y), bf16_pair(y.z, y.w));
          *reinterpret_cast<uint2*>(a + t * kATerm) = w;
          if (t < 2)
            x = make_float4(x.x - bf16_lo(w.x), x.y - bf16_hi(w.x), x.z - bf16_lo(w.y), x.w - bf16_hi(w.y));
          y = x;
        }
        low += (x.x + x.y) + (x.z + x.w);  // a value without a split: NaN from here on
      }
      sm100::fence_async_shared();
      sm100::mbar_arrive(&split[s]);
      if (kb + 1 < KB) load(kb + 1);
    }
  } else if (tid == kF32Split) {
    const uint32_t idesc = sm100::idesc_bf16_f32(kTileM, NT);
    auto weights = [&](int kb) {  // into the stage of k-block kb, which must be free
      uint8_t* st = smem + static_cast<size_t>(kb % S) * stage_bytes + 3 * kATerm;
      sm100::mbar_arrive_expect_tx(&full[kb % S], 3 * b_bytes);
      for (int u = 0; u < 3; ++u)
        sm100::tma_load_2d(st + u * b_bytes, &seg.tb, u * Kp + kb * kBoxK, n0, &full[kb % S]);
      ++loads;
    };
    for (int kb = 0; kb < KB && kb < S && !grp.skip_loads; ++kb) weights(kb);
    for (int kb = 0; kb < KB; ++kb) {
      const int s = kb % S;
      // (with one stage: this k-block's weights, once the last one's MMAs are done)
      if (S == 1 && kb > 0) {
        if (!(ok = sm100::mbar_wait(&empty[0], (kb - 1) & 1, grp.wait_ns))) break;
        weights(kb);
      }
      ok = sm100::mbar_wait(&full[s], (kb / S) & 1, grp.wait_ns) &&
           sm100::mbar_wait(&split[s], (kb / S) & 1, grp.wait_ns);
      if (!ok) break;
      sm100::tc_fence_after();
      const uint32_t x0 = sm100::smem_u32(smem + static_cast<size_t>(s) * stage_bytes), w0 = x0 + 3 * kATerm;
#pragma unroll
      for (int k = 0; k < kBoxK / 16; ++k) {
        auto mma = [&](uint32_t d, int xt, int wt, uint32_t acc) {
          sm100::umma_bf16(d, sm100::sdesc_sw128(x0 + xt * kATerm + k * 32),
                           sm100::sdesc_sw128(w0 + wt * b_bytes + k * 32), idesc, acc);
        };
        const uint32_t corr = tmem + NT, more = (kb | k) != 0 ? 1u : 0u;
        mma(tmem, 0, 0, more);
        mma(corr, 1, 2, more);
        mma(corr, 2, 1, 1u);
        mma(corr, 0, 2, 1u);
        mma(corr, 2, 0, 1u);
        mma(corr, 1, 1, 1u);
        mma(corr, 0, 1, 1u);
        mma(corr, 1, 0, 1u);
      }
      sm100::umma_commit(&empty[s]);
      issued = true;
      // while these run: the weights that follow those of the k-block before
      if (S > 1 && kb > 0 && kb - 1 + S < KB) {
        if (!(ok = sm100::mbar_wait(&empty[(kb - 1) % S], ((kb - 1) / S) & 1, grp.wait_ns))) break;
        weights(kb - 1 + S);
      }
    }
    if (issued) sm100::umma_commit(&bar_mma);
  }
  const int all_ok = __syncthreads_and(ok ? 1 : 0);
  const int any_mma = __syncthreads_or(issued ? 1 : 0);
  bool done = false;
  if (any_mma) done = sm100::mbar_wait(&bar_mma, 0);
  const int all_done = __syncthreads_and((done && all_ok) ? 1 : 0);
  const int plain = __syncthreads_or(low == low ? 0 : 1);
  sm100::tc_fence_after();
  if (all_done && plain) {
    if (tid < kF32Split) plain_tile(g, x_row, m0, n0, NT, tid);
  } else if (all_done && tid < kF32Split) {
    // warp w reads the accumulator lanes 32 (w mod 4) and every other 32-column chunk; rows
    // leave through a swizzled 4 KB tile per warp, as in k_umma_gemm
    const int quarter = warp & 3, r = m0 + quarter * 32 + lane;
    const bool write = r < g.rows;
    const long base = write ? static_cast<long>(r / g.rpn) * g.y_ns + g.y_off + static_cast<long>(r % g.rpn) * g.y_rs + n0
                            : 0;
    float* stg = reinterpret_cast<float*>(smem) + warp * 32 * 32;
    const int sub = lane >> 3, c4 = lane & 7;
    const uint32_t t0 = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    for (int c0 = (warp >> 2) * 32; c0 < NT; c0 += 64) {
      float a[32], b[32];
      sm100::tmem_ld32(t0 + static_cast<uint32_t>(c0), a);
      sm100::tmem_ld32(t0 + static_cast<uint32_t>(NT + c0), b);
#pragma unroll
      for (int q = 0; q < 32; ++q) a[q] += b[q];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        reinterpret_cast<float4*>(stg + lane * 32)[q ^ (lane & 7)] =
            make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int t = 4 * j + sub;
        const long yb = __shfl_sync(0xffffffffu, base, t);
        const int w = __shfl_sync(0xffffffffu, write ? 1 : 0, t);
        const float4 val = reinterpret_cast<const float4*>(stg + t * 32)[c4 ^ (t & 7)];
        if (w) reinterpret_cast<float4*>(g.Y + yb + c0)[c4] = val;
      }
      __syncwarp();
    }
  } else if (!all_done && tid == kF32Split) {
    record_timeout(status);
    for (int kb = loads - S > 0 ? loads - S : 0; kb < loads; ++kb) sm100::mbar_wait(&full[kb % S], (kb / S) & 1);
  }
  sm100::tc_fence_before();
  __syncthreads();
  if (warp == 0) sm100::tmem_dealloc(tmem, ncols);
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encoder() {
  static std::once_flag once;
  static EncodeTiledFn fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  if (!fn) throw std::runtime_error("cuTensorMapEncodeTiled is not available from the driver");
  return fn;
}

// 2-D bf16 tensor map over a row-major [rows][K] matrix, box = 64 x box_rows, 128-B swizzle.
CUtensorMap make_map(const void* base, long rows, int K, int box_rows) {
  if (reinterpret_cast<uintptr_t>(base) % 16 != 0) throw std::invalid_argument("tensor map base not 16-byte aligned");
  if (K % kBoxK != 0) throw std::invalid_argument("GEMM K must be a multiple of 64");
  CUtensorMap m;
  std::memset(&m, 0, sizeof(m));
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(kBoxK), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
                               estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed (" + std::to_string(r) + ")");
  return m;
}

}  // namespace

size_t umma_smem_bytes(int K, int NT, int stages, int terms) {
  stages = std::min(K / kBoxK, std::min(stages, kStages));
  return static_cast<size_t>(stages) * (split_xterms(terms) * kTileM + split_wterms(terms) * NT) * kBoxK * 2 + 1024;
}

// dynamic shared memory available next to the kernel's few static words
constexpr size_t kMaxDynSmem = 226 * 1024;

// (the launch lowers a schedule's ring depth until its stages fit)
bool umma_supported(int K, int NT, int terms) {
  return K % kBoxK == 0 && K > 0 && NT % 32 == 0 && NT >= 32 && NT <= 256 && terms >= 1 && terms <= 3 &&
         umma_smem_bytes(K, NT, 1, terms) <= kMaxDynSmem;
}

namespace {

// ring stages (see k_umma_f32)
int f32_stages(int K) { return K > 2 * kBoxK ? 2 : 1; }
// N-tile: the widest of 128, 96, 64, 32 that divides the columns
int f32_tile_n(int ncols) {
  for (int nt : {128, 96, 64})
    if (ncols % nt == 0) return nt;
  return 32;
}
size_t f32_smem_bytes(int NT, int stages) {
  return static_cast<size_t>(stages) * (3 * kATerm + 3 * static_cast<size_t>(NT) * kBoxK * 2) + 1024;
}
}  // namespace

// (K: the leading products' sums stay exact)
bool umma_f32_supported(int K, int ncols) {
  return K > 0 && K <= 1024 && K % 32 == 0 && ncols > 0 && ncols % 32 == 0;
}

int umma_f32_kp(int K) { return (K + kBoxK - 1) / kBoxK * kBoxK; }

void launch_umma_f32(const GemmBatch& b, const F32Weights* W, unsigned* status, cudaStream_t s,
                     bool test_timeout) {
  F32GroupDev grp;
  std::memset(&grp, 0, sizeof(grp));
  grp.skip_loads = test_timeout ? 1 : 0;
  grp.wait_ns = test_timeout ? 2000000ull : sm100::kWaitLimitNs;  // 2 ms when testing
  long gx = 0;
  size_t smem = 0;
  int used = 0;
  for (int q = 0; q < b.n; ++q) {
    const GemmSeg& g = b.s[q];
    if (!umma_f32_supported(g.K, g.ncols)) throw std::invalid_argument("unsupported tensor-core GEMM shape");
    if (g.rows <= 0) continue;
    F32SegDev& d = grp.s[used++];
    d.g = g;
    d.NT = f32_tile_n(g.ncols);
    d.stages = f32_stages(g.K);
    d.scale = W[q].scale;
    d.tb = make_map(W[q].terms, g.ncols, 3 * umma_f32_kp(g.K), d.NT);
    d.tiles_m = (g.rows + kTileM - 1) / kTileM;
    d.tiles_n = g.ncols / d.NT;
    gx = std::max(gx, static_cast<long>(d.tiles_m) * d.tiles_n);
    smem = std::max(smem, f32_smem_bytes(d.NT, d.stages));
  }
  if (used == 0) return;
  launch_pdl(k_umma_f32, dim3(static_cast<unsigned>(gx), 1, used), kF32Threads, smem, s, grp, status);
}

cudaError_t init_umma_kernels() {
  const cudaError_t e = cudaFuncSetAttribute(k_umma_f32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(f32_smem_bytes(128, 2)));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_umma_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(kMaxDynSmem));
}

void launch_umma_gemms(const UmmaGemm* g, int n, unsigned* status, cudaStream_t s, bool test_timeout) {
  if (n < 1 || n > 4) throw std::invalid_argument("1 to 4 tensor-core GEMMs per launch");
  UmmaGroupDev grp;
  std::memset(&grp, 0, sizeof(grp));
  grp.skip_loads = test_timeout ? 1 : 0;
  grp.wait_ns = test_timeout ? 2000000ull : sm100::kWaitLimitNs;  // 2 ms when testing
  long gx = 0;
  size_t smem = 0;
  int used = 0;
  for (int q = 0; q < n; ++q) {
    const UmmaGemm& a = g[q];
    if (!umma_supported(a.K, a.NT, a.terms) || a.nb_rows % a.NT != 0)
      throw std::invalid_argument("unsupported tensor-core GEMM shape");
    if (a.rows <= 0) continue;
    UmmaSegDev& d = grp.s[used++];
    d.ta = make_map(a.X, a.rows, split_xterms(a.terms) * a.K, kTileM);
    d.tb = make_map(a.B, a.nb_rows, split_wterms(a.terms) * a.K, a.NT);
    d.o = a.o;
    d.K = a.K;
    d.NT = a.NT;
    d.terms = a.terms;
    d.tiles_m = static_cast<int>((a.rows + kTileM - 1) / kTileM);
    d.tiles_n = a.nb_rows / a.NT;
    d.stages = a.stages >= 1 && a.stages <= kStages ? a.stages : kStages;
    while (d.stages > 1 && umma_smem_bytes(a.K, a.NT, d.stages, a.terms) > kMaxDynSmem) --d.stages;
    gx = std::max(gx, static_cast<long>(d.tiles_m) * d.tiles_n);
    smem = std::max(smem, umma_smem_bytes(a.K, a.NT, d.stages, a.terms));
  }
  if (used == 0) return;
  if (gx > 0x7fffffffL) throw std::invalid_argument("tensor-core GEMM too large for one launch");
  launch_pdl(k_umma_gemm, dim3(static_cast<unsigned>(gx), 1, used), 128, smem, s, grp, status);
}

}  // namespace smx
