// tc_contract.cu — the Wannier Fourier sums H(k), D(k) on the tcgen05 tensor
// cores (kind::f16 with exact BF16 integer slices) for mixed-precision batch
// instances.
//
// Real form of the complex sums: with A[k][.] = [cos(2 pi k.R_r) | sin(2 pi k.R_r)] / 2
// (K = 2 nr) and, per output element, the column pair
//   re: [ Re c_r ; -Im c_r ],   im: [ Im c_r ; Re c_r ]  (times 2),
// out = A . B^T gives Re / Im of sum_r e^{2 pi i k.R_r} c_r. Both operands are
// cut into 8-bit slices on a power-of-two scale (tc_contract.hpp): the GEMM
// depth holds one segment of 2 nr (padded to 64) per slice pair (a, b) with
// a + b <= 3. Within a segment every product is an integer times a common
// power of two and at most 2^14, so the tensor core's FP32 sums over a segment
// (at most 1024 deep) are exact; the segments are added in FP64 registers. The
// result is the FP64 sum to about 2^-32 of the terms, so the FP32 tables stored
// from it equal those of the FP64 CUDA-core build up to the last rounding.
//
// Three forms of the GEMM give the same planes bit for bit. k_tc_planes (the
// default) keeps the four slices of each operand once and forms the pair
// products itself (below). k_tc_gemm_tma (EDUS_TC_GEMM=tma) moves 128 x 64 and
// 64 x 64 operand tiles by TMA into 128-byte swizzled stages, four deep, all
// issued by thread 0. k_tc_gemm (EDUS_TC_GEMM=cpasync): one
// CTA (4 warps) per 128 x 32 tile of C. The 64-deep K slices
// (128-byte rows of BF16) are staged with cp.async into two shared-memory
// stages in the K-major canonical layout without swizzle (16-byte chunks of 8
// BF16, 8-row core matrices 128 bytes apart, the two 16-byte halves of one
// MMA's K = 16 one whole operand apart): slice s + 1 loads while the tensor
// core works on slice s. One elected thread issues four tcgen05.mma (M 128,
// N 32, K 16) per slice and commits them to the stage's mbarrier. Segments
// alternate between two TMEM accumulators (128 lanes x 32 FP32 columns each);
// a finished segment is read back with tcgen05.ld.32x32b into FP64 registers
// while the next one accumulates. All waits are bounded.
#include <cuda.h>
#include <stdint.h>

#include <cstdlib>
#include <cstring>

#include "batch.cuh"
#include "dev.cuh"
#include "tc_contract.hpp"

namespace edus {
namespace batch {
namespace {

constexpr int TM = 128, TN = 32, TK = 64;  // CTA tile and K slice (BF16 elements: 128-byte rows)
constexpr int kThreads = 128;
constexpr uint32_t kTmemCols = 32;

// A' rows: phases of k point m over the R vectors, [cos | sin] zero padded to
// the segment length. Four segments (kpad = 4 kseg): segment t holds slice t
// (k_tc_planes forms the pairs itself); ten: segment p holds slice tc_pair_a(p).
// One phase is evaluated once and written to every segment.
__global__ void k_phase_split(const double* __restrict__ kpt, const double* __restrict__ Rvec, int nk, int nr, int kseg,
                              int kpad, uint16_t* __restrict__ A) {
  const int m = blockIdx.x;
  const int K = 2 * nr;
  uint16_t* row = A + (size_t)m * kpad;
  for (int q = threadIdx.x; q < kseg; q += blockDim.x) {
    uint16_t sl[kTcSlices] = {0, 0, 0, 0};
    if (m < nk && q < K) {
      const int r = q < nr ? q : q - nr;
      const double kR = kpt[m * 3 + 0] * Rvec[r * 3 + 0] + kpt[m * 3 + 1] * Rvec[r * 3 + 1] + kpt[m * 3 + 2] * Rvec[r * 3 + 2];
      double sn, co;
      sincospi(2.0 * kR, &sn, &co);
      const double y = 0.5 * (q < nr ? co : sn);  // in [-1/2, 1/2]: every slice at most 128 in magnitude
#pragma unroll
      for (int t = 0; t < kTcSlices; t++) sl[t] = tc_bf16(tc_slice(y, t));  // at most 8 significant bits: exact in BF16
    }
    if (kpad == kTcSlices * kseg) {
#pragma unroll
      for (int t = 0; t < kTcSlices; t++) row[(size_t)t * kseg + q] = sl[t];
    } else {
#pragma unroll
      for (int p = 0; p < kTcPairs; p++) row[(size_t)p * kseg + q] = sl[tc_pair_a(p)];
    }
  }
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  // base offset 0, legacy LBO mode, no swizzle (layout type 0)
  return d;
}

// kind::tf32, D FP32, A and B TF32 K-major, M = 128, N = 32
// kind::f16: D FP32 (bits 4-5 = 1), A and B BF16 (bits 7-9 and 10-12 = 1), K-major, M = 128, N = 32
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);

// C (FP64) = A' B'^T. Each K segment (one slice pair) accumulates in FP32 in
// one of two TMEM regions, exactly (every product is an integer times the
// segment's power of two, at most 2^14, and a segment is at most 1024 deep);
// the segment is read back into FP64 registers while the next segment's MMAs
// run in the other region. The 32-deep K slices are staged with cp.async into
// two shared-memory stages: slice s + 1 loads while the tensor core works on
// slice s. Every wait is bounded; a wait that runs out ends the block
// uniformly after its own copies and MMAs have drained.
__device__ __forceinline__ void tc_cp16(uint32_t dst, const void* src, bool pred) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(pred ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(kThreads, 1) k_tc_gemm(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B, double* __restrict__ C,
                                                         int M, int N, int Kp, int kseg, int* err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr uint32_t kStageA = TM * TK * 2, kStageB = TN * TK * 2, kStage = kStageA + kStageB;
  __shared__ unsigned long long bar[2];  // MMAs of the slices staged in stage 0 / 1 have completed
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TN;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(2 * kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  const uint32_t base = smem_u32(smem);
  const int S = Kp / TK, SEG = kseg / TK;
  double acc[TN];
#pragma unroll
  for (int c = 0; c < TN; c++) acc[c] = 0.;

  // slice s -> stage b: row r, 16-byte chunk c at (c * rows + r) * 16 (K-major core matrices)
  auto load = [&](int s, int b) {
    const int k0 = s * TK;
    const uint32_t sa = base + (uint32_t)b * kStage, sb = sa + kStageA;
    for (int q = tid; q < TM * (TK / 8); q += kThreads) {
      const int r = q % TM, c = q / TM;
      const bool in = m0 + r < M;
      tc_cp16(sa + (uint32_t)((c * TM + r) * 16), in ? (const void*)(A + (size_t)(m0 + r) * Kp + k0 + 8 * c) : (const void*)A, in);
    }
    for (int q = tid; q < TN * (TK / 8); q += kThreads) {
      const int r = q % TN, c = q / TN;
      const bool in = n0 + r < N;
      tc_cp16(sb + (uint32_t)((c * TN + r) * 16), in ? (const void*)(B + (size_t)(n0 + r) * Kp + k0 + 8 * c) : (const void*)B, in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // segment p's accumulator (TMEM region p & 1) into FP64 registers: warp w reads
  // lanes 32w..32w+31 (rows m0 + 32w + lane), all TN columns
  auto readout = [&](int p) {
    asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
    for (int c0 = 0; c0 < TN; c0 += 8) {
      uint32_t v[8];
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((p & 1) * kTmemCols + c0);
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                   : "r"(taddr));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int u = 0; u < 8; u++) acc[c0 + u] += (double)__uint_as_float(v[u]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
  };
  // the MMAs of slice s have completed (commit number s >> 1 on bar[s & 1])
  auto mma_done = [&](int s) { return mbar_wait(&bar[s & 1], (uint32_t)((s >> 1) & 1), err); };

  bool ok = true;
  int issued = -1;  // last slice whose MMAs were committed
  load(0, 0);
  for (int s = 0; s < S; s++) {
    const int b = s & 1;
    if (s + 1 < S) {
      // stage b ^ 1 was last read by the MMAs of slice s - 1
      if (s >= 1) ok = mma_done(s - 1) && ok;
      if (__syncthreads_or(!ok)) break;
      load(s + 1, b ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    // this thread's copies of slice s are in; make every thread's visible to the tensor core
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t sa = base + (uint32_t)b * kStage, sb = sa + kStageA;
      const uint32_t dtm = tmem + (uint32_t)(((s / SEG) & 1) * kTmemCols);
#pragma unroll
      for (int j = 0; j < TK / 16; j++) {
        // K = 16 slice j: chunks 2j, 2j+1; LBO = one chunk plane, SBO = 8 rows x 16 bytes
        const uint64_t da = smem_desc(sa + (uint32_t)(2 * j * TM * 16), TM * 16, 128);
        const uint64_t db = smem_desc(sb + (uint32_t)(2 * j * TN * 16), TN * 16, 128);
        const uint32_t accum = (j > 0 || s % SEG != 0) ? 1u : 0u;  // each segment starts from zero
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(dtm),
            "l"(da), "l"(db), "r"(kIdesc), "r"(accum), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&bar[b])) : "memory");
    }
    issued = s;
    // the previous segment is complete once slice s - 1's MMAs are: read it back while
    // this segment's MMAs run in the other region
    // (the readout is warp-collective: the block decides on the wait together)
    if (s > 0 && s % SEG == 0) {
      const bool d = mma_done(s - 1);
      if (__syncthreads_or(!d)) {
        ok = false;
        break;
      }
      readout((s - 1) / SEG);
    }
  }
  if (__syncthreads_or(!ok)) ok = false;
  if (ok && issued == S - 1) {
    const bool d = mma_done(S - 1);
    if (__syncthreads_or(!d)) ok = false;
    else readout((S - 1) / SEG);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (!__syncthreads_or(!ok)) {
    const int row = m0 + warp * 32 + lane;
    if (row < M)
#pragma unroll
      for (int c = 0; c < TN; c++)
        if (n0 + c < N) C[(size_t)row * N + n0 + c] = acc[c];
  } else if (issued >= 0) {
    // drain: the last committed MMAs must finish before their TMEM is released (bounded)
    mma_done(issued);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kTmemCols));
}

// C[k][col] (col = (comp * ntri + e) * 2 + re/im) -> FP32 planes H [ntri][nk], D [3][ntri][nk];
// diagonal imaginary parts are zero (Wannier.h:489-492)
__global__ void k_scatter(const double* __restrict__ C, int nk, int n, int ntri, int ncols, float2* __restrict__ H,
                          float2* __restrict__ D) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int ce = blockIdx.y;  // comp * ntri + e
  if (k >= nk) return;
  const int comp = ce / ntri, e = ce - comp * ntri;
  float2 v = make_float2((float)C[(size_t)k * ncols + 2 * ce], (float)C[(size_t)k * ncols + 2 * ce + 1]);
  bool diag = false;
  for (int i = 0; i < n; i++) diag = diag || (e == i * n - (i * (i - 1)) / 2);
  if (diag) v.y = 0.f;
  if (comp == 0)
    H[(size_t)e * nk + k] = v;
  else
    D[((size_t)(comp - 1) * ntri + e) * nk + k] = v;
}

// FP64 band energies: Re sum_r e^{2 pi i k.R_r} H_ii(R_r), and the FP64 matrix the
// eigensolve uses: the tensor-core off-diagonal (as stored, FP32), diagonal from here.
__global__ void k_diag64(const double* __restrict__ kpt, const double* __restrict__ Rvec, const double2* __restrict__ hdiagR,
                         const float2* __restrict__ H32, int nk, int n, int nr, double* __restrict__ Hdiag,
                         double2* __restrict__ Hused) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y;
  if (k >= nk) return;
  double acc = 0.;
  for (int r = 0; r < nr; r++) {
    const double kR = kpt[k * 3 + 0] * Rvec[r * 3 + 0] + kpt[k * 3 + 1] * Rvec[r * 3 + 1] + kpt[k * 3 + 2] * Rvec[r * 3 + 2];
    double s, c;
    sincospi(2.0 * kR, &s, &c);
    const double2 h = hdiagR[(size_t)i * nr + r];
    acc += c * h.x - s * h.y;
  }
  Hdiag[(size_t)i * nk + k] = acc;
  for (int j = i; j < n; j++) {
    const int e = i * n - (i * (i - 1)) / 2 + (j - i);
    Hused[(size_t)e * nk + k] = (j == i) ? make_double2(acc, 0.) : make_double2(H32[(size_t)e * nk + k].x, H32[(size_t)e * nk + k].y);
  }
}

// ------------------------------------------------------------------ TMA-staged GEMM
// The same exact-slice GEMM with its operand tiles moved by TMA
// (cp.async.bulk.tensor.2d, no multicast; both tensor maps cover this GPU's
// own buffers) in the 128-byte swizzled K-major layout: one box of 64 BF16
// (128 bytes) x 128 rows of A' and one of 64 x 64 rows of B' per 64-deep K
// slice, each landing as 8-row x 128-byte swizzle atoms 1024 bytes apart; the
// MMA descriptors address K step j of the slice at +32 j bytes inside the
// atom. N tile 64, four shared-memory stages; thread 0 issues the MMAs of
// slice s, then the loads of slice s + 3 once slice s - 1's MMAs have freed
// their stage, so three slices are in flight while the tensor core works.
// Every wait is bounded; on a timeout the block waits (bounded) for its issued
// loads and MMAs, releases TMEM and ends.
constexpr int TN2 = 64, kStages2 = 4;
constexpr uint32_t kTmemCols2 = 64;
constexpr uint32_t kIdesc2 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN2 >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}

// K-major operand in 128-byte swizzle atoms (8 rows x 128 bytes, 1024-byte
// aligned, atoms 1024 bytes apart along M / N): stride byte offset 1024, the
// leading offset unused (encoded 1), layout type 2 (128-byte swizzle)
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  d |= (uint64_t)2 << 61;  // 128-byte swizzle
  return d;
}

__global__ void __launch_bounds__(kThreads, 1) k_tc_gemm_tma(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                                                             double* __restrict__ C, int M, int N, int Kp, int kseg, int* err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr uint32_t kStageA = TM * TK * 2, kStageB = TN2 * TK * 2, kStage = kStageA + kStageB;
  __shared__ unsigned long long full[kStages2], mmab[kStages2];
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TN2;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(2 * kTmemCols2));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int b = 0; b < kStages2; b++) {
      mbar_init(&full[b], 1);
      mbar_init(&mmab[b], 1);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  const uint32_t base = (smem_u32(smem) + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
  const int S = Kp / TK, SEG = kseg / TK;
  double acc[TN2];
#pragma unroll
  for (int c = 0; c < TN2; c++) acc[c] = 0.;

  // slice s into stage b: one 64 x 128 box of A', one 64 x 64 box of B' (rows past M, N read as zero)
  auto issue_load = [&](int s, int b) {
    const uint32_t sa = base + (uint32_t)b * kStage, sb = sa + kStageA;
    mbar_expect_tx(&full[b], kStage);
    tma_load_2d(sa, &mapA, s * TK, m0, smem_u32(&full[b]));
    tma_load_2d(sb, &mapB, s * TK, n0, smem_u32(&full[b]));
  };
  auto readout = [&](int p) {
    asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
    for (int c0 = 0; c0 < TN2; c0 += 8) {
      uint32_t v[8];
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((p & 1) * kTmemCols2 + c0);
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                   : "r"(taddr));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int u = 0; u < 8; u++) acc[c0 + u] += (double)__uint_as_float(v[u]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
  };
  // completion number (s / kStages2) of a stage's barrier belongs to slice s
  auto mma_done = [&](int s) { return mbar_wait(&mmab[s % kStages2], (uint32_t)((s / kStages2) & 1), err); };
  auto loaded = [&](int s) { return mbar_wait(&full[s % kStages2], (uint32_t)((s / kStages2) & 1), err); };

  bool ok = true;
  int issued = -1, loads = 0;  // last slice whose MMAs were committed; slices whose loads were issued
  if (tid == 0)
    for (; loads < kStages2 - 1 && loads < S; loads++) issue_load(loads, loads);
  for (int s = 0; s < S; s++) {
    if (tid == 0) {
      if (ok) ok = loaded(s);
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t sa = base + (uint32_t)(s % kStages2) * kStage, sb = sa + kStageA;
        const uint32_t dtm = tmem + (uint32_t)(((s / SEG) & 1) * kTmemCols2);
#pragma unroll
        for (int j = 0; j < TK / 16; j++) {
          // K step j: 16 BF16 = 32 bytes into every 128-byte swizzled row
          const uint64_t da = sw128_desc(sa + (uint32_t)(32 * j));
          const uint64_t db = sw128_desc(sb + (uint32_t)(32 * j));
          const uint32_t accum = (j > 0 || s % SEG != 0) ? 1u : 0u;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.b32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(dtm),
              "l"(da), "l"(db), "r"(kIdesc2), "r"(accum), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&mmab[s % kStages2]))
                     : "memory");
        issued = s;
      }
      // refill: slice s + 3 goes to the stage slice s - 1 used, once its MMAs are done
      // (slice s's MMAs are queued behind them meanwhile)
      if (ok && loads < S) {
        if (loads >= kStages2) ok = mma_done(loads - kStages2);
        if (ok) {
          issue_load(loads, loads % kStages2);
          loads++;
        }
      }
    }
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    // the previous segment is complete with slice s - 1: read it while this one accumulates
    if (s > 0 && s % SEG == 0) {
      const bool d = mma_done(s - 1);
      if (__syncthreads_or(!d)) {
        ok = false;
        break;
      }
      readout((s - 1) / SEG);
    }
  }
  if (__syncthreads_or(!ok)) ok = false;
  if (ok) {
    const bool d = mma_done(S - 1);
    if (__syncthreads_or(!d)) ok = false;
    else readout((S - 1) / SEG);
  }
  if (!__syncthreads_or(!ok)) {
    const int row = m0 + warp * 32 + lane;
    if (row < M)
#pragma unroll
      for (int c = 0; c < TN2; c++)
        if (n0 + c < N) C[(size_t)row * N + n0 + c] = acc[c];
  } else if (tid == 0) {
    // drain (bounded): issued loads land and committed MMAs finish before the stages and TMEM go away
    for (int s = issued + 1; s < loads; s++) loaded(s);
    if (issued >= 0) mma_done(issued);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kTmemCols2));
}

// ------------------------------------------------------- warp-specialised form
// H and D planes straight from the four slices of each operand. The pair
// segments of the forms above load every slice up to four times (983 KB per
// 128 x 64 tile at 121 R vectors), read the accumulator back into FP64
// registers after every pair, and write C for a second kernel to scatter. Here
// a 64-deep chunk of all four slices of both operands is loaded once and its
// ten pair products are formed from shared memory. Pairs of one a + b have the
// same power of two and share an accumulator: over a group of kGroup3 chunks
// its sums are at most 4 x 256 = 1024 deep, so they are still exact. The four
// accumulators are read back once per group (one group up to 128 R vectors) and
// added in FP64, exact too (25 bits each, 8 bits apart): the results have the
// bits of the other forms. They go to the planes, lanes along k.
// Tile 128 x 80: the 288 columns of 8 bands are four tiles, so 64 x 64 k points
// are 128 CTAs, one wave. A chunk is 104 KB, two of them one CTA's shared
// memory, whose bandwidth bounds the products: the B slices of a chunk lie one
// after another, and so do the accumulators, so that slice a of A meets up to
// three B slices in one MMA (N 160, 160, 240, 160, 80 for a = 0, 0, 1, 2, 3) and
// is read five times in all instead of ten. Read-back and stores take eight warps
// and rolled loops: unrolled, their instruction fetches took 40 % of the kernel.
// 8 bands, 121 R vectors, 64 x 64 k points: 11.1 us (16.4 with one MMA per
// pair, four read-back warps and unrolled loops); with pair segments and these
// roles 39.5 us and 6.6 us for the scatter.
// Roles: warp 8 (one lane) loads a chunk onto two barriers, first what the
// first MMAs need; warp 9 (one lane) issues the MMAs; warps 0-7 read back 32
// TMEM lanes and 40 columns each. Every wait is bounded; a role that times out
// raises a shared abort flag and stops, the others stop at their next wait, and
// before TMEM and shared memory are released the last loads and the last commit
// are waited for (bounded).
constexpr int kWsThreads = 320;
constexpr int TN3 = 80, kStages3 = 2, kGroup3 = 4, kTmemCols3 = 512;
constexpr uint32_t kSliceA3 = TM * TK * 2, kSliceB3 = TN3 * TK * 2, kStage3 = kTcSlices * (kSliceA3 + kSliceB3);
constexpr uint32_t kFirst3 = kSliceA3 + 2 * kSliceB3;  // A slice 0, B slices 0 and 1
constexpr size_t kPlanesSmem = (size_t)kStages3 * kStage3 + 1024;
static_assert(kSliceA3 % 1024 == 0 && kSliceB3 % 1024 == 0, "swizzle atoms are 1024 bytes");
static_assert(kTcSlices * kGroup3 * TK <= 1024, "exact FP32 sums");
static_assert(kTcSlices == 4 && kTcSlices * TN3 <= kTmemCols3 && 3 * TN3 <= 256 && TN3 % 16 == 0, "MMA shapes");

__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// T is double2 (velocity gauge) or float2 (batch tables); MULTI: more than one
// group, whose sums meet in registers
template <class T, bool MULTI>
__global__ void __launch_bounds__(kWsThreads, 1) k_tc_planes(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                                                             T* __restrict__ H, T* __restrict__ D, int nk, int n, int ntri, int kseg,
                                                             int* err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ unsigned long long full[kStages3][2], empty[kStages3], accf, acce;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag, loads_issued, commits;
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TN3, N = 8 * ntri;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(kTmemCols3));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mapA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mapB) : "memory");
    for (int b = 0; b < kStages3; b++) {
      mbar_init(&full[b][0], 1);
      mbar_init(&full[b][1], 1);
      mbar_init(&empty[b], 1);
    }
    mbar_init(&accf, 1);
    mbar_init(&acce, 8);  // one arrival per read-back warp
    abort_flag = 0;
    loads_issued = 0;
    commits = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  const uint32_t base = (smem_u32(smem) + 1023u) & ~1023u;
  pdl_wait();  // the coefficient slices; the set-up above overlaps the kernel that cuts them
  const int chunks = kseg / TK;
  volatile int* abortp = &abort_flag;

  if (warp == 8) {
    if (lane == 0) {
      int c = 0;
#pragma unroll 1
      for (; c < chunks; c++) {
        const int st = c % kStages3;
        if (*abortp) break;
        if (c >= kStages3 && !mbar_wait(&empty[st], (uint32_t)((c / kStages3 - 1) & 1), err)) {
          *abortp = 1;
          break;
        }
        const uint32_t sa = base + (uint32_t)st * kStage3, sb = sa + kTcSlices * kSliceA3;
        mbar_expect_tx(&full[st][0], kFirst3);
        mbar_expect_tx(&full[st][1], kStage3 - kFirst3);
#pragma unroll 1
        for (int q = 0; q < 2 * kTcSlices; q++) {
          // A0, B0, B1 | B2, B3, A1, A2, A3
          const bool isA = q == 0 || q > kTcSlices;
          const int t = isA ? (q == 0 ? 0 : q - kTcSlices) : q - 1;
          const uint32_t bar = smem_u32(&full[st][q < 3 ? 0 : 1]);
          if (isA)
            tma_load_2d(sa + (uint32_t)t * kSliceA3, &mapA, t * kseg + c * TK, m0, bar);
          else
            tma_load_2d(sb + (uint32_t)t * kSliceB3, &mapB, t * kseg + c * TK, n0, bar);
        }
      }
      loads_issued = c;
    }
  } else if (warp == 9) {
    if (lane == 0) {
      int c = 0;
#pragma unroll 1
      for (; c < chunks; c++) {
        const int st = c % kStages3;
        const uint32_t par = (uint32_t)((c / kStages3) & 1);
        if (*abortp) break;
        bool ok = true;
        // a group reuses the accumulators of the one before: wait for their read-back
        if (MULTI && c % kGroup3 == 0 && c > 0) ok = mbar_wait(&acce, (uint32_t)((c / kGroup3 - 1) & 1), err);
        const uint64_t da0 = sw128_desc(base + (uint32_t)st * kStage3);
        const uint64_t db0 = sw128_desc(base + (uint32_t)st * kStage3 + kTcSlices * kSliceA3);
#pragma unroll 1
        for (int p = 0; p <= kTcSlices && ok; p++) {
          // slice a of A with slices b .. b + nb - 1 of B into accumulators a + b ..
          const int a = p < 2 ? 0 : p - 1, b = p == 1 ? 2 : 0, nb = p < 2 ? 2 : kTcSlices - a;
          if (p < 2) ok = mbar_wait(&full[st][p], par, err);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t idesc =
              (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nb * (TN3 >> 3)) << 17) | ((uint32_t)(TM >> 4) << 24);
          const uint32_t dtm = tmem + (uint32_t)((a + b) * TN3);
          const uint64_t da = da0 + (uint64_t)(a * (kSliceA3 >> 4)), db = db0 + (uint64_t)(b * (kSliceB3 >> 4));
          const uint32_t first = c % kGroup3 == 0 && p < 2 ? 0u : 1u;  // starts two accumulators
#pragma unroll
          for (int j = 0; j < TK / 16; j++) {
            // K step j: 32 bytes into every 128-byte swizzled row
            const uint32_t accum = j > 0 ? 1u : first;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(dtm),
                "l"(da + (uint64_t)(2 * j)), "l"(db + (uint64_t)(2 * j)), "r"(idesc), "r"(accum), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
          }
        }
        // (also on the way out: what was issued ends before its stage and TMEM are released)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&empty[st]))
                     : "memory");
        commits = c + 1;
        if (!ok) {
          *abortp = 1;
          break;
        }
        if (c % kGroup3 == kGroup3 - 1 || c == chunks - 1)
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&accf)) : "memory");
      }
    }
  } else {
    // warp w: TMEM lanes 32 (w % 4) .. + 31, k points m0 + 32 (w % 4) + lane; columns 40 (w / 4) .. + 39
    constexpr int kCols = TN3 / 2;
    const int k = m0 + (warp % 4) * 32 + lane, col0 = (warp / 4) * kCols;
    const uint32_t trow = tmem + ((uint32_t)((warp % 4) * 32) << 16) + (uint32_t)col0;
    // column pair 2 ce, 2 ce + 1 = Re, Im of component and element ce = comp * ntri + e: planes
    // 0 .. ntri - 1 are H, the following D; e's row i of the upper triangle begins at its diagonal
    // element ed, whose imaginary part is zero (Wannier.h:489-492)
    int ce = (n0 + col0) / 2, e = ce % ntri, i = 0, ed = 0;
    while (e >= ed + n - i) ed += n - i++;
    auto store8 = [&](const double* z) {
#pragma unroll
      for (int u = 0; u < 8; u += 2, ce++) {
        T o;
        o.x = z[u];
        o.y = e == ed ? 0. : z[u + 1];
        if (k < nk && 2 * ce < N) (ce < ntri ? H + (size_t)ce * nk : D + (size_t)(ce - ntri) * nk)[k] = o;
        if (++e == ed + n - i) ed += n - i++;
        if (e == ntri) e = i = ed = 0;
      }
    };
    // the four accumulators of columns c0 .. c0 + 7, added to z
    auto read8 = [&](int c0, double* z) {
      uint32_t v[kTcSlices][8];
#pragma unroll
      for (int t = 0; t < kTcSlices; t++)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v[t][0]), "=r"(v[t][1]), "=r"(v[t][2]), "=r"(v[t][3]), "=r"(v[t][4]), "=r"(v[t][5]), "=r"(v[t][6]),
                       "=r"(v[t][7])
                     : "r"(trow + (uint32_t)(t * TN3 + c0)));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int t = 0; t < kTcSlices; t++)
#pragma unroll
        for (int u = 0; u < 8; u++) z[u] += (double)__uint_as_float(v[t][u]);
    };
    auto finished = [&](int g) {
      const bool ok = !*abortp && mbar_wait(&accf, (uint32_t)(g & 1), err);
      if (__any_sync(0xffffffffu, !ok)) {
        if (lane == 0) *abortp = 1;
        return false;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      return true;
    };
    if (!MULTI) {
      if (finished(0))
#pragma unroll 1
        for (int c0 = 0; c0 < kCols; c0 += 8) {
          double z[8] = {0., 0., 0., 0., 0., 0., 0., 0.};
          read8(c0, z);
          store8(z);
        }
    } else {
      const int groups = (chunks + kGroup3 - 1) / kGroup3;
      double acc[kCols];
#pragma unroll
      for (int c = 0; c < kCols; c++) acc[c] = 0.;
      int g = 0;
      for (; g < groups && finished(g); g++) {
#pragma unroll
        for (int c0 = 0; c0 < kCols; c0 += 8) read8(c0, acc + c0);
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acce);
      }
      if (g == groups)
#pragma unroll
        for (int c0 = 0; c0 < kCols; c0 += 8) store8(acc + c0);
    }
  }
  __syncthreads();
  if (*abortp) {
    // the last loads issued (one chunk per stage at most is outstanding) land before the stages go away
    if (tid == 256)
      for (int c = loads_issued - kStages3 < 0 ? 0 : loads_issued - kStages3; c < loads_issued; c++)
        for (int t = 0; t < 2; t++) mbar_wait(&full[c % kStages3][t], (uint32_t)((c / kStages3) & 1), err);
    // and the last committed MMAs finish before their TMEM is released
    if (tid == 288 && commits > 0) mbar_wait(&empty[(commits - 1) % kStages3], (uint32_t)(((commits - 1) / kStages3) & 1), err);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols3));
}

// Coefficient slices of c_A(R) = e^{2 pi i A.R} c(R) (velocity gauge; the model
// build of a batch instance has A = 0, where c_A = c exactly), one thread per
// (column, K entry); column 2 ce + part holds [Re c_A ; -Im c_A] (part 0) or
// [Im c_A ; Re c_A] (part 1), divided by the column's scale, cut and pre-multiplied
// by 2 scale (the phases enter halved); segments as in k_phase_split. 2.1 us for 8 bands and 121 R vectors; cut
// on the host for every admitted instance it was 3 ms of one core.
__global__ void k_bslices(const double2* __restrict__ coef, const double* __restrict__ Rvec, const double* __restrict__ colscale,
                             double A0, double A1, double A2, int ntri, int nr, int kseg, int kpad, uint16_t* __restrict__ B) {
  pdl_trigger();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;  // K entry
  const int col = blockIdx.y;                          // 2 (comp * ntri + e) + part
  const int K = 2 * nr;
  if (q >= K) return;
  const int ce = col / 2, part = col % 2;
  const int r = q < nr ? q : q - nr;
  const double* R = Rvec + (size_t)r * 3;
  double s, c;
  sincospi(2.0 * (A0 * R[0] + A1 * R[1] + A2 * R[2]), &s, &c);
  const double2 cf = coef[(size_t)ce * nr + r];
  const double re = c * cf.x - s * cf.y, im = c * cf.y + s * cf.x;
  const double v = part == 0 ? (q < nr ? re : -im) : (q < nr ? im : re);
  const double scale = colscale[col];
  uint16_t* row = B + (size_t)col * kpad;
  uint16_t sl[kTcSlices];
#pragma unroll
  for (int t = 0; t < kTcSlices; t++) sl[t] = tc_bf16(2.0 * scale * tc_slice(v / scale, t));
  if (kpad == kTcSlices * kseg) {
#pragma unroll
    for (int t = 0; t < kTcSlices; t++) row[(size_t)t * kseg + q] = sl[t];
  } else {
#pragma unroll
    for (int p = 0; p < kTcPairs; p++) row[(size_t)p * kseg + q] = sl[tc_pair_b(p)];
  }
}

// C[k][col] -> FP64 planes H [ntri][nk], D [3][ntri][nk]; diagonal imaginary parts zero
__global__ void k_scatter64(const double* __restrict__ C, int nk, int n, int ntri, int ncols, double2* __restrict__ H,
                            double2* __restrict__ D) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int ce = blockIdx.y;
  if (k >= nk) return;
  const int comp = ce / ntri, e = ce - comp * ntri;
  double2 v = make_double2(C[(size_t)k * ncols + 2 * ce], C[(size_t)k * ncols + 2 * ce + 1]);
  bool diag = false;
  for (int i = 0; i < n; i++) diag = diag || (e == i * n - (i * (i - 1)) / 2);
  if (diag) v.y = 0.;
  if (comp == 0)
    H[(size_t)e * nk + k] = v;
  else
    D[((size_t)(comp - 1) * ntri + e) * nk + k] = v;
}

}  // namespace

size_t tc_gemm_smem() { return 2 * sizeof(uint16_t) * (TM + TN) * TK + 1024; }

int tc_seg_k(int nr) { return ((2 * nr + TK - 1) / TK) * TK; }
int tc_depth(int nr, TcForm form) { return (form == TcForm::planes ? kTcSlices : kTcPairs) * tc_seg_k(nr); }
size_t tc_c_size(int nk, int ntri, TcForm form) { return form == TcForm::planes ? 0 : (size_t)nk * 8 * ntri; }

namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static const EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return (EncodeTiledFn)p;
    cudaGetLastError();
    return nullptr;
  }();
  return fn;
}

// rows x Kp BF16 operand (K contiguous; Kp a multiple of 64), boxes of 64 x
// box_rows in 128-byte swizzle atoms; out-of-range rows read as zero
cudaError_t encode_operand(CUtensorMap* map, const uint16_t* ptr, int rows, int Kp, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return cudaErrorNotSupported;
  const cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)Kp * sizeof(uint16_t)};
  const cuuint32_t box[2] = {(cuuint32_t)TK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1u, 1u};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

size_t tma_gemm_smem() { return (size_t)kStages2 * (TM + TN2) * TK * 2 + 1024; }

void launch_scatter(const double* C, int nk, int n, int ntri, float2* H, float2* D, cudaStream_t s) {
  k_scatter<<<dim3((nk + 255) / 256, 4 * ntri), 256, 0, s>>>(C, nk, n, ntri, 8 * ntri, H, D);
}
void launch_scatter(const double* C, int nk, int n, int ntri, double2* H, double2* D, cudaStream_t s) {
  k_scatter64<<<dim3((nk + 255) / 256, 4 * ntri), 256, 0, s>>>(C, nk, n, ntri, 8 * ntri, H, D);
}

// H and D planes from A' and B' in the layout of o.form
template <class T>
cudaError_t gemm_planes(const TcOperands& o, T* H, T* D, int nk, int n, int ntri, int nr, int* err, cudaStream_t s) {
  const int ncols = 8 * ntri, kpad = tc_depth(nr, o.form), kseg = tc_seg_k(nr);
  cudaError_t e;
  if (o.form == TcForm::planes) {
    auto kern = kseg > kGroup3 * TK ? k_tc_planes<T, true> : k_tc_planes<T, false>;
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlanesSmem)) != cudaSuccess) return e;
    return launch_pdl(kern, dim3((nk + TM - 1) / TM, (ncols + TN3 - 1) / TN3), dim3(kWsThreads), kPlanesSmem, s, o.mapA, o.mapB, H, D, nk, n,
                      ntri, kseg, err);
  }
  if (o.form == TcForm::tma) {
    if ((e = cudaFuncSetAttribute(k_tc_gemm_tma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tma_gemm_smem())) != cudaSuccess)
      return e;
    k_tc_gemm_tma<<<dim3((nk + TM - 1) / TM, (ncols + TN2 - 1) / TN2), kThreads, tma_gemm_smem(), s>>>(o.mapA, o.mapB, o.C, nk, ncols, kpad,
                                                                                                      kseg, err);
  } else {
    // about 55 KB of shared memory per CTA keeps at most four CTAs (256 of the 512 TMEM columns) per SM
    const size_t smem = std::max(tc_gemm_smem(), (size_t)56 * 1024);
    if ((e = cudaFuncSetAttribute(k_tc_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
    k_tc_gemm<<<dim3((nk + TM - 1) / TM, (ncols + TN - 1) / TN), kThreads, smem, s>>>(o.A, o.B, o.C, nk, ncols, kpad, kseg, err);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  launch_scatter(o.C, nk, n, ntri, H, D, s);
  return cudaGetLastError();
}

// phase slices of the grid, zero segment padding of the coefficient slices
cudaError_t prepare(const TcOperands& o, const double* kpt, const double* Rvec, int nk, int ntri, int nr, cudaStream_t s) {
  const int kpad = tc_depth(nr, o.form), ncols = 8 * ntri;
  k_phase_split<<<nk, 256, 0, s>>>(kpt, Rvec, nk, nr, tc_seg_k(nr), kpad, o.A);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemsetAsync(o.B, 0, sizeof(uint16_t) * (size_t)ncols * kpad, s);
  return e;
}

cudaError_t cut_coefficients(const TcOperands& o, const double2* coef, const double* Rvec, const double* colscale, const double A[3], int ntri,
                             int nr, cudaStream_t s) {
  k_bslices<<<dim3((2 * nr + 127) / 128, 8 * ntri), 128, 0, s>>>(coef, Rvec, colscale, A[0], A[1], A[2], ntri, nr, tc_seg_k(nr),
                                                                tc_depth(nr, o.form), o.B);
  return cudaGetLastError();
}

}  // namespace

// The warp-specialised form unless EDUS_TC_GEMM selects another (or the driver
// has no tensor maps: cp.async). 64 x 64 k points, 8 bands: 11.1 us against
// 61.9 us for the single-issuer TMA form and 93 us for the cp.async form,
// scatter included; all three give bit-identical planes (every FP32 sum is exact).
TcForm tc_gemm_form() {
  const char* form = std::getenv("EDUS_TC_GEMM");
  if ((form && std::strcmp(form, "cpasync") == 0) || !encode_fn()) return TcForm::cpasync;
  if (form && std::strcmp(form, "tma") == 0) return TcForm::tma;
  return TcForm::planes;
}

bool tc_maps(TcOperands& o, int nk, int ntri, int nr) {
  if (o.form == TcForm::cpasync) return true;
  const int kpad = tc_depth(nr, o.form);
  return encode_operand(&o.mapA, o.A, nk, kpad, TM) == cudaSuccess &&
         encode_operand(&o.mapB, o.B, 8 * ntri, kpad, o.form == TcForm::planes ? TN3 : TN2) == cudaSuccess;
}

cudaError_t tc_contract(const TcArgs& a, cudaStream_t s) {
  const double zero[3] = {0., 0., 0.};
  cudaError_t e = prepare(a.op, a.kpt, a.Rvec, a.nk, a.ntri, a.nr, s);
  if (e == cudaSuccess) e = cut_coefficients(a.op, a.coef, a.Rvec, a.colscale, zero, a.ntri, a.nr, s);
  if (e == cudaSuccess) e = gemm_planes(a.op, a.H32, a.D32, a.nk, a.n, a.ntri, a.nr, a.err, s);
  if (e != cudaSuccess) return e;
  k_diag64<<<dim3((a.nk + 127) / 128, a.n), 128, 0, s>>>(a.kpt, a.Rvec, a.hdiagR, a.H32, a.nk, a.n, a.nr, a.Hdiag, a.Hused);
  return cudaGetLastError();
}

cudaError_t tc_vg_prepare(const TcVgArgs& a, cudaStream_t s) { return prepare(a.op, a.kpt, a.Rvec, a.nk, a.ntri, a.nr, s); }

cudaError_t tc_vg_stage(const TcVgArgs& a, cudaStream_t s) {
  cudaError_t e = cut_coefficients(a.op, a.coef, a.Rvec, a.colscale, a.A, a.ntri, a.nr, s);
  if (e == cudaSuccess) e = gemm_planes(a.op, a.H, a.D, a.nk, a.n, a.ntri, a.nr, a.err, s);
  return e;
}

}  // namespace batch
}  // namespace edus
