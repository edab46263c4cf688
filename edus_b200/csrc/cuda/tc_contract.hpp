// tc_contract.hpp — tensor-core (tcgen05, exact BF16 slices) Wannier contraction.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstring>
#include <stddef.h>

#include <algorithm>

namespace edus {
namespace batch {

// GEMM forms (tc_contract.cu): `planes` has one K segment per slice in A and B and
// writes the planes itself, the others one per slice pair and a result C.
enum class TcForm { planes, tma, cpasync };
TcForm tc_gemm_form();
int tc_seg_k(int nr);                                   // K segment length: 2 nr padded to the 64-deep K slice
int tc_depth(int nr, TcForm form);                      // row length of A and B
size_t tc_c_size(int nk, int ntri, TcForm form);        // doubles in C

// Operands and scratch of a contraction, laid out for `form`
struct TcOperands {
  TcForm form = TcForm::cpasync;
  uint16_t* A = nullptr;  // [nk][tc_depth] phase slices (BF16)
  uint16_t* B = nullptr;  // [8 ntri][tc_depth] coefficient slices (BF16)
  double* C = nullptr;    // [nk][8 ntri], none for `planes`
  CUtensorMap mapA{}, mapB{};
};

struct TcArgs {
  int n, ntri, nk, nr;
  const double* kpt;     // [nk][3]
  const double* Rvec;    // [nr][3]
  const double2* coef;   // [4][ntri][nr]: H(R), (r_x(R) + r_x(R)^T) / 2 upper entries
  const double* colscale;  // [8 ntri] power-of-two scale of each GEMM column
  const double2* hdiagR; // [n][nr] H_ii(R) for the FP64 band energies
  TcOperands op;
  float2* H32;           // out [ntri][nk]
  float2* D32;           // out [3][ntri][nk]
  double* Hdiag;         // out [n][nk] FP64 band energies
  double2* Hused;        // out [ntri][nk] FP64 matrix the dynamics uses (for the eigensolve)
  int* err;              // device error word (bounded waits)
};

// Exact-slice form of the contraction. Every operand y (half a phase cos / sin,
// or a coefficient divided by its column's power-of-two scale) lies in
// [-1/2, 1/2] and is cut into kTcSlices slices of at most 8 significant bits,
// slice s a multiple of 2^-(8 s + 8) and at most 128 in magnitude:
// y = sum_s slice_s(y) + O(2^-33); every slice is exact in BF16. The GEMM runs
// one K segment per slice pair (or per value of a + b)
// (a, b) with a + b < kTcSlices; inside a segment every product is an integer
// times one power of two, at most 2^14 in magnitude, so the tensor core's FP32
// sums over a segment of up to 1024 are exact and the FP64 sum of the segments
// is the contraction to about 2^-32 of its terms.
constexpr int kTcSlices = 4;
constexpr int kTcPairs = 10;  // (a, b) with a + b <= 3
__host__ __device__ constexpr int tc_pair_a(int p) {
  return p == 0 ? 0 : p == 1 ? 0 : p == 2 ? 1 : p == 3 ? 0 : p == 4 ? 1 : p == 5 ? 2 : p == 6 ? 0 : p == 7 ? 1 : p == 8 ? 2 : 3;
}
__host__ __device__ constexpr int tc_pair_b(int p) {
  return p == 0 ? 0 : p == 1 ? 1 : p == 2 ? 0 : p == 3 ? 2 : p == 4 ? 1 : p == 5 ? 0 : p == 6 ? 3 : p == 7 ? 2 : p == 8 ? 1 : 0;
}
// slice s of y in [-1, 1] (FP64 arithmetic, exact at every step)
__host__ __device__ inline double tc_slice(double y, int s) {
  double r = y, v = 0.;
  double scale = 256.;
  for (int t = 0; t <= s; t++) {
    v = rint(r * scale) / scale;
    r -= v;
    scale *= 256.;
  }
  return v;
}
// BF16 bit pattern of a value with at most 8 significant bits (exact: the low
// 16 bits of its FP32 pattern are zero)
__host__ __device__ inline uint16_t tc_bf16(double v) {
  const float f = (float)v;
  uint32_t u;
  memcpy(&u, &f, 4);
  return (uint16_t)(u >> 16);
}
// Tensor maps of A and B. False where the driver has none for these operands: the
// caller then lays them out for `cpasync`, which needs no maps.
bool tc_maps(TcOperands& o, int nk, int ntri, int nr);
cudaError_t tc_contract(const TcArgs& a, cudaStream_t s);

// Velocity gauge on the tensor cores: H(k + A), D(k + A) of every k point for
// every RK4 stage as the exact-slice GEMM above. The phase slices of the grid
// (A' = [cos | sin](2 pi k.R) / 2) are cut once; each stage cuts the
// coefficient slices of c_A(R) = e^{2 pi i A.R} c(R) on the device (column
// scales fixed from |c(R)|, which bounds |Re c_A| and |Im c_A| for every A),
// runs the GEMM into FP64 planes (diagonal imaginary parts zero).
struct TcVgArgs {
  int n = 0, ntri = 0, nk = 0, nr = 0;
  const double* kpt = nullptr;       // [nk][3]
  const double* Rvec = nullptr;      // [nr][3]
  const double2* coef = nullptr;     // [4][ntri][nr]: H(R), (r_x(R) + r_x(R)^T) / 2 upper entries
  const double* colscale = nullptr;  // [8 ntri] power-of-two scale of each GEMM column
  double A[3] = {0, 0, 0};           // crystal coordinates
  TcOperands op;                     // phase slices and segment padding set by tc_vg_prepare
  double2* H = nullptr;              // out [ntri][nk]
  double2* D = nullptr;              // out [3][ntri][nk]
  int* err = nullptr;                // device error word (bounded waits)
};
cudaError_t tc_vg_prepare(const TcVgArgs& a, cudaStream_t s);
cudaError_t tc_vg_stage(const TcVgArgs& a, cudaStream_t s);

}  // namespace batch
}  // namespace edus
