// C[M,N] (+)= A[M,K] · W[N,K]^T in true 32-bit on the CUDA cores: the two fast bodies behind
// cretif_gemm_simt for float operands whose rows are 16-byte aligned (gemm_simt.cu takes the rest).
//
// Both use the two-wide multiply-add (fma.rn.f32x2) along k: one 16-byte load of a row is two
// operand pairs as it lies, and a sum is kept as two chains (even and odd k) that meet at the
// end, so no operand is ever duplicated or moved.
//
// * gemm_f32_few (M <= kFewRows): a step of few tokens is bound by reading W once.  A warp owns
//   kR = 4 rows of W and 1, 2, 4 or 8 rows of A; its lanes stride k by 16-byte loads (512 bytes of
//   a W row an instruction); WK warps of a CTA share a row group's k range when N alone gives
//   too few warps to keep loads in flight.  WK depends on N and K only, so a row's result does
//   not depend on how many rows are in the call.  More than 8 rows: the row tiles of one group
//   of W rows are neighbours in the grid and read it from L2.
// * gemm_f32_tile: WM x WN warps, 32 x 32 outputs a warp (8 x 4 a thread: 12 shared 16-byte
//   loads feed 64 two-wide FMAs), slabs of 32 k through a three-stage cp.async ring with rows of
//   36 floats (eight consecutive rows lie in different banks).  KS > 1: the warps of a CTA take
//   the slabs of one 32 x 32 tile in turn and their sums meet in shared memory; that is for
//   grids of so few tiles that 64 x 64 ones would leave SMs idle.
//   A slab's 32 products are summed in two chains of their own before they join the running sum.
//
// Measured beside the 64 x 64 kernel of gemm_simt.cu (one B200, weights not in L2, us before ->
// now; M x N x K).  Few rows: 1 x 49152 x 576 154 -> 22 (5.2 TB/s), 8 x 49152 x 576 157 -> 37,
// 3 x 576 x 1536 111 -> 3.8, 3 x 3072 x 576 43 -> 7.1, 8 x 2048 x 8192 589 -> 21.  Tiles:
// 578 x 3072 x 576 112 -> 72, 2048 x 3072 x 576 302 -> 189, 2048 x 16384 x 2048 5406 -> 3271
// (42 TFLOP/s of the 74 that 128 FMA lanes an SM give); 8 x 8 outputs a thread need 255 registers
// and are no faster.  The error against 64 bits is 0.6 to 0.8 of the old kernel's (8.6e-8 and
// 1.0e-7 against 1.3e-7 at K = 576).
#include "api.h"
#include "common.cuh"
#include "gemm_f32.h"

namespace cretif {

constexpr int kFewRows = 64;
constexpr int kR = 4;                 // rows of W a warp
constexpr int kFewWarps = 8;

// The sums of NV values over a warp's lanes; the lane whose number's top bits are i gets value i
// (NV = 32: lane i).  NV - 1 + log2(32 / NV) shuffles.
template <int NV>
__device__ __forceinline__ float warp_sums(float (&v)[NV], int lane) {
  int off = 16;
#pragma unroll
  for (int n = NV / 2; n > 0; n >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n];
      const float keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  float r = v[0];
  for (; off > 0; off >>= 1) r += __shfl_xor_sync(0xffffffffu, r, off);
  return r;
}

template <int MT>
__global__ void __launch_bounds__(kFewWarps * 32)
gemm_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                    int M, int N, int K, int lda, int ldw, int ldc, int accumulate, int WK) {
  dependent_begin();
  constexpr int NV = kR * MT;
  __shared__ float part[kFewWarps][NV];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / WK, wk = warp - group * WK;
  const int n0 = ((int)blockIdx.y * (kFewWarps / WK) + group) * kR;
  const int m0 = (int)blockIdx.x * MT;
  const float* wp[kR];
  const float* ap[MT];
#pragma unroll
  for (int r = 0; r < kR; ++r) wp[r] = W + (size_t)min(n0 + r, N - 1) * ldw;
#pragma unroll
  for (int m = 0; m < MT; ++m) ap[m] = A + (size_t)min(m0 + m, M - 1) * lda;
  float2 acc[kR][MT];
#pragma unroll
  for (int r = 0; r < kR; ++r)
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[r][m] = make_float2(0.f, 0.f);
  // rows beyond N or M read the last row's numbers; their sums are not stored
#pragma unroll 2
  for (int k = wk * 128 + lane * 4; k < K; k += WK * 128) {
    float4 w[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) w[r] = __ldg(reinterpret_cast<const float4*>(wp[r] + k));
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const float4 a = *reinterpret_cast<const float4*>(ap[m] + k);
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        acc[r][m] = __ffma2_rn(make_float2(a.x, a.y), make_float2(w[r].x, w[r].y), acc[r][m]);
        acc[r][m] = __ffma2_rn(make_float2(a.z, a.w), make_float2(w[r].z, w[r].w), acc[r][m]);
      }
    }
  }
  float v[NV];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int r = 0; r < kR; ++r) v[m * kR + r] = acc[r][m].x + acc[r][m].y;
  float s = warp_sums(v, lane);
  constexpr int kPer = 32 / NV;               // lanes that hold the same sum
  const int at = lane / kPer;
  if (WK > 1) {
    if (lane % kPer == 0) part[warp][at] = s;
    __syncthreads();
    if (wk != 0) return;
    s = 0.f;
    for (int i = 0; i < WK; ++i) s += part[warp + i][at];
  }
  const int m = m0 + at / kR, n = n0 + at % kR;
  if (lane % kPer == 0 && m < M && n < N) {
    float* c = C + (size_t)m * ldc + n;
    *c = accumulate ? *c + s : s;
  }
}

constexpr int kSlab = 32;             // k's a slab
constexpr int kRow = kSlab + 4;       // floats a row of it takes in shared memory
// stages of the ring: a CTA that shares a slab range among its warps takes two (74 KB, so that
// three of them share an SM and hide each other's loads), the other three
constexpr int ring_of(int KS) { return KS > 1 ? 2 : 3; }

__device__ __forceinline__ void copy16(float* dst, const float* src, bool real) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
               "r"(real ? 16 : 0) : "memory");
}

template <int WM, int WN, int KS>
__global__ void __launch_bounds__(32 * WM * WN * KS)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                     int M, int N, int K, int lda, int ldw, int ldc, int accumulate) {
  constexpr int BM = 32 * WM, BN = 32 * WN, kThreads = 32 * WM * WN * KS;
  constexpr int kStage = KS * (BM + BN) * kRow, kRing = ring_of(KS);       // (floats)
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ks = warp / (WM * WN), wm = (warp % (WM * WN)) / WN, wn = warp % WN;
  const int ty = lane >> 3, tx = lane & 7;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int rounds = (K + KS * kSlab - 1) / (KS * kSlab);

  auto fetch = [&](int round) {
    float* st = sm + (round % kRing) * kStage;
    // KS slabs of BM rows of A and BN rows of W, eight 16-byte pieces a row
#pragma unroll
    for (int i = tid; i < KS * (BM + BN) * 8; i += kThreads) {
      const int piece = i & 7, row = (i >> 3) % (BM + BN), s = (i >> 3) / (BM + BN);
      const int k = (round * KS + s) * kSlab + piece * 4;
      const bool is_a = row < BM;
      const int at = is_a ? m0 + row : n0 + row - BM;
      const bool real = k < K && at < (is_a ? M : N);
      const float* src = is_a ? A + (size_t)(real ? at : 0) * lda : W + (size_t)(real ? at : 0) * ldw;
      copy16(st + (s * (BM + BN) + row) * kRow + piece * 4, src + (real ? k : 0), real);
    }
  };

  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int r = 0; r < kRing - 1; ++r) {
    if (r < rounds) fetch(r);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int round = 0; round < rounds; ++round) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
    __syncthreads();            // this round's slabs are there, the last round's are read no more
    if (round + kRing - 1 < rounds) fetch(round + kRing - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* as = sm + (round % kRing) * kStage + (ks * (BM + BN) + wm * 32 + ty) * kRow;
    const float* ws = sm + (round % kRing) * kStage + (ks * (BM + BN) + BM + wn * 32 + tx) * kRow;
    float2 part[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) part[i][j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int kk = 0; kk < kSlab; kk += 4) {
      float4 w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const float4*>(ws + 8 * j * kRow + kk);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(as + 4 * i * kRow + kk);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          part[i][j] = __ffma2_rn(make_float2(a.x, a.y), make_float2(w[j].x, w[j].y), part[i][j]);
          part[i][j] = __ffma2_rn(make_float2(a.z, a.w), make_float2(w[j].z, w[j].w), part[i][j]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j].x + part[i][j].y;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (KS > 1) {
    __syncthreads();            // the ring is free: the warps' sums meet there, in their order
    if (ks > 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          sm[(((ks - 1) * WM * WN + warp % (WM * WN)) * 32 + i * 4 + j) * 32 + lane] = acc[i][j];
    }
    __syncthreads();
    if (ks > 0) return;
#pragma unroll
    for (int s = 1; s < KS; ++s)
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          acc[i][j] += sm[(((s - 1) * WM * WN + warp) * 32 + i * 4 + j) * 32 + lane];
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + wm * 32 + ty + 4 * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + wn * 32 + tx + 8 * j;
      if (n >= N) continue;
      float* c = C + (size_t)m * ldc + n;
      *c = accumulate ? *c + acc[i][j] : acc[i][j];
    }
  }
}

template <int MT>
static int launch_few(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                      int ldc, int accumulate, int WK, cudaStream_t st) {
  const int rows = kR * (kFewWarps / WK);               // of W, a CTA
  const dim3 grid((M + MT - 1) / MT, (N + rows - 1) / rows);
  launch_dependent(gemm_f32_few_kernel<MT>, grid, kFewWarps * 32, 0, st, A, W, C, M, N, K, lda, ldw,
                   ldc, accumulate, WK);
  return launch_status();
}

template <int WM, int WN, int KS>
static int launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int lda,
                       int ldw, int ldc, int accumulate, cudaStream_t st) {
  constexpr int BM = 32 * WM, BN = 32 * WN;
  constexpr int smem = ring_of(KS) * KS * (BM + BN) * kRow * (int)sizeof(float);
  auto kern = gemm_f32_tile_kernel<WM, WN, KS>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  kern<<<grid, 32 * WM * WN * KS, smem, st>>>(A, W, C, M, N, K, lda, ldw, ldc, accumulate);
  return launch_status();
}

bool gemm_f32_takes(const void* A, const void* W, int M, int N, int K, int lda, int ldw) {
  // 16-byte loads of whole rows; the grid's second dimension
  return K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 &&
         ((uintptr_t)W & 15) == 0 && N <= 4 * 65535 && M <= 32 * 65535;
}

int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
             int accumulate, cudaStream_t st) {
  // 17 to 64 rows: the few-row body reads W once per eight rows, the tiles once; the tiles need
  // enough columns to fill the chip (24 x 49152 x 576: 80 against 64 us, 64 x 49152 x 576: 199 against
  // 110, 64 x 576 x 576: 8.4 against 8.7).
  if (M <= 16 || (M <= kFewRows && M * N <= 64 * 576)) {
    // Enough warps for W's loads to be in flight everywhere (16 an SM); a warp of a shared k
    // range keeps at least one piece of 128.
    int WK = 1;
    while (WK < kFewWarps && (long long)((N + kR - 1) / kR) * WK < 148 * 16 && WK * 128 < K) WK *= 2;
    if (M == 1) return launch_few<1>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, WK, st);
    if (M == 2) return launch_few<2>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, WK, st);
    if (M <= 4) return launch_few<4>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, WK, st);
    return launch_few<8>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, WK, st);
  }
  // The tile whose waves of 148 SMs cost less: a 64 x 64 tile is four 32 x 32 ones, and about a
  // seventh cheaper than those (fewer shared-memory fills a product).
  auto waves = [&](int b) {
    return ((long long)((M + b - 1) / b) * ((N + b - 1) / b) + 147) / 148;
  };
  if (waves(32) * 8 < waves(64) * 4 * 7)
    return launch_tile<1, 1, 4>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
  return launch_tile<2, 2, 1>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
}

}  // namespace cretif
