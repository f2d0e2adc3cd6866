// C[M,N] (+)= A[M,K] · W[N,K]^T in true 32-bit on the CUDA cores: the two fast bodies behind
// cretif_gemm_simt for float operands whose rows are 16-byte aligned (gemm_simt.cu takes the rest).
//
// Both use the two-wide multiply-add (fma.rn.f32x2) along k: one 16-byte load of a row is two
// operand pairs as it lies, and a sum is kept as two chains (even and odd k) that meet at the
// end, so no operand is ever duplicated or moved.
//
// Both sum an output in one order, whatever M and N are, so that a row's result does not depend on how
// many rows the call has: a slab of 32 k in two chains of its own, the slabs with the same number
// mod 4 in ascending order, then the four totals in theirs.
//
// * gemm_f32_few: a step of few tokens is bound by reading W once, and small matrices by the latency of
//   that.  A CTA has NT columns and MT rows, a warp the slabs with one number mod 4, U = 32 / NT at a
//   time: a lane sums one slab of one column for all MT rows.  W and A come through a cp.async ring of
//   the warp's own (no barrier before the totals meet), slabs 36 floats a row so that neighbouring
//   columns read different banks.  Fewer columns a CTA put more CTAs and shorter chains on a small
//   matrix; they read A more often.  More than 8 rows: the row tiles of one group of columns are
//   neighbours in the grid and read W from L2.
// * gemm_f32_tile: WM x WN warps, 32 x 32 outputs a warp (8 x 4 a thread: 12 shared 16-byte
//   loads feed 64 two-wide FMAs), slabs through a cp.async ring with rows of 36 floats (eight
//   consecutive rows lie in different banks).  KS = 4: the warps of a CTA take the slabs of one
//   32 x 32 tile in turn and the totals meet in shared memory; that is for grids of so few tiles that
//   64 x 64 ones would leave SMs idle.  KS = 1 visits the slabs 0, 4, 8, .., 1, 5, .. for the same order.
//
// Measured beside the 64 x 64 kernel of gemm_simt.cu (one B200, weights not in L2, us before ->
// now; M x N x K).  Few rows: 1 x 49152 x 576 154 -> 21 (5.3 TB/s), 8 x 49152 x 576 157 -> 31,
// 3 x 576 x 1536 111 -> 4.0, 3 x 3072 x 576 43 -> 4.5, 8 x 2048 x 8192 589 -> 31, 8 x 16384 x 2048 34.  Tiles:
// 578 x 3072 x 576 112 -> 67, 2048 x 3072 x 576 302 -> 196, 2048 x 16384 x 2048 5406 -> 3361
// (41 TFLOP/s of the 74 that 128 FMA lanes an SM give); 8 x 8 outputs a thread need 255 registers
// and are no faster.  Lanes that take pieces of 8 k of a row as 16-byte loads lie (no shared memory, and
// sums the tiles can follow piece by piece) cost the tiles a third; a block barrier a chunk of slabs
// cost the few rows a third.
#include "api.h"
#include "common.cuh"
#include "gemm_f32.h"

namespace cretif {

constexpr int kFewRows = 64;
constexpr int kSlab = 32;             // k's a slab
constexpr int kRow = kSlab + 4;       // floats it takes in shared memory

__device__ __forceinline__ void copy16(float* dst, const float* src, bool real) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
               "r"(real ? 16 : 0) : "memory");
}

// Steps a warp's ring holds (a step: 32 / NT slabs).
constexpr int few_depth(int NT) { return NT <= 16 ? 3 : 4; }
// Floats of a slab in it: MT rows of A, NT of W; where two slabs meet in one shared-memory phase (four
// columns) they lie 16 banks apart.
constexpr int few_slab(int MT, int NT) {
  return (MT + NT) * kRow + (NT == 4 ? (48 - 4 * (MT + NT) % 32) % 32 : 0);
}
constexpr int few_smem(int MT, int NT) {
  return 4 * (4 * few_depth(NT) * (32 / NT) * few_slab(MT, NT) + 4 * MT * NT);
}

template <int MT, int NT>
__global__ void __launch_bounds__(128)
gemm_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                    int M, int N, int K, int lda, int ldw, int ldc, int accumulate, int m_tiles) {
  dependent_begin();
  constexpr int D = few_depth(NT), U = 32 / NT, kOne = few_slab(MT, NT), kRows = (MT + NT + 3) / 4;
  static_assert(U * NT == 32, "a lane has a column of one of U slabs");
  extern __shared__ __align__(16) float sm[];
  const int ks = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned bn = blockIdx.x / (unsigned)m_tiles;
  const int n0 = (int)bn * NT, m0 = (int)(blockIdx.x - bn * m_tiles) * MT;
  const int slabs = (K + kSlab - 1) / kSlab, mine = (slabs - ks + 3) / 4, steps = (mine + U - 1) / U;
  float* ring = sm + ks * D * U * kOne;
  float* totals = sm + 4 * D * U * kOne;           // [4][MT][NT]
  // a lane copies piece lane & 7 of every fourth row: NT of W, then MT of A (rows beyond N or M are
  // the last row again; their sums are not stored)
  const int piece = (lane & 7) * 4, row0 = lane >> 3;
  const float* src[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int row = row0 + 4 * i;
    src[i] = row < NT ? W + (size_t)min(n0 + row, N - 1) * ldw
                      : A + (size_t)min(m0 + row - NT, M - 1) * lda;
  }
  auto fetch = [&](int step) {
    if (step < steps) {
      float* st = ring + step % D * U * kOne;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = (ks + 4 * (step * U + u)) * kSlab + piece;
#pragma unroll
        for (int i = 0; i < kRows; ++i)
          if ((MT + NT) % 4 == 0 || row0 + 4 * i < MT + NT)
            copy16(st + u * kOne + (row0 + 4 * i) * kRow + piece, src[i] + (k < K ? k : 0), k < K);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int j = 0; j < D - 1; ++j) fetch(j);
  const int tx = lane % NT, u = lane / NT;
  float acc[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[m] = 0.f;
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory");
    __syncwarp();               // this step's slabs are there, the last one's are read no more
    fetch(step + D - 1);
    const float* one = ring + (step % D * U + u) * kOne;
    float2 part[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) part[m] = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kSlab; k += 4) {
      const float4 w = *reinterpret_cast<const float4*>(one + tx * kRow + k);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const float4 a = *reinterpret_cast<const float4*>(one + (NT + m) * kRow + k);
        part[m] = __ffma2_rn(make_float2(a.x, a.y), make_float2(w.x, w.y), part[m]);
        part[m] = __ffma2_rn(make_float2(a.z, a.w), make_float2(w.z, w.w), part[m]);
      }
    }
    // (slabs beyond K are zero)
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const float sum = part[m].x + part[m].y;
      if (U == 1) {
        acc[m] += sum;
      } else {
#pragma unroll
        for (int v = 0; v < U; ++v) acc[m] += __shfl_sync(0xffffffffu, sum, v * NT + tx);
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (u == 0) {
#pragma unroll
    for (int m = 0; m < MT; ++m) totals[(ks * MT + m) * NT + tx] = acc[m];
  }
  __syncthreads();
  for (int o = threadIdx.x; o < MT * NT; o += 128) {
    const int m = m0 + o / NT, n = n0 + o % NT;
    float sum = totals[o];
#pragma unroll
    for (int g = 1; g < 4; ++g) sum += totals[g * MT * NT + o];
    if (m < M && n < N) {
      float* c = C + (size_t)m * ldc + n;
      *c = accumulate ? *c + sum : sum;
    }
  }
}

// stages of the ring: a CTA that shares a slab range among its warps takes two (74 KB, so that
// three of them share an SM and hide each other's loads), the other three
constexpr int ring_of(int KS) { return KS > 1 ? 2 : 3; }

template <int WM, int WN, int KS>
__global__ void __launch_bounds__(32 * WM * WN * KS)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                     int M, int N, int K, int lda, int ldw, int ldc, int accumulate, int n_tiles) {
  constexpr int BM = 32 * WM, BN = 32 * WN, kThreads = 32 * WM * WN * KS;
  constexpr int kStage = KS * (BM + BN) * kRow, kRing = ring_of(KS);       // (floats)
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ks = warp / (WM * WN), wm = (warp % (WM * WN)) / WN, wn = warp % WN;
  const int ty = lane >> 3, tx = lane & 7;
  const unsigned bm = blockIdx.x / (unsigned)n_tiles;
  const int m0 = (int)bm * BM, n0 = (int)(blockIdx.x - bm * n_tiles) * BN;
  const int slabs = (K + kSlab - 1) / kSlab, quarter = (slabs + 3) / 4;
  const int rounds = KS == 1 ? slabs : quarter;
  // KS == 1: the slab of a round; slabs with 0 mod 4 first (`longer`: how many mod 4 have `quarter` slabs)
  const int longer = slabs - 4 * (quarter - 1);
  auto slab_of = [&](int round, bool* last = nullptr) {
    const int of_longer = longer * quarter;
    const bool in_longer = round < of_longer;
    const int n = in_longer ? quarter : quarter - 1, at = in_longer ? round : round - of_longer;
    const int g = at / n, i = at - g * n;
    if (last) *last = i == n - 1;
    return 4 * i + g + (in_longer ? 0 : longer);
  };

  auto fetch = [&](int round) {
    float* st = sm + (round % kRing) * kStage;
    const int slab0 = KS == 1 ? slab_of(round) : round * KS;
    // KS slabs of BM rows of A and BN rows of W, eight 16-byte pieces a row
#pragma unroll
    for (int i = tid; i < KS * (BM + BN) * 8; i += kThreads) {
      const int piece = i & 7, row = (i >> 3) % (BM + BN), s = (i >> 3) / (BM + BN);
      const int k = (slab0 + s) * kSlab + piece * 4;
      const bool is_a = row < BM;
      const int at = is_a ? m0 + row : n0 + row - BM;
      const bool real = k < K && at < (is_a ? M : N);
      const float* src = is_a ? A + (size_t)(real ? at : 0) * lda : W + (size_t)(real ? at : 0) * ldw;
      copy16(st + (s * (BM + BN) + row) * kRow + piece * 4, src + (real ? k : 0), real);
    }
  };

  // KS == 1: the four totals are added one after the other into `whole`
  float acc[8][4], whole[KS == 1 ? 8 : 1][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[i][j] = 0.f;
      if (KS == 1) whole[i][j] = 0.f;
    }
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
    if (KS == 1) {
      bool last;
      slab_of(round, &last);
      if (last) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            whole[i][j] += acc[i][j];
            acc[i][j] = 0.f;
          }
      }
    }
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
      const float v = KS == 1 ? whole[KS == 1 ? i : 0][j] : acc[i][j];
      *c = accumulate ? *c + v : v;
    }
  }
}


template <int MT, int NT>
static int launch_few(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                      int ldc, int accumulate, cudaStream_t st) {
  constexpr int smem = few_smem(MT, NT);
  count_variant(kVarF32Few);
  auto kern = gemm_f32_few_kernel<MT, NT>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
  }
  const int m_tiles = (M + MT - 1) / MT;
  launch_dependent(kern, (unsigned)((N + NT - 1) / NT) * m_tiles, 128, smem, st, A, W, C, M, N, K, lda,
                   ldw, ldc, accumulate, m_tiles);
  return launch_status();
}

template <int WM, int WN, int KS>
static int launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int lda,
                       int ldw, int ldc, int accumulate, cudaStream_t st) {
  constexpr int BM = 32 * WM, BN = 32 * WN;
  constexpr int smem = ring_of(KS) * KS * (BM + BN) * kRow * (int)sizeof(float);
  count_variant(KS == 1 ? kVarF32Tile64 : kVarF32Tile32);
  auto kern = gemm_f32_tile_kernel<WM, WN, KS>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const int n_tiles = (N + BN - 1) / BN;
  kern<<<(unsigned)n_tiles * ((M + BM - 1) / BM), 32 * WM * WN * KS, smem, st>>>(
      A, W, C, M, N, K, lda, ldw, ldc, accumulate, n_tiles);
  return launch_status();
}

bool gemm_f32_takes(const void* A, const void* W, int M, int N, int K, int lda, int ldw) {
  // 16-byte loads of whole rows; the grids have one dimension (few rows: at most 64 of them, four
  // columns a CTA and more)
  return K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 &&
         ((uintptr_t)W & 15) == 0 && N <= 1 << 26 &&
         (M + 31LL) / 32 * ((N + 31) / 32) <= 0x7fffffffLL;
}

int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
             int accumulate, cudaStream_t st) {
  auto tiles = [&](int m, int n) { return ((long long)(M + m - 1) / m) * ((N + n - 1) / n); };
  // The few-row body reads W once per eight rows, the tiles once; the tiles need enough columns to fill
  // the chip (us, few rows and tiles: 24 x 49152 x 576 85 and 57, 64 x 3072 x 576 17 and 14,
  // 24 x 3072 x 576 6.7 and 8.8, 64 x 576 x 576 5.0 and 8.8).
  if (M <= 8 || (M <= kFewRows && tiles(8, 32) <= 512)) {
    // 32 columns a CTA while that leaves enough CTAs, more of them for a long K, whose chains are the
    // time then (3 x 3072 x 576: 4.5 us, 6.3 with 8 columns; 3 x 576 x 1536: 7.1 and 4.0; 8 x 2048 x 8192:
    // 43 and 31); 8 rows only where half as many CTAs still fill the chip (8 x 576 x 1536: 6.8 us, 4.3
    // as two times four).
    const int wide = K > 4096 ? 512 : 96;
    if (M == 1) {
      if (tiles(1, 32) >= wide) return launch_few<1, 32>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
      if (tiles(1, 8) >= 96) return launch_few<1, 8>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
      return launch_few<1, 4>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
    }
    if (M == 2) {
      if (tiles(2, 32) >= wide) return launch_few<2, 32>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
      if (tiles(2, 8) >= 96) return launch_few<2, 8>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
      return launch_few<2, 4>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
    }
    if (M > 4 && tiles(8, 32) >= (wide > kSmCount ? wide : kSmCount))
      return launch_few<8, 32>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
    if (tiles(4, 32) >= wide) return launch_few<4, 32>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
    return launch_few<4, 8>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
  }
  // The tile whose waves of SMs cost less: a 64 x 64 tile is four 32 x 32 ones, and about a
  // seventh cheaper than those (fewer shared-memory fills a product).
  auto waves = [&](int b) { return (tiles(b, b) + kSmCount - 1) / kSmCount; };
  if (waves(32) * 8 < waves(64) * 4 * 7)
    return launch_tile<1, 1, 4>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
  return launch_tile<2, 2, 1>(A, W, C, M, N, K, lda, ldw, ldc, accumulate, st);
}

}  // namespace cretif
