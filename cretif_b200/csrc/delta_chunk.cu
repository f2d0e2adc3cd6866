// The delta rules over whole prompts, a chunk of 32 tokens at a time.
//
// Inside a chunk the recurrences of delta_rule.cu are linear in the state M0 at its start, so
// what depends on the tokens alone is worked out for all chunks side by side and only what meets
// the state walks them in order:
//
// * prepare (a CTA per chunk and head): the products of the chunk's keys and queries with each
//   other, times the decay between the two tokens, and a forward substitution (a thread per
//   column, the rows so far in its registers) give row vectors with which
//       x_t = X_t + W_t M0        what token t writes along its key,
//       o_t = O_t + Q_t M0        its read-out,
//       M   = diag(Gamma) M0 + sum_t K_t x_t^T (+ K2_t v_t^T).
//   The decay between two tokens is the running product of the decays in between, never a
//   quotient of cumulated ones: a decay of 0 stays exact and nothing overflows.
// * state (a CTA per sequence, head and slice of EC columns): the two products with M0 as one
//   64 x d by d x EC product whose k range is shared among the warps (4 x 4 outputs a thread,
//   two-wide FMAs), then the rank-32 update of the state the threads hold in registers.  A
//   chunk's operands arrive by cp.async a chunk ahead; three barriers a chunk.
//
// The prepared vectors lie in a workspace; a step that it does not hold goes span by span of
// its tokens, the state passing from one to the next through memory.
//
// All arithmetic is 32-bit FMA.  A token-by-token walk is a chain of two dependent reductions and
// an update, 0.47 us a token (0.54 to 1.1 for the general rule, whose five vectors a token load
// the shared memory) whatever the chip has idle.  Microseconds a layer with the norm of the
// read-outs, walk -> chunks: 16 heads of 128 x 128, one sequence of 2,048 tokens 996 -> 242 (the
// general rule 1,468 -> 360), four of 300 to 1,500 870 -> 408 (1,668 -> 610), sixteen of 256
// 468 -> 339 (866 -> 558); 9 heads of 64 x 64, one of 2,048 822 -> 125 (1,091 -> 189).  What
// bounds the state kernel is shared memory's pipe (ncu: stalls on it 4.1 an issue, the FMA pipe busy 39 %
// of the time with two CTAs an SM).
#include "api.h"
#include "common.cuh"

namespace cretif {
namespace {

constexpr int kC = 32;                       // tokens a chunk
constexpr int kA = kC + 4;                   // row stride of the chunk's token x token matrices

__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(dst);
  const int n = ok ? 16 : 0;                 // 0: the destination is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(src), "r"(n)
               : "memory");
}

// Row offsets (floats) of a token's prepared vectors; a chunk's decays lie in its first row.
struct Rows {
  long long ld;
  int w, q, k, k2, x, o, gamma;
};
__host__ __device__ __forceinline__ Rows rows_of(int H, int d, int e, bool general) {
  Rows r;
  r.w = 0;
  r.q = H * d;
  r.k = 2 * H * d;
  r.k2 = 3 * H * d;
  r.x = (general ? 4 : 3) * H * d;
  r.o = r.x + H * e;
  r.gamma = r.o + H * e;
  r.ld = r.gamma + (general ? H * d : (H + 3) / 4 * 4);
  return r;
}

// Which tokens chunk `x` of the grid holds (none of sequences of fewer than `from` tokens: those are
// walked by delta_rule.cu).  The launch takes the tokens s0 .. s1 - 1, of sequence b those from lo to
// hi - 1; its chunks are numbered from (lo - s0) / kC + b: the ranges of two sequences do not meet,
// and the last number is below (s1 - s0) / kC + B.
struct Span {
  int t0, n;
};
__device__ __forceinline__ Span find_span(const int* cu, int B, int x, int from, int s0, int s1,
                                          Span* shared) {
  if (threadIdx.x == 0) shared->n = 0;
  __syncthreads();
  for (int b = threadIdx.x; b < B; b += blockDim.x) {
    const int lo = max(cu[b], s0), hi = min(cu[b + 1], s1), at = x - ((lo - s0) / kC + b);
    if (cu[b + 1] - cu[b] >= from && lo < hi && at >= 0 && at < (hi - lo + kC - 1) / kC) {
      shared->t0 = lo + at * kC;
      shared->n = min(kC, hi - shared->t0);
    }
  }
  __syncthreads();
  return *shared;
}

// A thread's two neighbouring columns of
//     x_t = rhs_t + sum_{s<t} A[t][s] x_s (+ sum_{s<t} B[t][s] v_s),
//     y_t = out_t + sum_{s<=t} E[t][s] x_s (+ sum_{s<=t} F[t][s] v_s),
// eight tokens at a time.  The matrices are stored with s first, so that eight tokens' factors
// are two 16-byte reads that the whole warp shares, for sixteen two-wide FMAs; a token's sums
// never touch later tokens' values.  rhs_t, the larger part of x_t, joins its corrections when they are
// summed: as the first term of the chain it was rounded with each of them.  (With that, the prepared rows
// first in the state's products and one chain over a head's channels, state and read-outs of the gated
// rule were 1.65e-7 and 2.1e-7 from 64 bits, now 0.95e-7 and 1.5e-7, the token walk's figures.)  x
// goes to shared memory (X, row stride ldx) for the rows to come.  (The whole substitution unrolled with
// x in registers ran at a third of this: 50 KB of straight-line code, and 160 registers a thread.)
template <bool TWO, typename Rhs, typename Out, typename Store>
__device__ __forceinline__ void substitute(float* X, int ldx, const float* V, int ldv,
                                           const float* A, const float* E, const float* Bv,
                                           const float* F, int n, Rhs rhs, Out out, Store store) {
#pragma unroll 1
  for (int t8 = 0; t8 < n; t8 += 8) {
    float2 x[8], y[8], own[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      own[j] = rhs(t8 + j), x[j] = make_float2(0.f, 0.f), y[j] = out(t8 + j);
    auto add = [&](const float* m, float2* acc, float2 z, int from) {
      const float4 lo = *reinterpret_cast<const float4*>(m);
      const float4 hi = *reinterpret_cast<const float4*>(m + 4);
      const float f[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j >= from) acc[j] = __ffma2_rn(make_float2(f[j], f[j]), z, acc[j]);
    };
#pragma unroll 2
    for (int s = 0; s < t8; ++s) {
      const float2 xs = *reinterpret_cast<const float2*>(X + s * ldx);
      add(A + s * kA + t8, x, xs, 0);
      add(E + s * kA + t8, y, xs, 0);
      if (TWO) {
        const float2 vs = *reinterpret_cast<const float2*>(V + s * ldv);
        add(Bv + s * kA + t8, x, vs, 0);
        add(F + s * kA + t8, y, vs, 0);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int s = t8 + j;
      x[j] = make_float2(own[j].x + x[j].x, own[j].y + x[j].y);
      if (TWO) {
        const float2 vs = *reinterpret_cast<const float2*>(V + s * ldv);
        add(Bv + s * kA + t8, x, vs, j + 1);
        add(F + s * kA + t8, y, vs, j);
      }
      add(A + s * kA + t8, x, x[j], j + 1);
      add(E + s * kA + t8, y, x[j], j);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      *reinterpret_cast<float2*>(X + (t8 + j) * ldx) = x[j];
      if (t8 + j < n) store(t8 + j, x[j], y[j]);
    }
  }
}
__device__ __forceinline__ float2 times(float a, float2 b) { return make_float2(a * b.x, a * b.y); }
__device__ __forceinline__ float2 at2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ void put2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }

// prep row: [q (G d) | k (G d) | v (H e) | beta (H) | g (H)], see delta_rule.cu.
template <int D>
__global__ void __launch_bounds__(128, 4)
delta_chunk_prepare_kernel(const float* __restrict__ prep, int ldp, float* __restrict__ ws,
                           const int* __restrict__ cu, int B, int H, int G, int e, int from,
                           int s0, int s1) {
  constexpr int LD = D + 4;
  extern __shared__ __align__(16) float sm[];
  float* Ks = sm;                            // [kC][LD], then W
  float* Qs = Ks + kC * LD;                  // [kC][LD]
  float* A = Qs + kC * LD;                   // [s][t]: -beta_t decay(s, t) k_s . k_t, s < t
  float* E = A + kC * kA;                    // [s][t]: decay(s, t) k_s . q_t, s <= t
  float* R = E + kC * kA;                    // [s][t]: decay(s, t)
  float* beta = R + kC * kA;
  float* g = beta + kC;
  float* Vs = g + kC;                        // [kC][e], then X
  __shared__ Span span;
  const int tid = threadIdx.x, h = blockIdx.y, grp = h / (H / G);
  const Span sp = find_span(cu, B, blockIdx.x, from, s0, s1, &span);
  const int n = sp.n;
  if (n == 0) return;
  const int C0 = 2 * G * D + H * e;
  const float* base = prep + (size_t)sp.t0 * ldp;
  for (int i = tid; i < kC * (D / 4); i += 128) {
    const int t = i / (D / 4), c = (i % (D / 4)) * 4;
    const float* row = base + (size_t)min(t, n - 1) * ldp;
    cp16(Qs + t * LD + c, row + (size_t)grp * D + c, t < n);
    cp16(Ks + t * LD + c, row + (size_t)(G + grp) * D + c, t < n);
  }
  if (tid < kC) {
    beta[tid] = tid < n ? base[(size_t)tid * ldp + C0 + h] : 0.f;
    g[tid] = tid < n ? base[(size_t)tid * ldp + C0 + H + h] : 1.f;
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int t = tid >> 5; t < kC; t += 4) {
    const float* row = base + (size_t)min(t, n - 1) * ldp + 2 * G * D + (size_t)h * e;
    for (int c = (tid & 31) * 4; c < e; c += 128) cp16(Vs + t * e + c, row + c, t < n);
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;" ::: "memory");
  __syncthreads();
  if (tid < kC) {
    float run = 1.f;
    for (int t = 0; t < kC; ++t) {
      if (t > tid) run *= g[t];
      R[tid * kA + t] = t < tid ? 0.f : run;
    }
  }
  __syncthreads();
  {
    // a warp gives eight tokens' products with all earlier ones; the four warps take the
    // chunk's quarters
    const int t = tid >> 2, s0 = tid & 3, last = (tid >> 5) * 2 + 2;
    float kk[8], qk[8];
#pragma unroll
    for (int y = 0; y < 8; ++y) kk[y] = qk[y] = 0.f;
#pragma unroll 1
    for (int i0 = 0; i0 < D; i0 += 32) {     // (32 channels on their own: eight terms a chain)
      float2 k2[8], q2[8];
#pragma unroll
      for (int y = 0; y < 8; ++y) k2[y] = q2[y] = make_float2(0.f, 0.f);
#pragma unroll 2
      for (int i = i0; i < i0 + 32; i += 4) {
        const float4 kt = *reinterpret_cast<const float4*>(Ks + t * LD + i);
        const float4 qt = *reinterpret_cast<const float4*>(Qs + t * LD + i);
#pragma unroll
        for (int y = 0; y < 8; ++y) {
          if (y >= last) break;
          const float4 ks = *reinterpret_cast<const float4*>(Ks + (s0 + 4 * y) * LD + i);
          k2[y] = __ffma2_rn(make_float2(kt.x, kt.y), make_float2(ks.x, ks.y), k2[y]);
          k2[y] = __ffma2_rn(make_float2(kt.z, kt.w), make_float2(ks.z, ks.w), k2[y]);
          q2[y] = __ffma2_rn(make_float2(qt.x, qt.y), make_float2(ks.x, ks.y), q2[y]);
          q2[y] = __ffma2_rn(make_float2(qt.z, qt.w), make_float2(ks.z, ks.w), q2[y]);
        }
      }
#pragma unroll
      for (int y = 0; y < 8; ++y) kk[y] += k2[y].x + k2[y].y, qk[y] += q2[y].x + q2[y].y;
    }
#pragma unroll
    for (int y = 0; y < 8; ++y) {
      const int s = s0 + 4 * y;
      const float r = R[s * kA + t];
      A[s * kA + t] = s < t ? -beta[t] * (r * kk[y]) : 0.f;
      E[s * kA + t] = s <= t ? r * qk[y] : 0.f;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const Rows at = rows_of(H, D, e, false);
  float* out = ws + (size_t)(sp.t0 - s0) * at.ld;
  const float g0 = g[0];
  if (tid == 0) out[at.gamma + h] = g0 * R[n - 1];
  for (int c = 2 * tid; c < D + e; c += 256) {
    if (c < D) {
      float* col = out + (size_t)h * D + c;
      substitute<false>(
          Ks + c, LD, nullptr, 0, A, E, nullptr, nullptr, n,
          [&](int t) {
            const float2 k = at2(Ks + t * LD + c);
            if (t < n) put2(col + (size_t)t * at.ld + at.k, times(R[t * kA + n - 1], k));
            return times(-beta[t] * (g0 * R[t]), k);
          },
          [&](int t) { return times(g0 * R[t], at2(Qs + t * LD + c)); },
          [&](int t, float2 x, float2 y) {
            put2(col + (size_t)t * at.ld + at.w, x);
            put2(col + (size_t)t * at.ld + at.q, y);
          });
    } else {
      float* col = out + (size_t)h * e + (c - D);
      substitute<false>(
          Vs + (c - D), e, nullptr, 0, A, E, nullptr, nullptr, n,
          [&](int t) { return times(beta[t], at2(Vs + t * e + c - D)); },
          [&](int) { return make_float2(0.f, 0.f); },
          [&](int t, float2 x, float2 y) {
            put2(col + (size_t)t * at.ld + at.x, x);
            put2(col + (size_t)t * at.ld + at.o, y);
          });
    }
  }
}

// proj row: [r (H d) | k (H d) | v (H e) | ...]; prep row: [u (H d) | -b (H d) | w (H d)].
// Four lanes hold k_s and -b_s of one token s and carry them through the later tokens' decays;
// at every token t they give the four products with u_t (before its decay) and r_t (after).
template <int D>
__global__ void __launch_bounds__(128, 2)
general_chunk_prepare_kernel(const float* __restrict__ proj, int ldp,
                             const float* __restrict__ prep, int ldq, float* __restrict__ ws,
                             const int* __restrict__ cu, int B, int H, int e, int from, int s0,
                             int s1) {
  constexpr int LD = D + 4, V = D / 16;      // V: 16-byte pieces a lane holds
  extern __shared__ __align__(16) float sm[];
  float* Us = sm;                            // [kC][LD], then W
  float* Ws = Us + kC * LD;                  // [kC][LD]
  float* Rs = Ws + kC * LD;                  // [kC][LD]
  float* M = Rs + kC * LD;                   // [4][s][t]: u.(-b), u.k (s < t); r.(-b), r.k (s <= t)
  float* Vs = M + 4 * kC * kA;               // [kC][e]
  float* Xs = Vs + kC * e;                   // [kC][e]
  __shared__ Span span;
  const int tid = threadIdx.x, h = blockIdx.y;
  const Span sp = find_span(cu, B, blockIdx.x, from, s0, s1, &span);
  const int n = sp.n;
  if (n == 0) return;
  const size_t Hd = (size_t)H * D;
  const float* pj = proj + (size_t)sp.t0 * ldp + (size_t)h * D;
  const float* pp = prep + (size_t)sp.t0 * ldq + (size_t)h * D;
  for (int i = tid; i < kC * (D / 4); i += 128) {
    const int t = i / (D / 4), c = (i % (D / 4)) * 4;
    const size_t tt = min(t, n - 1);
    cp16(Us + t * LD + c, pp + tt * ldq + c, t < n);
    cp16(Ws + t * LD + c, pp + tt * ldq + 2 * Hd + c, t < n);
    cp16(Rs + t * LD + c, pj + tt * ldp + c, t < n);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int t = tid >> 5; t < kC; t += 4) {
    const float* row = proj + (size_t)(sp.t0 + min(t, n - 1)) * ldp + 2 * Hd + (size_t)h * e;
    for (int c = (tid & 31) * 4; c < e; c += 128) cp16(Vs + t * e + c, row + c, t < n);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int i = tid; i < 4 * kC * kA; i += 128) M[i] = 0.f;
  const int s = tid >> 2, l = tid & 3;
  float4 ck[V], cb[V];
#pragma unroll
  for (int m = 0; m < V; ++m) {
    const int c = 4 * (l + 4 * m);
    ck[m] = cb[m] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s < n) {
      ck[m] = *reinterpret_cast<const float4*>(pj + (size_t)s * ldp + Hd + c);
      cb[m] = *reinterpret_cast<const float4*>(pp + (size_t)s * ldq + Hd + c);
    }
  }
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();
  for (int t = (tid >> 5) * 8; t < n; ++t) {
    float2 ub = make_float2(0.f, 0.f), uk = ub, rb = ub, rk = ub;
#pragma unroll
    for (int m = 0; m < V; ++m) {
      const int c = t * LD + 4 * (l + 4 * m);
      const float4 u = *reinterpret_cast<const float4*>(Us + c);
      float4 w = *reinterpret_cast<const float4*>(Ws + c);
      const float4 r = *reinterpret_cast<const float4*>(Rs + c);
      if (t <= s) w = make_float4(1.f, 1.f, 1.f, 1.f);
      const float2 u0 = make_float2(u.x, u.y), u1 = make_float2(u.z, u.w);
      const float2 w0 = make_float2(w.x, w.y), w1 = make_float2(w.z, w.w);
      const float2 r0 = make_float2(r.x, r.y), r1 = make_float2(r.z, r.w);
      float2 k0 = make_float2(ck[m].x, ck[m].y), k1 = make_float2(ck[m].z, ck[m].w);
      float2 b0 = make_float2(cb[m].x, cb[m].y), b1 = make_float2(cb[m].z, cb[m].w);
      ub = __ffma2_rn(u0, b0, ub);
      uk = __ffma2_rn(u0, k0, uk);
      ub = __ffma2_rn(u1, b1, ub);
      uk = __ffma2_rn(u1, k1, uk);
      k0 = __fmul2_rn(k0, w0);
      k1 = __fmul2_rn(k1, w1);
      b0 = __fmul2_rn(b0, w0);
      b1 = __fmul2_rn(b1, w1);
      rb = __ffma2_rn(r0, b0, rb);
      rk = __ffma2_rn(r0, k0, rk);
      rb = __ffma2_rn(r1, b1, rb);
      rk = __ffma2_rn(r1, k1, rk);
      ck[m] = make_float4(k0.x, k0.y, k1.x, k1.y);
      cb[m] = make_float4(b0.x, b0.y, b1.x, b1.y);
    }
    // four sums over four lanes in three shuffles: lane 0 keeps u.b, 1 u.k, 2 r.b, 3 r.k
    const float v0 = ub.x + ub.y, v1 = uk.x + uk.y, v2 = rb.x + rb.y, v3 = rk.x + rk.y;
    const bool hi = l & 2, od = l & 1;
    const float p0 = (hi ? v2 : v0) + __shfl_xor_sync(0xffffffffu, hi ? v0 : v2, 2);
    const float p1 = (hi ? v3 : v1) + __shfl_xor_sync(0xffffffffu, hi ? v1 : v3, 2);
    const float p = (od ? p1 : p0) + __shfl_xor_sync(0xffffffffu, od ? p0 : p1, 1);
    if (hi ? t >= s : t > s) M[(l * kC + s) * kA + t] = p;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const float *A = M, *Bv = M + kC * kA, *E = Bv + kC * kA, *F = E + kC * kA;
  const Rows at = rows_of(H, D, e, true);
  float* out = ws + (size_t)(sp.t0 - s0) * at.ld;
  for (int c = 2 * tid; c < D + e; c += 256) {
    if (c < D) {
      float* col = out + (size_t)h * D + c;
      // the products of decays up to a token, before it (rhs) and with it (out), token by token
      float2 before = make_float2(1.f, 1.f), with = before;
      substitute<false>(
          Us + c, LD, nullptr, 0, A, E, nullptr, nullptr, n,
          [&](int t) {
            const float2 r = __fmul2_rn(before, at2(Us + t * LD + c));
            before = __fmul2_rn(before, at2(Ws + t * LD + c));
            return r;
          },
          [&](int t) {
            const float2 w = __fmul2_rn(with, at2(Ws + t * LD + c));
            if (t < n) with = w;
            return __fmul2_rn(w, at2(Rs + t * LD + c));
          },
          [&](int t, float2 x, float2 y) {
            put2(col + (size_t)t * at.ld + at.w, x);
            put2(col + (size_t)t * at.ld + at.q, y);
          });
      put2(col + at.gamma, with);
      float2 run = make_float2(1.f, 1.f);
#pragma unroll 8
      for (int t = n - 1; t >= 0; --t) {
        float* p = col + (size_t)t * at.ld;
        put2(p + at.k, __fmul2_rn(run, at2(pp + (size_t)t * ldq + Hd + c)));
        put2(p + at.k2, __fmul2_rn(run, at2(pj + (size_t)t * ldp + Hd + c)));
        run = __fmul2_rn(run, at2(Ws + t * LD + c));
      }
    } else {
      float* col = out + (size_t)h * e + (c - D);
      substitute<true>(
          Xs + (c - D), e, Vs + (c - D), e, A, E, Bv, F, n,
          [&](int) { return make_float2(0.f, 0.f); }, [&](int) { return make_float2(0.f, 0.f); },
          [&](int t, float2 x, float2 y) {
            put2(col + (size_t)t * at.ld + at.x, x);
            put2(col + (size_t)t * at.ld + at.o, y);
          });
    }
  }
}

template <int D, int EC, bool GENERAL>
struct StatePlan {
  static constexpr int LD = D + 4;
  static constexpr int KS = 128 / EC / 2;                   // warps' shares of the k range
  static constexpr int kWQ = 2 * kC * LD;
  static constexpr int kK = (GENERAL ? 2 : 1) * kC * LD + (GENERAL ? kC * EC + D : 4);
  static constexpr int kXO = 2 * kC * EC;
  static constexpr int kRed = KS * 2 * kC * (EC + 4);
  static constexpr int kFloats = kWQ + kK + 2 * kXO + EC * LD + kRed + kC * EC;
};

// One buffer for what the products read (W, Q), refilled while the update runs, one for what the
// update reads (K, K2, V, decays), refilled while the products run: two CTAs share an SM and hide
// each other's barriers (with two stages of everything one CTA filled it: 490 us against 456 for eight
// prompts; of the general rule with heads of 128 one CTA of 32 columns fits all the same).
template <int D, int EC, bool GENERAL>
__global__ void __launch_bounds__(256, 2)
delta_chunk_state_kernel(const float* __restrict__ ws, const float* __restrict__ v, int ldv,
                         float* __restrict__ state, size_t state_stride,
                         const int* __restrict__ cu, const int* __restrict__ seq_slot, int B, int H,
                         int e, float* __restrict__ o_raw, int write_state, int from, int s0,
                         int s1) {
  using P = StatePlan<D, EC, GENERAL>;
  constexpr int LD = P::LD, KS = P::KS, J = EC / 4, I = D / 64;
  extern __shared__ __align__(16) float sm[];
  float* WQ = sm;                            // [2 kC][LD]
  float* Kh = WQ + P::kWQ;                   // [kC][LD] (, K2 [kC][LD], V [kC][EC]), decays
  float* Vs = Kh + (GENERAL ? 2 : 1) * kC * LD;
  float* gam = Vs + (GENERAL ? kC * EC : 0);
  float* XO = Kh + P::kK;                    // two of [2 kC][EC]
  float* ST = XO + 2 * P::kXO;               // the state's slice, a row per column: [EC][LD]
  float* red = ST + EC * LD;                 // [KS][2 kC][EC + 4]
  float* X = red + P::kRed;                  // [kC][EC]
  // the grid: heads, slices of columns, sequences (the slowest)
  const unsigned part = blockIdx.x / (unsigned)H, slices = (unsigned)(e / EC);
  const int h = (int)(blockIdx.x - part * H), col0 = (int)(part % slices) * EC;
  const int b = sequence_by_length(cu, B, (int)(part / slices));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t0 = max(cu[b], s0), t1 = min(cu[b + 1], s1);
  if (cu[b + 1] - cu[b] < from || t0 >= t1) return;
  const Rows at = rows_of(H, D, e, GENERAL);

  // A thread copies the same 16 bytes of every kStep-th row, and the same of every cStep-th row
  // of the column slices.
  constexpr int kStep = 256 / (D / 4), cStep = 256 / (EC / 4);
  const int rt = tid / (D / 4), rc = (tid % (D / 4)) * 4;
  const int ct = tid / (EC / 4), cc = (tid % (EC / 4)) * 4;
  auto copy_rows = [&](float* dst, const float* base, int first, int n) {
#pragma unroll
    for (int i = 0; i < kC / kStep; ++i) {   // first: W and Q (0) or K and K2 (2)
      const int t = rt + i * kStep;
      const float* src = base + (size_t)min(t, n - 1) * at.ld + (size_t)h * D + rc;
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (first == 0 || x == 0 || GENERAL)
          cp16(dst + (x * kC + t) * LD + rc, src + (size_t)(first + x) * H * D, t < n);
    }
  };
  auto issue_wq = [&](int c0, int half) {
    const int n = min(kC, t1 - c0);
    const float* base = ws + (size_t)(c0 - s0) * at.ld;
    copy_rows(WQ, base, 0, n);
    float* dst = XO + half * P::kXO;
#pragma unroll
    for (int i = 0; i < (2 * kC + cStep - 1) / cStep; ++i) {
      const int r = ct + i * cStep, t = r & (kC - 1);
      cp16(dst + r * EC + cc,
           base + (size_t)min(t, n - 1) * at.ld + (r < kC ? at.x : at.o) + (size_t)h * e + col0 + cc,
           t < n);
    }
  };
  auto issue_k = [&](int c0) {
    const int n = min(kC, t1 - c0);
    const float* base = ws + (size_t)(c0 - s0) * at.ld;
    copy_rows(Kh, base, 2, n);
    if constexpr (GENERAL) {
      for (int t = ct; t < kC; t += cStep)
        cp16(Vs + t * EC + cc,
             v + (size_t)(c0 + min(t, n - 1)) * ldv + (size_t)h * e + col0 + cc, t < n);
      if (tid < D / 4) cp16(gam + tid * 4, base + at.gamma + (size_t)h * D + tid * 4, true);
    } else if (tid == 0) {
      const unsigned a = (unsigned)__cvta_generic_to_shared(gam);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(a), "l"(base + at.gamma + h)
                   : "memory");
    }
  };
  issue_wq(t0, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");

  // the thread's part of the state: columns jb .. jb+J-1 (in pairs), rows ib .. ib+I-1
  const int jb = (lane >> 3) * J, ib = (warp * 8 + (lane & 7)) * I;
  float* Mg = state + (size_t)seq_slot[b] * state_stride + (size_t)h * D * e + col0;
  float2 S[J / 2][I];
#pragma unroll
  for (int y = 0; y < I; ++y)
#pragma unroll
    for (int x = 0; x < J / 2; ++x) S[x][y] = at2(Mg + (size_t)(ib + y) * e + jb + 2 * x);
  auto publish = [&] {
#pragma unroll
    for (int x = 0; x < J / 2; ++x)
#pragma unroll
      for (int y = 0; y < I; ++y) {
        ST[(jb + 2 * x) * LD + ib + y] = S[x][y].x;
        ST[(jb + 2 * x + 1) * LD + ib + y] = S[x][y].y;
      }
  };
  publish();
  // the warp's tile of the products: 32 rows, 16 columns, D / KS of the k range
  constexpr int TB = 8 / KS;
  const int ks = warp / TB, rb = (warp % TB) & 1, cb = (warp % TB) >> 1;
  const int row = rb * 32 + (lane >> 2), col = cb * 16 + (lane & 3);   // + 8 x, + 4 y

  int half = 0;
  for (int c0 = t0; c0 < t1; c0 += kC, half ^= 1) {
    const int n = min(kC, t1 - c0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();          // W, Q, X, O and the state have arrived; K's buffer is free
    issue_k(c0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    {
      float2 acc[4][4];
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) acc[x][y] = make_float2(0.f, 0.f);
      const float* wp = WQ + row * LD + ks * (D / KS);
      const float* sp = ST + col * LD + ks * (D / KS);
#pragma unroll 4
      for (int k = 0; k < D / KS; k += 4) {
        float4 a[4], m[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          a[x] = *reinterpret_cast<const float4*>(wp + 8 * x * LD + k);
          m[x] = *reinterpret_cast<const float4*>(sp + 4 * x * LD + k);
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            acc[x][y] = __ffma2_rn(make_float2(a[x].x, a[x].y), make_float2(m[y].x, m[y].y),
                                   acc[x][y]);
            acc[x][y] = __ffma2_rn(make_float2(a[x].z, a[x].w), make_float2(m[y].z, m[y].w),
                                   acc[x][y]);
          }
      }
      float* rp = red + (ks * 2 * kC + row) * (EC + 4) + col;
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) rp[8 * x * (EC + 4) + 4 * y] = acc[x][y].x + acc[x][y].y;
    }
    __syncthreads();          // the shares are there; W's and Q's buffer is free
    if (c0 + kC < t1) issue_wq(c0 + kC, half ^ 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* xo = XO + half * P::kXO;
#pragma unroll
    for (int i = 0; i < (2 * kC + cStep - 1) / cStep; ++i) {
      const int r = ct + i * cStep;
      const float* rp = red + r * (EC + 4) + cc;
      float4 sum = *reinterpret_cast<const float4*>(rp);
#pragma unroll
      for (int k = 1; k <= KS; ++k) {
        const float4 p = *reinterpret_cast<const float4*>(
            k < KS ? rp + k * 2 * kC * (EC + 4) : xo + r * EC + cc);
        sum.x += p.x, sum.y += p.y, sum.z += p.z, sum.w += p.w;
      }
      if (r < kC)
        *reinterpret_cast<float4*>(X + r * EC + cc) = sum;
      else if (r - kC < n)
        *reinterpret_cast<float4*>(o_raw + (size_t)(c0 + r - kC) * H * e + (size_t)h * e + col0 +
                                   cc) = sum;
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();          // X is written, K has arrived
#pragma unroll
    for (int y = 0; y < I; ++y) {
      const float gm = GENERAL ? gam[ib + y] : gam[0];
#pragma unroll
      for (int x = 0; x < J / 2; ++x) S[x][y] = times(gm, S[x][y]);
    }
    auto update = [&](const float* K, const float* Y) {
#pragma unroll 8
      for (int s = 0; s < kC; ++s) {
        float2 xs[J / 2];
#pragma unroll
        for (int x = 0; x < J / 4; ++x) {
          const float4 f = *reinterpret_cast<const float4*>(Y + s * EC + jb + 4 * x);
          xs[2 * x] = make_float2(f.x, f.y), xs[2 * x + 1] = make_float2(f.z, f.w);
        }
        float kv[2];
        if constexpr (I == 2) {
          const float2 f = at2(K + s * LD + ib);
          kv[0] = f.x, kv[1] = f.y;
        } else {
          kv[0] = K[s * LD + ib];
        }
#pragma unroll
        for (int y = 0; y < I; ++y)
#pragma unroll
          for (int x = 0; x < J / 2; ++x)
            S[x][y] = __ffma2_rn(make_float2(kv[y], kv[y]), xs[x], S[x][y]);
      }
    };
    update(Kh, X);
    if constexpr (GENERAL) update(Kh + kC * LD, Vs);
    publish();
  }
  if (write_state) {
#pragma unroll
    for (int y = 0; y < I; ++y)
#pragma unroll
      for (int x = 0; x < J / 2; ++x) put2(Mg + (size_t)(ib + y) * e + jb + 2 * x, S[x][y]);
  }
}

template <int D, int EC, bool GENERAL>
int launch_state_t(const float* ws, const float* v, int ldv, float* state, size_t stride,
                   const int* cu, const int* slot, int B, int H, int e, float* o_raw,
                   int write_state, int from, int s0, int s1, cudaStream_t st) {
  constexpr int bytes = StatePlan<D, EC, GENERAL>::kFloats * 4;
  static_assert(bytes <= 227 * 1024, "a chunk's stages do not fit");
  auto kern = delta_chunk_state_kernel<D, EC, GENERAL>;
  cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (err != cudaSuccess) return (int)err;
  count_variant(EC == 32 ? kVarDeltaSlices32 : kVarDeltaSlices16);
  kern<<<(unsigned)B * H * (e / EC), 256, bytes, st>>>(ws, v, ldv, state, stride, cu, slot, B, H, e,
                                                       o_raw, write_state, from, s0, s1);
  return launch_status();
}

template <int D, bool GENERAL>
int launch_state(const float* ws, const float* v, int ldv, float* state, size_t stride,
                 const int* cu, const int* slot, int B, int H, int e, float* o_raw,
                 int write_state, int from, int s0, int s1, cudaStream_t st) {
  // Slices of 32 columns halve the reads of a chunk's rows; slices of 16 while there are fewer than two
  // of 32 an SM (four sequences of 300 to 1,500 tokens, 16 heads of 128: 408 us in slices of 16, 439 in
  // slices of 32).  Of the general rule with heads of 128 one CTA of 32 columns fits an SM (128 KB) and
  // is still the faster one from there on: 5 x 512 tokens 419 us in slices of 32, 417 of 16, 8 x 512 589
  // and 599, 32 x 256 1,099 and 1,185.
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
  }();
  if (e % 32 == 0 && (long long)B * H * (e / 32) >= 2LL * sms)
    return launch_state_t<D, 32, GENERAL>(ws, v, ldv, state, stride, cu, slot, B, H, e, o_raw,
                                          write_state, from, s0, s1, st);
  return launch_state_t<D, 16, GENERAL>(ws, v, ldv, state, stride, cu, slot, B, H, e, o_raw,
                                        write_state, from, s0, s1, st);
}

template <typename K>
int allow_smem(K kern, int bytes) {
  return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

bool takes(int B, int H, int d, int e, const float* state, long long stride) {
  return (d == 64 || d == 128) && e > 0 && e <= 256 && e % 16 == 0 && H > 0 && H <= 65535 &&
         (long long)B * H * (e / 16) <= 0x7fffffffLL && stride % 4 == 0 && ((uintptr_t)state & 15) == 0;
}

}  // namespace
}  // namespace cretif

using namespace cretif;

// Floats of workspace a token needs, or 0 where the sizes are not taken.
extern "C" long long cretif_delta_chunk_row(int H, int d, int e, int general) {
  if (H <= 0 || (d != 64 && d != 128) || e <= 0 || e > 256 || e % 16) return 0;
  return rows_of(H, d, e, general != 0).ld;
}

namespace cretif {
namespace {
// Tokens of a span, whole chunks of them, for a workspace of that many floats; 0: it is too small, or
// the step needs several spans and may not write the state that passes between them.
int span_tokens(long long ws_floats, const Rows& at, int T, int write_state) {
  const long long rows = ws_floats / at.ld;
  if (rows >= T) return T;
  return write_state ? (int)(rows / kC * kC) : 0;
}
}  // namespace
}  // namespace cretif

extern "C" int cretif_delta_chunks(const float* prep, int ldp, float* state, long long stride,
                                   const int* cu, const int* seq_slot, int B, int H, int G, int d,
                                   int e, float* ws, long long ws_floats, float* o_raw,
                                   int write_state, int T, int from, void* stream) {
  if (B <= 0 || T <= 0) return kOk;
  if (!takes(B, H, d, e, state, stride) || G <= 0 || H % G || ldp < 2 * G * d + H * e + 2 * H)
    return kBadArgument;
  if (ldp % 4 || (((uintptr_t)prep | (uintptr_t)ws | (uintptr_t)o_raw) & 15)) return kMisaligned;
  const int step = span_tokens(ws_floats, rows_of(H, d, e, false), T, write_state);
  if (step <= 0) return kBadArgument;
  cudaStream_t st = (cudaStream_t)stream;
  const int bytes = 4 * (2 * kC * (d + 4) + 3 * kC * kA + 2 * kC + kC * e);
  int rc = d == 64 ? allow_smem(delta_chunk_prepare_kernel<64>, bytes)
                   : allow_smem(delta_chunk_prepare_kernel<128>, bytes);
  for (int s0 = 0; s0 < T && !rc; s0 += step) {
    const int s1 = T - s0 < step ? T : s0 + step;
    const dim3 grid((s1 - s0) / kC + B, H);
    if (d == 64)
      delta_chunk_prepare_kernel<64><<<grid, 128, bytes, st>>>(prep, ldp, ws, cu, B, H, G, e, from,
                                                               s0, s1);
    else
      delta_chunk_prepare_kernel<128><<<grid, 128, bytes, st>>>(prep, ldp, ws, cu, B, H, G, e, from,
                                                                s0, s1);
    if ((rc = launch_status())) return rc;
    rc = d == 64 ? launch_state<64, false>(ws, nullptr, 0, state, (size_t)stride, cu, seq_slot, B, H,
                                           e, o_raw, write_state, from, s0, s1, st)
                 : launch_state<128, false>(ws, nullptr, 0, state, (size_t)stride, cu, seq_slot, B,
                                            H, e, o_raw, write_state, from, s0, s1, st);
  }
  return rc;
}

extern "C" int cretif_general_delta_chunks(const float* proj, int ldp, const float* prep, int ldq,
                                           float* state, long long stride, const int* cu,
                                           const int* seq_slot, int B, int H, int d, int e,
                                           float* ws, long long ws_floats, float* o_raw,
                                           int write_state, int T, int from, void* stream) {
  if (B <= 0 || T <= 0) return kOk;
  if (!takes(B, H, d, e, state, stride) || ldp < 2 * H * d + H * e || ldq < 3 * H * d)
    return kBadArgument;
  if (ldp % 4 || ldq % 4 ||
      (((uintptr_t)proj | (uintptr_t)prep | (uintptr_t)ws | (uintptr_t)o_raw) & 15))
    return kMisaligned;
  const int step = span_tokens(ws_floats, rows_of(H, d, e, true), T, write_state);
  if (step <= 0) return kBadArgument;
  cudaStream_t st = (cudaStream_t)stream;
  const int bytes = 4 * (3 * kC * (d + 4) + 4 * kC * kA + 2 * kC * e);
  int rc = d == 64 ? allow_smem(general_chunk_prepare_kernel<64>, bytes)
                   : allow_smem(general_chunk_prepare_kernel<128>, bytes);
  const float* v = proj + 2 * (size_t)H * d;
  for (int s0 = 0; s0 < T && !rc; s0 += step) {
    const int s1 = T - s0 < step ? T : s0 + step;
    const dim3 grid((s1 - s0) / kC + B, H);
    if (d == 64)
      general_chunk_prepare_kernel<64><<<grid, 128, bytes, st>>>(proj, ldp, prep, ldq, ws, cu, B, H,
                                                                 e, from, s0, s1);
    else
      general_chunk_prepare_kernel<128><<<grid, 128, bytes, st>>>(proj, ldp, prep, ldq, ws, cu, B, H,
                                                                  e, from, s0, s1);
    if ((rc = launch_status())) return rc;
    rc = d == 64 ? launch_state<64, true>(ws, v, ldp, state, (size_t)stride, cu, seq_slot, B, H, e,
                                          o_raw, write_state, from, s0, s1, st)
                 : launch_state<128, true>(ws, v, ldp, state, (size_t)stride, cu, seq_slot, B, H, e,
                                           o_raw, write_state, from, s0, s1, st);
  }
  return rc;
}
