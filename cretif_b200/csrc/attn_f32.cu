// Causal attention of the 32-bit path over the block cache, heads of 64 channels and blocks of 64
// tokens (the maths of attn_simt.cu, which takes every other size, the learned bias by distance and
// pooled entries).
//
// Two bodies, both 32-bit FMA (fma.rn.f32x2 where operands pair up as they lie):
//
// * attn_f32_row, a CTA of eight warps per (token, head): decode steps.  It is bound by the
//   latency of a few dependent loads, so everything a warp needs of 32 keys is asked for at once:
//   four lanes share a key (four 16-byte loads each), eight keys an instruction; sixteen lanes
//   share a value.  The warps take tiles of 32 keys in turn.
// * attn_f32_tile, a CTA of four warps per (32 packed tokens, head): prompts.  Blocks of 64 keys and
//   values come through two cp.async stages; a thread holds 4 x 4 scores and 4 rows x 4 channels
//   of the output.  A row belongs to half a warp from its scores to its output, so the
//   probabilities cross lanes through shared memory without a block barrier.
//   Tokens of several sequences in one tile are walked run by run (a run: neighbouring tokens of
//   one sequence); with `leave_short` runs of fewer than kShortRun are left to attn_f32_row, which
//   is launched over the same tokens and takes exactly those.
//
// Which body takes a token depends on its neighbours in the step, its output does not: both sum in one
// order.  Keys go in tiles of 32 from a multiple of 32.  A score: the sixteen channels 16 i + 4 c + (0 .. 3)
// of every c in a chain of two-wide FMAs, the four c as (0 + 2) + (1 + 3).  A tile's sum of probabilities:
// the tree of warp_sum over lanes that hold key 8 (lane & 3) + (lane >> 2).  A tile's output: its even
// and its odd keys, each as a chain, then their sum.  Tiles join the running sums in ascending order.
// The exponential is taken apart (Power): a probability is a number near 1 times a power of two, the
// maximum is one of the exponents, and so every rescaling is exact and it does not matter which keys
// it has seen.
//
// Measured beside attn_simt.cu (one B200, 9 heads on 3, us a launch, before -> now).  Decode: three
// sequences of 90 to 300 keys 33 -> 4.7, eight of 2,048 125 -> 23, one of 4,000 232 -> 35 (a chain of
// 16 dependent rounds a warp), 64 of 1,000 271 -> 27.  Prompts: 90, 164 and 300 tokens 288 -> 35,
// 2,048 tokens 4,630 -> 296 (the order costs a tenth: sums by channel group and by tile), 33 tokens
// 20 -> 8.4.  Error against 64 bits 1.0 to 1.6e-7 there, of attn_simt.cu 1.4 to 2.8e-7.
#include "api.h"
#include "common.cuh"

namespace cretif {

constexpr int kHd = 64;
constexpr int kRowWarps = 8;
constexpr int kTile = 32;             // keys that are summed on their own
constexpr int kRowTiles = 64;         // tiles whose sums the row body keeps before it adds them up
constexpr int kTileRows = 32, kTileKeys = 64;      // the prompt body's stage is a cache block
constexpr int kLd = kHd + 4;          // floats a row takes in shared memory
constexpr int kShortRun = 8;

struct AttnF32 {
  const float* q;
  float* out;
  const float* kc;
  const float* vc;
  const int* table;
  const int* tok_pos;
  const int* tok_seq;
  const int* seq_slot;
  const float* sink;
  const float* slope;
  int ldq, ldo, table_stride, nh, nkv, window, T;
  float scale;
};

// e^s = f 2^n with n whole (kept as a float: scores are not bounded) and f between 2^-0.5 and 2^0.5.
// s log2 e is taken in two parts, so that f is as exact for a large score as for a small one (of
// numbers from 2^22 on a part below their last place is dropped).  s = -inf: f = 0.
struct Power {
  float f, n;
};
__device__ __forceinline__ Power power_of(float s) {
  const float l2e = 1.44269502f, l2e_rest = 1.92596299e-8f;         // log2 e
  const float hi = __fmul_rn(s, l2e);
  const float lo = fabsf(hi) < 4194304.f ? fmaf(s, l2e_rest, fmaf(s, l2e, -hi)) : 0.f;
  Power p;
  p.n = hi == hi ? rintf(hi) : 0.f;              // (no number stays none in f)
  p.f = s == -INFINITY ? 0.f : exp2f(__fadd_rn(__fsub_rn(hi, p.n), lo));
  return p;
}
// 2^x for whole x <= 0 and -inf; 0 from -127 on
__device__ __forceinline__ float two_to(float x) {
  return __int_as_float(((int)fmaxf(x, -127.f) + 127) << 23);
}

// Running sums of a row; a tile's join them.  (All factors are powers of two.)
__device__ __forceinline__ float join(float sum, float keep, float tile, float take) {
  return fmaf(tile, take, __fmul_rn(sum, keep));
}

// The run of tokens of one sequence around token t inside its tile of kTileRows: [lo, hi).
__device__ __forceinline__ void run_of(const AttnF32& a, int t, int& lo, int& hi) {
  const int t0 = t - t % kTileRows, t1 = min(t0 + kTileRows, a.T), s = a.tok_seq[t];
  for (lo = t; lo > t0 && a.tok_seq[lo - 1] == s; --lo) {}
  for (hi = t + 1; hi < t1 && a.tok_seq[hi] == s; ++hi) {}
}

__global__ void __launch_bounds__(kRowWarps * 32)
attn_f32_row_kernel(const AttnF32 a, int only_short) {
  dependent_begin();
  __shared__ __align__(16) float part_o[kRowTiles][kHd];
  __shared__ float part_m[kRowTiles], part_l[kRowTiles], keep_s[kRowTiles], take_s[kRowTiles];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = (int)(blockIdx.x / a.nh), h = (int)(blockIdx.x - (unsigned)t * a.nh);
  if (only_short) {
    int lo, hi;
    run_of(a, t, lo, hi);
    if (hi - lo >= kShortRun) return;
  }
  const int kvh = h / (a.nh / a.nkv);
  const int pos = a.tok_pos[t];
  const int* tab = a.table + (size_t)a.seq_slot[a.tok_seq[t]] * a.table_stride;
  const int first = first_visible_key(pos, a.window);
  const float tilt = a.slope ? a.slope[h] : 0.f;
  // scores: a lane's channels 16 i + 4 c + (0 .. 3) of key kk of eight; softmax: key 8 c + kk of the tile
  const int kk = lane >> 2, c = lane & 3;
  // values: a lane's channels 4 cv .. + 3 of the even (gv = 0) or odd keys
  const int gv = lane >> 4, cv = lane & 15;
  float4 q[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    q[i] = *reinterpret_cast<const float4*>(a.q + (size_t)t * a.ldq + (size_t)h * kHd + 16 * i + 4 * c);
  const int tile0 = first / kTile, tile1 = pos / kTile;
  // the output so far of channel threadIdx.x (the first kHd threads)
  float m = -INFINITY, l = 0.f, o = 0.f;
  int next = tile0 + warp <= tile1 ? tab[(tile0 + warp) >> 1] : -1;
  for (int from = tile0; from <= tile1; from += kRowTiles) {
    const int till = min(from + kRowTiles - 1, tile1);
    for (int tile = from + warp; tile <= till; tile += kRowWarps) {
      const int blk = next;
      next = tile + kRowWarps <= tile1 ? tab[(tile + kRowWarps) >> 1] : -1;   // (64 keys a block)
      if (blk < 0) {                       // keys without a place
        if (lane == 0) part_m[tile - from] = -INFINITY;
        continue;
      }
      const size_t row0 = ((size_t)blk * a.nkv + kvh) * kTileKeys + (tile & 1) * kTile;
      float4 kv[16];
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          kv[4 * x + i] = *reinterpret_cast<const float4*>(a.kc + (row0 + 8 * x + kk) * kHd + 16 * i + 4 * c);
      float s = 0.f;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float2 d2 = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 k4 = kv[4 * x + i];
          d2 = __ffma2_rn(make_float2(q[i].x, q[i].y), make_float2(k4.x, k4.y), d2);
          d2 = __ffma2_rn(make_float2(q[i].z, q[i].w), make_float2(k4.z, k4.w), d2);
        }
        float d = d2.x + d2.y;
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        if (c == x) s = d;
      }
      // the values' loads do not wait for the softmax
#pragma unroll
      for (int i = 0; i < 16; ++i)
        kv[i] = *reinterpret_cast<const float4*>(a.vc + (row0 + 2 * i + gv) * kHd + 4 * cv);
      const int key = tile * kTile + 8 * c + kk;
      const bool seen = key >= first && key <= pos;
      const Power e = power_of(fmaf(-tilt, (float)(pos - key), __fmul_rn(s, a.scale)));
      const float mt = warp_max(seen ? e.n : -INFINITY);
      const float p = seen ? e.f * two_to(e.n - mt) : 0.f;
      const float lt = warp_sum(p);
      float2 x0 = make_float2(0.f, 0.f), x1 = x0;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int key_of = 2 * i + gv;
        const float w = __shfl_sync(0xffffffffu, p, (key_of & 7) * 4 + (key_of >> 3));
        if (w != 0.f) {                    // (a value may be anything where the probability is none)
          x0 = __ffma2_rn(make_float2(w, w), make_float2(kv[i].x, kv[i].y), x0);
          x1 = __ffma2_rn(make_float2(w, w), make_float2(kv[i].z, kv[i].w), x1);
        }
      }
      x0.x += __shfl_xor_sync(0xffffffffu, x0.x, 16);
      x0.y += __shfl_xor_sync(0xffffffffu, x0.y, 16);
      x1.x += __shfl_xor_sync(0xffffffffu, x1.x, 16);
      x1.y += __shfl_xor_sync(0xffffffffu, x1.y, 16);
      if (gv == 0)
        *reinterpret_cast<float4*>(&part_o[tile - from][4 * cv]) = make_float4(x0.x, x0.y, x1.x, x1.y);
      if (lane == 0) {
        part_m[tile - from] = mt;
        part_l[tile - from] = lt;
      }
    }
    __syncthreads();
    // the tiles' sums join in their order; thread i works out tile i's two factors first
    const int n = till - from + 1;
    if (threadIdx.x < n) {
      float before = m;
      for (int i = 0; i < (int)threadIdx.x; ++i) before = fmaxf(before, part_m[i]);
      const float now = fmaxf(before, part_m[threadIdx.x]);
      keep_s[threadIdx.x] = two_to(before - now);
      take_s[threadIdx.x] = two_to(part_m[threadIdx.x] - now);
    }
    __syncthreads();
    if (threadIdx.x < kHd) {
      for (int i = 0; i < n; ++i) {
        const float mt = part_m[i];
        if (mt == -INFINITY) continue;     // nothing seen there
        m = fmaxf(m, mt);
        l = join(l, keep_s[i], part_l[i], take_s[i]);
        o = join(o, keep_s[i], part_o[i][threadIdx.x], take_s[i]);
      }
    }
    if (till < tile1) __syncthreads();     // the tiles' sums have been read
  }
  if (threadIdx.x >= kHd) return;
  float f = 1.f;
  if (a.sink) {
    // one more term exp(sink) in the denominator, with no key and no value
    const Power e = power_of(a.sink[h]);
    const float top = fmaxf(m, e.n);
    f = two_to(m - top);
    l = join(l, f, e.f, two_to(e.n - top));
  }
  a.out[(size_t)t * a.ldo + (size_t)h * kHd + threadIdx.x] = o * f * (1.0f / l);
}

__device__ __forceinline__ void copy16_or_zero(float* dst, const float* src, bool real) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
               "r"(real ? 16 : 0) : "memory");
}

constexpr int kTileSmem = (4 * kTileKeys + 2 * kTileRows) * kLd * (int)sizeof(float);

// A thread (tx of 16) has four keys of a stage, two of each tile: key_at(tx, j), j >> 1 the tile.
// They are the ones of row body lanes tx and tx + 16, so that both sum a row's probabilities alike.
__device__ __forceinline__ int key_at(int tx, int j) {
  return kTile * (j >> 1) + 8 * (tx & 3) + 4 * (j & 1) + (tx >> 2);
}

__global__ void __launch_bounds__(128, 2)
attn_f32_tile_kernel(const AttnF32 a, int leave_short) {
  extern __shared__ __align__(16) float sm[];
  float* kv = sm;                                    // two stages of [keys | values]
  float* qs = sm + 4 * kTileKeys * kLd;
  float* ps = qs + kTileRows * kLd;
  __shared__ int pos_s[kTileRows], first_s[kTileRows];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;            // rows ty + 8 i; channels 4 tx
  const int t0 = blockIdx.x * kTileRows, t1 = min(t0 + kTileRows, a.T);
  const int h = blockIdx.y, kvh = h / (a.nh / a.nkv);
  const float tilt = a.slope ? a.slope[h] : 0.f;
  for (int lo = t0; lo < t1;) {
    const int seq = a.tok_seq[lo];
    int hi = lo + 1;
    while (hi < t1 && a.tok_seq[hi] == seq) ++hi;
    const int n = hi - lo;
    if (leave_short && n < kShortRun) {
      lo = hi;
      continue;
    }
    const int* tab = a.table + (size_t)a.seq_slot[seq] * a.table_stride;
    // positions rise by one inside a run
    const int p0 = a.tok_pos[lo], p1 = p0 + n - 1;
    const int key0 = first_visible_key(p0, a.window) / kTileKeys * kTileKeys;
    const int tiles = (p1 - key0) / kTileKeys + 1;
    __syncthreads();                                 // an earlier run is done with shared memory
    if (tid < kTileRows) {
      pos_s[tid] = tid < n ? p0 + tid : -1;          // a row beyond the run sees nothing
      first_s[tid] = tid < n ? first_visible_key(p0 + tid, a.window) : 0;
    }
    for (int i = tid; i < kTileRows * (kHd / 4); i += 128) {
      const int r = i >> 4, d = (i & 15) * 4;
      copy16_or_zero(qs + r * kLd + d,
                     a.q + (size_t)(lo + (r < n ? r : 0)) * a.ldq + (size_t)h * kHd + d, r < n);
    }
    auto fetch = [&](int tile) {
      const int blk = tab[key0 / kTileKeys + tile];
      const size_t at = ((size_t)max(blk, 0) * a.nkv + kvh) * kTileKeys * kHd;
      const float *kb = a.kc + at, *vb = a.vc + at;
      float* st = kv + (tile & 1) * 2 * kTileKeys * kLd;
      for (int i = tid; i < kTileKeys * (kHd / 4); i += 128) {
        const int r = i >> 4, d = (i & 15) * 4;
        // row tx + 16 j of the keys holds key_at(tx, j); values lie in their own order
        const int key = key_at(r & 15, r >> 4), last = p1 - key0 - tile * kTileKeys;
        copy16_or_zero(st + r * kLd + d, kb + key * kHd + d, blk >= 0 && key <= last);
        copy16_or_zero(st + (kTileKeys + r) * kLd + d, vb + i * 4, blk >= 0 && r <= last);
      }
    };
    fetch(0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    float m[4], l[4], o[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m[i] = -INFINITY;
      l[i] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) o[i][j] = 0.f;
    }
    for (int tile = 0; tile < tiles; ++tile) {
      if (tile + 1 < tiles) fetch(tile + 1);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      const bool mapped = tab[key0 / kTileKeys + tile] >= 0;
      const float* ks = kv + (tile & 1) * 2 * kTileKeys * kLd;
      const float* vs = ks + kTileKeys * kLd;
      float s[4][4], s1[4][4];
#pragma unroll
      for (int part = 0; part < 4; ++part) {         // the score's channels c = 0, 2, 1, 3
        const int c = ((part & 1) << 1) | (part >> 1);
        float2 s2[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) s2[i][j] = make_float2(0.f, 0.f);
#pragma unroll
        for (int d = 4 * c; d < kHd; d += 16) {
          float4 kf[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            kf[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * kLd + d);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 qf = *reinterpret_cast<const float4*>(qs + (ty + 8 * i) * kLd + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              s2[i][j] = __ffma2_rn(make_float2(qf.x, qf.y), make_float2(kf[j].x, kf[j].y), s2[i][j]);
              s2[i][j] = __ffma2_rn(make_float2(qf.z, qf.w), make_float2(kf[j].z, kf[j].w), s2[i][j]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float d = s2[i][j].x + s2[i][j].y;
            if (part == 0) s[i][j] = d;
            if (part == 1) s[i][j] += d;
            if (part == 2) s1[i][j] = d;
            if (part == 3) s[i][j] += s1[i][j] + d;
          }
      }
      float mt[4][2], lt[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = ty + 8 * i, pos = pos_s[r], first = first_s[r];
        Power e[4];
        bool seen[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = key0 + tile * kTileKeys + key_at(tx, j);
          seen[j] = key <= pos && key >= first && mapped;
          e[j] = power_of(fmaf(-tilt, (float)(pos - key), __fmul_rn(s[i][j], a.scale)));
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          float top = fmaxf(seen[2 * u] ? e[2 * u].n : -INFINITY,
                            seen[2 * u + 1] ? e[2 * u + 1].n : -INFINITY);
#pragma unroll
          for (int x = 8; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
          float p[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            p[j] = seen[2 * u + j] ? e[2 * u + j].f * two_to(e[2 * u + j].n - top) : 0.f;
            ps[r * kLd + key_at(tx, 2 * u + j)] = p[j];
          }
          float sum = p[0] + p[1];
#pragma unroll
          for (int x = 8; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
          mt[i][u] = top;
          lt[i][u] = sum;
        }
      }
      __syncwarp();                                  // a row's probabilities stay in its half warp
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float2 x2[2][4][2];                          // even and odd keys
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
          for (int i = 0; i < 4; ++i) x2[g][i][0] = x2[g][i][1] = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int key = kTile * u; key < kTile * (u + 1); key += 4) {
          float4 vf[4];
#pragma unroll
          for (int w = 0; w < 4; ++w)
            vf[w] = *reinterpret_cast<const float4*>(vs + (key + w) * kLd + 4 * tx);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 pf = *reinterpret_cast<const float4*>(ps + (ty + 8 * i) * kLd + key);
            const float pu[4] = {pf.x, pf.y, pf.z, pf.w};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const float2 pp = make_float2(pu[w], pu[w]);
              x2[w & 1][i][0] = __ffma2_rn(pp, make_float2(vf[w].x, vf[w].y), x2[w & 1][i][0]);
              x2[w & 1][i][1] = __ffma2_rn(pp, make_float2(vf[w].z, vf[w].w), x2[w & 1][i][1]);
            }
          }
        }
        float x[4][4], odd = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[i][0] = x2[0][i][0].x + x2[1][i][0].x;
          x[i][1] = x2[0][i][0].y + x2[1][i][0].y;
          x[i][2] = x2[0][i][1].x + x2[1][i][1].x;
          x[i][3] = x2[0][i][1].y + x2[1][i][1].y;
          odd += 0.f * ((x[i][0] + x[i][1]) + (x[i][2] + x[i][3]));
        }
        // A key that a row does not see has probability 0, and 0 times an infinite value is no
        // number: where one turns up the sums are taken again over the seen keys alone.
        if (odd != 0.f) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            for (int key = kTile * u; key < kTile * (u + 1); key += 2)
#pragma unroll
              for (int g = 0; g < 2; ++g) {
                const float p = ps[(ty + 8 * i) * kLd + key + g];
                if (p != 0.f)
#pragma unroll
                  for (int d = 0; d < 4; ++d)
                    y[g][d] = fmaf(p, vs[(key + g) * kLd + 4 * tx + d], y[g][d]);
              }
#pragma unroll
            for (int d = 0; d < 4; ++d) x[i][d] = y[0][d] + y[1][d];
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (mt[i][u] == -INFINITY) continue;       // nothing seen there
          const float now = fmaxf(m[i], mt[i][u]);
          const float keep = two_to(m[i] - now), take = two_to(mt[i][u] - now);
          m[i] = now;
          l[i] = join(l[i], keep, lt[i][u], take);
#pragma unroll
          for (int d = 0; d < 4; ++d) o[i][d] = join(o[i][d], keep, x[i][d], take);
        }
      }
      __syncthreads();                               // the stage may be filled again
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty + 8 * i;
      if (r >= n) continue;
      float f = 1.0f, total = l[i];
      if (a.sink) {                                  // (see the row body)
        const Power e = power_of(a.sink[h]);
        const float top = fmaxf(m[i], e.n);
        f = two_to(m[i] - top);
        total = join(total, f, e.f, two_to(e.n - top));
      }
      const float inv = 1.0f / total;
      *reinterpret_cast<float4*>(a.out + (size_t)(lo + r) * a.ldo + (size_t)h * kHd + 4 * tx) =
          make_float4(o[i][0] * f * inv, o[i][1] * f * inv, o[i][2] * f * inv, o[i][3] * f * inv);
    }
    lo = hi;
  }
}

}  // namespace cretif

using namespace cretif;

// rows: 0 every sequence brings one token; 1 each brings kShortRun or more; 2 a mixture.
extern "C" int cretif_attn_f32(const float* q, int ldq, float* out, int ldo, const float* kc,
                               const float* vc, const int* table, int table_stride,
                               const int* tok_pos, const int* tok_seq, const int* seq_slot, int nh,
                               int nkv, int hd, float scale, int window, int bt, int T,
                               const float* sink, const float* slope, int rows, void* stream) {
  if (T <= 0) return kOk;
  if (nh <= 0 || nkv <= 0 || nh % nkv || hd != kHd || bt != kTileKeys || rows < 0 || rows > 2 ||
      (long long)T * nh > 0x7fffffffLL || nh > 65535)
    return kBadArgument;
  if (ldq % 4 || ldo % 4 || ((uintptr_t)q | (uintptr_t)out | (uintptr_t)kc | (uintptr_t)vc) & 15)
    return kMisaligned;
  const AttnF32 a{q,    out, kc, vc,           table, tok_pos, tok_seq, seq_slot, sink, slope,
                  ldq,  ldo, table_stride, nh, nkv,   window,  T,       scale};
  cudaStream_t st = (cudaStream_t)stream;
  if (rows != 0) {
    const cudaError_t e = cudaFuncSetAttribute(
        attn_f32_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem);
    if (e != cudaSuccess) return (int)e;
    attn_f32_tile_kernel<<<dim3((T + kTileRows - 1) / kTileRows, nh), 128, kTileSmem, st>>>(
        a, rows == 2);
    if (const int r = launch_status()) return r;
  }
  if (rows != 1) {
    launch_dependent(attn_f32_row_kernel, (unsigned)T * nh, kRowWarps * 32, 0, st, a, rows == 2);
    return launch_status();
  }
  return kOk;
}
