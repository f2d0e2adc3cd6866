// Causal attention of the 32-bit path over the block cache, heads of 64 channels and blocks
// of 64 tokens (the maths of attn_simt.cu, which takes every other size, the learned bias by distance and pooled entries).
//
// Two bodies, both 32-bit FMA (fma.rn.f32x2 where operands pair up as they lie) and expf:
//
// * attn_f32_row, a CTA of eight warps per (token, head): decode steps.  It is bound by the
//   latency of a few dependent loads, so everything a warp needs of 32 keys is asked for at once:
//   eight lanes share a key (two 16-byte loads each), four keys an instruction, the same for the
//   values.  The warps take blocks of 32 keys in turn and are merged in their order.
// * attn_f32_tile, a CTA of four warps per (32 packed tokens, head): prompts.  Tiles of 64 keys and
//   values come through two cp.async stages; a thread holds 4 x 4 scores and 4 rows x 4 channels
//   of the output.  A row belongs to half a warp from its scores to its output, so the
//   probabilities cross lanes through shared memory without a block barrier.  A tile's share of
//   the output is summed on its own and joins the rescaled running sum with one FMA.
//   Tokens of several sequences in one tile are walked run by run (a run: neighbouring tokens of
//   one sequence); with `leave_short` runs of fewer than kShortRun are left to attn_f32_row, which
//   is launched over the same tokens and takes exactly those.
//
// Measured beside attn_simt.cu (one B200, 9 heads on 3, us a launch, before -> now).  Decode: three
// sequences of 90 to 300 keys 33 -> 5.9, eight of 2,048 125 -> 18, one of 4,000 232 -> 29 (a chain
// of 16 dependent rounds a warp), 64 of 1,000 271 -> 34.  Prompts: 90, 164 and 300 tokens
// 288 -> 32, 2,048 tokens 4,630 -> 274, 33 tokens 20 -> 8.8.
#include "api.h"
#include "common.cuh"

namespace cretif {

constexpr int kHd = 64;
constexpr int kRowWarps = 8;
constexpr int kTileRows = 32, kTileKeys = 64;      // a tile of keys is a cache block
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

// The run of tokens of one sequence around token t inside its tile of kTileRows: [lo, hi).
__device__ __forceinline__ void run_of(const AttnF32& a, int t, int& lo, int& hi) {
  const int t0 = t - t % kTileRows, t1 = min(t0 + kTileRows, a.T), s = a.tok_seq[t];
  for (lo = t; lo > t0 && a.tok_seq[lo - 1] == s; --lo) {}
  for (hi = t + 1; hi < t1 && a.tok_seq[hi] == s; ++hi) {}
}

__global__ void __launch_bounds__(kRowWarps * 32)
attn_f32_row_kernel(const AttnF32 a, int only_short) {
  dependent_begin();
  __shared__ float part_acc[kRowWarps][kHd];
  __shared__ float part_m[kRowWarps], part_l[kRowWarps];
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
  // a lane's eight channels: four at 4c, four at 32 + 4c
  const int g = lane >> 3, c = lane & 7;
  const float* qrow = a.q + (size_t)t * a.ldq + (size_t)h * kHd + 4 * c;
  const float4 q0 = *reinterpret_cast<const float4*>(qrow);
  const float4 q1 = *reinterpret_cast<const float4*>(qrow + 32);
  float m = -INFINITY, l = 0.f;
  float4 o0 = make_float4(0.f, 0.f, 0.f, 0.f), o1 = o0;
  // Lane (g, c) of the softmax holds key base + 4 c + g; the cache row it lies in, or -1.  The rows
  // of the next 32 keys are looked up while these are worked on.
  auto row_of = [&](int base) {
    const int key = base + 4 * c + g;
    const int blk = key <= pos ? tab[key >> 6] : -1;
    return blk < 0 ? -1 : (blk * a.nkv + kvh) * 64 + (key & 63);
  };
  int next = row_of(first + 32 * warp);
  for (int base = first + 32 * warp; base <= pos; base += 32 * kRowWarps) {
    const int key = base + 4 * c + g, row = next;
    next = row_of(base + 32 * kRowWarps);
    float4 k0[8], k1[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {        // four keys an instruction: base + 4 i + g
      const int r = __shfl_sync(0xffffffffu, row, 8 * g + i);
      const float* p = a.kc + (size_t)max(r, 0) * kHd + 4 * c;
      k0[i] = *reinterpret_cast<const float4*>(p);
      k1[i] = *reinterpret_cast<const float4*>(p + 32);
    }
    float s = -INFINITY;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float d = k0[i].x * q0.x;
      d = fmaf(k0[i].y, q0.y, d);
      d = fmaf(k0[i].z, q0.z, d);
      d = fmaf(k0[i].w, q0.w, d);
      float e = k1[i].x * q1.x;
      e = fmaf(k1[i].y, q1.y, e);
      e = fmaf(k1[i].z, q1.z, e);
      e = fmaf(k1[i].w, q1.w, e);
      d += e;
      d += __shfl_xor_sync(0xffffffffu, d, 4);
      d += __shfl_xor_sync(0xffffffffu, d, 2);
      d += __shfl_xor_sync(0xffffffffu, d, 1);
      if (c == i) s = d;
    }
    // the values' loads do not wait for the softmax; a key without a place is not read
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = __shfl_sync(0xffffffffu, row, 8 * g + i);
      k0[i] = k1[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r >= 0) {
        const float* p = a.vc + (size_t)r * kHd + 4 * c;
        k0[i] = *reinterpret_cast<const float4*>(p);
        k1[i] = *reinterpret_cast<const float4*>(p + 32);
      }
    }
    s = row < 0 ? -INFINITY : s * a.scale - tilt * (float)(pos - key);
    const float m_new = fmaxf(m, warp_max(s));
    const float p = row < 0 ? 0.f : expf(s - m_new);
    const float corr = m == -INFINITY ? 0.f : expf(m - m_new);
    l = l * corr + warp_sum(p);
    m = m_new;
    o0.x *= corr; o0.y *= corr; o0.z *= corr; o0.w *= corr;
    o1.x *= corr; o1.y *= corr; o1.z *= corr; o1.w *= corr;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float w = __shfl_sync(0xffffffffu, p, 8 * g + i);
      if (w != 0.f) {                    // (a value may be anything where the probability is none)
        o0.x = fmaf(w, k0[i].x, o0.x); o0.y = fmaf(w, k0[i].y, o0.y);
        o0.z = fmaf(w, k0[i].z, o0.z); o0.w = fmaf(w, k0[i].w, o0.w);
        o1.x = fmaf(w, k1[i].x, o1.x); o1.y = fmaf(w, k1[i].y, o1.y);
        o1.z = fmaf(w, k1[i].z, o1.z); o1.w = fmaf(w, k1[i].w, o1.w);
      }
    }
  }
  // the four groups of lanes hold shares of the same channels
  float o[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    o[i] += __shfl_xor_sync(0xffffffffu, o[i], 8);
    o[i] += __shfl_xor_sync(0xffffffffu, o[i], 16);
  }
  if (g == 0) {
    *reinterpret_cast<float4*>(&part_acc[warp][4 * c]) = make_float4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<float4*>(&part_acc[warp][32 + 4 * c]) = make_float4(o[4], o[5], o[6], o[7]);
  }
  if (lane == 0) {
    part_m[warp] = m;
    part_l[warp] = l;
  }
  __syncthreads();
  if (threadIdx.x >= kHd) return;
  const int d = threadIdx.x;
  float m_all = a.sink ? a.sink[h] : -INFINITY;
#pragma unroll
  for (int w = 0; w < kRowWarps; ++w) m_all = fmaxf(m_all, part_m[w]);
  float l_all = a.sink ? expf(a.sink[h] - m_all) : 0.f, acc = 0.f;
#pragma unroll
  for (int w = 0; w < kRowWarps; ++w) {
    if (part_m[w] == -INFINITY) continue;
    const float f = expf(part_m[w] - m_all);
    l_all += part_l[w] * f;
    acc = fmaf(part_acc[w][d], f, acc);
  }
  a.out[(size_t)t * a.ldo + (size_t)h * kHd + d] = acc * (1.0f / l_all);
}

__device__ __forceinline__ void copy16_or_zero(float* dst, const float* src, bool real) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
               "r"(real ? 16 : 0) : "memory");
}

constexpr int kTileSmem = (4 * kTileKeys + 2 * kTileRows) * kLd * (int)sizeof(float);

__global__ void __launch_bounds__(128)
attn_f32_tile_kernel(const AttnF32 a, int leave_short) {
  extern __shared__ __align__(16) float sm[];
  float* kv = sm;                                    // two stages of [keys | values]
  float* qs = sm + 4 * kTileKeys * kLd;
  float* ps = qs + kTileRows * kLd;
  __shared__ int pos_s[kTileRows], first_s[kTileRows];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;            // rows ty + 8 i; keys tx + 16 j, channels 4 tx
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
        const bool real = blk >= 0 && key0 + tile * kTileKeys + r <= p1;
        copy16_or_zero(st + r * kLd + d, kb + i * 4, real);
        copy16_or_zero(st + (kTileKeys + r) * kLd + d, vb + i * 4, real);
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
      float2 s2[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s2[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
      for (int d = 0; d < kHd; d += 4) {
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
      float corr[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = ty + 8 * i, pos = pos_s[r], first = first_s[r];
        float s[4], top = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = key0 + tile * kTileKeys + tx + 16 * j;
          const bool seen = key <= pos && key >= first && mapped;
          s[j] = seen ? (s2[i][j].x + s2[i][j].y) * a.scale - tilt * (float)(pos - key) : -INFINITY;
          top = fmaxf(top, s[j]);
        }
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
        const float m_new = fmaxf(m[i], top);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float p = s[j] == -INFINITY ? 0.f : expf(s[j] - m_new);
          ps[r * kLd + tx + 16 * j] = p;
          sum += p;
        }
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
        corr[i] = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
        l[i] = l[i] * corr[i] + sum;
        m[i] = m_new;
      }
      __syncwarp();                                  // a row's probabilities stay in its half warp
      float2 x2[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) x2[i][0] = x2[i][1] = make_float2(0.f, 0.f);
#pragma unroll 2
      for (int key = 0; key < kTileKeys; key += 4) {
        float4 vf[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          vf[u] = *reinterpret_cast<const float4*>(vs + (key + u) * kLd + 4 * tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 pf = *reinterpret_cast<const float4*>(ps + (ty + 8 * i) * kLd + key);
          const float pu[4] = {pf.x, pf.y, pf.z, pf.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 pp = make_float2(pu[u], pu[u]);
            x2[i][0] = __ffma2_rn(pp, make_float2(vf[u].x, vf[u].y), x2[i][0]);
            x2[i][1] = __ffma2_rn(pp, make_float2(vf[u].z, vf[u].w), x2[i][1]);
          }
        }
      }
      // A key that a row does not see has probability 0, and 0 times an infinite value is no
      // number: where one turns up the sums are taken again over the seen keys alone.
      float odd = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        odd += 0.f * ((x2[i][0].x + x2[i][0].y) + (x2[i][1].x + x2[i][1].y));
      if (odd != 0.f) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float y[4] = {0.f, 0.f, 0.f, 0.f};
          for (int key = 0; key < kTileKeys; ++key) {
            const float p = ps[(ty + 8 * i) * kLd + key];
            if (p != 0.f)
              for (int d = 0; d < 4; ++d) y[d] = fmaf(p, vs[key * kLd + 4 * tx + d], y[d]);
          }
          x2[i][0] = make_float2(y[0], y[1]);
          x2[i][1] = make_float2(y[2], y[3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[i][0] = fmaf(o[i][0], corr[i], x2[i][0].x);
        o[i][1] = fmaf(o[i][1], corr[i], x2[i][0].y);
        o[i][2] = fmaf(o[i][2], corr[i], x2[i][1].x);
        o[i][3] = fmaf(o[i][3], corr[i], x2[i][1].y);
      }
      __syncthreads();                               // the stage may be filled again
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty + 8 * i;
      if (r >= n) continue;
      float f = 1.0f, total = l[i];
      if (a.sink) {
        // one more term exp(sink) in the denominator, with no key and no value
        const float sk = a.sink[h], top = fmaxf(m[i], sk);
        f = m[i] == -INFINITY ? 0.f : expf(m[i] - top);
        total = l[i] * f + expf(sk - top);
      }
      f *= 1.0f / total;
      *reinterpret_cast<float4*>(a.out + (size_t)(lo + r) * a.ldo + (size_t)h * kHd + 4 * tx) =
          make_float4(o[i][0] * f, o[i][1] * f, o[i][2] * f, o[i][3] * f);
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
