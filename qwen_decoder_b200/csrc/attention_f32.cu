// Paged attention of the float32 path, for head sizes up to 128 in multiples of 4: prompt portions and decoded tokens alike,
// one CTA per (token, kv head, up to 8 of its query heads, share of the keys).  (attention_generic.cu takes the rest.)
//
// A warp takes four keys at a time: its lanes hold 16 bytes of the head size each, so a key and a value are one coalesced
// 512-byte read, asked for one round ahead; the four keys meet all query heads of the group (read once per group, not once
// per head), and the 4 x 8 dot products are folded over the lanes by halving, which leaves lane (4 h + j) with the score of
// head h and key j: 31 shuffles where a lane per key would read 32 rows at once, uncoalesced.  The running maximum and sum
// live in those lanes, the output in all of them.  The CTA's 8 warps merge through shared memory; shares of the keys merge
// through scratch memory, by the CTA that finishes last.  Everything is float32.
//
// Bound by latency at the sizes of a step (8 MB of keys and values per layer for 4 tokens at context 1,000).  Measured on a
// B200 at the 3B sizes: that decode 2,395 us a layer with a warp per (token, head) in attention_generic.cu -> 11.6; a prompt of
// 203 tokens 398 -> 25.6.
#include "common.cuh"
#include <math.h>

#define AF_WARPS 8
#define AF_KEYS 4

template <int M>
__device__ __forceinline__ float fold_lanes(float (&v)[M], int lane) {      // as in gemm_f32.cu, M <= 32
  int m = M;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    if (m > 1) {
      const int half = m >> 1;
      const bool upper = lane & o;
#pragma unroll
      for (int i = 0; i < M / 2; i++) {
        if (i < half) {
          const float send = upper ? v[i] : v[i + half];
          const float keep = upper ? v[i + half] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      m = half;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];
}

template <int NH>
__global__ void __launch_bounds__(AF_WARPS * 32)
attention_f32_kernel(const float* __restrict__ q, long long q_stride, float* __restrict__ out, const float* __restrict__ kv,
                     const int* __restrict__ block_table, int max_blocks, const int* __restrict__ token_req,
                     const int* __restrict__ positions, int H, int G, int d, int page_size, float scale, int window,
                     int splits, int blocks, float* __restrict__ part_o, float* __restrict__ part_ml,
                     unsigned* __restrict__ tickets) {
  constexpr int M = AF_KEYS * NH, DUP = 32 / M;
  __shared__ float4 so[AF_WARPS][NH][32];
  __shared__ float sm[AF_WARPS][NH], sl[AF_WARPS][NH];
  __shared__ bool last;
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.z, split = blockIdx.x, g = blockIdx.y / blocks, hb = blockIdx.y - g * blocks;
  const int group = H / G, h0 = g * group + hb * NH, nh = min(NH, group - hb * NH);
  const bool on = lane * 4 < d;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 qv[NH], o[NH];
#pragma unroll
  for (int h = 0; h < NH; h++) {
    qv[h] = on && h < nh ? *reinterpret_cast<const float4*>(q + (size_t)t * q_stride + (size_t)(h0 + h) * d + lane * 4) : zero;
    o[h] = zero;
  }
  const int pos = positions[t];
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  // whole rounds of the CTA (32 keys) to a share
  const int rounds = (pos - lo) / (AF_WARPS * AF_KEYS) + 1;
  const int k_begin = lo + (int)((long long)rounds * split / splits) * AF_WARPS * AF_KEYS;
  const int k_end = min(pos + 1, lo + (int)((long long)rounds * (split + 1) / splits) * AF_WARPS * AF_KEYS);
  const int* bt = block_table + (size_t)token_req[t] * max_blocks;
  const size_t page_elems = (size_t)2 * G * page_size * d, v_off = (size_t)G * page_size * d;
  const float* base = kv + (size_t)g * page_size * d + lane * 4;

  float4 kc[AF_KEYS], vc[AF_KEYS];
  auto fetch = [&](int key0) {
    // lane j & 3 finds the row of key j; a key past the end reads the last one and counts for nothing
    const int key = min(key0 + (lane & 3), pos);
    const int in_table = key / page_size;
    const size_t at = (size_t)bt[in_table] * page_elems + (size_t)(key - in_table * page_size) * d;
#pragma unroll
    for (int j = 0; j < AF_KEYS; j++) {
      const float* r = base + __shfl_sync(0xffffffffu, (unsigned long long)at, j);
      kc[j] = on ? __ldg(reinterpret_cast<const float4*>(r)) : zero;
      vc[j] = on ? __ldg(reinterpret_cast<const float4*>(r + v_off)) : zero;
    }
  };
  float m = -INFINITY, l = 0.f;
  int k0 = k_begin + warp * AF_KEYS;
  if (k0 < k_end) fetch(k0);
  for (; k0 < k_end; k0 += AF_WARPS * AF_KEYS) {
    float s[M];
#pragma unroll
    for (int h = 0; h < NH; h++)
#pragma unroll
      for (int j = 0; j < AF_KEYS; j++) {
        float a = qv[h].x * kc[j].x;
        a = fmaf(qv[h].y, kc[j].y, a); a = fmaf(qv[h].z, kc[j].z, a); a = fmaf(qv[h].w, kc[j].w, a);
        s[h * AF_KEYS + j] = a;
      }
    float4 v[AF_KEYS];
#pragma unroll
    for (int j = 0; j < AF_KEYS; j++) v[j] = vc[j];
    if (k0 + AF_WARPS * AF_KEYS < k_end) fetch(k0 + AF_WARPS * AF_KEYS);
    float sc = fold_lanes<M>(s, lane) * scale;       // head lane / DUP / 4, key lane / DUP % 4
    const bool valid = k0 + (lane / DUP) % AF_KEYS < k_end;
    sc = valid ? sc : -INFINITY;
    float top = fmaxf(sc, __shfl_xor_sync(0xffffffffu, sc, DUP));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2 * DUP));
    const float m_new = fmaxf(m, top);               // finite: the first key of a round is always there
    const float c = expf(m - m_new), p = valid ? expf(sc - m_new) : 0.f;
    float sum = p + __shfl_xor_sync(0xffffffffu, p, DUP);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2 * DUP);
    l = l * c + sum;
    const bool grown = __any_sync(0xffffffffu, m_new != m);
    m = m_new;
#pragma unroll
    for (int h = 0; h < NH; h++) {
      if (grown) {
        const float ch = __shfl_sync(0xffffffffu, c, h * AF_KEYS * DUP);
        o[h].x *= ch; o[h].y *= ch; o[h].z *= ch; o[h].w *= ch;
      }
#pragma unroll
      for (int j = 0; j < AF_KEYS; j++) {
        const float pj = __shfl_sync(0xffffffffu, p, (h * AF_KEYS + j) * DUP);
        o[h].x = fmaf(pj, v[j].x, o[h].x); o[h].y = fmaf(pj, v[j].y, o[h].y);
        o[h].z = fmaf(pj, v[j].z, o[h].z); o[h].w = fmaf(pj, v[j].w, o[h].w);
      }
    }
  }
#pragma unroll
  for (int h = 0; h < NH; h++) so[warp][h][lane] = o[h];
  if (lane % (AF_KEYS * DUP) == 0) { sm[warp][lane / (AF_KEYS * DUP)] = m; sl[warp][lane / (AF_KEYS * DUP)] = l; }
  __syncthreads();
  // warp w: heads w, w + 8, ... (NH <= 8: one head); a warp without keys has the maximum -inf and adds nothing
  if (warp < nh) {
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < AF_WARPS; w++) top = fmaxf(top, sm[w][warp]);
    float4 a = zero;
    float sum = 0.f;
    if (top != -INFINITY) {
#pragma unroll
      for (int w = 0; w < AF_WARPS; w++) {
        const float f = expf(sm[w][warp] - top);
        const float4 b = so[w][warp][lane];
        sum = fmaf(sl[w][warp], f, sum);
        a.x = fmaf(b.x, f, a.x); a.y = fmaf(b.y, f, a.y); a.z = fmaf(b.z, f, a.z); a.w = fmaf(b.w, f, a.w);
      }
    }
    if (splits == 1) {
      const float inv = 1.0f / sum;
      if (on)
        *reinterpret_cast<float4*>(out + ((size_t)t * H + h0 + warp) * d + lane * 4) =
            make_float4(a.x * inv, a.y * inv, a.z * inv, a.w * inv);
    } else {
      const size_t at = ((size_t)t * H + h0 + warp) * splits + split;
      if (on) *reinterpret_cast<float4*>(part_o + at * d + lane * 4) = a;
      if (lane == 0) { part_ml[at * 2] = top; part_ml[at * 2 + 1] = sum; }
      __threadfence();
    }
  }
  if (splits == 1) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned* ticket = tickets + (size_t)t * gridDim.y + blockIdx.y;
    last = atomicAdd(ticket, 1u) == (unsigned)splits - 1;
    if (last) *ticket = 0;                           // as it was found
  }
  __syncthreads();
  if (!last || warp >= nh) return;
  __threadfence();
  const size_t at = ((size_t)t * H + h0 + warp) * splits;
  float top = -INFINITY, sum = 0.f;
  float4 a = zero;
  constexpr int PB = 8;                              // shares in flight: each would be a trip to L2 of its own
  for (int s0 = 0; s0 < splits; s0 += PB) {
    float2 mlv[PB];
    float4 pv[PB];
#pragma unroll
    for (int u = 0; u < PB; u++) {
      const bool in = s0 + u < splits;
      mlv[u] = in ? __ldcg(reinterpret_cast<const float2*>(part_ml) + at + s0 + u) : make_float2(-INFINITY, 0.f);
      pv[u] = in && on ? __ldcg(reinterpret_cast<const float4*>(part_o + (at + s0 + u) * d + lane * 4)) : zero;
    }
    float best = top;
#pragma unroll
    for (int u = 0; u < PB; u++) best = fmaxf(best, mlv[u].x);
    if (best == -INFINITY) continue;                 // none of these shares had a key
    const float old = expf(top - best);
    top = best;
    sum *= old; a.x *= old; a.y *= old; a.z *= old; a.w *= old;
#pragma unroll
    for (int u = 0; u < PB; u++) {
      const float f = expf(mlv[u].x - best);
      sum = fmaf(mlv[u].y, f, sum);
      a.x = fmaf(pv[u].x, f, a.x); a.y = fmaf(pv[u].y, f, a.y); a.z = fmaf(pv[u].z, f, a.z); a.w = fmaf(pv[u].w, f, a.w);
    }
  }
  const float inv = 1.0f / sum;
  if (on)
    *reinterpret_cast<float4*>(out + ((size_t)t * H + h0 + warp) * d + lane * 4) =
        make_float4(a.x * inv, a.y * inv, a.z * inv, a.w * inv);
}

// q rows ``q_stride`` apart, out [T, H * d]; kv [pages, 2, G, page_size, d].  ``splits`` > 1: scratch part_o
// [T * H * splits, d], part_ml [T * H * splits, 2] and zeroed tickets [T * G * ceil(H / G / 8)], left zero.
extern "C" int qd_attention_f32(const float* q, long long q_stride, float* out, const float* kv, const int* block_table,
                                int max_blocks, const int* token_req, const int* positions, int T, int H, int G, int d,
                                int page_size, float scale, int window, int splits, float* part_o, float* part_ml,
                                unsigned* tickets, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (d <= 0 || d > 128 || d % 4 || G <= 0 || H <= 0 || H % G || page_size <= 0 || splits < 1 || T > 65535 || q_stride % 4 ||
      (((uintptr_t)q | (uintptr_t)out | (uintptr_t)kv | (uintptr_t)part_o) & 15))
    return QD_ERR_UNSUPPORTED;
  if (splits > 1 && (!part_o || !part_ml || !tickets)) return QD_ERR_UNSUPPORTED;
  const int group = H / G, nh = group >= 5 ? 8 : group >= 3 ? 4 : group, blocks = (group + nh - 1) / nh;
  if ((long long)G * blocks > 65535) return QD_ERR_UNSUPPORTED;
  const dim3 grid(splits, G * blocks, T);
#define AF(NH)                                                                                                        \
  qd_launch(attention_f32_kernel<NH>, grid, dim3(AF_WARPS * 32), 0, stream, q, q_stride, out, kv, block_table, max_blocks, \
            token_req, positions, H, G, d, page_size, scale, window, splits, blocks, part_o, part_ml, tickets)
  if (nh == 8) AF(8); else if (nh == 4) AF(4); else if (nh == 2) AF(2); else AF(1);
#undef AF
  return qd_last_error();
}
