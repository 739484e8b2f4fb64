// Paged attention of the float32 path, for head sizes up to 128 in multiples of 4: prompt portions and decoded tokens alike,
// a cluster of up to 8 CTAs per (token, kv head, up to 8 of its query heads).  (attention_generic.cu takes the rest.)
//
// A warp takes four keys at a time: its lanes hold 16 bytes of the head size each, so a key and a value are one coalesced
// 512-byte read, asked for one round ahead; the four keys meet all query heads of the group (read once per group, not once
// per head), and the dot products, 4 keys x 4 heads at a time, are folded over the lanes by halving, which leaves two lanes with
// the score of each head and key: 16 shuffles where a lane per key would read 32 rows at once, uncoalesced.  The running maximum and sum
// live in those lanes, the output in all of them.  Everything is float32.
//
// The order of every sum depends on the token's own position (and the window) alone, so the result does not depend on how the
// prompt was cut or on what else is in the batch: a token's n keys are 128 runs of 8 ceil(n / 1,024) keys; the 16 warps of a CTA
// take 16 neighbouring runs, merged in their order (a wave, at most 8 of them), and the waves are merged in theirs.  Which CTA of
// the cluster took a wave (wave w the CTA w mod size) does not matter: the waves' results lie in its shared memory, from where
// the others read them.  No memory is shared beyond the cluster.
//
// Bound by latency at the sizes of a step (8 MB of keys and values per layer for 4 tokens at context 1,000).  Measured on a
// B200 at the 3B sizes: that decode 2,395 us a layer with a warp per (token, head) in attention_generic.cu -> 10.2; a prompt of 203
// tokens 398 -> 29.4.  With shares of the keys that go by the batch (and scratch memory shared by all steps of the device) they were
// 10.0 and 24.6; one request at 2,048 tokens 11.2, now 14.7.
#include "common.cuh"
#include <math.h>

#define AF_WARPS 16
#define AF_KEYS 4
#define AF_WAVES 8

template <int M>
__device__ __forceinline__ float fold_lanes(float (&v)[M], int lane) {      // M <= 32: lane l has value l * M / 32 afterwards
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

// reads 16 bytes / 4 bytes at the same place in the shared memory of the cluster's CTA ``rank``
__device__ __forceinline__ unsigned af_at(const void* p, unsigned rank) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 af_ld4(unsigned a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 af_own4(unsigned a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float2 af_ld2(unsigned a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void af_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// what exponents are taken from: the maximum, or 0 where nothing was above minus infinity
__device__ __forceinline__ float af_base(float top) { return top == -INFINITY ? 0.f : top; }

template <int NH>
__global__ void __launch_bounds__(AF_WARPS * 32)
attention_f32_kernel(const float* __restrict__ q, long long q_stride, float* __restrict__ out, const float* __restrict__ kv,
                     const int* __restrict__ block_table, int max_blocks, const int* __restrict__ token_req,
                     const int* __restrict__ positions, int H, int G, int d, int page_size, float scale, int window,
                     int ctas, int blocks) {
  constexpr int HB = NH < 4 ? NH : 4, NF = NH / HB, M = AF_KEYS * HB, DUP = 32 / M;      // heads whose scores are folded together
  extern __shared__ float4 af_smem[];
  float4 (*so)[NH][32] = reinterpret_cast<float4 (*)[NH][32]>(af_smem);                        // [AF_WARPS]: a wave's runs
  float4 (*wave_o)[NH][32] = so + AF_WARPS;                                                    // [AF_WAVES / ctas]: this CTA's waves
  __shared__ float4 qs[NH][32];
  __shared__ float sm[AF_WARPS][NH], sl[AF_WARPS][NH];
  __shared__ float2 wave_ml[AF_WAVES][NH];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.z, rank = blockIdx.x, g = blockIdx.y / blocks, hb = blockIdx.y - g * blocks;
  const int group = H / G, h0 = g * group + hb * NH, nh = min(NH, group - hb * NH);
  const bool on = lane * 4 < d;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  // (eight heads' queries would not fit the registers beside the eight sums)
  if (warp < NH)
    qs[warp][lane] = on && warp < nh ? *reinterpret_cast<const float4*>(q + (size_t)t * q_stride + (size_t)(h0 + warp) * d + lane * 4) : zero;
  __syncthreads();
  const unsigned qs_at = (unsigned)__cvta_generic_to_shared(&qs[0][lane]);
  const int pos = positions[t];
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  const int n = pos + 1 - lo;
  const int run = 8 * ((n + 8 * AF_WAVES * AF_WARPS - 1) / (8 * AF_WAVES * AF_WARPS));
  const int waves = (n + run * AF_WARPS - 1) / (run * AF_WARPS);
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
  for (int wave = rank; wave < waves; wave += ctas) {
    float4 o[NH];
#pragma unroll
    for (int h = 0; h < NH; h++) o[h] = zero;
    float m[NF], l[NF];
#pragma unroll
    for (int f = 0; f < NF; f++) { m[f] = -INFINITY; l[f] = 0.f; }
    int k0 = lo + (wave * AF_WARPS + warp) * run;
    const int k_end = min(pos + 1, k0 + run);
    if (k0 < k_end) fetch(k0);
    for (; k0 < k_end; k0 += AF_KEYS) {
      float sc[NF];                                  // head f HB + lane / DUP / 4, key lane / DUP % 4
#pragma unroll
      for (int f = 0; f < NF; f++) {
        float s[M];
#pragma unroll
        for (int h = 0; h < HB; h++) {
          const float4 x = af_own4(qs_at + (f * HB + h) * 512);
#pragma unroll
          for (int j = 0; j < AF_KEYS; j++) {
            float a = x.x * kc[j].x;
            a = fmaf(x.y, kc[j].y, a); a = fmaf(x.z, kc[j].z, a); a = fmaf(x.w, kc[j].w, a);
            s[h * AF_KEYS + j] = a;
          }
        }
        sc[f] = fold_lanes<M>(s, lane) * scale;
      }
      float4 v[AF_KEYS];
#pragma unroll
      for (int j = 0; j < AF_KEYS; j++) v[j] = vc[j];
      if (k0 + AF_KEYS < k_end) fetch(k0 + AF_KEYS);
      const bool valid = k0 + (lane / DUP) % AF_KEYS < k_end;
#pragma unroll
      for (int f = 0; f < NF; f++) {
        const float x = valid ? sc[f] : -INFINITY;
        float top = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, DUP));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2 * DUP));
        const float m_new = fmaxf(m[f], top), from = af_base(m_new);
        const float c = expf(m[f] - from), p = valid ? expf(x - from) : 0.f;
        float sum = p + __shfl_xor_sync(0xffffffffu, p, DUP);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2 * DUP);
        l[f] = l[f] * c + sum;
        const bool grown = __any_sync(0xffffffffu, m_new != m[f]);
        m[f] = m_new;
#pragma unroll
        for (int i = 0; i < HB; i++) {
          float4& acc = o[f * HB + i];
          if (grown) {
            const float ch = __shfl_sync(0xffffffffu, c, i * AF_KEYS * DUP);
            acc.x *= ch; acc.y *= ch; acc.z *= ch; acc.w *= ch;
          }
#pragma unroll
          for (int j = 0; j < AF_KEYS; j++) {
            const float pj = __shfl_sync(0xffffffffu, p, (i * AF_KEYS + j) * DUP);
            acc.x = fmaf(pj, v[j].x, acc.x); acc.y = fmaf(pj, v[j].y, acc.y);
            acc.z = fmaf(pj, v[j].z, acc.z); acc.w = fmaf(pj, v[j].w, acc.w);
          }
        }
      }
    }
    if (wave != rank) __syncthreads();               // the wave before is merged
#pragma unroll
    for (int h = 0; h < NH; h++) so[warp][h][lane] = o[h];
    if (lane % (AF_KEYS * DUP) == 0)
#pragma unroll
      for (int f = 0; f < NF; f++) { sm[warp][f * HB + lane / (AF_KEYS * DUP)] = m[f]; sl[warp][f * HB + lane / (AF_KEYS * DUP)] = l[f]; }
    __syncthreads();
    // warp h: head h; a run without keys has the maximum -inf and adds nothing
    if (warp < nh) {
      float top = -INFINITY;
#pragma unroll
      for (int w = 0; w < AF_WARPS; w++) top = fmaxf(top, sm[w][warp]);
      const float from = af_base(top);
      float4 a = zero;
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < AF_WARPS; w++) {
        const float f = expf(sm[w][warp] - from);
        const float4 b = so[w][warp][lane];
        sum = fmaf(sl[w][warp], f, sum);
        a.x = fmaf(b.x, f, a.x); a.y = fmaf(b.y, f, a.y); a.z = fmaf(b.z, f, a.z); a.w = fmaf(b.w, f, a.w);
      }
      wave_o[wave / ctas][warp][lane] = a;
      if (lane == 0) wave_ml[wave / ctas][warp] = make_float2(top, sum);
    }
  }
  if (ctas > 1) af_cluster_sync(); else __syncthreads();
  const int h = warp * ctas + rank;                  // the heads are shared among the cluster's CTAs
  if (h < nh) {
    float top = -INFINITY, sum = 0.f;
    float4 a = zero;
    float2 ml[AF_WAVES];
    float4 b[AF_WAVES];
#pragma unroll
    for (int w = 0; w < AF_WAVES; w++) {
      const int cta = w % ctas, at = w / ctas;
      ml[w] = w < waves ? af_ld2(af_at(&wave_ml[at][h], cta)) : make_float2(-INFINITY, 0.f);
      b[w] = w < waves ? af_ld4(af_at(&wave_o[at][h][lane], cta)) : zero;
    }
#pragma unroll
    for (int w = 0; w < AF_WAVES; w++) {
      if (w >= waves) break;
      const float best = fmaxf(top, ml[w].x), from = af_base(best);
      const float fa = expf(top - from), fb = expf(ml[w].x - from);
      top = best;
      sum = fmaf(ml[w].y, fb, sum * fa);
      a.x = fmaf(b[w].x, fb, a.x * fa); a.y = fmaf(b[w].y, fb, a.y * fa);
      a.z = fmaf(b[w].z, fb, a.z * fa); a.w = fmaf(b[w].w, fb, a.w * fa);
    }
    const float inv = 1.0f / sum;
    if (on)
      *reinterpret_cast<float4*>(out + ((size_t)t * H + h0 + h) * d + lane * 4) =
          make_float4(a.x * inv, a.y * inv, a.z * inv, a.w * inv);
  }
  if (ctas > 1) af_cluster_sync();                   // nobody leaves while its shared memory is read
}

template <int NH>
static int launch_attention_f32(dim3 grid, cudaStream_t stream, const float* q, long long q_stride, float* out, const float* kv,
                                const int* block_table, int max_blocks, const int* token_req, const int* positions, int H, int G,
                                int d, int page_size, float scale, int window, int ctas, int blocks) {
  const int smem = (AF_WARPS + AF_WAVES / ctas) * NH * 32 * (int)sizeof(float4);
  const cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(AF_WARPS * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = qd_pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&cfg, attention_f32_kernel<NH>, q, q_stride, out, kv, block_table, max_blocks, token_req, positions, H, G, d,
                     page_size, scale, window, ctas, blocks);
  return qd_last_error();
}

// q rows ``q_stride`` apart, out [T, H * d]; kv [pages, 2, G, page_size, d].  ``ctas``: CTAs of a cluster, 1, 2, 4 or 8; the
// result does not depend on it.
extern "C" int qd_attention_f32(const float* q, long long q_stride, float* out, const float* kv, const int* block_table,
                                int max_blocks, const int* token_req, const int* positions, int T, int H, int G, int d,
                                int page_size, float scale, int window, int ctas, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (d <= 0 || d > 128 || d % 4 || G <= 0 || H <= 0 || H % G || page_size <= 0 || q_stride % 4 ||
      (ctas != 1 && ctas != 2 && ctas != 4 && ctas != 8) || (((uintptr_t)q | (uintptr_t)out | (uintptr_t)kv) & 15))
    return QD_ERR_UNSUPPORTED;
  const int group = H / G, nh = group >= 5 ? 8 : group >= 3 ? 4 : group, blocks = (group + nh - 1) / nh;
  if ((long long)G * blocks > 65535) return QD_ERR_UNSUPPORTED;
  for (int t0 = 0; t0 < T; t0 += 65535) {            // as many tokens as a grid takes
    const dim3 grid(ctas, G * blocks, T - t0 < 65535 ? T - t0 : 65535);
    const float* qt = q + (long long)t0 * q_stride;
    float* ot = out + (size_t)t0 * H * d;
    int rc = 0;
#define AF(NH)                                                                                                              \
    rc = launch_attention_f32<NH>(grid, stream, qt, q_stride, ot, kv, block_table, max_blocks, token_req + t0, positions + t0, \
                                  H, G, d, page_size, scale, window, ctas, blocks)
    if (nh == 8) AF(8); else if (nh == 4) AF(4); else if (nh == 2) AF(2); else AF(1);
#undef AF
    if (rc) return rc;
  }
  return 0;
}
