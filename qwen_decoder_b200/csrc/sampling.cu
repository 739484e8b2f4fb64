// Sampling over float32 logits on the device: greedy, temperature, top-k.
//
// Semantics of the reference's host sampler (common.cpp:564-629): temperature 0 is
// argmax with the lowest index winning ties (common.cpp:564-574); otherwise
// p_i = exp((l_i - max) / T) over the kept entries, normalised, and the first index
// whose running sum reaches the uniform draw r is returned (common.cpp:590-598);
// with 0 < k < V only entries >= the k-th largest logit are kept, ties included
// (common.cpp:600-618).  The draw r is given per row by the caller, so that a request's
// draws do not depend on the batch it is in.
#include "common.cuh"
#include <math.h>

#define SB 1024
#define S_AHEAD 8          // loads of a thread in flight: a row is one multiprocessor's 600 KB from L2, several times
#define S_LIST 2048        // entries that may be among the k largest, at most
#define S_WALK 256         // a list up to here is searched by every thread, once for each of its entries; else the row's segments

// One CTA per row.  The k-th largest logit: the k-th largest of the 1,024 threads' own maxima is a lower bound of it (each is an
// entry of its own), so one more pass collects the entries that reach the bound, usually little more than k, and what follows
// works on that list; four passes with counts in shared memory (most logits share a few leading bytes, and their counters) remain
// for k above 1,024 and for lists that overflow.  Four rows of 151,936 logits, k = 40, the whole kernel: 132 us with those passes, 60 so.

__device__ __forceinline__ unsigned order_key(float f) {
  unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // ascending in float order
}
__device__ __forceinline__ float key_to_float(unsigned k) {
  unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

__global__ void __launch_bounds__(SB)
sample_kernel(const float* __restrict__ logits, int V, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ draws, int* __restrict__ out) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float s_val[SB];
  __shared__ int s_idx[SB];
  __shared__ unsigned s_hist[256];
  __shared__ float s_scratch[40];
  __shared__ unsigned s_prefix, s_remaining;
  __shared__ int s_result, s_count;
  __shared__ unsigned list_key[S_LIST], s_some[SB / 32];
  __shared__ int list_idx[S_LIST];
  int r = blockIdx.x, tid = threadIdx.x;
  const float* row = logits + (size_t)r * V;

  // 1. maximum and its lowest index
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int i0 = tid; i0 < V; i0 += S_AHEAD * SB) {
    float v[S_AHEAD];
#pragma unroll
    for (int u = 0; u < S_AHEAD; u++) v[u] = i0 + u * SB < V ? row[i0 + u * SB] : 0.0f;
#pragma unroll
    for (int u = 0; u < S_AHEAD; u++) {
      const int i = i0 + u * SB;
      if (i < V && (v[u] > best || bi == 0x7fffffff)) { best = v[u]; bi = i; }
    }
  }
  const unsigned own_key = order_key(best);
  s_val[tid] = best; s_idx[tid] = bi;
  __syncthreads();
  for (int s = SB / 2; s > 0; s >>= 1) {
    if (tid < s) {
      float ov = s_val[tid + s]; int oi = s_idx[tid + s];
      if (oi != 0x7fffffff && (s_idx[tid] == 0x7fffffff || ov > s_val[tid] ||
                               (ov == s_val[tid] && oi < s_idx[tid]))) {
        s_val[tid] = ov; s_idx[tid] = oi;
      }
    }
    __syncthreads();
  }
  float mx = s_val[0];
  int amax = s_idx[0];
  float temp = temperature[r];
  if (temp == 0.0f) {
    if (tid == 0) out[r] = amax;
    return;
  }

  // 2. threshold = k-th largest logit (radix select on order-preserving keys)
  int k = top_k[r];
  float threshold = -INFINITY;
  bool listed = false;
  if (k > 0 && k < V && k <= SB) {
    // the k-th largest of the threads' maxima, then of the list, by the same selection on keys
    auto select = [&](int n, auto&& key_at) {
      if (tid == 0) { s_prefix = 0; s_remaining = (unsigned)k; }
      __syncthreads();
      for (int shift = 24; shift >= 0; shift -= 8) {
        if (tid < 256) s_hist[tid] = 0;
        __syncthreads();
        const unsigned prefix = s_prefix, mask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
        for (int i = tid; i < n; i += SB) {
          const unsigned key = key_at(i);
          if ((key & mask) == prefix) atomicAdd(&s_hist[(key >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (tid < 32) {
          // lane l holds the eight digits below 256 - 8 l: the digit where the count from above reaches the rest
          unsigned c[8], sum = 0;
#pragma unroll
          for (int u = 0; u < 8; u++) { c[u] = s_hist[255 - (tid * 8 + u)]; sum += c[u]; }
          unsigned incl = sum;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
            if (tid >= o) incl += v;
          }
          const unsigned rem = s_remaining, before = incl - sum;
          __syncwarp();
          if (before < rem && rem <= incl) {
            unsigned left = rem - before;
            int u = 0;
            while (left > c[u]) left -= c[u++];
            s_prefix = prefix | ((unsigned)(255 - (tid * 8 + u)) << shift);
            s_remaining = left;
          }
        }
        __syncthreads();
      }
      return s_prefix;
    };
    unsigned bound = select(SB, [&](int) { return own_key; });
    // kept is what reaches the threshold by value, and -0 reaches +0 though its key lies below
    if (bound == order_key(0.0f)) bound = order_key(-0.0f);
    if (tid == 0) s_count = 0;
    __syncthreads();
    for (int i0 = tid; i0 < V; i0 += S_AHEAD * SB) {
      float v[S_AHEAD];
#pragma unroll
      for (int u = 0; u < S_AHEAD; u++) v[u] = i0 + u * SB < V ? row[i0 + u * SB] : 0.0f;
#pragma unroll
      for (int u = 0; u < S_AHEAD; u++) {
        const int i = i0 + u * SB;
        const unsigned key = order_key(v[u]);
        if (i < V && key >= bound) {
          const int at = atomicAdd(&s_count, 1);
          if (at < S_LIST) { list_key[at] = key; list_idx[at] = i; }
        }
      }
    }
    __syncthreads();
    listed = s_count <= S_LIST;
    if (listed) threshold = key_to_float(select(s_count, [&](int i) { return list_key[i]; }));
  }
  if (k > 0 && k < V && !listed) {
    if (tid == 0) { s_prefix = 0; s_remaining = (unsigned)k; }
    __syncthreads();
    for (int shift = 24; shift >= 0; shift -= 8) {
      if (tid < 256) s_hist[tid] = 0;
      __syncthreads();
      unsigned prefix = s_prefix;
      unsigned mask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
      for (int i = tid; i < V; i += SB) {
        unsigned key = order_key(row[i]);
        if ((key & mask) == prefix) atomicAdd(&s_hist[(key >> shift) & 255u], 1u);
      }
      __syncthreads();
      if (tid == 0) {
        unsigned rem = s_remaining;
        int dgt = 255;
        for (; dgt > 0; dgt--) {
          unsigned c = s_hist[dgt];
          if (c >= rem) break;
          rem -= c;
        }
        s_prefix = prefix | ((unsigned)dgt << shift);
        s_remaining = rem;
      }
      __syncthreads();
    }
    threshold = key_to_float(s_prefix);
  }

  // 3. each thread owns a contiguous segment; segment sums of the kept probabilities
  int seg = (V + SB - 1) / SB;
  int lo = tid * seg, hi = lo + seg < V ? lo + seg : V;
  float part = 0.0f;
  const int n = s_count;
  if (listed && n <= S_WALK) {
    // every entry that is kept is in the list: those of the segment in their order
    for (int last = lo - 1; last < hi;) {
      int next = hi;
      float v = 0.0f;
      for (int j = 0; j < n; j++) {
        const int i = list_idx[j];
        if (i > last && i < next) {
          const float w = key_to_float(list_key[j]);
          if (w >= threshold) { next = i; v = w; }
        }
      }
      if (next < hi) part += expf((v - mx) / temp);
      last = next;
    }
  } else {
    for (int i = lo; i < hi; i++) {
      float v = row[i];
      if (v >= threshold) part += expf((v - mx) / temp);
    }
  }
  s_val[tid] = part;
  // which segments hold anything: the search below passes over the others
  {
    const unsigned some = __ballot_sync(0xffffffffu, part > 0.0f);
    if ((tid & 31) == 0) s_some[tid >> 5] = some;
  }
  __syncthreads();
  float total = block_sum(part, s_scratch);
  // 4. first index whose running sum reaches r * total
  if (tid == 0) {
    float target = draws[r] * total;
    float cum = 0.0f;
    int found = -1;
    for (int word = 0; word < SB / 32 && found < 0; word++)
    for (unsigned bits = s_some[word]; bits && found < 0; bits &= bits - 1) {
      const int sgi = word * 32 + __ffs(bits) - 1;
      float next = cum + s_val[sgi];
      if (target <= next) {
        int a = sgi * seg, b = a + seg < V ? a + seg : V;
        for (int i = a; i < b; i++) {
          float v = row[i];
          if (v >= threshold) {
            cum += expf((v - mx) / temp);
            if (target <= cum) { found = i; break; }
          }
        }
        if (found < 0) cum = next;  // rounding: go on with the next segment
      } else {
        cum = next;
      }
    }
    s_result = found >= 0 ? found : amax;
  }
  __syncthreads();
  if (tid == 0) out[r] = s_result;
}

extern "C" int qd_sample(const float* logits, int R, int V, const float* temperature, const int* top_k,
                         const float* draws, int* out, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (V <= 0) return QD_ERR_UNSUPPORTED;
  qd_launch(sample_kernel, dim3(R), dim3(SB), 0, stream, logits, V, temperature, top_k, draws, out);
  return qd_last_error();
}
