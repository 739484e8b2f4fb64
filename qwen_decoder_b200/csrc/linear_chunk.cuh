// Linear attention over portions in chunks of LC tokens, on the tensor cores (the general kernels of linear_scan.cu go token by
// token: a serial chain of 0.1 us a token that leaves most of the GPU waiting).  For heads of 64 x 64 or 128 x 128 (keys x values)
// without the delta rule.  With S0 the state before a chunk, g_i the decays, G_p = g_0 .. g_p, d(s, p) = g_(s+1) .. g_p:
//
//   o_p = G_p S0^T q_p + sum_(s <= p) d(s, p) (k_s . q_p) v_s,   S <- G S0 + sum_s d(s, last) k_s v_s^T
//
// Three launches a pass of as many chunks as the scratch holds: what a chunk adds to the state, sum_s d(s, last) k_s v_s^T, all chunks at once; the states before the chunks, one
// after the other; the outputs with norm and gate, all chunks at once.
//
// The delta rule has no such form here.  There the values' place is taken by the solution of a triangular system a chunk, and rounded
// to float32 it was further from float64 than the kernels that go four tokens at a time: 512 tokens, keys and queries whose common part
// is 0.9, decays from 0.9 on: outputs 2.8e-7 against 1.3e-7, states 2.2e-7 against 1.3e-7; decays from 0.99 on: outputs 4.6e-7 against
// 1.6e-7 (266 us against 316 a call of 1,500 tokens, 32 heads of 128).  In a restatement with every sum rounded once the system's matrix,
// its right sides, its solution and the products of keys and queries all had to carry more than float32 to come below.
//
// Numbers stay float32: every operand is cut into three bfloat16 pieces that sum to it exactly, and of the nine products of pieces
// the six above 2^-24 are taken, the large one and the five small ones in sums of their own.  The tensor cores cut a running sum off at
// every addition: the large product of 16 k is made from zero and joins its sum by a rounded addition.  A decay's error is the same
// for all that a token left in the state and does not average out: a product of decays is rounded once.  Error from float64 of 512
// tokens of heads of 64, outputs and states, token by token / so / with running sums and every product of decays rounded (4 % less time):
// random keys, decays from 0.3 on 1.3e-7, 4.2e-8 / 9.3e-8, 6.1e-8 / 9.2e-8, 5.9e-8; from 0.99 on 3.1e-7, 3.5e-7 / 1.1e-7, 7.3e-8 /
// 1.5e-7, 2.6e-7; keys and queries whose common part is 0.99, decays from 0.99 on (700 tokens) 1.0e-7, 3.5e-7 / 1.1e-7, 5.9e-8 /
// 1.8e-7, 2.6e-7.
// A chunk that holds an infinity, NaN or a number beyond bfloat16's range takes its triangular products by FMA over s <= p only, so
// that tokens before it stay as they are.
#pragma once
#include "common.cuh"
#include "mma_sync.cuh"

#define LC 64                 // tokens of a chunk
#define LC_THREADS 256
#define LC_DEC 68             // numbers per (chunk, head): d(s, last) of the LC tokens, then the chunk's whole decay

struct LinearChunk {
  const float *q, *k;                     // [T, G, D]
  const float* v; long long ldv;
  const float* g; int g_ld;
  int T, R, H, G;
  float* state; long long state_stride, s_off;
  const int *cu_tokens, *slots; int write_state;
  float* dec;                             // [chunk, H, LC_DEC]
  float* s0;                              // [chunk, H, DV, D]: what the chunk adds to the state, then the state before it
  // The pass: chunks c0 .. c0 + pass - 1 of all (the arrays above hold these), and the state of the request that is cut between two
  // passes, [H, DV, D]: as the pass before left it, and for the next one (another place: two requests may meet in one pass).
  int c0, pass;
  const float* from; float* to;
  // norm, gate and result, as LinearFinish in linear_scan.cu
  const float* gate; long long gate_ld; const float* norm; int norm_ld; float eps, out_scale; int gate_kind;
  void* out; int out_dtype; long long out_stride;
};

// The pass's chunk ``b``: its request, its first token and how many it has; false past the last one.
__device__ __forceinline__ bool lc_find(const LinearChunk& a, int b, int& r, int& t0, int& n) {
  int at = 0;
  b += a.c0;
  for (r = 0; r < a.R; r++) {
    const int begin = a.cu_tokens[r], end = a.cu_tokens[r + 1], chunks = (end - begin + LC - 1) / LC;
    if (b < at + chunks) {
      t0 = begin + (b - at) * LC;
      n = min(LC, end - t0);
      return true;
    }
    at += chunks;
  }
  return false;
}

__device__ __forceinline__ unsigned lc_round2(float lo, float hi) {
  unsigned r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// the pieces of (x, y) as bfloat16 pairs
__device__ __forceinline__ void lc_cut(float x, float y, unsigned (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    p[i] = lc_round2(x, y);
    x -= __uint_as_float(p[i] << 16);
    y -= __uint_as_float(p[i] & 0xFFFF0000u);
  }
}
__device__ __forceinline__ bool lc_odd(float x) { return !(fabsf(x) <= 3.38e38f); }

// A tile of pieces in shared memory: [3][ROWS][W + 8] bfloat16 (eight rows of a matrix of ldmatrix fall on different banks)
template <int ROWS, int W>
struct LcTile {
  static constexpr int LD = W + 8, PIECE = ROWS * LD, ELEMS = 3 * PIECE;
};
// Rows of W numbers ``ld`` apart on their way into registers, the rows from ``n`` on zero, and from there into a tile; true if one of
// this thread's is odd.
template <int ROWS, int W, int THREADS>
__device__ __forceinline__ void lc_ask(float4 (&x)[ROWS * W / 4 / THREADS], const float* src, long long ld, int n) {
#pragma unroll
  for (int i = 0; i < ROWS * W / 4 / THREADS; i++) {
    const int e = threadIdx.x + i * THREADS, row = e / (W / 4), c = (e - row * (W / 4)) * 4;
    x[i] = row < n ? *reinterpret_cast<const float4*>(src + row * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
template <int ROWS, int W, int THREADS>
__device__ __forceinline__ bool lc_put(bf16* tile, const float4 (&x)[ROWS * W / 4 / THREADS]) {
  using L = LcTile<ROWS, W>;
  bool odd = false;
#pragma unroll
  for (int k = 0; k < ROWS * W / 4 / THREADS; k++) {
    const int e = threadIdx.x + k * THREADS, row = e / (W / 4), c = (e - row * (W / 4)) * 4;
    odd = odd || lc_odd(x[k].x) || lc_odd(x[k].y) || lc_odd(x[k].z) || lc_odd(x[k].w);
    unsigned lo[3], hi[3];
    lc_cut(x[k].x, x[k].y, lo);
    lc_cut(x[k].z, x[k].w, hi);
#pragma unroll
    for (int i = 0; i < 3; i++) *reinterpret_cast<uint2*>(tile + i * L::PIECE + row * L::LD + c) = make_uint2(lo[i], hi[i]);
  }
  return odd;
}
// both at once, eight pieces of 16 bytes a thread at a time
template <int ROWS, int W, int THREADS = LC_THREADS>
__device__ __forceinline__ bool lc_fill(bf16* tile, const float* src, long long ld, int n) {
  constexpr int TURN = ROWS * W / 4 / THREADS < 8 ? ROWS * W / 4 / THREADS : 8, STEP = TURN * THREADS * 4 / W;      // rows a turn
  static_assert(ROWS % STEP == 0 && TURN * THREADS * 4 % W == 0, "whole turns");
  bool odd = false;
#pragma unroll 1
  for (int row = 0; row < ROWS; row += STEP) {
    float4 x[TURN];
#pragma unroll
    for (int i = 0; i < TURN; i++) {
      const int e = threadIdx.x + i * THREADS, r = row + e / (W / 4), c = e % (W / 4) * 4;
      x[i] = r < n ? *reinterpret_cast<const float4*>(src + r * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    using L = LcTile<ROWS, W>;
#pragma unroll
    for (int k = 0; k < TURN; k++) {
      const int e = threadIdx.x + k * THREADS, r = row + e / (W / 4), c = e % (W / 4) * 4;
      odd = odd || lc_odd(x[k].x) || lc_odd(x[k].y) || lc_odd(x[k].z) || lc_odd(x[k].w);
      unsigned lo[3], hi[3];
      lc_cut(x[k].x, x[k].y, lo);
      lc_cut(x[k].z, x[k].w, hi);
#pragma unroll
      for (int i = 0; i < 3; i++) *reinterpret_cast<uint2*>(tile + i * L::PIECE + r * L::LD + c) = make_uint2(lo[i], hi[i]);
    }
  }
  return odd;
}

// Fragments of one piece.  A: 16 x 16 at (m, k), B: 16 (k) x 16 (n, two tiles of the MMA), from tiles whose rows run over the other
// index of the matrix (_t) or not.
__device__ __forceinline__ void lc_a(unsigned (&r)[4], const bf16* t, int ld, int m, int k, int lane) {        // rows m
  ts_ldmatrix_x4(r, t + (m + (lane & 7) + 8 * ((lane >> 3) & 1)) * ld + k + 8 * (lane >> 4));
}
__device__ __forceinline__ void lc_a_t(unsigned (&r)[4], const bf16* t, int ld, int m, int k, int lane) {      // rows k
  ts_ldmatrix_x4_trans(r, t + (k + (lane & 7) + 8 * (lane >> 4)) * ld + m + 8 * ((lane >> 3) & 1));
}
__device__ __forceinline__ void lc_b(unsigned (&r)[4], const bf16* t, int ld, int k, int n, int lane) {        // rows n
  ts_ldmatrix_x4(r, t + (n + (lane & 7) + 8 * (lane >> 4)) * ld + k + 8 * ((lane >> 3) & 1));
}
__device__ __forceinline__ void lc_b_t(unsigned (&r)[4], const bf16* t, int ld, int k, int n, int lane) {      // rows k
  ts_ldmatrix_x4_trans(r, t + (k + (lane & 7) + 8 * ((lane >> 3) & 1)) * ld + n + 8 * (lane >> 4));
}
__device__ __forceinline__ void lc_zero(float (&c)[2][4]) {
#pragma unroll
  for (int n = 0; n < 2; n++) c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0.f;
}
// Two tiles of 16 x 8: the large products into ``c``, the small ones into ``s`` (an MMA waits for the one before it into the same sum:
// the two tiles' take turns).
__device__ __forceinline__ void lc_mma(float (&c)[2][4], float (&s)[2][4], const unsigned (&a)[3][4], const unsigned (&b)[3][4]) {
  auto both = [&](float (&d)[2][4], int i, int j) {
#pragma unroll
    for (int n = 0; n < 2; n++) ts_mma(d[n], a[i], b[j][2 * n], b[j][2 * n + 1]);
  };
  float t[2][4];
  lc_zero(t);
  both(s, 0, 1);
  both(t, 0, 0);
  both(s, 1, 0);
  both(s, 1, 1);
  both(s, 0, 2);
  both(s, 2, 0);
#pragma unroll
  for (int n = 0; n < 2; n++)
#pragma unroll
    for (int e = 0; e < 4; e++) c[n][e] += t[n][e];
}

// A product of decays, rounded once: what the roundings on the way lose is carried along.
struct LcDecay {
  float d = 1.f, lost = 0.f;
  __device__ __forceinline__ void times(float x) {
    const float y = d * x;
    lost = fmaf(lost, x, fmaf(d, x, -y));
    d = y;
  }
  __device__ __forceinline__ float value() const { return fabsf(d) <= 3.402823466e38f ? d + lost : d; }      // (infinities stay)
};

// dm[p][s] = d(s, p) for s <= p < LC from the chunk's decays (1 past its end), dm's rows LC_DM apart
#define LC_DM (LC + 2)
__device__ __forceinline__ void lc_decays(const LinearChunk& a, int t0, int n, int h, float* gs, float* dm) {
  if (threadIdx.x < LC) gs[threadIdx.x] = (int)threadIdx.x < n ? a.g[(a.g_ld ? (size_t)(t0 + threadIdx.x) * a.g_ld : 0) + h] : 1.f;
  __syncthreads();
  if (threadIdx.x < 4 * LC) {                         // four threads a column: a quarter of its rows each
    const int s = threadIdx.x & (LC - 1), p0 = (threadIdx.x / LC) * (LC / 4);
    LcDecay d;
    for (int p = s + 1; p < p0; p++) d.times(gs[p]);
#pragma unroll
    for (int p1 = 0; p1 < LC / 4; p1 += 8) {
      float x[8];
#pragma unroll
      for (int i = 0; i < 8; i++) x[i] = gs[p0 + p1 + i];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int p = p0 + p1 + i;
        if (p > s) d.times(x[i]);
        dm[p * LC_DM + s] = p >= s ? d.value() : 0.f;
      }
    }
  }
  __syncthreads();
}

// ------------------------------------------------------------------------------------- what a chunk contributes
// s0[chunk, h, j, i] = sum_s d(s, last) v_s[j] k_s[i].  grid (chunks, H)
template <int D, int DV>
__global__ void __launch_bounds__(LC_THREADS)
linear_chunk_add_kernel(LinearChunk a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char lc_sm[];
  using TK = LcTile<LC, D>;
  using TV = LcTile<LC, DV>;
  bf16* ks = reinterpret_cast<bf16*>(lc_sm);
  bf16* vs = ks + TK::ELEMS;
  __shared__ float gs[LC], dl[LC];
  int r, t0, n;
  if (!lc_find(a, blockIdx.x, r, t0, n)) return;
  const int h = blockIdx.y, gk = h / (a.H / a.G), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < LC) gs[tid] = tid < n ? a.g[(a.g_ld ? (size_t)(t0 + tid) * a.g_ld : 0) + h] : 1.f;
  lc_fill<LC, D>(ks, a.k + ((size_t)t0 * a.G + gk) * D, (long long)a.G * D, n);
  __syncthreads();
  float* dec = a.dec + ((size_t)blockIdx.x * a.H + h) * LC_DEC;
  if (tid <= LC) {                                    // d(s, last); thread LC: the whole decay
    LcDecay d;
    for (int p = LC - 1; p > (tid < LC ? tid : -1); p--) d.times(gs[p]);
    if (tid < LC) dl[tid] = d.value();
    dec[tid] = d.value();
  }
  __syncthreads();
  const float* v = a.v + (size_t)t0 * a.ldv + (size_t)h * DV;
  for (int e = tid; e < LC * (DV / 4); e += LC_THREADS) {
    const int row = e / (DV / 4), c = (e - row * (DV / 4)) * 4;
    const float4 x = row < n ? *reinterpret_cast<const float4*>(v + row * a.ldv + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float d = dl[row];
    unsigned lo[3], hi[3];
    lc_cut(d * x.x, d * x.y, lo);
    lc_cut(d * x.z, d * x.w, hi);
#pragma unroll
    for (int i = 0; i < 3; i++) *reinterpret_cast<uint2*>(vs + i * TV::PIECE + row * TV::LD + c) = make_uint2(lo[i], hi[i]);
  }
  __syncthreads();
  // a warp: 16 rows (j) at a time by a share of the columns (i)
  constexpr int MT = DV / 16, NW = 8 / (MT < 8 ? MT : 8), NP = D / 16 / NW;      // warps to a row of tiles; pairs of tiles a warp
  float* out = a.s0 + ((size_t)blockIdx.x * a.H + h) * DV * D;
  const int m = (warp / NW) * 16, n0 = (warp % NW) * NP * 16;
#pragma unroll
  for (int np = 0; np < NP; np++) {
    float c[2][4], s[2][4];
    lc_zero(c);
    lc_zero(s);
#pragma unroll
    for (int kk = 0; kk < LC / 16; kk++) {
      unsigned fa[3][4], fb[3][4];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        lc_a_t(fa[i], vs + i * TV::PIECE, TV::LD, m, kk * 16, lane);
        lc_b_t(fb[i], ks + i * TK::PIECE, TK::LD, kk * 16, n0 + np * 16, lane);
      }
      lc_mma(c, s, fa, fb);
    }
#pragma unroll
    for (int t = 0; t < 2; t++) {
      float* o = out + (size_t)(m + (lane >> 2)) * D + n0 + np * 16 + t * 8 + (lane & 3) * 2;
      *reinterpret_cast<float2*>(o) = make_float2(c[t][0] + s[t][0], c[t][1] + s[t][1]);
      *reinterpret_cast<float2*>(o + 8 * D) = make_float2(c[t][2] + s[t][2], c[t][3] + s[t][3]);
    }
  }
}

// ----------------------------------------------------------------------------------- the states before the chunks
// grid (DV D / 4 / LC_THREADS, H, requests)
template <int D, int DV>
__global__ void __launch_bounds__(LC_THREADS)
linear_chunk_states_kernel(LinearChunk a) {
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.y, req = blockIdx.z, e = blockIdx.x * LC_THREADS + threadIdx.x;
  int at = -a.c0;                                     // where the request's first chunk is in the pass, or would be
  for (int r = 0; r < req; r++) at += (a.cu_tokens[r + 1] - a.cu_tokens[r] + LC - 1) / LC;
  const int end = at + (a.cu_tokens[req + 1] - a.cu_tokens[req] + LC - 1) / LC, first = max(at, 0), chunks = min(end, a.pass) - first;
  if (chunks <= 0) return;
  float4* S = reinterpret_cast<float4*>(a.state + (size_t)a.slots[req] * a.state_stride + a.s_off + (size_t)h * DV * D) + e;
  float4 s = at < 0 ? reinterpret_cast<const float4*>(a.from + (size_t)h * DV * D)[e] : *S;
  constexpr int AHEAD = 8;
  for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
    float4 add[AHEAD];
    float G[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
      if (c0 + i < chunks) {
        const size_t at = (size_t)(first + c0 + i) * a.H + h;
        add[i] = reinterpret_cast<const float4*>(a.s0 + at * DV * D)[e];
        G[i] = a.dec[at * LC_DEC + LC];
      }
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
      if (c0 + i < chunks) {
        reinterpret_cast<float4*>(a.s0 + ((size_t)(first + c0 + i) * a.H + h) * DV * D)[e] = s;
        s = make_float4(fmaf(G[i], s.x, add[i].x), fmaf(G[i], s.y, add[i].y), fmaf(G[i], s.z, add[i].z), fmaf(G[i], s.w, add[i].w));
      }
  }
  if (end > a.pass) reinterpret_cast<float4*>(a.to + (size_t)h * DV * D)[e] = s;      // goes on in the next pass
  else if (a.write_state) *S = s;
}

// ------------------------------------------------------------------------------------------------ the outputs
// out[t, h] = o / sqrt(mean(o^2) + eps) (* norm) * gate * out_scale with o as above.  grid (chunks, H); a warp has 16 tokens by a
// quarter of the columns, and of the products of q and k 16 tokens by 16.
#define LC_OUT_THREADS 512
template <int D, int DV>
__global__ void __launch_bounds__(LC_OUT_THREADS)
linear_chunk_out_kernel(LinearChunk a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char lc_sm[];
  using TK = LcTile<LC, D>;
  using TS = LcTile<DV, D>;
  using TX = LcTile<LC, DV>;
  using TP = LcTile<LC, LC>;
  constexpr int FIRST = TS::ELEMS > TK::ELEMS + TX::ELEMS ? TS::ELEMS : TK::ELEMS + TX::ELEMS;
  static_assert(TP::ELEMS <= TK::ELEMS, "");
  bf16* qs = reinterpret_cast<bf16*>(lc_sm);
  bf16* ss = qs + TK::ELEMS;                          // the state; after it K and V
  bf16* ks = ss;
  bf16* xs = ks + TK::ELEMS;
  bf16* ps = ks;                                      // d(s, p) (k_s . q_p), in the keys' place
  float* dm = reinterpret_cast<float*>(ss + FIRST);   // [LC][LC_DM]
  float* os = reinterpret_cast<float*>(qs);           // [LC][LO]: the outputs take the queries' place
  constexpr int LO = DV + 4;
  static_assert(LC * LO * 4 <= TK::ELEMS * 2, "the outputs fit where the queries were");
  __shared__ float gs[LC];
  int r, t0, n;
  if (!lc_find(a, blockIdx.x, r, t0, n)) return;
  const int h = blockIdx.y, gk = h / (a.H / a.G), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t2 = (lane & 3) * 2;
  const size_t at = (size_t)blockIdx.x * a.H + h;
  const float* xg = a.v + (size_t)t0 * a.ldv + (size_t)h * DV;
  lc_fill<LC, D, LC_OUT_THREADS>(qs, a.q + ((size_t)t0 * a.G + gk) * D, (long long)a.G * D, n);
  lc_fill<DV, D, LC_OUT_THREADS>(ss, a.s0 + at * DV * D, D, DV);
  lc_decays(a, t0, n, h, gs, dm);
  // K and V are on their way while the state's product is made
  float4 kx[LC * D / 4 / LC_OUT_THREADS], xx[LC * DV / 4 / LC_OUT_THREADS];
  lc_ask<LC, D, LC_OUT_THREADS>(kx, a.k + ((size_t)t0 * a.G + gk) * D, (long long)a.G * D, n);
  lc_ask<LC, DV, LC_OUT_THREADS>(xx, xg, a.ldv, n);
  constexpr int NP = DV / 64;
  // (a scheduler's four warps have all four rows of tiles: their triangular products are of different lengths)
  const int part = warp >> 2, m = ((warp + part) & 3) * 16, c0 = part * (DV / 4);
  float o[NP][2][4], s2[NP][2][4];
  const float g0 = gs[0], G0 = dm[(m + g) * LC_DM] * g0, G1 = dm[(m + g + 8) * LC_DM] * g0;
#pragma unroll
  for (int np = 0; np < NP; np++) { lc_zero(o[np]); lc_zero(s2[np]); }
#pragma unroll 2
  for (int kk = 0; kk < D / 16; kk++) {               // G_p S0^T q_p
    unsigned fa[3][4];
#pragma unroll
    for (int i = 0; i < 3; i++) lc_a(fa[i], qs + i * TK::PIECE, TK::LD, m, kk * 16, lane);
#pragma unroll
    for (int np = 0; np < NP; np++) {
      unsigned fb[3][4];
#pragma unroll
      for (int i = 0; i < 3; i++) lc_b(fb[i], ss + i * TS::PIECE, TS::LD, kk * 16, c0 + np * 16, lane);
      lc_mma(o[np], s2[np], fa, fb);
    }
  }
#pragma unroll
  for (int np = 0; np < NP; np++)
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        o[np][t][e] = (e < 2 ? G0 : G1) * (o[np][t][e] + s2[np][t][e]);
        s2[np][t][e] = 0.f;
      }
  __syncthreads();
  lc_put<LC, D, LC_OUT_THREADS>(ks, kx);
  const bool odd = __syncthreads_or(lc_put<LC, DV, LC_OUT_THREADS>(xs, xx));
  // the gate of what this thread stores in the end
  constexpr int LANES = DV / 4, PER = LC_OUT_THREADS / LANES;
  const int j = (tid % LANES) * 4;
  float2 z[LC / PER][2];
  float4 w = make_float4(1.f, 1.f, 1.f, 1.f);
  if (a.norm) {
    const float* norm = a.norm + (size_t)h * a.norm_ld + j;
    w = make_float4(norm[0], norm[1], norm[2], norm[3]);
  }
#pragma unroll
  for (int i = 0; i < LC / PER; i++) {
    const int p = min(tid / LANES + i * PER, n - 1);
    const float2* gate = reinterpret_cast<const float2*>(a.gate + (size_t)(t0 + p) * a.gate_ld + (size_t)h * DV + j);
    z[i][0] = gate[0];
    z[i][1] = gate[1];
  }
  float c[2][4], s[2][4];
  lc_zero(c);
  lc_zero(s);
  if (part * 16 <= m) {                               // tokens s part * 16 .. + 15 for tokens p m .. m + 15
#pragma unroll 2
    for (int kk = 0; kk < D / 16; kk++) {
      unsigned fa[3][4], fb[3][4];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        lc_a(fa[i], qs + i * TK::PIECE, TK::LD, m, kk * 16, lane);
        lc_b(fb[i], ks + i * TK::PIECE, TK::LD, kk * 16, part * 16, lane);
      }
      lc_mma(c, s, fa, fb);
    }
  }
  __syncthreads();
  if (part * 16 <= m) {
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int p = m + g + 4 * e, q = part * 16 + t * 8 + t2;
        float2* d = reinterpret_cast<float2*>(dm + p * LC_DM + q);      // (this thread's alone)
        const float x = q <= p ? d->x * (c[t][e] + s[t][e]) : 0.f, y = q + 1 <= p ? d->y * (c[t][e + 1] + s[t][e + 1]) : 0.f;
        if (odd) *d = make_float2(x, y);
        unsigned cut[3];
        lc_cut(x, y, cut);
#pragma unroll
        for (int i = 0; i < 3; i++) *reinterpret_cast<unsigned*>(ps + i * TP::PIECE + p * TP::LD + q) = cut[i];
      }
  }
  __syncthreads();
  if (odd) {                                          // only what lies at or before a token joins its sum
#pragma unroll
    for (int np = 0; np < NP; np++)
#pragma unroll
      for (int t = 0; t < 2; t++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int p = m + g + 8 * (e >> 1), j = c0 + np * 16 + t * 8 + t2 + (e & 1);
          float y = 0.f;
          for (int s = 0; s <= p && s < n; s++) y = fmaf(dm[p * LC_DM + s], xg[s * a.ldv + j], y);
          s2[np][t][e] = y;
        }
  } else {
#pragma unroll 1
    for (int kb = 0; kb * 16 <= m; kb++) {
      unsigned fa[3][4];
#pragma unroll
      for (int i = 0; i < 3; i++) lc_a(fa[i], ps + i * TP::PIECE, TP::LD, m, kb * 16, lane);
#pragma unroll
      for (int np = 0; np < NP; np++) {
        unsigned fb[3][4];
#pragma unroll
        for (int i = 0; i < 3; i++) lc_b_t(fb[i], xs + i * TX::PIECE, TX::LD, kb * 16, c0 + np * 16, lane);
        lc_mma(o[np], s2[np], fa, fb);
      }
    }
  }
#pragma unroll
  for (int np = 0; np < NP; np++)
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        *reinterpret_cast<float2*>(os + (m + g + 4 * e) * LO + c0 + np * 16 + t * 8 + t2) =
            make_float2(o[np][t][e] + s2[np][t][e], o[np][t][e + 1] + s2[np][t][e + 1]);
  __syncthreads();
  // norm, gate, store: a group of DV / 4 lanes has a token
#pragma unroll
  for (int i = 0; i < LC / PER; i++) {
    const int p = tid / LANES + i * PER;
    const float4 y = *reinterpret_cast<const float4*>(os + p * LO + j);
    float ss = y.x * y.x + y.y * y.y + y.z * y.z + y.w * y.w;
#pragma unroll
    for (int l = LANES / 2; l > 0; l >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, l);
    const float f = a.out_scale / sqrtf(ss / (float)DV + a.eps);
    auto gated = [&](float o, float w, float z) { return o * (f * w) * ((a.gate_kind ? 1.0f : z) / (1.0f + expf(-z))); };
    const float r0 = gated(y.x, w.x, z[i][0].x), r1 = gated(y.y, w.y, z[i][0].y), r2 = gated(y.z, w.z, z[i][1].x), r3 = gated(y.w, w.w, z[i][1].y);
    if (p < n) {
      const size_t dst = (size_t)(t0 + p) * a.out_stride + (size_t)h * DV + j;
      if (a.out_dtype == QD_F32) {
        float2* to = reinterpret_cast<float2*>(reinterpret_cast<float*>(a.out) + dst);
        to[0] = make_float2(r0, r1);
        to[1] = make_float2(r2, r3);
      } else {
        unsigned* to = reinterpret_cast<unsigned*>(reinterpret_cast<bf16*>(a.out) + dst);
        to[0] = lc_round2(r0, r1);
        to[1] = lc_round2(r2, r3);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ host
// Whether the sizes are taken: whole heads of 64 x 64 or 128 x 128 without the delta rule, and portions that are long enough on the
// average.
#define LC_MEAN 192
static bool lc_takes(int T, int R, int d, int dv, int DP, bool delta, int nrm) {
  return !nrm && !delta && d == DP && dv == d && (d == 128 || d == 64) && (long long)T >= (long long)LC_MEAN * R;
}
// Whether they are the faster form, the longest portion having ``longest`` tokens: in chunks every (chunk, head) is work for itself, token
// by token only every (request, head), which is enough where there are many of these.  us, fitted to captured calls with 4 to 128
// heads.  Measured on a B200, chunks / token by token, 32 heads of 64: 256 tokens 19.5 / 29.3, 1,500 67.4 / 155, three portions of 200 36.8 /
// 41.7, eight of 400 154 / 127; 64 heads, three of 200 67.9 / 53.4; 32 heads of 128: 256 tokens 35.6 / 49.9, 1,500 172 / 275, three of 200
// 84.5 / 73.8, eight of 400 399 / 326; 128 heads of 128, 1,500 tokens 726 / 674.
static bool lc_pays(int T, int R, int H, int d, int longest) {
  const double work = (T / 64.0 + 0.5 * R) * H, side_by_side = (double)H * T / longest;
  const double chunks = d == 64 ? 14 + 0.07 * work + 0.018 * fmax(0.0, work - 800) : 20 + 0.15 * work + 0.1 * fmax(0.0, work - 280);
  const double tokens = 4 + longest * (d == 64 ? fmax(0.0965, 0.09 + 0.00095 * side_by_side) : fmax(0.155, 0.09 + 0.0029 * side_by_side));
  return chunks <= tokens;
}
static long long lc_chunks(int T, int R) { return (long long)T / LC + R; }      // no fewer than there are

// Scratch.  A chunk of 32 heads of 128 takes 2.1 MB, 33 KB a token: a step of 32,768 tokens would take 1.1 GB beside a cache that was
// given the rest of the memory.  So there are no more chunks at a time than LC_SCRATCH floats hold (64 MB: 1,800 of those tokens, 7,900
// of 32 heads of 64), and where that is not one chunk, none.  A pass more costs 6 to 10 us where all fits into L2 and gives some back
// where it does not: 1,500 tokens of 32 heads of 64 in one, two and four passes 69, 75 and 102 us, 6,000 of 128 734, 750 and 681.
#define LC_SCRATCH (16ll << 20)
static long long lc_floats(int H, int d) { return (long long)H * (LC_DEC + d * d); }       // of a chunk
static long long lc_carry(int H, int d) { return 2ll * H * d * d; }                        // with more than one pass
// chunks of a pass with ``floats`` of scratch, 0: too few
static long long lc_pass(int T, int R, int H, int d, long long floats) {
  const long long all = lc_chunks(T, R), one = lc_floats(H, d);
  if (floats / one >= all) return all;
  return floats < lc_carry(H, d) + one ? 0 : (floats - lc_carry(H, d)) / one;
}
static long long lc_scratch(int T, int R, int H, int d) {
  const long long pass = lc_pass(T, R, H, d, LC_SCRATCH);
  return pass * lc_floats(H, d) + (pass > 0 && pass < lc_chunks(T, R) ? lc_carry(H, d) : 0);
}

template <int D>
static int lc_launch(LinearChunk a, float* scratch, long long floats, cudaStream_t stream) {
  const long long all = lc_chunks(a.T, a.R), c = lc_pass(a.T, a.R, a.H, D, floats);
  if (c < 1 || all > 65535 || a.H > 65535 || a.R > 65535) return QD_ERR_UNSUPPORTED;
  a.s0 = scratch;
  a.dec = a.s0 + c * a.H * D * D;
  float* carry = a.dec + c * a.H * LC_DEC;
  constexpr size_t tile = LcTile<LC, D>::ELEMS * sizeof(bf16), state = LcTile<D, D>::ELEMS * sizeof(bf16), dm = LC * LC_DM * sizeof(float);
  constexpr size_t out = tile + (state > 2 * tile ? state : 2 * tile) + dm;
  auto go = [&](auto kernel, dim3 g, size_t smem, int threads = LC_THREADS) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    qd_launch(kernel, g, dim3(threads), smem, stream, a);
  };
  for (long long c0 = 0, i = 0; c0 < all; c0 += c, i++) {
    a.c0 = (int)c0;
    a.pass = (int)(all - c0 < c ? all - c0 : c);
    a.from = carry + (i & 1) * a.H * D * D;
    a.to = carry + (~i & 1) * a.H * D * D;
    const dim3 grid(a.pass, a.H);
    go(linear_chunk_add_kernel<D, D>, grid, 2 * tile);
    go(linear_chunk_states_kernel<D, D>, dim3(D * D / 4 / LC_THREADS, a.H, a.R), 0);
    go(linear_chunk_out_kernel<D, D>, grid, out, LC_OUT_THREADS);
  }
  return qd_last_error();
}
