// The float32 path's contractions Y[T, N] = X[T, K] * W[N, K]^T (+ bias[N]) in float32 FMA (no TF32, no tensor cores), for
// rows of whole 16-byte pieces (K and the row stride of X multiples of 4, both 16-byte aligned; gemm_generic.cu takes the
// rest).  Two kernels, by what bounds them:
//
// * up to 8 tokens: reading W once.  A warp owns 8 rows of W and a share of K: its lanes read 16 bytes of each row at a
//   time (512 contiguous bytes per row and warp) past L1, every piece meets the same 16 bytes of each token's row (L1), and
//   the 8 x T sums stay in registers.  The warps of a CTA are KG shares of K of RG blocks of 8 rows; the lanes' sums are
//   folded together by halving (31 shuffles for 32 sums), the shares through shared memory, and the CTA stores whole sums.
//   Up to 4 tokens the first pieces of W are asked for before the wait for the kernel before, and every piece one round ahead.
// * more tokens: the FMA units (64 TFLOP/s is what a loop of FMAs alone reaches).  Tiles of up to 128 tokens x 128 or 256
//   features; stages of 32 k arrive by cp.async, four deep, the first ones' weights before the wait.  A thread's sums are
//   pairs, over even and over odd k: two neighbouring k of a row, as they lie in memory, are one operand of fma.rn.f32x2, so
//   nothing is rearranged, and it takes half the issue slots of single FMAs.  The tile's rows are chosen for T so that less
//   than a sixteenth to an eighth of a tile is padding; K is cut into shares where the tiles would leave multiprocessors
//   idle (gemm_f32_splits), whose partial sums are added up in the order of the shares.
//
// Measured on a B200 at the 3B sizes (all products of a step): 4 tokens 58.3 ms through the 64 x 64 tiles of
// gemm_generic.cu -> 2.5; gate/up alone 33.6 us = 5.4 TB/s (8 tokens: 43.7; through the second kernel 53).  203 tokens 82 ->
// 29.7 ms; gate/up alone 476 us = 38 TFLOP/s.
#include "common.cuh"

#define F32_ROWS 8           // rows of W per warp
#define F32_WARPS 8

__device__ __forceinline__ float4 ld_stream(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// The sums of M values over the 32 lanes of a warp: afterwards lane l holds, for M >= 32, the values
// (l * M / 32) .. + M / 32 - 1 in v[0 ..], and for M < 32 value l * M / 32 in v[0].
template <int M>
__device__ __forceinline__ void fold_lanes(float (&v)[M], int lane) {
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
}

template <int TT, int RG>
__global__ void __launch_bounds__(F32_WARPS * 32, 2)
gemm_f32_few_kernel(const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ bias,
                    float* __restrict__ Y, int T, int N, int K, long long ldx, long long ldy) {
  constexpr int KG = F32_WARPS / RG, M = F32_ROWS * TT;
  constexpr bool AHEAD = TT <= 4;                    // with more sums there are no registers for the next pieces of W beside these
  __shared__ float red[KG][RG][M];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = warp % RG, kg = warp / RG;
  const int row0 = (blockIdx.x * RG + rg) * F32_ROWS;
  const float* wr[F32_ROWS];
#pragma unroll
  for (int r = 0; r < F32_ROWS; r++) wr[r] = W + (size_t)min(row0 + r, N - 1) * K;
  float acc[M];                                      // [token][row]
#pragma unroll
  for (int i = 0; i < M; i++) acc[i] = 0.f;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 w[F32_ROWS];
  int k = (kg * 32 + lane) * 4;
#pragma unroll
  for (int r = 0; r < F32_ROWS; r++) w[r] = AHEAD && k < K ? ld_stream(wr[r] + k) : zero;
  pdl_wait();
  for (; k < K; k += KG * 128) {
    float4 next[F32_ROWS];
    const bool more = AHEAD && k + KG * 128 < K;
#pragma unroll
    for (int r = 0; r < F32_ROWS; r++) {
      if (!AHEAD) w[r] = ld_stream(wr[r] + k);
      next[r] = more ? ld_stream(wr[r] + k + KG * 128) : zero;
    }
#pragma unroll
    for (int t = 0; t < TT; t++) {
      const float4 x = __ldg(reinterpret_cast<const float4*>(X + (size_t)min(t, T - 1) * ldx + k));
#pragma unroll
      for (int r = 0; r < F32_ROWS; r++) {
        float& a = acc[t * F32_ROWS + r];
        a = fmaf(w[r].x, x.x, a); a = fmaf(w[r].y, x.y, a); a = fmaf(w[r].z, x.z, a); a = fmaf(w[r].w, x.w, a);
      }
    }
#pragma unroll
    for (int r = 0; r < F32_ROWS; r++) w[r] = next[r];
  }
  fold_lanes<M>(acc, lane);
  if (M >= 32) {
#pragma unroll
    for (int i = 0; i < (M >= 32 ? M / 32 : 1); i++) red[kg][rg][lane * (M / 32) + i] = acc[i];
  } else if (lane % (32 / (M < 32 ? M : 32)) == 0) {
    red[kg][rg][lane * M / 32] = acc[0];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < RG * M; i += F32_WARPS * 32) {
    const int g = i / M, v = i - g * M, t = v / F32_ROWS, row = (blockIdx.x * RG + g) * F32_ROWS + v % F32_ROWS;
    float s = red[0][g][v];
#pragma unroll
    for (int q = 1; q < KG; q++) s += red[q][g][v];
    if (t < T && row < N) Y[(size_t)t * ldy + row] = bias ? s + bias[row] : s;
  }
}

// ---------------------------------------------------------------------------------------------- more tokens
#define F32_BK 32
#define F32_LD (F32_BK + 4)       // floats from one row of a stage to the next: 16 bytes of 8 neighbouring rows hit 32 banks once
#define F32_STAGES 4

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pair_sum(unsigned long long v) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
  return x + y;
}
__device__ __forceinline__ void copy16(unsigned dst, const float* src, bool in) {     // zeros where ``in`` is false
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// A CTA: BM = RM * TYN tokens x BN = RN * (256 / TYN) features over a share of K.  out: [T, N] with row stride ldy
// (splits 1), or partial sums [splits, T, N].
template <int RM, int TYN, int RN>
__global__ void __launch_bounds__(256, 1)
gemm_f32_tile_kernel(const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ out, int T, int N, int K, long long ldx, long long ldy, int splits) {
  constexpr int TXN = 256 / TYN, BM = RM * TYN, BN = RN * TXN, ROWS = BM + BN;
  extern __shared__ __align__(16) float tile_smem[];         // [stage][BN rows of W, BM rows of X][F32_LD]
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // a warp covers 4 places of ty and 8 of tx
  const int ty = (warp % (TYN / 4)) * 4 + (lane >> 3), tx = (warp / (TYN / 4)) * 8 + (lane & 7);
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
  const int steps = (K + F32_BK - 1) / F32_BK;
  const int s_begin = (int)((long long)steps * blockIdx.z / splits), s_end = (int)((long long)steps * (blockIdx.z + 1) / splits);
  const unsigned base = (unsigned)__cvta_generic_to_shared(tile_smem);
  const int piece = (tid & 7) * 4, lr = tid >> 3;            // a thread copies 16 bytes of every 32nd row
  auto fetch_w = [&](int s) {
    const int k = s * F32_BK + piece;
    const bool in = s < s_end && k < K;
    const unsigned dst = base + (unsigned)(((s - s_begin) % F32_STAGES * ROWS + lr) * F32_LD + piece) * 4;
#pragma unroll
    for (int v = 0; v < BN / 32; v++)
      copy16(dst + v * 32 * F32_LD * 4, W + (size_t)min(n0 + lr + 32 * v, N - 1) * K + (in ? k : 0), in);
  };
  auto fetch_x = [&](int s) {
    const int k = s * F32_BK + piece;
    const bool in = s < s_end && k < K;
    const unsigned dst = base + (unsigned)(((s - s_begin) % F32_STAGES * ROWS + BN + lr) * F32_LD + piece) * 4;
#pragma unroll
    for (int v = 0; v < (BM + 31) / 32; v++)
      if (BM % 32 == 0 || lr + 32 * v < BM)
        copy16(dst + v * 32 * F32_LD * 4, X + (size_t)min(m0 + lr + 32 * v, T - 1) * ldx + (in ? k : 0), in);
  };
  unsigned long long acc[RM][RN];                            // sums over even k and over odd k
#pragma unroll
  for (int i = 0; i < RM; i++)
#pragma unroll
    for (int j = 0; j < RN; j++) acc[i][j] = 0ull;
  // weights are written by no kernel of the step: the first stages' are asked for before the tokens are there
#pragma unroll
  for (int s = 0; s < F32_STAGES - 1; s++) fetch_w(s_begin + s);
  pdl_wait();
#pragma unroll
  for (int s = 0; s < F32_STAGES - 1; s++) {
    fetch_x(s_begin + s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int s = s_begin; s < s_end; s++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(F32_STAGES - 2) : "memory");
    __syncthreads();                                         // everybody's copies are there, and the stage before is free
    fetch_w(s + F32_STAGES - 1);
    fetch_x(s + F32_STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* st = tile_smem + (size_t)((s - s_begin) % F32_STAGES) * ROWS * F32_LD;
    const float* ws = st + tx * F32_LD;
    const float* xs = st + (BN + ty) * F32_LD;
#pragma unroll
    for (int k = 0; k < F32_BK; k += 4) {
      ulonglong2 a[RM];
#pragma unroll
      for (int i = 0; i < RM; i++) a[i] = *reinterpret_cast<const ulonglong2*>(xs + i * TYN * F32_LD + k);
#pragma unroll
      for (int j = 0; j < RN; j++) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + j * TXN * F32_LD + k);
#pragma unroll
        for (int i = 0; i < RM; i++) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
        for (int i = 0; i < RM; i++) fma2(acc[i][j], a[i].y, b.y);
      }
    }
  }
  float* o = out + (splits > 1 ? (size_t)blockIdx.z * T * N : 0);
  const long long ld = splits > 1 ? N : ldy;
#pragma unroll
  for (int j = 0; j < RN; j++) {
    const int col = n0 + tx + j * TXN;
    if (col >= N) continue;
    const float b = bias && splits == 1 ? bias[col] : 0.f;
#pragma unroll
    for (int i = 0; i < RM; i++) {
      const int row = m0 + ty + i * TYN;
      if (row < T) o[(size_t)row * ld + col] = pair_sum(acc[i][j]) + b;
    }
  }
}

template <int RM, int TYN, int RN>
static int launch_tile(const float* X, const float* W, const float* bias, float* out, int T, int N, int K, long long ldx,
                       long long ldy, int splits, cudaStream_t stream) {
  constexpr int BM = RM * TYN, BN = RN * (256 / TYN);
  constexpr int smem = F32_STAGES * (BM + BN) * F32_LD * 4;
  const dim3 grid((N + BN - 1) / BN, (T + BM - 1) / BM, splits);
  if (grid.y > 65535 || grid.z > 65535) return QD_ERR_UNSUPPORTED;
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<RM, TYN, RN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  qd_launch(gemm_f32_tile_kernel<RM, TYN, RN>, grid, dim3(256), smem, stream, X, W, bias, out, T, N, K, ldx, ldy, splits);
  return qd_last_error();
}

// Y[t, n] = sum of the shares' partial sums (+ bias), in the order of the shares; N a multiple of 4
__global__ void __launch_bounds__(256)
f32_shares_kernel(const float* __restrict__ part, const float* __restrict__ bias, float* __restrict__ Y, size_t n4, int N4,
                  int splits, long long ldy) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  const size_t t = i / N4, c = i - t * N4;
  float4 s = reinterpret_cast<const float4*>(part)[i];
  for (int p = 1; p < splits; p++) {
    const float4 v = reinterpret_cast<const float4*>(part)[(size_t)p * n4 + i];
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  if (bias) { s.x += bias[4 * c]; s.y += bias[4 * c + 1]; s.z += bias[4 * c + 2]; s.w += bias[4 * c + 3]; }
  float* y = Y + t * ldy + 4 * c;
  y[0] = s.x; y[1] = s.y; y[2] = s.z; y[3] = s.w;
}

// ``splits`` > 1 (more than 16 tokens only): ``part`` [splits, T, N] takes the shares' partial sums; with ``Y`` they are
// added up into it (N a multiple of 4), without it they are the result and ``bias`` must be null.
extern "C" int qd_gemm_f32(const float* X, const float* W, const float* bias, float* Y, float* part, int T, int N, int K,
                           long long ldx, long long ldy, int splits, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 4 || ldx % 4 || (((uintptr_t)X | (uintptr_t)W) & 15) || splits < 1) return QD_ERR_UNSUPPORTED;
  if (T <= 8) {
    if (splits != 1 || !Y) return QD_ERR_UNSUPPORTED;
    // two blocks of 8 rows to a CTA where that still gives every multiprocessor several CTAs: each token's row is then
    // read half as often (a down projection of 2,048 features has 256 CTAs of 8 rows, and needs them)
    const int rg = N >= 8192 ? 2 : 1;
    const dim3 grid((N + rg * F32_ROWS - 1) / (rg * F32_ROWS));
#define FEW(TT)                                                                                                       \
    do {                                                                                                              \
      if (rg == 2) qd_launch(gemm_f32_few_kernel<TT, 2>, grid, dim3(F32_WARPS * 32), 0, stream, X, W, bias, Y, T, N, K, ldx, ldy); \
      else qd_launch(gemm_f32_few_kernel<TT, 1>, grid, dim3(F32_WARPS * 32), 0, stream, X, W, bias, Y, T, N, K, ldx, ldy);         \
    } while (0)
    if (T == 1) FEW(1); else if (T == 2) FEW(2); else if (T <= 4) FEW(4); else FEW(8);
#undef FEW
    return qd_last_error();
  }
  if (splits > 1 && (!part || ((uintptr_t)part & 15) || (Y && N % 4) || (!Y && bias))) return QD_ERR_UNSUPPORTED;
  if (splits == 1 && !Y) return QD_ERR_UNSUPPORTED;
  float* out = splits > 1 ? part : Y;
  int rc = QD_ERR_UNSUPPORTED;
#define TILE(RM, TYN, RN) rc = launch_tile<RM, TYN, RN>(X, W, bias, out, T, N, K, ldx, ldy, splits, stream)
  if (T <= 64) {
    // 8 tokens at a time with 4 places of ty up to 32 tokens, 8 places above
    if (T <= 8) TILE(2, 4, 4); else if (T <= 16) TILE(4, 4, 4); else if (T <= 24) TILE(6, 4, 4); else if (T <= 32) TILE(8, 4, 4);
    else if (T <= 40) TILE(5, 8, 4); else if (T <= 48) TILE(6, 8, 4); else if (T <= 56) TILE(7, 8, 4); else TILE(8, 8, 4);
  } else {
    // equal tiles of at most 128 tokens
    const int m_tiles = (T + 127) / 128;
    switch (((T + m_tiles - 1) / m_tiles + 15) / 16) {
      case 5: TILE(5, 16, 8); break;
      case 6: TILE(6, 16, 8); break;
      case 7: TILE(7, 16, 8); break;
      default: TILE(8, 16, 8);
    }
  }
#undef TILE
  if (rc) return rc;
  if (splits > 1 && Y) {
    const size_t n4 = (size_t)T * N / 4;
    qd_launch(f32_shares_kernel, dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, stream, part, bias, Y, n4, N / 4, splits, ldy);
  }
  return qd_last_error();
}
