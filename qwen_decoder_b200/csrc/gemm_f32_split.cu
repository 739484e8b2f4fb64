// The float32 path's contractions of many tokens on the tensor cores, without losing a bit of the operands:
// Y[T, N] = X[T, K] * W[N, K]^T (+ bias[N]).
//
// A float32 number is the sum of three bfloat16 numbers exactly: its leading 8 bits, the next 8, and the rest (cut off, not
// rounded, so that nothing overflows and each remainder is exact).  Of the nine products of pieces the six with weights down
// to 2^-16 are taken, x1 w1 + (x1 w2 + x2 w1) + (x1 w3 + x2 w2 + x3 w1); what is left out is below 2^-23 of |x| |w|, and
// products of two pieces are exact in the tensor cores' float32 sums.  Those sums are cut off at 24 bits at every
// addition, which costs about 1.6e-8 of the result per MMA (2.1e-6 over K = 2048, measured); so the large products x1 w1 have
// an accumulator of their own, moved to registers and added there, rounded, every FS_CHUNK blocks of k, and the small ones
// another.  Measured error of a product against float64: 1.4e-7 to 3.1e-7 (K from 516 to 2052; 5e-7 when moved half as often),
// the FMA tiles of gemm_f32.cu 1.2e-7 to 3.1e-7; a whole prompt's logits 9.2e-7 (one FMA chain over K: 2.7e-6).  (An infinite operand gives NaN where an FMA chain may give infinity: infinity
// times a piece that is zero.)
//
// The weights are the MMA's 128 rows, the tokens its columns (up to 224): a CTA takes 128 features x a tile of tokens x a
// share of K, one CTA per multiprocessor, in turn.  Warps 0-7 read W (float32, 64 of k per block, the next block while this
// one is worked on), cut it into three tiles as the tensor cores read them (K-major, 128-byte swizzle) and, between
// blocks, move the accumulator; warp 8 fetches the tokens' pieces (cut beforehand by a kernel of their own) by TMA, one ring
// slot per piece; warp 9 issues the MMAs, the small products first, so that the large ones of a block find their accumulator
// moved.  At 203 tokens a block takes 2.8 us, fetching 3 x 28 KB of tokens and 32 KB of W (the MMAs 1.4); at 64 and fewer 1.9,
// reading and cutting W.  Gate and up of the 3B sizes at 203 tokens: 478 us with FMA -> 160; all products of that prompt 29.5
// -> 10.4 ms; the prompt 31.9 -> 12.7 ms.
// Every wait is bounded, as in gemm_mid.cu.
#include "common.cuh"
#include "tc5_ops.cuh"

#define FS_THREADS 320
#define FS_BK 64
#define FS_CHUNK 4              // blocks of 64 k between two moves of the accumulator
#define FS_XSLOTS 4
#define FS_WPIECE (128 * 128)   // bytes of a piece of W: 128 rows of 64 bfloat16
#define FS_MAX_COLS 224

// a: pieces of (x, y) packed as bfloat16 pairs
__device__ __forceinline__ void cut3(float x, float y, unsigned& p1, unsigned& p2, unsigned& p3) {
  const unsigned xi = __float_as_uint(x), yi = __float_as_uint(y);
  p1 = __byte_perm(xi, yi, 0x7632);                          // the upper halves
  const float xr = x - __uint_as_float(xi & 0xFFFF0000u), yr = y - __uint_as_float(yi & 0xFFFF0000u);
  const unsigned xj = __float_as_uint(xr), yj = __float_as_uint(yr);
  p2 = __byte_perm(xj, yj, 0x7632);
  const float xs = xr - __uint_as_float(xj & 0xFFFF0000u), ys = yr - __uint_as_float(yj & 0xFFFF0000u);
  p3 = __byte_perm(__float_as_uint(xs), __float_as_uint(ys), 0x7632);      // at most 8 bits are left
}

// pieces[p][t][Kp] of X [T, K], zeros from K to Kp (a multiple of 64)
__global__ void __launch_bounds__(256)
f32_cut_kernel(const float* __restrict__ X, long long ldx, bf16* __restrict__ pieces, int T, int K, int Kp) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t plane = (size_t)T * Kp;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < plane / 4; i += (size_t)gridDim.x * 256) {
    const size_t t = i / (Kp / 4);
    const int k = (int)(i - t * (Kp / 4)) * 4;
    const float4 v = k < K ? *reinterpret_cast<const float4*>(X + t * ldx + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    uint2 a, b, c;
    cut3(v.x, v.y, a.x, b.x, c.x);
    cut3(v.z, v.w, a.y, b.y, c.y);
    bf16* o = pieces + t * Kp + k;
    *reinterpret_cast<uint2*>(o) = a;
    *reinterpret_cast<uint2*>(o + plane) = b;
    *reinterpret_cast<uint2*>(o + 2 * plane) = c;
  }
}

struct FsArgs {
  const float* W; const float* bias; float* out; long long ldy;      // out: [T, N], or with splits > 1 partial sums [splits, T, N]
  int T, N, K, kb, splits, n_tiles, t_tiles, t_rows;                 // t_rows: tokens of a tile
  int* status;
};

template <int NT>
__global__ void __launch_bounds__(FS_THREADS, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_x, const FsArgs a) {
  constexpr int HALF = NT / 2;                               // token columns of a warp in the moves
  constexpr int XBYTES = NT * 128;
  constexpr unsigned COLS = 2 * NT <= 64 ? 64 : 2 * NT <= 128 ? 128 : 2 * NT <= 256 ? 256 : 512;
  extern __shared__ unsigned char smem_raw[];
  __shared__ unsigned long long wfull[2], wempty[2], xfull[FS_XSLOTS], xempty[FS_XSLOTS], moved;
  __shared__ unsigned tmem_slot;
  __shared__ int dead;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* wbuf = smem_raw + ((1024 - (tc_smem(smem_raw) & 1023)) & 1023);      // [2][3 pieces][128 rows][128 bytes]
  unsigned char* xring = wbuf + 2 * 3 * FS_WPIECE;
  if (threadIdx.x == 0) {
    dead = 0;
    for (int i = 0; i < 2; i++) { tc_bar_init(&wfull[i], 8); tc_bar_init(&wempty[i], 1); }
    for (int i = 0; i < FS_XSLOTS; i++) { tc_bar_init(&xfull[i], 1); tc_bar_init(&xempty[i], 1); }
    tc_bar_init(&moved, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) tc_alloc(&tmem_slot, COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_slot;                           // columns 0 .. NT - 1: x1 w1; NT .. 2 NT - 1: the small products
  pdl_launch_dependents();
  const int n_items = a.n_tiles * a.t_tiles * a.splits;
  // neighbouring CTAs: neighbouring features of the same tokens and share of K
  auto decode = [&](int item, int& n0, int& t0, int& share, int& k0, int& k1) {
    n0 = item % a.n_tiles * 128;
    const int rest = item / a.n_tiles;
    t0 = rest % a.t_tiles * a.t_rows;
    share = rest / a.t_tiles;
    k0 = (int)((long long)a.kb * share / a.splits);
    k1 = (int)((long long)a.kb * (share + 1) / a.splits);
  };

  if (warp < 8) {
    // ------------------------------------------------------------------ W: read, cut, store; the accumulator's moves
    const int quarter = warp & 3, half = warp >> 2;
    const unsigned t_main = tmem + ((unsigned)quarter << 21) + half * HALF, t_small = t_main + NT;
    const int row = threadIdx.x >> 4, chunk = threadIdx.x & 15;      // rows row + 16 j, floats 4 chunk .. + 3 of a block
    const unsigned at = row * 128 + (((chunk >> 1) ^ (row & 7)) << 4) + (chunk & 1) * 8;      // (16 j rows on: + 2048 j)
    float sum[HALF];
    float4 w[8];
    unsigned g = 0;                                          // blocks stored so far
    bool waited = false;
    auto fetch = [&](int n0, int kb) {
      const int k = kb * FS_BK + chunk * 4;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int r = min(n0 + row + 16 * j, a.N - 1);
        w[j] = k < a.K ? __ldg(reinterpret_cast<const float4*>(a.W + (size_t)r * a.K + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    auto block_done = [&](unsigned b) {                      // the MMAs of block b (counted over all items) are complete
      if (!tc_wait(&wempty[b & 1], (b >> 1) & 1, &dead) && lane == 0) atomicExch(a.status, 1);
    };
    auto move = [&]() {                                      // x1 w1 of a chunk into the registers
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < HALF; c += 16) {
        unsigned v[16];
        tc_ld16(t_main + c, v);
        tc_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i++) sum[c + i] += __uint_as_float(v[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) tc_arrive(&moved);
    };
    int item = blockIdx.x;
    {
      int n0, t0, share, k0, k1;
      if (item < n_items) { decode(item, n0, t0, share, k0, k1); fetch(n0, k0); }
    }
    for (; item < n_items; item += gridDim.x) {
      int n0, t0, share, k0, k1;
      decode(item, n0, t0, share, k0, k1);
#pragma unroll
      for (int i = 0; i < HALF; i++) sum[i] = 0.f;
      bool pending = false;                                  // a chunk ended with block g - 2 or g - 1 and is not moved yet
      for (int kb = k0; kb < k1; kb++, g++) {
        if (g >= 2) block_done(g - 2);
        if (pending && (kb - 2 - k0) % FS_CHUNK == FS_CHUNK - 1) { move(); pending = false; }
        unsigned char* dst = wbuf + (g & 1) * (3 * FS_WPIECE) + at;
#pragma unroll
        for (int j = 0; j < 8; j++) {
          uint2 p1, p2, p3;
          cut3(w[j].x, w[j].y, p1.x, p2.x, p3.x);
          cut3(w[j].z, w[j].w, p1.y, p2.y, p3.y);
          *reinterpret_cast<uint2*>(dst + j * 2048) = p1;
          *reinterpret_cast<uint2*>(dst + j * 2048 + FS_WPIECE) = p2;
          *reinterpret_cast<uint2*>(dst + j * 2048 + 2 * FS_WPIECE) = p3;
        }
        asm volatile("fence.proxy.async;" ::: "memory");     // read by the tensor cores
        __syncwarp();
        if (lane == 0) tc_arrive(&wfull[g & 1]);
        if ((kb - k0) % FS_CHUNK == FS_CHUNK - 1 && kb + 1 < k1) pending = true;
        if (kb + 1 < k1) {
          fetch(n0, kb + 1);
        } else if (item + (int)gridDim.x < n_items) {
          int n1, t1, s1, q0, q1;
          decode(item + gridDim.x, n1, t1, s1, q0, q1);
          fetch(n1, q0);
        }
      }
      if (pending) {                                         // a chunk that ended with the last block but one
        block_done(g - 2);
        move();
      }
      block_done(g - 1);
      tc_fence_after();
      if (!waited) pdl_wait();
      waited = true;
      const int n = n0 + quarter * 32 + lane;
      const float b = a.bias && a.splits == 1 && n < a.N ? a.bias[n] : 0.f;
      float* o = a.out + (a.splits > 1 ? (size_t)share * a.T * a.N : 0) + n;
      const long long ld = a.splits > 1 ? a.N : a.ldy;
      const int t_end = min(a.t_rows, a.T - t0);
#pragma unroll
      for (int c = 0; c < HALF; c += 16) {
        unsigned v[16], u[16];
        __syncwarp();
        tc_ld16(t_main + c, v);
        tc_ld16(t_small + c, u);
        tc_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i++) {
          const int t = half * HALF + c + i;
          const float s = (sum[c + i] + __uint_as_float(v[i])) + __uint_as_float(u[i]) + b;
          if (t < t_end && n < a.N) o[(size_t)(t0 + t) * ld] = s;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) tc_arrive(&moved);
    }
    if (!waited) pdl_wait();
  } else if (warp == 8) {
    // ------------------------------------------------------------------ the tokens' pieces, in the order x2, x3, x1
    pdl_wait();
    if (lane == 0) {
      asm volatile("fence.proxy.async;" ::: "memory");
      unsigned s = 0, ph = 0;
      for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
        int n0, t0, share, k0, k1;
        decode(item, n0, t0, share, k0, k1);
        for (int kb = k0; kb < k1; kb++)
#pragma unroll
          for (int i = 0; i < 3; i++) {
            if (!tc_wait(&xempty[s], ph ^ 1, &dead)) atomicExch(a.status, 2);
            tc_expect_tx(&xfull[s], XBYTES);
            tc_load_2d(xring + s * XBYTES, &map_x, kb * FS_BK, (i == 2 ? 0 : i + 1) * a.T + t0, &xfull[s]);
            if (++s == FS_XSLOTS) { s = 0; ph ^= 1; }
          }
      }
    }
  } else if (lane == 0) {
    // ------------------------------------------------------------------ MMA issuer
    const unsigned idesc = tc_idesc_bf16(128, NT);
    const unsigned long long dw0 = tc_desc_sw128(tc_smem(wbuf)), dx0 = tc_desc_sw128(tc_smem(xring));
    const unsigned small = tmem + NT;
    unsigned s = 0, ph = 0, g = 0, moves = 0;
    auto product = [&](unsigned d, unsigned long long dw, unsigned long long dx, bool fresh) {
      tc_mma_bf16(d, dw, dx, idesc, !fresh);
#pragma unroll
      for (int k = 1; k < FS_BK / 16; k++) tc_mma_bf16(d, dw + 2 * k, dx + 2 * k, idesc, true);
    };
    auto wait_moved = [&]() {
      if (!tc_wait(&moved, moves & 1, &dead)) atomicExch(a.status, 3);
      moves++;
      tc_fence_after();
    };
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
      int n0, t0, share, k0, k1;
      decode(item, n0, t0, share, k0, k1);
      if (item != (int)blockIdx.x) wait_moved();             // the item before is written
      for (int kb = k0; kb < k1; kb++, g++) {
        if (!tc_wait(&wfull[g & 1], (g >> 1) & 1, &dead)) atomicExch(a.status, 4);
        const unsigned long long dw = dw0 + (g & 1) * (3 * FS_WPIECE >> 4);
        constexpr unsigned P = FS_WPIECE >> 4;
#pragma unroll
        for (int i = 0; i < 3; i++) {
          if (!tc_wait(&xfull[s], ph, &dead)) atomicExch(a.status, 5);
          tc_fence_after();
          const unsigned long long dx = dx0 + s * (XBYTES >> 4);
          if (i == 0) {
            product(small, dw, dx, kb == k0);                // x2 w1
            product(small, dw + P, dx, false);               // x2 w2
          } else if (i == 1) {
            product(small, dw, dx, false);                   // x3 w1
          } else {
            product(small, dw + P, dx, false);               // x1 w2
            product(small, dw + 2 * P, dx, false);           // x1 w3
            const bool fresh = (kb - k0) % FS_CHUNK == 0;
            if (fresh && kb > k0) wait_moved();
            product(tmem, dw, dx, fresh);                    // x1 w1
          }
          tc_commit(&xempty[s]);
          if (++s == FS_XSLOTS) { s = 0; ph ^= 1; }
        }
        tc_commit(&wempty[g & 1]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tc_dealloc(tmem, COLS);
  }
}

// Y[t, n] = sum of the shares' partial sums (+ bias), in the order of the shares; N a multiple of 4
__global__ void __launch_bounds__(256)
f32_split_shares_kernel(const float* __restrict__ part, const float* __restrict__ bias, float* __restrict__ Y, size_t n4, int N4,
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

static int* fs_status_word() {
  static int* words[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!words[dev]) {
    int* w = nullptr;
    if (cudaMalloc(&w, sizeof(int)) != cudaSuccess) return nullptr;
    cudaMemset(w, 0, sizeof(int));
    words[dev] = w;
  }
  return words[dev];
}

template <int NT>
static int launch_split(const CUtensorMap& map, const FsArgs& a, cudaStream_t stream) {
  constexpr int smem = 2 * 3 * FS_WPIECE + FS_XSLOTS * NT * 128 + 1024;
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_split_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int items = a.n_tiles * a.t_tiles * a.splits;
  qd_launch(gemm_f32_split_kernel<NT>, dim3(items < sms ? items : sms), dim3(FS_THREADS), smem, stream, map, a);
  return qd_last_error();
}

// ``pieces``: scratch of 3 * T * ceil(K / 64) * 64 bfloat16; ``part``: with splits > 1, scratch of splits * T * N floats (N then a
// multiple of 4).  K and ldx multiples of 4, X and W 16-byte aligned.
extern "C" int qd_gemm_f32_split(const float* X, const float* W, const float* bias, float* Y, void* pieces, float* part, int T,
                                 int N, int K, long long ldx, long long ldy, int splits, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 4 || ldx % 4 || (((uintptr_t)X | (uintptr_t)W | (uintptr_t)pieces | (uintptr_t)part) & 15) || splits < 1 ||
      !Y || !pieces || (splits > 1 && (!part || N % 4)))
    return QD_ERR_UNSUPPORTED;
  FsArgs a = {};
  a.W = W; a.bias = bias; a.T = T; a.N = N; a.K = K; a.kb = (K + FS_BK - 1) / FS_BK; a.splits = splits;
  a.out = splits > 1 ? part : Y; a.ldy = ldy;
  a.n_tiles = (N + 127) / 128;
  a.t_tiles = (T + FS_MAX_COLS - 1) / FS_MAX_COLS;
  a.t_rows = (T + a.t_tiles - 1) / a.t_tiles;
  const int cols = (a.t_rows + 31) / 32 * 32;
  a.status = fs_status_word();
  if (!a.status || splits > a.kb || (long long)3 * T > 0x7fffffff) return QD_ERR_UNSUPPORTED;
  const int Kp = a.kb * FS_BK;
  CUtensorMap map;
  if (!tc_make_map(&map, pieces, 3ll * T, Kp, Kp, cols)) return QD_ERR_UNSUPPORTED;
  const size_t quads = (size_t)T * Kp / 4;
  const unsigned blocks = (unsigned)((quads + 255) / 256 < 1184 ? (quads + 255) / 256 : 1184);
  qd_launch(f32_cut_kernel, dim3(blocks), dim3(256), 0, stream, X, ldx, (bf16*)pieces, T, K, Kp);
  int rc = qd_last_error();
  if (rc) return rc;
  switch (cols) {
    case 32: rc = launch_split<32>(map, a, stream); break;
    case 64: rc = launch_split<64>(map, a, stream); break;
    case 96: rc = launch_split<96>(map, a, stream); break;
    case 128: rc = launch_split<128>(map, a, stream); break;
    case 160: rc = launch_split<160>(map, a, stream); break;
    case 192: rc = launch_split<192>(map, a, stream); break;
    case 224: rc = launch_split<224>(map, a, stream); break;
    default: return QD_ERR_UNSUPPORTED;
  }
  if (rc || splits == 1) return rc;
  const size_t n4 = (size_t)T * N / 4;
  qd_launch(f32_split_shares_kernel, dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, stream, part, bias, Y, n4, N / 4, splits, ldy);
  return qd_last_error();
}

// 0 if no bounded wait of this library has run out on the current device.  Reported once.  Synchronises.
QD_DEFINE_WAIT_PROBE(qd_gemm_f32_split_wait_probe, tc_wait(bar, 0, dead, 0, poll_limit), fs_status_word, 99)

extern "C" int qd_gemm_f32_split_status() {
  int* status = fs_status_word();
  if (!status) return -1;
  int v = 0;
  if (cudaMemcpy(&v, status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (v) cudaMemset(status, 0, sizeof(int));
  return v;
}
