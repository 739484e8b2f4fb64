// The float32 path's contractions on the tensor cores, without losing a bit of the operands: Y[T, N] = X[T, K] * W[N, K]^T
// (+ bias[N]), for rows of whole 16-byte pieces (K and the row stride of X multiples of 4, X and W 16-byte aligned;
// gemm_generic.cu takes the rest).
//
// A float32 number x is the sum of three bfloat16 numbers: x1 = x rounded, x2 = the remainder rounded, x3 = what is left, at most
// 8 bits (each remainder is exact; numbers below 2^-109 lose bits at the end of bfloat16's range).  Of the nine products of pieces
// of x and w all but x3 w3 (below 2^-34 of |x| |w|) are taken.  Products of pieces are exact in the tensor cores' float32 sums, but
// these are cut off, not rounded, at every addition: the sum of the large products x1 w1 is taken out after every block of 64 k and
// added to a register, rounded; that of the small ones (2^-8 of it) runs on.  (Cutting operands into bfloat16 pieces: Henry, Tang
// and Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations", 2019.)
//
// A row's sums do not depend on the other rows or on their number.  The blocks of 64 k of all tiles of 128 features are cut into
// ``runs`` equal runs, one per multiprocessor, by N and K alone; where a run ends inside a tile, the runs' sums of that tile are
// added up in their order by a kernel of its own.  A result that is not finite, or so small (2^-80) that pieces may have left
// bfloat16's range, is made again as one FMA chain over k, which is what gemm_generic.cu computes.  (What that does not see: a row
// whose terms are all a number below 2^-109 times one above 2^29; the lost bits are worth 2^-134 of the latter each.)
//
// The weights are the MMA's 128 rows, the tokens its columns.  Warps 0-7 cut W (float32) into tiles as the tensor cores read them
// (K-major, 128-byte swizzle), warp 16 issues TMA loads, warp 17 the MMAs, warps 8-15 add up the blocks' sums (cutting and adding in
// the same warps took turns: 2,500 cycles a block at 4 tokens, of which 1,300 were the sums').  Two forms:
//  * up to 64 tokens, bound by reading W (the projection over the vocabulary at 5.5 TB/s) and by ramps and tails where a run is short:
//    W comes by TMA, the first blocks before the wait for the kernel before; its pieces go to tensor memory, from where the MMAs take
//    them (in shared memory their 32 reads of a piece's 4 KB, the stores and W itself took 2,000 cycles a block: gate and up 48 us
//    at 4 tokens, now 40); warps 0-7 read and cut the tokens too.
//  * more tokens: W is read by warps 0-7, the tokens' pieces are made by a kernel beforehand and come by TMA, a piece a slot; bound by
//    shared memory too (203 tokens: 3,300 cycles of MMAs a block, 4,200 of reads and writes, 5,100 taken).
// Measured on a B200 at the 3B sizes, us a product, at 4 / 64 / 203 tokens: gate and up 40 / 55 / 129, output projection 8.6 / 13 / 27,
// all products of a step 3,200 at 4 tokens, 9,800 at 203.  With kernels and shares of K chosen by the number of tokens, and six products
// of pieces that were cut off, they had been 34 / 96 / 165 and 4.9 / 17 / 27: the smallest steps pay for sums that do not go by the
// batch.  Error against float64 1.2e-7 (gate and up; the FMA tiles of 9 to 32 tokens: 3.3e-7).
// Every wait is bounded; after one has run out nothing new is asked for and what is in flight is waited for.
#include "common.cuh"
#include "tc5_ops.cuh"

#define FS_THREADS 640          // five warpgroups, 96 registers a thread at launch; what one takes more the others give
#define FS_TAKE(n) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(n))
#define FS_GIVE(n) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(n))
#define FS_TMA_WARP 16
#define FS_MMA_WARP 17
#define FS_BK 64
#define FS_WPIECE (128 * 128)   // bytes of a piece of W: 128 rows of 64 bfloat16
#define FS_WBLOCK (3 * FS_WPIECE)
#define FS_FEW 64               // tokens that the first form takes
#define FS_MANY 224             // tokens of a tile of the second: their sums are 112 registers a thread
#define FS_XSLOTS 4             // pieces of a block's tokens on their way or in use (second form)

// pieces of (x, y), packed as bfloat16 pairs
__device__ __forceinline__ void cut3(float x, float y, unsigned& p1, unsigned& p2, unsigned& p3) {
  auto round2 = [](float a, float b) {
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
  };
  p1 = round2(x, y);
  const float xr = x - __uint_as_float(p1 << 16), yr = y - __uint_as_float(p1 & 0xFFFF0000u);
  p2 = round2(xr, yr);
  p3 = round2(xr - __uint_as_float(p2 << 16), yr - __uint_as_float(p2 & 0xFFFF0000u));
}

__device__ __forceinline__ bool fs_doubtful(float s) { return !(fabsf(s) >= 0x1p-80f && fabsf(s) <= 3.4e38f) && s != 0.f; }

struct FsArgs {
  const float* X; const float* W; const float* bias; float* Y; float* part;      // part [shares, T, N]
  long long ldx, ldy;
  int T, N, K, kb, runs, total;                      // kb: blocks of 64 k; total = tiles of 128 features * kb
  int t_tiles, t_rows, n_cols;                       // the second form: tiles of tokens, MMA columns (t_rows in whole 16)
  int* status;
};

// A result (bias included) that pieces cannot be trusted with is the FMA chain's.  (A row of zeros stays as it is.)
__device__ __noinline__ void fs_chain(const float* x, const float* w, int K, const float* bias, float* y) {
  if (!fs_doubtful(*y)) return;
  float s = 0.f;
  for (int k = 0; k < K; k++) s = fmaf(x[k], w[k], s);
  *y = bias ? s + *bias : s;
}
__device__ __forceinline__ void fs_settle(const FsArgs& a, int t, int n, float* y) {
  fs_chain(a.X + (size_t)t * a.ldx, a.W + (size_t)n * a.K, a.K, a.bias ? a.bias + n : nullptr, y);
}

// the run that has block b
__host__ __device__ __forceinline__ int fs_run_of(long long b, int runs, int total) { return (int)(((b + 1) * runs + total - 1) / total) - 1; }
__host__ __device__ __forceinline__ int fs_run_begin(long long r, int runs, int total) { return (int)(r * total / runs); }

// Where the sums of a run's part of tile ``tile`` go: row 0 of a [T, N] matrix with rows ``ld`` apart; ``whole``: they are the results.
__device__ __forceinline__ float* fs_dest(const FsArgs& a, int run, int tile, long long& ld, bool& whole) {
  const int first = fs_run_of((long long)tile * a.kb, a.runs, a.total);
  whole = first == fs_run_of((long long)tile * a.kb + a.kb - 1, a.runs, a.total);
  ld = whole ? a.ldy : a.N;
  return whole ? a.Y : a.part + (size_t)(run - first) * a.T * a.N;
}

// The blocks of a CTA in its order: its runs, each once for every tile of tokens.
struct FsAt {
  int run, tt, left, tile, k;                        // left: blocks of the run that are not passed, this one among them
  __device__ __forceinline__ void begin(const FsArgs& a) {
    const int b = fs_run_begin(run, a.runs, a.total);
    left = fs_run_begin(run + 1, a.runs, a.total) - b;
    tile = b / a.kb;
    k = b - tile * a.kb;
  }
  __device__ __forceinline__ FsAt(const FsArgs& a) : run(blockIdx.x), tt(0) { begin(a); }
  __device__ __forceinline__ bool ends_part(const FsArgs& a) const { return left == 1 || k + 1 == a.kb; }      // of a tile
  __device__ __forceinline__ void next(const FsArgs& a) {
    if (--left) {
      if (++k == a.kb) { k = 0; tile++; }
      return;
    }
    if (++tt == a.t_tiles) { tt = 0; run += gridDim.x; }
    if (run < a.runs) begin(a);
  }
};
__device__ __forceinline__ int fs_blocks(const FsArgs& a) {
  int n = 0;
  for (int run = blockIdx.x; run < a.runs; run += gridDim.x) n += fs_run_begin(run + 1, a.runs, a.total) - fs_run_begin(run, a.runs, a.total);
  return n * a.t_tiles;
}

// Stores a thread's sums of feature n, tokens t0 .. t_end - 1, and sets them to zero.  (What is doubtful is looked for once all are
// stored: this code is unrolled, runs once a tile and comes from memory, 10 us of it when it held the chain's call.)
template <int M>
__device__ __forceinline__ void fs_store(const FsArgs& a, int run, int tile, int n, int t0, int t_end, float (&sum)[M]) {
  long long ld;
  bool whole;
  float* const o = fs_dest(a, run, tile, ld, whole) + n;
  const bool in = n < a.N;
  if (whole && a.bias) {
    const float b = in ? a.bias[n] : 0.f;
#pragma unroll
    for (int c = 0; c < M; c++) sum[c] += b;
  }
  bool doubtful = false;
  float* p = o + t0 * ld;
#pragma unroll
  for (int c = 0; c < M; c++) {
    if (in && t0 + c < t_end) {
      *p = sum[c];
      doubtful = doubtful || fs_doubtful(sum[c]);
    }
    p += ld;
    sum[c] = 0.f;
  }
  if (doubtful && whole)
    for (int t = t0; t < min(t0 + M, t_end); t++) fs_settle(a, t, n, o + t * ld);
}

// the product of two pieces over a block of k, by one thread: 4 MMAs into the columns at d; W's piece in shared memory or in
// tensor memory (the same sums)
__device__ __forceinline__ void fs_product(unsigned d, unsigned long long w, unsigned long long x, unsigned idesc, bool fresh) {
  tc_mma_bf16(d, w, x, idesc, !fresh);
#pragma unroll
  for (int k = 1; k < FS_BK / 16; k++) tc_mma_bf16(d, w + 2 * k, x + 2 * k, idesc, true);
}
__device__ __forceinline__ void fs_product(unsigned d, unsigned w, unsigned long long x, unsigned idesc, bool fresh) {
  tc_mma_bf16_tmem(d, w, x, idesc, !fresh);
#pragma unroll
  for (int k = 1; k < FS_BK / 16; k++) tc_mma_bf16_tmem(d, w + 8 * k, x + 2 * k, idesc, true);
}
// What the small products' sum consists of, in this order in both forms, and then x1 w2, x1 w3 (P: from one piece of W to the next)
#define FS_WITH_X2(small, w, x, idesc, fresh) \
  do { fs_product(small, w, x, idesc, fresh); fs_product(small, w + P, x, idesc, false); fs_product(small, w + 2 * P, x, idesc, false); } while (0)
#define FS_WITH_X3(small, w, x, idesc) do { fs_product(small, w, x, idesc, false); fs_product(small, w + P, x, idesc, false); } while (0)

// adds 8 columns at ``t`` to ``sum``
__device__ __forceinline__ void fs_add8(unsigned t, float* sum) {
  unsigned v[8];
  __syncwarp();
  tc_ld8(t, v);
  tc_ld_wait();
#pragma unroll
  for (int i = 0; i < 8; i++) sum[i] += __uint_as_float(v[i]);
}
// a float4 of W or X as the thread (row tid / 16 and rows + 16, floats 4 (tid % 16) of a block) stores its pieces
__device__ __forceinline__ void fs_put(unsigned char* dst, unsigned piece, const float4& v) {
  uint2 p1, p2, p3;
  cut3(v.x, v.y, p1.x, p2.x, p3.x);
  cut3(v.z, v.w, p1.y, p2.y, p3.y);
  *reinterpret_cast<uint2*>(dst) = p1;
  *reinterpret_cast<uint2*>(dst + piece) = p2;
  *reinterpret_cast<uint2*>(dst + 2 * piece) = p3;
}

// A CTA's end.  After a wait that ran out nobody may have waited for the last MMAs, or for the last of the ``asked`` loads of a ring
// of ``slots`` (the count is the TMA warp's): both are waited for, with a limit of their own, before anything is given back.
__device__ __forceinline__ void fs_end(volatile int& dead, int warp, int lane, unsigned tmem, unsigned cols, unsigned long long* loaded,
                                       unsigned slots, unsigned asked) {
  __shared__ unsigned long long fin;
  tc_fence_before();
  __syncthreads();
  if (dead) {
    int late = 0;
    if (warp == FS_MMA_WARP && tc_elect()) {         // (the lane that issued the MMAs)
      tc_bar_init(&fin, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      tc_commit(&fin);
      tc_wait_inline(&fin, 0, &late);
    }
    if (warp == FS_TMA_WARP && lane == 0)
      for (unsigned i = asked > slots ? asked - slots : 0; i < asked; i++) tc_wait_inline(&loaded[i % slots], (i / slots) & 1, &late);
    __syncthreads();
  }
  if (warp == FS_MMA_WARP) {
    tc_fence_after();
    tc_dealloc(tmem, cols);
  }
}

// ---------------------------------------------------------------------------------------------- up to 64 tokens
// NT tokens (a multiple of 16); F blocks of W as they are (float32) on their way or in use, two blocks of pieces (W's in tensor
// memory, 32 columns each, the tokens' in shared memory), each with its own NT columns for the large products' sum
template <int NT, int F>
__global__ void __launch_bounds__(FS_THREADS, 1)
gemm_f32_few_kernel(const __grid_constant__ CUtensorMap map_w, const FsArgs a) {
  constexpr int HALF = NT / 2, XP = NT / 16, XPIECE = NT * 128, RAW = 128 * FS_BK * 4;
  constexpr unsigned P = FS_BK / 2, COLS = 6 * P + 3 * NT <= 256 ? 256 : 512;
  static_assert(NT % 16 == 0 && 6 * P + 3 * NT <= 512, "");
  extern __shared__ unsigned char smem_raw[];
  __shared__ unsigned long long raw_full[F], raw_free[F], full[2], done[2], part_read;
  __shared__ unsigned tmem_slot;
  __shared__ int dead;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* raw = smem_raw + ((1024 - (tc_smem(smem_raw) & 1023)) & 1023);        // [F][2 halves of k][128 rows][32 floats, swizzled]
  unsigned char* ring = raw + F * RAW;                                                 // [2][3 pieces][tokens][128 bytes]
  if (threadIdx.x == 0) {
    dead = 0;
    // a block's pieces are there (warps 0-7) and the sums that lay in its columns are read (warps 8-15): one wait for the MMA warp,
    // whose waits take 300 cycles each beside the others' stores
    for (int i = 0; i < 2; i++) { tc_bar_init(&full[i], 16); tc_bar_init(&done[i], 1); }
    tc_bar_init(&part_read, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == FS_MMA_WARP) tc_alloc(&tmem_slot, COLS);
  const int blocks = fs_blocks(a);
  unsigned asked = 0;
  FsAt at(a);
  auto ask_w = [&]() {                               // W (written by no kernel of the step: not waited for)
    const unsigned r = asked % F;
    tc_expect_tx(&raw_full[r], RAW);
    tc_load_2d(raw + r * RAW, &map_w, at.k * FS_BK, at.tile * 128, &raw_full[r]);
    tc_load_2d(raw + r * RAW + RAW / 2, &map_w, at.k * FS_BK + FS_BK / 2, at.tile * 128, &raw_full[r]);
    at.next(a);
    asked++;
  };
  if (warp == FS_TMA_WARP && lane == 0) {
    for (int i = 0; i < F; i++) { tc_bar_init(&raw_full[i], 1); tc_bar_init(&raw_free[i], 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    while ((int)asked < F && (int)asked < blocks) ask_w();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_slot, main = tmem + 6 * P, small = main + 2 * NT;
  pdl_launch_dependents();
  if (warp < 8) {
    // ------------------------------------------------------------------ cut, store
    const int quarter = warp & 3, half = warp >> 2, w_row = quarter * 32 + lane;       // of W: a row, half of the block's k
    const unsigned w_to = tmem + ((unsigned)quarter << 21) + half * (P / 2);
    const int row = threadIdx.x >> 4, chunk = threadIdx.x & 15;      // of the tokens: rows row + 16 j, floats 4 chunk .. + 3
    const unsigned at_x = row * 128 + (((chunk >> 1) ^ (row & 7)) << 4) + (chunk & 1) * 8;
    float4 x[XP];
    auto ask_x = [&]() {
      const int k = at.k * FS_BK + chunk * 4;
#pragma unroll
      for (int j = 0; j < XP; j++) {
        const int t = row + 16 * j;
        x[j] = k < a.K && t < a.T ? __ldg(reinterpret_cast<const float4*>(a.X + (size_t)t * a.ldx + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      at.next(a);
    };
    pdl_wait();
    ask_x();
    for (int g = 0, r = 0, ph = 0; g < blocks; g++) {
      const int s = g & 1;
      if (!tc_wait(&raw_full[r], ph, &dead) && lane == 0) atomicExch(a.status, 1);
      float4 w[8];
#pragma unroll
      for (int j = 0; j < 8; j++)
        w[j] = *reinterpret_cast<const float4*>(raw + r * RAW + half * (RAW / 2) + w_row * 128 + ((j ^ (w_row & 7)) << 4));
      if (!tc_wait(&done[s], ((g >> 1) & 1) ^ 1, &dead) && lane == 0) atomicExch(a.status, 2);       // the stage is free
      tc_fence_after();
#pragma unroll
      for (int j = 0; j < XP; j++) fs_put(ring + s * 3 * XPIECE + at_x + j * 2048, XPIECE, x[j]);
#pragma unroll
      for (int j = 0; j < 8; j += 4) {               // 16 floats: 8 columns of each piece
        unsigned p1[8], p2[8], p3[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          cut3(w[j + i].x, w[j + i].y, p1[2 * i], p2[2 * i], p3[2 * i]);
          cut3(w[j + i].z, w[j + i].w, p1[2 * i + 1], p2[2 * i + 1], p3[2 * i + 1]);
        }
        __syncwarp();
        tc_st8(w_to + s * 3 * P + 2 * j, p1);
        tc_st8(w_to + s * 3 * P + P + 2 * j, p2);
        tc_st8(w_to + s * 3 * P + 2 * P + 2 * j, p3);
      }
      tc_st_wait();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tokens are read by the tensor cores
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { tc_arrive(&full[s]); tc_arrive(&raw_free[r]); }
      if (++r == F) { r = 0; ph ^= 1; }
      if (g + 1 < blocks) ask_x();
    }
  } else if (warp < 16) {
    // ------------------------------------------------------------------ the blocks' sums, and the results
    const int quarter = warp & 3, half = (warp >> 2) & 1;
    const unsigned mine = ((unsigned)quarter << 21) + half * HALF;
    float sum[HALF];
#pragma unroll
    for (int i = 0; i < HALF; i++) sum[i] = 0.f;
    if (lane == 0) { tc_arrive(&full[0]); tc_arrive(&full[1]); }
    pdl_wait();
    for (int g = 0; g < blocks; g++, at.next(a)) {
      const int s = g & 1;
      if (!tc_wait(&done[s], (g >> 1) & 1, &dead, 32) && lane == 0) atomicExch(a.status, 3);
      tc_fence_after();
      const bool end = at.ends_part(a);
#pragma unroll
      for (int c = 0; c < HALF; c += 8) fs_add8(main + s * NT + mine + c, sum + c);
      if (end) {
#pragma unroll
        for (int c = 0; c < HALF; c += 8) fs_add8(small + mine + c, sum + c);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) tc_arrive(&full[s]);
      if (!end) continue;
      if (lane == 0) tc_arrive(&part_read);
      fs_store(a, at.run, at.tile, at.tile * 128 + quarter * 32 + lane, half * HALF, a.T, sum);
    }
  } else if (warp == FS_TMA_WARP) {
    if (lane == 0)
      while ((int)asked < blocks) {
        if (!tc_wait(&raw_free[asked % F], (asked / F & 1) ^ 1, &dead)) { atomicExch(a.status, 4); break; }
        ask_w();
      }
  } else if (warp == FS_MMA_WARP) {
    const unsigned idesc = tc_idesc_bf16(128, NT);
    const unsigned long long x0 = tc_desc_sw128(tc_smem(ring));
    const bool one = tc_elect();
    bool first = true;                               // of a part: the small products' sum begins anew
    unsigned parts = 0;
    for (int g = 0; g < blocks; g++) {
      const int s = g & 1;
      if (!tc_wait(&full[s], (g >> 1) & 1, &dead) && one) atomicExch(a.status, 5);
      if (first && g > 0) {
        if (!tc_wait(&part_read, parts & 1, &dead) && one) atomicExch(a.status, 6);
        parts++;
      }
      tc_fence_after();
      __syncwarp();
      const unsigned w = tmem + s * 3 * P;
      const unsigned long long x = x0 + s * (3 * XPIECE >> 4);
      if (one) {
        FS_WITH_X2(small, w, x + (XPIECE >> 4), idesc, first);
        FS_WITH_X3(small, w, x + 2 * (XPIECE >> 4), idesc);
        fs_product(small, w + P, x, idesc, false);
        fs_product(small, w + 2 * P, x, idesc, false);
        fs_product(main + s * NT, w, x, idesc, true);
        tc_commit(&done[s]);
      }
      first = at.ends_part(a);
      at.next(a);
    }
  }
  fs_end(dead, warp, lane, tmem, COLS, raw_full, F, asked);
}

// ---------------------------------------------------------------------------------------------- more tokens
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
    fs_put(reinterpret_cast<unsigned char*>(pieces + t * Kp + k), plane * 2, v);
  }
}

// up to NT tokens to a tile
template <int NT>
__global__ void __launch_bounds__(FS_THREADS, 1)
gemm_f32_many_kernel(const __grid_constant__ CUtensorMap map_x, const FsArgs a) {
  constexpr int HALF = NT / 2, XPIECE = NT * 128;
  constexpr unsigned COLS = 2 * NT <= 256 ? 256 : 512, P = FS_WPIECE >> 4;
  extern __shared__ unsigned char smem_raw[];
  __shared__ unsigned long long wfull[2], wfree[2], xfull[FS_XSLOTS], xfree[FS_XSLOTS], done, sfree;
  __shared__ unsigned tmem_slot;
  __shared__ int dead;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* wring = smem_raw + ((1024 - (tc_smem(smem_raw) & 1023)) & 1023);      // [2][3 pieces][128 rows][128 bytes]
  unsigned char* xring = wring + 2 * FS_WBLOCK;                                        // [FS_XSLOTS][tokens][128 bytes]
  if (threadIdx.x == 0) {
    dead = 0;
    for (int i = 0; i < 2; i++) { tc_bar_init(&wfull[i], 8); tc_bar_init(&wfree[i], 1); }
    for (int i = 0; i < FS_XSLOTS; i++) { tc_bar_init(&xfull[i], 1); tc_bar_init(&xfree[i], 1); }
    tc_bar_init(&done, 1);
    tc_bar_init(&sfree, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == FS_MMA_WARP) tc_alloc(&tmem_slot, COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_slot, small = tmem + NT;
  pdl_launch_dependents();
  const int blocks = fs_blocks(a);
  unsigned asked = 0;                                // loads of the tokens' pieces so far
  if (warp < 8) {
    // ------------------------------------------------------------------ W: read, cut, store
    FS_GIVE(64);
    const int row = threadIdx.x >> 4, chunk = threadIdx.x & 15;      // rows row + 16 j, floats 4 chunk .. + 3 of a block
    const unsigned at = row * 128 + (((chunk >> 1) ^ (row & 7)) << 4) + (chunk & 1) * 8;
    float4 w[8];
    FsAt ask(a);
    auto ask_w = [&]() {
      const int k = ask.k * FS_BK + chunk * 4;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int r = min(ask.tile * 128 + row + 16 * j, a.N - 1);
        w[j] = k < a.K ? __ldg(reinterpret_cast<const float4*>(a.W + (size_t)r * a.K + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      ask.next(a);
    };
    ask_w();
    for (int g = 0; g < blocks; g++) {
      if (!tc_wait_inline(&wfree[g & 1], ((g >> 1) & 1) ^ 1, &dead, 32) && lane == 0) atomicExch(a.status, 1);
      unsigned char* dst = wring + (g & 1) * FS_WBLOCK + at;
#pragma unroll
      for (int j = 0; j < 8; j++) fs_put(dst + j * 2048, FS_WPIECE, w[j]);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // read by the tensor cores
      __syncwarp();
      if (lane == 0) tc_arrive(&wfull[g & 1]);
      if (g + 1 < blocks) ask_w();
    }
  } else if (warp < 16) {
    // ------------------------------------------------------------------ the blocks' sums, and the results
    FS_TAKE(152);
    const int quarter = warp & 3, half = (warp >> 2) & 1;
    const unsigned mine = ((unsigned)quarter << 21) + half * HALF;
    float sum[HALF];
#pragma unroll
    for (int i = 0; i < HALF; i++) sum[i] = 0.f;
    FsAt at(a);
    pdl_wait();
    for (int g = 0; g < blocks; g++, at.next(a)) {
      if (!tc_wait_inline(&done, g & 1, &dead, 32) && lane == 0) atomicExch(a.status, 2);
      tc_fence_after();
      const bool end = at.ends_part(a);
#pragma unroll
      for (int c = 0; c < HALF; c += 8) fs_add8(tmem + mine + c, sum + c);
      if (end) {
#pragma unroll
        for (int c = 0; c < HALF; c += 8) fs_add8(small + mine + c, sum + c);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) tc_arrive(&sfree);
      if (!end) continue;
      const int t0 = at.tt * a.t_rows;
      fs_store(a, at.run, at.tile, at.tile * 128 + quarter * 32 + lane, t0 + half * HALF, min(a.T, t0 + a.t_rows), sum);
    }
  } else {
    FS_GIVE(48);
    if (warp == FS_TMA_WARP) {
      // ---------------------------------------------------------------- the tokens' pieces, in the order x2, x3, x1
      pdl_wait();
      if (lane == 0) {
        asm volatile("fence.proxy.async;" ::: "memory");
        FsAt at(a);
        unsigned s = 0, ph = 0;
        for (int g = 0; g < blocks; g++, at.next(a))
          for (int i = 0; i < 3; i++) {
            if (!tc_wait_inline(&xfree[s], ph ^ 1, &dead)) { atomicExch(a.status, 3); g = blocks; break; }
            tc_expect_tx(&xfull[s], a.n_cols * 128);
            tc_load_2d(xring + s * XPIECE, &map_x, at.k * FS_BK, (i == 2 ? 0 : i + 1) * a.T + at.tt * a.t_rows, &xfull[s]);
            asked++;
            if (++s == FS_XSLOTS) { s = 0; ph ^= 1; }
          }
      }
    } else if (warp == FS_MMA_WARP) {
      // ---------------------------------------------------------------- MMA issuer
      // Each wait takes 200 to 300 cycles beside the others' stores, so what comes next is waited for one product ahead, while
      // the tensor cores still have the last ones to do.
      const unsigned idesc = tc_idesc_bf16(128, a.n_cols);
      const unsigned long long dw0 = tc_desc_sw128(tc_smem(wring)), dx0 = tc_desc_sw128(tc_smem(xring));
      const bool one = tc_elect();
      FsAt at(a);
      unsigned s = 0, ph = 0;
      auto x_there = [&](unsigned code) {
        if (!tc_wait_inline(&xfull[s], ph, &dead) && one) atomicExch(a.status, code);
        const unsigned long long x = dx0 + s * (XPIECE >> 4);
        return x;
      };
      auto x_read = [&]() {
        if (one) tc_commit(&xfree[s]);
        if (++s == FS_XSLOTS) { s = 0; ph ^= 1; }
      };
      auto go = [&]() { tc_fence_after(); __syncwarp(); };
      auto w_there = [&](int g) {
        if (!tc_wait_inline(&wfull[g & 1], (g >> 1) & 1, &dead) && one) atomicExch(a.status, 4);
      };
      auto sums_read = [&](int g) {                  // of the block before
        if (g > 0 && !tc_wait_inline(&sfree, (g - 1) & 1, &dead) && one) atomicExch(a.status, 8);
      };
      w_there(0);
      unsigned long long x = x_there(5);
      bool first = true;                             // of a part: the small products' sum begins anew
      for (int g = 0; g < blocks; g++) {
        const unsigned long long w = dw0 + (g & 1) * (FS_WBLOCK >> 4);
        const bool end = at.ends_part(a);
        at.next(a);
        if (first) sums_read(g);
        go();
        if (one) FS_WITH_X2(small, w, x, idesc, first);
        x_read();
        x = x_there(6);
        go();
        if (one) FS_WITH_X3(small, w, x, idesc);
        x_read();
        x = x_there(7);
        go();
        if (one) fs_product(small, w + P, x, idesc, false);
        if (!first) sums_read(g);
        if (one) fs_product(small, w + 2 * P, x, idesc, false);
        if (g + 1 < blocks) w_there(g + 1);
        go();
        if (one) {
          fs_product(tmem, w, x, idesc, true);
          tc_commit(&done);
          tc_commit(&wfree[g & 1]);
        }
        x_read();
        if (g + 1 < blocks) x = x_there(5);
        first = end;
      }
    }
  }
  fs_end(dead, warp, lane, tmem, COLS, xfull, FS_XSLOTS, asked);
}

// Y[t, n] = the sums of the runs that have a part of n's tile, in the order of the runs (+ bias); whole tiles are written already.
// A block: a tile and 8 R tokens, a warp R of them, 8 apart; a thread has four features (V = 4) or one, and its loads of FR_RUNS runs'
// sums in flight together: one run after the other they took 4.7 us for the 10 runs of a tile at 4 tokens.
#define FR_RUNS 4
template <int V, int R>
__global__ void __launch_bounds__(256)
f32_runs_kernel(const FsArgs a) {
  pdl_launch_dependents();
  const int tile = blockIdx.x, t0 = blockIdx.y * 8 * R + (threadIdx.x >> 5);
  const int first = fs_run_of((long long)tile * a.kb, a.runs, a.total);
  const int shares = fs_run_of((long long)tile * a.kb + a.kb - 1, a.runs, a.total) - first + 1;
  pdl_wait();
  if (shares == 1) return;
  const size_t step = (size_t)a.T * a.N;
#pragma unroll
  for (int c = 0; c < 128; c += 32 * V) {
    const int n = tile * 128 + c + (threadIdx.x & 31) * V;
    if (n >= a.N) continue;
    const float* from = a.part + (size_t)t0 * a.N + n;
    float s[R][V];
    for (int i0 = 0; i0 < shares; i0 += FR_RUNS) {
      float v[FR_RUNS][R][V];
#pragma unroll
      for (int i = 0; i < FR_RUNS; i++)
#pragma unroll
        for (int r = 0; r < R; r++) {
          const float* p = from + (i0 + i) * step + (size_t)(8 * r) * a.N;
          const bool in = i0 + i < shares && t0 + 8 * r < a.T;
          if constexpr (V == 4) {
            const float4 q = in ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i][r][0] = q.x; v[i][r][1] = q.y; v[i][r][2] = q.z; v[i][r][3] = q.w;
          } else {
            v[i][r][0] = in ? *p : 0.f;
          }
        }
#pragma unroll
      for (int i = 0; i < FR_RUNS; i++)
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
          for (int u = 0; u < V; u++)
            if (i0 + i == 0) s[r][u] = v[i][r][u];
            else if (i0 + i < shares) s[r][u] += v[i][r][u];
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int t = t0 + 8 * r;
      if (t >= a.T) continue;
      float* y = a.Y + t * a.ldy + n;
      bool doubtful = false;
#pragma unroll
      for (int u = 0; u < V; u++) {
        const float q = a.bias ? s[r][u] + a.bias[n + u] : s[r][u];
        y[u] = q;
        doubtful = doubtful || fs_doubtful(q);
      }
      if (doubtful)
        for (int u = 0; u < V; u++) fs_settle(a, t, n + u, y + u);
    }
  }
}
static void launch_runs(const FsArgs& a, cudaStream_t stream) {
  const int tiles = (a.N + 127) / 128;
  if (a.N % 4) qd_launch(f32_runs_kernel<1, 4>, dim3(tiles, (a.T + 31) / 32), dim3(256), 0, stream, a);
  else if (a.T <= 8) qd_launch(f32_runs_kernel<4, 1>, dim3(tiles, 1), dim3(256), 0, stream, a);
  else qd_launch(f32_runs_kernel<4, 2>, dim3(tiles, (a.T + 15) / 16), dim3(256), 0, stream, a);
}

// ---------------------------------------------------------------------------------------------- host
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
static int fs_sms() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int NT, int F>
static int launch_few(const FsArgs& a, int grid, cudaStream_t stream) {
  constexpr int smem = 2 * 3 * NT * 128 + F * 128 * FS_BK * 4 + 1024;
  CUtensorMap map;
  if (!tc_make_map(&map, a.W, false, a.N, a.K, 128)) return QD_ERR_UNSUPPORTED;
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_kernel<NT, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  qd_launch(gemm_f32_few_kernel<NT, F>, dim3(grid), dim3(FS_THREADS), smem, stream, map, a);
  return qd_last_error();
}
static int fs_few(const FsArgs& a, int grid, cudaStream_t stream) {
  if (a.T <= 16) return launch_few<16, 5>(a, grid, stream);
  if (a.T <= 32) return launch_few<32, 5>(a, grid, stream);
  return launch_few<64, 4>(a, grid, stream);
}

template <int NT>
static int launch_many(const FsArgs& a, void* pieces, int grid, cudaStream_t stream) {
  constexpr int smem = 2 * FS_WBLOCK + FS_XSLOTS * NT * 128 + 1024;
  CUtensorMap map;
  if (!tc_make_map(&map, pieces, true, 3ll * a.T, (long long)a.kb * FS_BK, a.n_cols)) return QD_ERR_UNSUPPORTED;
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_many_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  qd_launch(gemm_f32_many_kernel<NT>, dim3(grid), dim3(FS_THREADS), smem, stream, map, a);
  return qd_last_error();
}
static int fs_many(FsArgs a, void* pieces, int grid, cudaStream_t stream) {
  a.t_tiles = (a.T + FS_MANY - 1) / FS_MANY;
  a.t_rows = (a.T + a.t_tiles - 1) / a.t_tiles;
  a.n_cols = (a.t_rows + 15) / 16 * 16;
  const int Kp = a.kb * FS_BK;
  const size_t quads = (size_t)a.T * Kp / 4;
  const unsigned blocks = (unsigned)((quads + 255) / 256 < 1184 ? (quads + 255) / 256 : 1184);
  qd_launch(f32_cut_kernel, dim3(blocks), dim3(256), 0, stream, a.X, a.ldx, (bf16*)pieces, a.T, a.K, Kp);
  const int rc = qd_last_error();
  if (rc) return rc;
  if (a.t_rows <= 96) return launch_many<96>(a, pieces, grid, stream);
  if (a.t_rows <= 128) return launch_many<128>(a, pieces, grid, stream);
  if (a.t_rows <= 160) return launch_many<160>(a, pieces, grid, stream);
  if (a.t_rows <= 192) return launch_many<192>(a, pieces, grid, stream);
  return launch_many<224>(a, pieces, grid, stream);
}

// ``pieces``: scratch of 3 * min(T, seg) * ceil(K / 64) * 64 bfloat16, for more than 64 tokens; ``part``: scratch of
// shares * min(T, seg) * N floats where runs end inside tiles, shares = ceil(runs / tiles) + 1.  ``seg``: tokens that are worked on
// at once (what bounds the scratch).  ``runs``: at most ceil(N / 128) * ceil(K / 64).
extern "C" int qd_gemm_f32(const float* X, const float* W, const float* bias, float* Y, void* pieces, float* part, int T, int N,
                           int K, long long ldx, long long ldy, int runs, int seg, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return 0;
  const long long kb = ((long long)K + FS_BK - 1) / FS_BK, total = (N + 127ll) / 128 * kb;
  if (K <= 0 || K % 4 || ldx % 4 || (((uintptr_t)X | (uintptr_t)W | (uintptr_t)pieces | (uintptr_t)part) & 15) || !Y || runs < 1 || runs > total ||
      total * (runs + 1) > 0x7fffffffffll || total > 0x3fffffff || seg < 1 || seg > 65535)
    return QD_ERR_UNSUPPORTED;
  const bool cut = total % runs || total / runs % kb;        // whether runs end inside tiles
  if ((cut && !part) || (T > FS_FEW && !pieces)) return QD_ERR_UNSUPPORTED;
  FsArgs a = {};
  a.W = W; a.bias = bias; a.part = part; a.ldx = ldx; a.ldy = ldy; a.N = N; a.K = K;
  a.kb = (int)kb; a.runs = runs; a.total = (int)total; a.t_tiles = 1;
  a.status = fs_status_word();
  if (!a.status) return QD_ERR_UNSUPPORTED;
  const int sms = fs_sms(), grid = runs < sms ? runs : sms;
  for (int t0 = 0; t0 < T; t0 += seg) {
    a.X = X + (long long)t0 * ldx;
    a.Y = Y + (long long)t0 * ldy;
    a.T = T - t0 < seg ? T - t0 : seg;
    int rc = a.T <= FS_FEW ? fs_few(a, grid, stream) : fs_many(a, pieces, grid, stream);
    if (rc) return rc;
    if (cut) {
      launch_runs(a, stream);
      if ((rc = qd_last_error())) return rc;
    }
  }
  return 0;
}

// 0 if no bounded wait of this library has run out on the current device.  Reported once.  Synchronises.
QD_DEFINE_WAIT_PROBE(qd_gemm_f32_wait_probe, tc_wait(bar, 0, dead, 0, poll_limit), fs_status_word, 99)

extern "C" int qd_gemm_f32_status() {
  int* status = fs_status_word();
  if (!status) return -1;
  int v = 0;
  if (cudaMemcpy(&v, status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (v) cudaMemset(status, 0, sizeof(int));
  return v;
}
