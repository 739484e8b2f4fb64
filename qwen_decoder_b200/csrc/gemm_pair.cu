// Contraction Y[T, N] = X[T, K] * W[N, K]^T of more than a few tokens on pairs of multiprocessors: tcgen05.mma with
// cta_group::2, bfloat16 in, float32 sums in tensor memory, operands by TMA tensor copies (128-byte swizzle).
//
// A cluster of two CTAs works on a tile of up to 256 tokens (the MMA's rows, 128 a CTA) by ``bn`` rows of W (its columns, 32 to
// 256): each CTA brings its own tokens and half of the weights' rows, the tensor cores of both read both halves.  A byte brought
// into shared memory thereby serves twice as many products as with one CTA, which is what bounds a tile of 256 x 256 (64 bytes a
// clock and multiprocessor against 512 clocks of MMAs a block of 64 k).  Few tokens: a CTA brings only the rows there are (the
// rest of the MMA's rows are never looked at), and the launch is bound by reading W.
//
// Warps of a CTA: 0..7 epilogue (two for each quarter of the lanes, columns halved between them), 8 producer, 9 MMAs (only the
// pair's first CTA issues them).  A pair goes through its items (feature tile x token tile x share of K) one after the other;
// the accumulator is double-buffered, so that an item's epilogue runs under the next one's MMAs.  The producer asks for the first
// stages' weights before the programmatic-dependency wait and for the tokens after it.
//
// Epilogues: whole sums (+ bias) as bfloat16 or float32; float32 partial sums of a share of K; the gated activation, where a
// pair's first CTA brings rows of the gate matrix and the second the same rows of the up matrix, so that both sums of a feature
// lie in one thread's lane.
//
// Every mbarrier wait is bounded; after one that ran out all roles run on to their ends with void results and a status word says
// which wait it was.
//
// The reference calls cublasHgemm for these products (gpu_kernels.cu:431-436) and adds bias and SwiGLU in kernels of their own
// (gpu_kernels.cu:70-79, 149-160).
#include "tc5_ops.cuh"
#include "entry_points.h"

#define GP_EPI_WARPS 8
#define GP_THREADS (GP_EPI_WARPS * 32 + 64)
#define GP_MAX_STAGES 16
#define GP_SMEM (206 * 1024)          // of stages: with 128 KB the products of 64 tokens took 4 % longer, with 94 KB (two CTAs to a
                                      // multiprocessor, the next product's beside this one's) 11 %
#define GP_STAGE_ROWS (32 * 64)       // of a warp's epilogue: 64 bytes of each of its rows
#define GP_BK 64

#define GP_PLAIN_TOKENS 256           // beyond these only the gated product is taken
#define GP_STORE_FEATURES 10240       // of whole sums at least

#define GP_STORE 0
#define GP_PARTIAL 1
#define GP_GATED 2

struct GpParams {
  int act, T, N, K;
  int bn;                  // rows of W of a tile, of both CTAs together
  int mrows;               // tokens of a CTA
  int n_ft, n_tt, splits;
  int kb_total, stages;
  int acc_stride, tmem_cols;
  int feats;               // columns of the result
  int vec;                 // rows of the result take 16-byte stores
  long long ldo;
};

// ---- what a pair needs beyond tc5_ops.cuh
__device__ __forceinline__ unsigned gp_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
// where the first CTA of the pair has what this one has at ``p``: bit 24 of a shared-memory address is the place in the pair (what
// mapa gives, too, but the compiler sees that all lanes have the same: a copy took 125 cycles of the producer with mapa, 16 so)
__device__ __forceinline__ unsigned gp_leader(const void* p) { return tc_smem(p) & 0xFEFFFFFFu; }
__device__ __forceinline__ void gp_arrive_at(unsigned bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void gp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// into this CTA's shared memory, the bytes counted on a barrier of either CTA
__device__ __forceinline__ void gp_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(tc_smem(dst)), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void gp_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n}\n"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u) : "memory");
}
// arrives at the barrier of both CTAs once the MMAs so far are done
__device__ __forceinline__ void gp_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(tc_smem(bar)), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ void gp_alloc(unsigned* slot, unsigned cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void gp_ld16(unsigned addr, float (&v)[16]) {
  unsigned r[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(addr));
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// A place in a pair's sequence of (item, block of 64 k)
struct GpPos { int item, kb, kb1, ya, yb; };

template <int EPI, int CG>
__device__ __forceinline__ void gp_open(const GpParams& p, int rank, GpPos& q) {
  const int sp = q.item % p.splits, rest = q.item / p.splits, tt = rest % p.n_tt, ft = rest / p.n_tt;
  q.kb = p.kb_total * sp / p.splits;
  q.kb1 = p.kb_total * (sp + 1) / p.splits;
  q.ya = (CG * tt + rank) * p.mrows;
  q.yb = EPI == GP_GATED ? ft * (p.bn >> 1) + rank * p.feats : ft * p.bn + rank * (p.bn >> 1);
}

__device__ __forceinline__ void gp_bias16(float (&v)[16], const float* bias, int col, int feats) {
#pragma unroll
  for (int i = 0; i < 16; i++)
    if (col + i < feats) v[i] += bias[col + i];
}
// v = act(v) u.  A gate of minus infinity goes as the largest finite one does, to zero: as it stands, the quotient by an infinite
// exponential would be no number.  Which activation is asked once: a launch's epilogue is bound by its instructions on their way (with a
// selection at each number, though without the maximum, a prompt of 101 tokens at the 3B sizes took 2,464 us, so 2,447).
template <int ACT>
__device__ __forceinline__ void gp_gated16(float (&v)[16], const float (&u)[16]) {
#pragma unroll
  for (int i = 0; i < 16; i++) {
    asm("max.NaN.f32 %0, %0, 0fFF7FFFFF;" : "+f"(v[i]));
    v[i] = __fdividef(v[i], 1.0f + __expf(-qd_gate_arg(v[i], ACT))) * u[i];
  }
}
__device__ __forceinline__ void gp_gated16(float (&v)[16], const float (&u)[16], int act) {
  if (act == QD_ACT_GELU_TANH) gp_gated16<QD_ACT_GELU_TANH>(v, u);
  else gp_gated16<QD_ACT_SILU>(v, u);
}
// 16 numbers as pieces of 16 bytes of a row of 64 in a warp's part of shared memory.  Rows lie side by side, the pieces of rows
// 2 i and 2 i + 1 turned by i: eight lanes that write or read together meet no bank twice.
template <typename TO>
__device__ __forceinline__ void gp_stage16(unsigned char* rows, int row, int piece, const float (&v)[16]) {
  uint4 u[sizeof(TO)];
  if (sizeof(TO) == 4) {
#pragma unroll
    for (int i = 0; i < 4; i++)
      u[i] = make_uint4(__float_as_uint(v[4 * i]), __float_as_uint(v[4 * i + 1]), __float_as_uint(v[4 * i + 2]), __float_as_uint(v[4 * i + 3]));
  } else {
    unsigned h[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      h[i] = *reinterpret_cast<const unsigned*>(&b);
    }
    u[0] = make_uint4(h[0], h[1], h[2], h[3]);
    u[1] = make_uint4(h[4], h[5], h[6], h[7]);
  }
#pragma unroll
  for (int i = 0; i < (int)sizeof(TO); i++)
    *reinterpret_cast<uint4*>(rows + row * 64 + (((piece + i) ^ (row >> 1 & 3)) << 4)) = u[i];
}

template <int EPI, typename TO, int CG>
__global__ void __launch_bounds__(GP_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                 const float* __restrict__ bias, TO* __restrict__ out, const GpParams p, int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long full[GP_MAX_STAGES], empty[GP_MAX_STAGES], acc_ready[2], acc_free[2];
  __shared__ unsigned tmem_slot;
  __shared__ int dead;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CG == 2 ? (int)gp_rank() : 0;
  unsigned char* base = smem_raw + ((1024 - (tc_smem(smem_raw) & 1023)) & 1023);
  // The stages' tokens lie before the stages' weights: an MMA reads 128 rows of tokens whatever a CTA has, and what lies behind
  // them is then always there.
  const int a_bytes = p.mrows * 128, b_bytes = p.bn / CG * 128;
  unsigned char* a_s = base;
  unsigned char* b_s = base + (size_t)p.stages * a_bytes;
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    dead = 0;
    for (int s = 0; s < p.stages; s++) { tc_bar_init(&full[s], 1); tc_bar_init(&empty[s], 1); }
    for (int b = 0; b < 2; b++) { tc_bar_init(&acc_ready[b], 1); tc_bar_init(&acc_free[b], CG * GP_EPI_WARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (CG == 2) gp_cluster_sync();

  const int worker = blockIdx.x / CG, n_workers = gridDim.x / CG, n_items = p.n_ft * p.n_tt * p.splits;

  if (warp == GP_EPI_WARPS) {
    // ------------------------------------------------------------------ producer
    // The whole warp goes through the loop, one lane of it issues: the compiler then knows that addresses and coordinates are the
    // same for all lanes (with the loop in one lane alone a copy cost 100 cycles, a block of k 480).
    const bool one = tc_elect();
    const unsigned bytes = (unsigned)(CG * (a_bytes + b_bytes));
    const int half = p.bn >> 1;
    auto load = [&](unsigned char* dst, const CUtensorMap* map, int x, int y, int s) {
      if (CG == 2) gp_load_2d(dst, map, x, y, gp_leader(&full[s]));
      else tc_load_2d(dst, map, x, y, &full[s]);
    };
    auto tokens = [&](int s, const GpPos& q) { load(a_s + s * a_bytes, &map_x, q.kb * GP_BK, q.ya, s); };
    auto weights = [&](int s, const GpPos& q) {
      if (CG == 1 || rank == 0) tc_expect_tx(&full[s], bytes);
      load(b_s + s * b_bytes, &map_w, q.kb * GP_BK, q.yb, s);
      if (CG == 1 && EPI == GP_GATED) load(b_s + s * b_bytes + half * 128, &map_w, q.kb * GP_BK, q.yb + p.feats, s);
    };
    auto next = [&](GpPos& q) {
      if (++q.kb < q.kb1) return;
      q.item += n_workers;
      if (q.item < n_items) gp_open<EPI, CG>(p, rank, q);
    };
    GpPos q = {worker, 0, 0, 0, 0};
    gp_open<EPI, CG>(p, rank, q);
    GpPos first = q;
    int n = 0;
    for (; n < p.stages && q.item < n_items; n++, next(q))
      if (one) weights(n, q);
    pdl_wait();
    for (int s = 0; s < n; s++, next(first))
      if (one) tokens(s, first);
    int s = n == p.stages ? 0 : n;
    unsigned ph = 0;
    for (; q.item < n_items; next(q)) {
      if (!tc_wait(&empty[s], ph, &dead)) atomicExch(status, 1);
      if (one) {
        weights(s, q);
        tokens(s, q);
      }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
    // the commits' last arrivals at this CTA's barriers come before it may go
    for (int i = 0; i < n; i++) {
      if (n == p.stages) {
        if (!tc_wait(&empty[s], ph, &dead)) atomicExch(status, 1);
        if (++s == p.stages) { s = 0; ph ^= 1; }
      } else if (!tc_wait(&empty[i], 0, &dead)) {
        atomicExch(status, 1);
      }
    }
    __syncwarp();
  } else if (warp == GP_EPI_WARPS + 1) {
    // ------------------------------------------------------------------ MMAs
    if (CG == 2) gp_alloc(&tmem_slot, p.tmem_cols);
    else tc_alloc(&tmem_slot, p.tmem_cols);
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(GP_EPI_WARPS * 32 + 32) : "memory");
    tc_fence_after();
    if (rank == 0) {
      const bool one = tc_elect();
      const unsigned tmem = tmem_slot;
      const unsigned idesc = tc_idesc_bf16(128 * CG, p.bn);
      const unsigned long long a0 = tc_desc_sw128(tc_smem(a_s)), b0 = tc_desc_sw128(tc_smem(b_s));
      const unsigned a_step = (unsigned)a_bytes >> 4, b_step = (unsigned)b_bytes >> 4;
      int s = 0;
      unsigned ph = 0, buf = 0, use = 1;              // use: parity of the accumulators' "free" barriers
      for (int item = worker; item < n_items; item += n_workers) {
        const int sp = item % p.splits, kb0 = p.kb_total * sp / p.splits, kb1 = p.kb_total * (sp + 1) / p.splits;
        if (!tc_wait(&acc_free[buf], use, &dead)) atomicExch(status, 3);
        tc_fence_after();
        const unsigned d = tmem + buf * (unsigned)p.acc_stride;
        for (int kb = kb0; kb < kb1; kb++) {
          if (!tc_wait(&full[s], ph, &dead)) atomicExch(status, 2);
          tc_fence_after();
          const unsigned long long da = a0 + s * a_step, db = b0 + s * b_step;
          if (one) {
#pragma unroll
            for (int k = 0; k < GP_BK / 16; k++) {
              if (CG == 2) gp_mma(d, da + 2 * k, db + 2 * k, idesc, k > 0 || kb > kb0);
              else tc_mma_bf16(d, da + 2 * k, db + 2 * k, idesc, k > 0 || kb > kb0);
            }
            if (CG == 2) gp_commit(&empty[s]); else tc_commit(&empty[s]);
          }
          if (++s == p.stages) { s = 0; ph ^= 1; }
        }
        if (one) {
          if (CG == 2) gp_commit(&acc_ready[buf]); else tc_commit(&acc_ready[buf]);
        }
        if (++buf == 2) { buf = 0; use ^= 1; }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue
    asm volatile("bar.sync 1, %0;" ::"n"(GP_EPI_WARPS * 32 + 32) : "memory");
    tc_fence_after();
    constexpr int E = 16 / (int)sizeof(TO), PASS = 2 * 16 / (int)sizeof(TO) >= 16 ? 2 : 1;      // elements of a piece; 16s of a pass
    const int quarter = (warp & 3) * 32;
    const unsigned tmem = tmem_slot + ((unsigned)quarter << 16);
    unsigned char* rows = b_s + (size_t)p.stages * b_bytes + warp * GP_STAGE_ROWS;
    const int half = p.bn >> 1;
    const int groups = (EPI == GP_GATED ? half : p.bn) / 16;          // of 16 columns of the result
    const int g0 = groups * (warp >> 2) / 2, g1 = groups * ((warp >> 2) + 1) / 2;
    unsigned buf = 0, ph = 0;
    for (int item = worker; item < n_items; item += n_workers) {
      const int sp = item % p.splits, rest = item / p.splits, tt = rest % p.n_tt, ft = rest / p.n_tt;
      const int tok0 = (CG * tt + rank) * p.mrows + quarter;          // of this warp's rows the first, and how many there are
      const int n_rows = min(32, min(p.mrows - quarter, p.T - tok0));
      const int n0 = ft * (EPI == GP_GATED ? half : p.bn);
      TO* dst = out + (EPI == GP_PARTIAL ? ((size_t)sp * p.T + tok0) * p.N : (size_t)tok0 * p.ldo);
      const long long ld = EPI == GP_PARTIAL ? (long long)p.N : p.ldo;
      if (!tc_wait(&acc_ready[buf], ph, &dead, 64) && lane == 0) atomicExch(status, 4);
      tc_fence_after();
      const unsigned acc = tmem + buf * (unsigned)p.acc_stride;
      if (n_rows > 0) {                               // whole warps: the loads are collective
        for (int g = g0; g < g1; g += PASS) {
          const int w = min(PASS, g1 - g);            // 64 bytes of every row, or what is left of the columns
          float v[PASS][16], u[EPI == GP_GATED ? PASS : 1][16];
#pragma unroll
          for (int i = 0; i < PASS; i++)
            if (i < w) {
              gp_ld16(acc + 16 * (g + i), v[i]);
              if (EPI == GP_GATED) gp_ld16(acc + half + 16 * (g + i), u[i]);
            }
          tc_ld_wait();
          __syncwarp();
#pragma unroll
          for (int i = 0; i < PASS; i++)
            if (i < w) {
              const int col = n0 + 16 * (g + i);
              if (EPI != GP_PARTIAL && bias) gp_bias16(v[i], bias, col, p.feats);
              if (EPI == GP_GATED) {
                if (bias) gp_bias16(u[i], bias + p.feats, col, p.feats);
                gp_gated16(v[i], u[EPI == GP_GATED ? i : 0], p.act);
              }
              gp_stage16<TO>(rows, lane, i * (int)sizeof(TO), v[i]);
            }
          __syncwarp();
          const int piece = lane & 3, col = n0 + 16 * g + piece * E;
          if (piece < w * (int)sizeof(TO)) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const int r = 8 * i + (lane >> 2);
              if (r >= n_rows) break;
              const unsigned char* src = rows + r * 64 + ((piece ^ (r >> 1 & 3)) << 4);
              TO* to = dst + (size_t)r * ld + col;
              if (p.vec && col + E <= p.feats) *reinterpret_cast<uint4*>(to) = *reinterpret_cast<const uint4*>(src);
              else
                for (int e = 0; e < E && col + e < p.feats; e++) to[e] = reinterpret_cast<const TO*>(src)[e];
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) gp_arrive_at(gp_leader(&acc_free[buf]));
        else tc_arrive(&acc_free[buf]);
      }
      if (++buf == 2) { buf = 0; ph ^= 1; }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (CG == 2) gp_cluster_sync();
  if (warp == GP_EPI_WARPS + 1) {
    tc_fence_after();
    if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot), "r"((unsigned)p.tmem_cols) : "memory");
    else tc_dealloc(tmem_slot, p.tmem_cols);
  }
}

// ------------------------------------------------------------------------------------ host
static int* g_status[64];
static int* status_word() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!g_status[dev]) {
    int* ptr = nullptr;
    if (cudaMalloc(&ptr, sizeof(int)) != cudaSuccess) return nullptr;
    cudaMemset(ptr, 0, sizeof(int));
    g_status[dev] = ptr;
  }
  return g_status[dev];
}

static int up(int a, int b) { return (a + b - 1) / b; }

// The gated product of more than GP_PLAIN_TOKENS tokens: one multiprocessor to a tile of 128 tokens or two to one of 256, whichever leaves
// fewer of the MMA's rows empty, or the library's product with the activation after it.  Clocks of 1.9 GHz, fitted to times of 257 to 2,048
// tokens in captured graphs, cold weights, at the 3B, 7B and mixed sizes and two more (6 % rms): a worker's rounds of blocks of 64 k, or W's
// bytes, the longer of both and some of the other; the library's: 1.62 times what the tensor cores need and 12 us, about its best, less 5 %
// (a 3B prompt of 300 tokens took 1.4 % longer so where the estimates were 4 % apart the other way).  Measured on a B200, us, as chosen ("-": the library) / two multiprocessors to every tile / the library:
//   tokens          3B                       7B                      mixed
//     257     - / 34.6 / 31.9          - / 91.5 / 70.1         17.3 / 20.4 / 17.6
//     300     - / 34.8 / 33.3          - / 96.2 / 77.7         17.4 / 20.3 / 18.5
//     340  31.7 / 35.0 / 32.6          - / 92.7 / 82.3         17.5 / 20.4 / 20.3
//     384  32.0 / 35.3 / 33.4       86.5 / 93.6 / 84.8         17.5 / 20.6 / 19.5
//     400  35.9 / 35.9 / 37.7          - / 93.6 / 91.5         20.5 / 20.8 / 22.1
//     450  35.6 / 35.6 / 42.1       93.9 / 93.9 / 101.1        20.9 / 20.9 / 22.9
//     512  37.0 / 37.0 / 43.9       95.3 / 95.3 / 110.0        21.0 / 21.0 / 25.3
//     513  45.5 / 50.5 / 49.3          - / 134.8 / 115.7       23.8 / 27.0 / 25.6
//     600  45.9 / 50.1 / 53.1      128.3 / 137.3 / 127.5       24.3 / 27.0 / 28.3
//     769     - / 63.9 / 62.6          - / 186.8 / 180.4       32.7 / 34.2 / 34.5
//   1,025  75.3 / 76.4 / 78.6          - / 236.6 / 235.6       40.4 / 40.4 / 42.2
static int gp_plan_many(int T, int N, int K, int sms, int* cg_out, int* bn_out) {
  const double dram = 2.0 * N * K / 3300.0, lib = 23000.0 + fmax(1.62 * T * N * K / (4096.0 * sms), 1.03 * dram);
  const int kb = up(K, GP_BK);
  double best = 0;
  for (int cg = 1; cg <= 2; cg++) {
    const int n_tt = up(T, 128 * cg), mrows = up(up(T, cg * n_tt), 8) * 8, workers = sms / cg;
    for (int bn = 96; bn <= 256; bn += 32) {
      const long long rounds = ((long long)up(N / 2, bn / 2) * n_tt + workers - 1) / workers;
      const double block = cg == 1 ? fmax((bn < 256 ? 3.0 : 2.85) * bn, 120 + 1.9 * bn + 0.8 * mrows)
                                   : fmax((bn < 256 ? 2.65 : 2.6) * bn, 350.0 + bn);
      const double work = rounds * (double)kb * block, cost = fmax(work, dram) + 0.18 * fmin(work, dram) + 20.0 * bn;
      if (best == 0 || cost < best) { best = cost; *cg_out = cg; *bn_out = bn; }
    }
  }
  return best <= 0.95 * lib;
}

// How a product is cut, and whether it belongs here: *cg, *bn, *splits; 0 if the library's product is the faster one.  ``epi`` as
// below; GP_PARTIAL: the caller takes whole bfloat16 sums (splits 1) or float32 partial sums.
//
// Up to 128 tokens one multiprocessor to a tile, beyond two.  The rest by what a worker's busiest share takes: rounds over its items
// times blocks of k, a block being the longest of its MMAs (2 bn clocks), its bytes (60 a clock into shared memory) and the 350
// clocks that one costs anyway; or W's bytes at 6.3 TB/s; the longer of both and some of the other; plus an item's epilogue and the partial sums' way through L2.
// Measured on a B200, us, here / the library (the gated product with its activation, the others with the norm that follows), 3B and 7B:
//   tokens       gate and up                down                 output projection
//     64      18.1 / 21.7 45.0/51.8  14.0 / 19.0 29.0/33.9   7.3 / 8.2    - /11.2
//    192      21.7 / 25.9 55.2/60.6  16.8 / 19.9 36.4/47.1     - / 8.7    - /12.4
//    512      37.0 / 43.9 95.3/110     - / 27.1    - /60.5     - /10.8    - /17.4
// Sums for a norm, where the library shares K well enough by itself: 3,584 x 3,584, 17, 64, 112 and 128 tokens 10.6 / 10.9, 11.3 / 11.2,
// 11.7 / 10.6 and 12.3 / 11.4; 5,120 x 5,120, 64 tokens 16.4 / 15.3; 4,096 x 14,336, 144 and 256 tokens 31.7 / 29.2 and 36.9 / 33.8.
// Whole sums, float32: a projection over the vocabulary, 151,936 x 2,048 and 152,064 x 3,584: 17 rows 99 / 107 and 166 / 185, 128 rows 117 / 140
// and 202 / 219, 256 rows 145 / 187 and 248 / 325; 32,000 x 2,048: 64 rows 26.5 / 27.8, 128 rows 28.3 / 30.9, 160 rows 31.9 / 31.2.
// Layers' own: 12,352 x 2,048, 64 and 129 tokens 11.6 / 11.8 and 15.1 / 13.1.  These stay here up to 256 tokens all the same: steps of so
// few tokens through such layers wait for the host, where a call of the library's costs 19 us more (a prompt of 130 tokens through eight
// mixed layers 2,115 us, with the library's eight products 2,220; in 64 requests' replayed step, where the host does not count, 1,010 and
// 968).  2,048 x 4,096 of 193 to 256 tokens for a norm for the same reason: 12.2 / 11.6, 200 tokens through eight layers 2,100 us and 2,270.
// Beyond 256 tokens the library's are up to 16 % faster and never more than 5 % slower: 12,352 x 2,048, 1,025 and 1,500 tokens 49.2 / 41.3 and
// 57.8 / 57.7.  So they are with fewer features: 8,192 x 2,048 in bfloat16, 32 and 129 tokens 10.3 / 8.5 and 11.6 / 9.9; q/k/v of the 3B
// sizes, 64 tokens 7.5 / 5.8.
extern "C" int qd_gemm_pair_plan(int T, int N, int K, int epi, int sms, int* cg_out, int* bn_out, int* splits_out) {
  epi &= 255;
  if (T <= 0 || N <= 0 || K <= 0 || sms < 2) return 0;
  if ((long long)N * K < (1 << 20)) return 0;        // small models: a launch's own time
  if (epi != GP_GATED && T > GP_PLAIN_TOKENS) return 0;
  if (epi == GP_STORE && N < GP_STORE_FEATURES) return 0;
  if (epi == GP_PARTIAL && (T <= 128 ? K < 2 * N && N > 3072 : K < 2 * N || N >= 4096)) return 0;
  if (epi == GP_GATED && T > GP_PLAIN_TOKENS) {
    *splits_out = 1;
    return gp_plan_many(T, N, K, sms, cg_out, bn_out);
  }
  const int cg = T <= 128 ? 1 : 2, workers = sms / cg, n_tt = up(T, 128 * cg), mrows = up(up(T, cg * n_tt), 8) * 8;
  const int feats = epi == GP_GATED ? N / 2 : N, kb = up(K, GP_BK);
  const double dram = 2.0 * N * K / 3300.0;          // clocks of 1.9 GHz
  double best = 0, best_work = 0;
  for (int bn = 64; bn <= 256; bn += 32) {
    const long long tiles = (long long)up(feats, epi == GP_GATED ? bn / 2 : bn) * n_tt;
    for (int splits = 1; splits <= (epi == GP_PARTIAL ? 8 : 1) && (splits == 1 || splits * 8 <= kb); splits++) {
      const long long rounds = (tiles * splits + workers - 1) / workers;
      const double bytes = (mrows + bn / cg) * 128 / 60.0;
      double block = 2.0 * bn;
      if (block < bytes) block = bytes;
      if (block < 350) block = 350;
      if (bn == 256 && rounds > 4) block *= 1.12;    // (all of tensor memory in turn: 139 us where 224 takes 123)
      const double work = (double)rounds * up(kb, splits) * block;
      double cost = work > dram ? work + 0.15 * dram : dram + 0.15 * work;
      cost += 12.0 * bn + (splits > 1 ? 8.0 * splits * T * N / 4000.0 : 2.0 * T * N / 4000.0);
      if (best == 0 || cost < best) { best = cost; best_work = work; *cg_out = cg; *bn_out = bn; *splits_out = splits; }
    }
  }
  // whole sums of a long k by few workers: the library shares k
  return epi != GP_STORE || best_work < 1.2 * dram;
}

template <int EPI, typename TO, int CG>
static int gp_launch(const CUtensorMap& map_w, const CUtensorMap& map_x, const float* bias, void* out, const GpParams& p, int* status,
                     int ctas, size_t smem, cudaStream_t stream) {
  cudaFuncSetAttribute(gemm_pair_kernel<EPI, TO, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(GP_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CG;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = qd_pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&cfg, gemm_pair_kernel<EPI, TO, CG>, map_w, map_x, bias, (TO*)out, p, status);
  return qd_last_error();
}

// epi 0: out [T, N] = X W^T (+ bias float32 [N]), bfloat16 or float32, rows ``ldo`` apart; 1: out float32 [splits, T, N], the sums of
// ``splits`` shares of K; 2 (+ 256 * QD_ACT_*): W [2F, K] the gate's rows, then up's, out bfloat16 [T, F] = act(X Wg^T) * (X Wu^T).
// X rows ``ldx`` apart; K and ldx multiples of 8, W and X 16-byte aligned.  ``cg``: multiprocessors to a tile, 1 (up to 128 tokens
// a tile) or 2 (up to 256); ``bn``: rows of W to a tile, a multiple of 32 up to 256.
extern "C" int qd_gemm_pair(const void* W, const void* X, long long ldx, const float* bias, void* out, int out_dtype,
                            long long ldo, int T, int N, int K, int cg, int bn, int splits, int epi, int sms, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return 0;
  const int act = epi >> 8;
  epi &= 255;
  if (K <= 0 || K % 8 || ldx % 8 || ldx < K || (cg != 1 && cg != 2) || bn < 32 || bn > 256 || bn % 32 || splits < 1 || sms < 2)
    return QD_ERR_UNSUPPORTED;
  if (((uintptr_t)W & 15) || ((uintptr_t)X & 15) || !out) return QD_ERR_UNSUPPORTED;
  if (epi == GP_GATED && ((N & 1) || out_dtype != QD_BF16)) return QD_ERR_UNSUPPORTED;
  if ((epi == GP_PARTIAL && (out_dtype != QD_F32 || bias)) || (epi != GP_PARTIAL && splits != 1)) return QD_ERR_UNSUPPORTED;
  GpParams p;
  p.act = act; p.T = T; p.N = N; p.K = K; p.bn = bn; p.splits = splits; p.ldo = ldo;
  p.kb_total = up(K, GP_BK);
  if (splits > p.kb_total || (long long)p.kb_total * splits > (1ll << 30)) return QD_ERR_UNSUPPORTED;
  p.feats = epi == GP_GATED ? N / 2 : N;
  p.n_tt = up(T, 128 * cg);
  p.mrows = up(up(T, cg * p.n_tt), 8) * 8;           // the tokens evenly over the token tiles and their CTAs
  p.n_ft = up(p.feats, epi == GP_GATED ? bn / 2 : bn);
  const long long items = (long long)p.n_ft * p.n_tt * splits;
  if (items > (1ll << 30)) return QD_ERR_UNSUPPORTED;
  const int workers = (int)(items < sms / cg ? items : sms / cg);
  const int stage_bytes = (p.mrows + bn / cg) * 128;
  p.stages = GP_SMEM / stage_bytes;
  if (p.stages > GP_MAX_STAGES) p.stages = GP_MAX_STAGES;
  p.acc_stride = bn <= 32 ? 32 : bn <= 64 ? 64 : bn <= 128 ? 128 : 256;
  p.tmem_cols = items > workers ? 2 * p.acc_stride : p.acc_stride;
  p.vec = !((uintptr_t)out & 15) && (epi == GP_PARTIAL ? N : ldo) % (out_dtype == QD_F32 ? 4 : 8) == 0;
  // An MMA reads 128 rows of the last stage's tokens.  With fewer there are more stages, and the weights' stages behind them
  // hold at least 12 x 16 rows.
  const size_t smem = (size_t)p.stages * stage_bytes + GP_EPI_WARPS * GP_STAGE_ROWS + 1024;
  int* status = status_word();
  CUtensorMap map_w, map_x;
  const int box = epi == GP_GATED || cg == 2 ? bn / 2 : bn;
  if (!status || !tc_make_map(&map_w, W, true, N, K, box) || !tc_make_map(&map_x, X, true, T, K, p.mrows, ldx))
    return QD_ERR_UNSUPPORTED;
#define GO(E, TO)                                                                                                      \
  return cg == 2 ? gp_launch<E, TO, 2>(map_w, map_x, bias, out, p, status, 2 * workers, smem, stream)                   \
                 : gp_launch<E, TO, 1>(map_w, map_x, bias, out, p, status, workers, smem, stream)
  if (epi == GP_GATED) GO(GP_GATED, bf16);
  if (epi == GP_PARTIAL) GO(GP_PARTIAL, float);
  if (epi == GP_STORE && out_dtype == QD_BF16) GO(GP_STORE, bf16);
  if (epi == GP_STORE && out_dtype == QD_F32) GO(GP_STORE, float);
#undef GO
  return QD_ERR_UNSUPPORTED;
}

// 0 if no bounded wait of this library's kernel has run out on the current device (1: producer, for a free stage; 2: MMAs, for
// data; 3: MMAs, for a drained accumulator; 4: epilogue).  Synchronises the device.
QD_DEFINE_WAIT_PROBE(qd_gemm_pair_wait_probe, tc_wait(bar, 0, dead, 0, poll_limit), status_word, 99)

extern "C" int qd_gemm_pair_status() {
  int* status = status_word();
  if (!status) return -1;
  int v = 0;
  if (cudaMemcpy(&v, status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  if (v) cudaMemset(status, 0, sizeof(int));
  return v;
}
