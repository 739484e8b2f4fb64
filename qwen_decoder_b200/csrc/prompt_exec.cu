// The layers of a prompt step launched from native code.
//
// A step with a prompt portion is no replayed graph: its kernels are launched one by one, about nine
// per layer, and from Python each launch costs some 15 us of interpreter, argument conversion and
// tensor bookkeeping -- more than the device needs for portions of a few hundred tokens.  For a model
// whose layers are all the common composition (pre-norm block, grouped-query attention with one
// rotary table, SwiGLU, RMSNorm; bfloat16) this file runs the same kernels, in the same order, with
// the same arguments as the parts do, from one C++ loop:
//
//   per layer:  h = rmsnorm(x += delta) ; qkv = h Wqkv^T ; bias, rotation, cache write ; attention over
//               the pages (the decode kernel for the single tokens of a mixed step, a prompt kernel for the
//               rest) ; delta = attn Wo^T ; h = rmsnorm(x += delta) ; gu = h Wgu^T ; act = silu(gate) * up (one kernel
//               where gemm_pair.cu takes it) ; delta = act Wd^T
//   at the end: hrows = rmsnorm(x += delta) at the wanted rows          (the output projection stays outside)
//
// It holds no kernel of its own.  The launchers live in the other libraries of this directory and the matrix
// products that gemm_pair.cu does not take in cuBLAS (as the reference's do, gpu_kernels.cu:431-436); the caller hands over their
// addresses, so this library links against none of them and uses whatever cuBLAS the process has loaded.
// The reference launches its layers from C++ as well (gpu_decoder.cu:321-497).
#include "common.cuh"
#include "entry_points.h"
#include <cublas_v2.h>

struct PeLayer {
  const float* norm1_w; const float* norm2_w;
  const void* wqkv; const float* bqkv; const void* wo; const void* wgu; const void* wd;
  void* kv;                        // this layer's pages [pages, 2, G, page_size, d]
  float eps1, eps2;
  int write_kv, pad;
};

// cublasGemmEx (the 32-bit form; the header overloads the name for C++)
typedef cublasStatus_t (*PeGemmEx)(cublasHandle_t, cublasOperation_t, cublasOperation_t, int, int, int, const void*,
                                   const void*, cudaDataType, int, const void*, cudaDataType, int, const void*, void*,
                                   cudaDataType, int, cublasComputeType_t, cublasGemmAlgo_t);

// cublasGemmStridedBatchedEx (32-bit form)
typedef cublasStatus_t (*PeGemmBatched)(cublasHandle_t, cublasOperation_t, cublasOperation_t, int, int, int, const void*,
                                        const void*, cudaDataType, int, long long, const void*, cudaDataType, int,
                                        long long, const void*, void*, cudaDataType, int, long long, int,
                                        cublasComputeType_t, cublasGemmAlgo_t);

struct PeFns {
  decltype(&qd_add_rmsnorm) add_rmsnorm;
  decltype(&qd_rope_kv_write_biased) rope_kv_write;
  decltype(&qd_swiglu) swiglu;
  decltype(&qd_prefill_attention) attention_regs;       // mma.sync, any supported head size
  decltype(&qd_prefill_attention_tc5) attention_tc5;    // tcgen05, head size 64 or 128
  decltype(&qd_decode_attention) attention_decode;      // split-KV, for the single tokens of a mixed step
  decltype(&qd_decode_attention_tma) attention_decode_tma;      // the same by TMA copies, the same bits (null: not at this head size)
  PeGemmEx gemm_ex;
  cublasHandle_t blas;             // the caller's handle, bound to ``stream``
  PeGemmBatched gemm_batched;
  decltype(&qd_elementwise_plain_next) plain_next;      // the elementwise library's next launch without the attribute
  decltype(&qd_gemm_pair) gemm_pair;                    // products on pairs of multiprocessors, where a plan below says so
  decltype(&qd_decode_shares) decode_shares;            // the list of shares by length of a mixed step's single tokens
  decltype(&qd_decode_attention_shares) attention_shares;       // the single tokens' attention with shares by length
};

// How a product is cut (``qd_gemm_pair_plan``); cg 0: the library's product
struct PePlan { int cg, bn, splits; };

struct PeParams {
  PeFns fn;
  const PeLayer* layers; int n_layers;
  int T, R, D, H, G, d, F, page_size, window, rotary_dim, pairing, max_blocks, use_tc5, n_wanted;
  float scale, final_eps;
  long long n_pages;
  const int* positions; const int* slot_map; const int* block_table; const int* cu_tokens; const int* start_pos;
  const int* logit_rows;
  const float* cos_t; const float* sin_t; const float* final_w;
  float* x;                        // [T, D] residual sum, float32
  const void* delta0;              // null: nothing pending on entry
  void* h; void* qkv; void* attn; void* delta; void* gu; void* act;   // bfloat16 scratch: [T,D] [T,(H+2G)d] [T,Hd] [T,D] [T,2F] [T,F]
  void* hrows;                     // [n_wanted, D] bfloat16
  // a mixed step: requests and tokens 0 .. n_decode-1 are single tokens and go to the decode kernel
  int n_decode, decode_splits;
  const int* token_req; float* part_o; float* part_ml; unsigned* tickets;
  // the down projection over ``down_shares`` equal shares of F as one batched product that leaves float32 partial
  // sums [down_shares, T, D] in ``down_part`` for the next norm's kernel (0: the plain product into ``delta``).
  // With few tokens, a long K and few output features the plain product fills the GPU with too few CTAs.
  float* down_part; int down_shares, pad2;
  // the output projection, gate and up with the activation, the down projection; their partial sums go to ``o_part`` [splits, T, D]
  // and ``down_part``
  PePlan wo_plan, wgu_plan, wd_plan;
  int sms;
  float* o_part;
  // the single tokens' shares of decode attention (null: ``decode_splits`` for each); ``part_o`` and ``part_ml`` are theirs then
  void* shares;
  int n_shares, scratch_row;
};

extern "C" int qd_prompt_exec_struct_sizes(int* layer_bytes, int* params_bytes) {
  *layer_bytes = (int)sizeof(PeLayer);
  *params_bytes = (int)sizeof(PeParams);
  return 0;
}

// Y[T, N] = X[T, K] W[N, K]^T, all bfloat16 row-major, float32 accumulation
static int product(const PeParams& p, const void* W, const void* X, void* Y, int T, int N, int K) {
  const float one = 1.f, zero = 0.f;
  cublasStatus_t st = p.fn.gemm_ex(p.fn.blas, CUBLAS_OP_T, CUBLAS_OP_N, N, T, K, &one, W, CUDA_R_16BF, K, X, CUDA_R_16BF,
                                   K, &zero, Y, CUDA_R_16BF, N, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT);
  return st == CUBLAS_STATUS_SUCCESS ? 0 : 20000 + (int)st;
}

// part[s][T, N] = X[T, share s of K] W[N, share s of K]^T in float32, for `shares` equal shares of K
static int product_shares(const PeParams& p, const void* W, const void* X, float* part, int T, int N, int K, int shares) {
  const float one = 1.f, zero = 0.f;
  const int kc = K / shares;
  cublasStatus_t st = p.fn.gemm_batched(p.fn.blas, CUBLAS_OP_T, CUBLAS_OP_N, N, T, kc, &one, W, CUDA_R_16BF, K, kc, X,
                                        CUDA_R_16BF, K, kc, &zero, part, CUDA_R_32F, N, (long long)T * N, shares,
                                        CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT);
  return st == CUBLAS_STATUS_SUCCESS ? 0 : 20000 + (int)st;
}

// The same into ``Y`` or, in shares, into ``part``; what was left: the tensor, its dtype and its parts.
static int product_for_norm(const PeParams& p, const PePlan& plan, const void* W, const void* X, void* Y, float* part, int T, int N,
                            int K, const void** left, int* dtype, int* parts, cudaStream_t stream) {
  *left = Y; *dtype = QD_BF16; *parts = 1;
  if (!plan.cg) return product(p, W, X, Y, T, N, K);
  if (plan.splits == 1) return p.fn.gemm_pair(W, X, K, nullptr, Y, QD_BF16, N, T, N, K, plan.cg, plan.bn, 1, 0, p.sms, stream);
  *left = part; *dtype = QD_F32; *parts = plan.splits;
  return p.fn.gemm_pair(W, X, K, nullptr, part, QD_F32, N, T, N, K, plan.cg, plan.bn, plan.splits, 1, p.sms, stream);
}

#define PE_TRY(call)            \
  do {                          \
    int rc_ = (call);           \
    if (rc_ != 0) return rc_;   \
  } while (0)

extern "C" int qd_prompt_exec(const PeParams* pp, cudaStream_t stream) {
  const PeParams& p = *pp;
  if (p.T <= 0 || p.n_layers < 0 || p.n_decode < 0 || p.n_decode >= p.R) return QD_ERR_UNSUPPORTED;
  const int shares = p.down_shares;
  if (shares < 0 || shares == 1 ||
      (shares > 1 && (!p.down_part || !p.fn.gemm_batched || !p.fn.plain_next || p.F % (8 * shares))))
    return QD_ERR_UNSUPPORTED;
  if (p.shares && (!p.fn.attention_shares || !p.fn.decode_shares)) return QD_ERR_UNSUPPORTED;
  if ((p.wo_plan.cg || p.wgu_plan.cg || p.wd_plan.cg) && !p.fn.gemm_pair) return QD_ERR_UNSUPPORTED;
  if ((p.wo_plan.cg && p.wo_plan.splits > 1 && !p.o_part) || (p.wd_plan.cg && p.wd_plan.splits > 1 && !p.down_part)) return QD_ERR_UNSUPPORTED;
  const int T = p.T, D = p.D, H = p.H, G = p.G, d = p.d, F = p.F;
  const int n_qkv = (H + 2 * G) * d;
  const long long xn = (long long)T * D;
  const void* delta = p.delta0;
  int delta_dtype = QD_BF16, delta_parts = 1;          // what the previous layer's down projection left
  const void* o;
  int o_dtype, o_parts;
  for (int l = 0; l < p.n_layers; l++) {
    const PeLayer& L = p.layers[l];
    if (shares > 1 && delta_parts > 1) p.fn.plain_next();     // the norm that reads the batched product waits for all of it
    PE_TRY(p.fn.add_rmsnorm(p.x, delta, delta ? delta_dtype : -1, L.norm1_w, p.h, QD_BF16, nullptr, T, D, L.eps1, 1,
                            delta_parts, xn, stream));
    PE_TRY(product(p, L.wqkv, p.h, p.qkv, T, n_qkv, D));
    PE_TRY(p.fn.rope_kv_write(p.qkv, L.bqkv, T, H, G, d, p.rotary_dim, p.pairing, p.cos_t, p.sin_t, p.positions, L.kv,
                              p.slot_map, p.page_size, L.write_kv, stream));
    const int nd = p.n_decode;
    if (nd > 0 && p.shares && l == 0) PE_TRY(p.fn.decode_shares(p.positions, p.slot_map, p.scratch_row, nd, p.n_shares, p.shares, stream));
    if (nd > 0 && p.shares)
      PE_TRY(p.fn.attention_shares(p.qkv, n_qkv, p.attn, L.kv, p.n_pages, p.block_table, p.max_blocks, nd, H, G, d, p.page_size,
                                   p.scale, p.shares, p.n_shares, l == 0, p.part_o, p.part_ml, p.tickets, stream));
    else if (nd > 0 && p.fn.attention_decode_tma && (p.decode_splits == 1 || p.tickets))
      PE_TRY(p.fn.attention_decode_tma(p.qkv, n_qkv, p.attn, L.kv, p.n_pages, p.block_table, p.max_blocks, p.token_req,
                                       p.positions, nd, H, G, d, p.page_size, p.scale, p.window, p.decode_splits, p.part_o,
                                       p.part_ml, p.tickets, stream));
    else if (nd > 0)
      PE_TRY(p.fn.attention_decode(p.qkv, n_qkv, p.attn, L.kv, p.block_table, p.max_blocks, p.token_req, p.positions,
                                   nd, H, G, d, p.page_size, p.scale, p.window, p.decode_splits, p.part_o, p.part_ml,
                                   p.tickets, stream));
    const int* bt = p.block_table + (size_t)nd * p.max_blocks;
    if (p.use_tc5)
      PE_TRY(p.fn.attention_tc5(p.qkv, n_qkv, p.attn, L.kv, p.n_pages, bt, p.max_blocks, p.cu_tokens + nd,
                                p.start_pos + nd, p.R - nd, T - nd, H, G, d, p.page_size, p.scale, p.window, nullptr,
                                stream));
    else
      PE_TRY(p.fn.attention_regs(p.qkv, n_qkv, p.attn, L.kv, bt, p.max_blocks, p.cu_tokens + nd, p.start_pos + nd,
                                 p.R - nd, T - nd, H, G, d, p.page_size, p.scale, p.window, stream));
    PE_TRY(product_for_norm(p, p.wo_plan, L.wo, p.attn, p.delta, p.o_part, T, D, H * d, &o, &o_dtype, &o_parts, stream));
    PE_TRY(p.fn.add_rmsnorm(p.x, o, o_dtype, L.norm2_w, p.h, QD_BF16, nullptr, T, D, L.eps2, 1, o_parts, xn, stream));
    if (p.wgu_plan.cg) {
      PE_TRY(p.fn.gemm_pair(L.wgu, p.h, D, nullptr, p.act, QD_BF16, F, T, 2 * F, D, p.wgu_plan.cg, p.wgu_plan.bn, 1, 2, p.sms, stream));
    } else {
      PE_TRY(product(p, L.wgu, p.h, p.gu, T, 2 * F, D));
      PE_TRY(p.fn.swiglu(p.gu, p.act, QD_BF16, T, F, stream));
    }
    if (shares > 1) {
      PE_TRY(product_shares(p, L.wd, p.act, p.down_part, T, D, F, shares));
      delta = p.down_part; delta_dtype = QD_F32; delta_parts = shares;
    } else {
      PE_TRY(product_for_norm(p, p.wd_plan, L.wd, p.act, p.delta, p.down_part, T, D, F, &delta, &delta_dtype, &delta_parts, stream));
    }
  }
  if (p.n_wanted > 0 && shares > 1 && delta_parts > 1) p.fn.plain_next();
  if (p.n_wanted > 0)
    PE_TRY(p.fn.add_rmsnorm(p.x, delta, delta ? delta_dtype : -1, p.final_w, p.hrows, QD_BF16, p.logit_rows, p.n_wanted,
                            D, p.final_eps, 0, delta_parts, xn, stream));     // only the wanted rows: x itself stays as it is
  return 0;
}
