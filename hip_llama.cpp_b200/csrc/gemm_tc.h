// Host-side interface of the tcgen05 weight matmul (gemm_tc.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tha {

struct TcArgs {
  int n_mats;                 // 1..3 stacked weight matrices with the same K
  const float* W[3]; int M[3]; int out_off[3];   // rows of matrix i land at out[n*ldo + out_off[i] + row]
  int K;
  const float* Xhi; const float* Xlo; int N; long long ldx;   // activations [N, ldx] split: hi = tf32(x), lo = x - hi
  float* out; long long ldo; long long zstride;  // split z writes out + z*zstride (partials, summed by the consumer)
  int splits;                 // split-K factor (>= 1); must divide the k-blocks into exactly `splits` non-empty parts
  const float* colscale;      // nullable [N]: out *= colscale[n]  (the 1/rms factor of a folded RMSNorm)
};

struct TcP {                  // kernel parameter block
  int M[3]; int tiles[3]; int out_off[3];
  int K, N, ny, kblocks_total, kblocks_per_split;   // ny = column tiles
  float* out; long long ldo; long long zstride;
  const float* colscale;
  int* error_flag;
  int splits, n_items;          // work items = (tiles of all matrices) x column tiles x splits, walked by persistent CTAs
  long long* trace;           // development aid (tha_gemm_trace)
};

// fp32 weights x activations split into fp16 hi and lo (gemm_f16x3.cu)
struct X3Args {
  int n_mats; const float* W[3]; int M[3]; int out_off[3];
  int K;
  const uint16_t* Xhi; const uint16_t* Xlo; int N;             // planes [N, K]
  const float* colscale;                                       // [N], 16-byte aligned: what a product with row n is multiplied by
  float* out; long long ldo; long long zstride; int splits;
};
bool gemm_f16x3_width_ok(int K);
int gemm_f16x3_splits(int tiles256, int rows_out, int K, int N);   // tiles256: 256-row weight tiles of all matrices, rows_out: their rows
int gemm_f16x3_launch(cudaStream_t st, const X3Args& a, bool pdl);
struct X3RowsP {                                               // rows -> planes
  float* x; long long ld;                                      // rows to be split [rows, ld] (the norm: ld = n); SwiGLU: ld of the partials
  const float* part; int nz; long long zstride;
  const float* emb; const int* token; const int* pos; const float* gain;
  int n;                                                       // values a row
  uint16_t *hi, *lo; float* scale;
};
int x3_norm_launch(cudaStream_t st, bool pdl, int rows, const X3RowsP& p);
int x3_swiglu_launch(cudaStream_t st, bool pdl, int rows, const X3RowsP& p);
int x3_split_launch(cudaStream_t st, bool pdl, int rows, const X3RowsP& p);

// What the attention of such prompts reads (attn_prefill_x3.cu): q [rows][dim], k / v [rows staged][kv_dim] as planes, inverse scales [rows][heads] and
// [kv head][rows staged].  row: the staged row of every row; pad: staged rows behind it that are zeroed in v (non-zero for a sequence's last row only).
struct X3Staged { uint16_t *qh, *ql, *kh, *kl, *vh, *vl; float *qs, *ks, *vs; const int *row, *pad; int rows; };

// Q8_0 weights x Q8_0 activations on the int8 tensor cores (gemm_q8i_kernel)
struct Q8iArgs {
  int n_mats; const int8_t* Wq[3]; const float* Ws[3]; int M[3]; int out_off[3];
  int K, gs;
  const int8_t* Xq; const float* xsT; int ldxs; int N;   // activations int8 [N, K]; scales transposed [K/gs, ldxs]
  float* out; long long ldo; long long zstride; int splits;   // split over 128-value slots
};
bool gemm_q8i_ok(const Q8iArgs& a);
int gemm_q8i_pick_nt(int N, int gs);
int gemm_q8i_launch(cudaStream_t st, const Q8iArgs& a, bool pdl);

// What the kernel that rotates prompt rows leaves for the tensor-core attention besides the cache: q [rows][dim], k / v
// [staged row][kv_dim] in bf16; row: the staged row of every row; pad: staged rows behind it that are zeroed in v (non-zero
// for a sequence's last row only).  All null: none of it.
struct RopeBf16 { uint16_t *q, *k, *v; const int *row, *pad; };

// bf16 weights x bf16 activations (gemm_bf16.cu): both operands straight from TMA-written shared memory
constexpr int BF_MAX_MATS = 8;
struct BfArgs {
  int n_mats; const uint16_t* W[3]; int M[BF_MAX_MATS]; int out_off[BF_MAX_MATS];
  int K;
  const uint16_t* X; int N; long long ldx;       // activations [N, ldx] bf16
  float* out; long long ldo; long long zstride; int splits;
  const float* colscale;
  // A feed-forward's activation in the read-out (prompt-sized N, no split-K); its result, rounded to bf16, goes to act_out[n * ld_act + row]
  // (the input of the down product) and `out` is not written at all.  ff_act 0: SwiGLU of the llama block, silu(w1 x) * (w3 x); else
  // 1 + THA_ACT_* of a layer program.  Gated ones (SwiGLU too) take two matrices of equal height, w1 = gate and w3 = up: a work item
  // multiplies 128 rows of the one AND the same 128 rows of the other.  Ungated ones take one matrix.
  uint16_t* act_out; long long ld_act;
  int ff_act; float act_limit, act_alpha;
  // stacked: up to BF_MAX_MATS matrices that are row ranges of ONE matrix W[0], each with activation rows of its own: matrix i =
  // rows w_row[i] .. + M[i] of W[0], its activations rows x_row[i] .. + N of X
  int stacked; int w_row[BF_MAX_MATS]; int x_row[BF_MAX_MATS];
};
bool gemm_bf16_act_ok(const BfArgs& a);   // the launch can take the activation into its read-out, and that is the faster way
bool gemm_bf16_ok(const BfArgs& a);
struct BfTile { int nt, mt; };
BfTile gemm_bf16_tile(int tiles, int N, int splits);   // output tile: 128 mt weight rows (of `tiles` 128-row tiles) x nt activation rows; K in `splits` shares
int gemm_bf16_launch(cudaStream_t st, const BfArgs& a, bool pdl);

bool gemm_tc_ok(const TcArgs& a);
int gemm_tc_pick_nt(int N);
int gemm_tc_launch(cudaStream_t st, const TcArgs& a, bool pdl);
int gemm_tc_check_error();
int gemm_tc_init(int** flag_out);   // allocate the per-device error flag (outside any stream capture)
void gemm_tc_forget();

}  // namespace tha
