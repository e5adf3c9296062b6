// Matrix products with few batch columns (beam decoding of a sentence or two, scoring of small minibatches): every weight
// is used for a handful of columns, so a launch is a stream of the weights through the SMs with a short latency, and
// what costs is the fixed part of a launch.  See skinny_gemm.cu.
#pragma once
#include <cuda_runtime.h>

namespace zrnn {

enum { SK_BF16 = 0, SK_F16X2 = 1 };  // operand arithmetic, as TC_BF16 / TC_F16X2
enum { SK_EPI_STORE = 0, SK_EPI_LSTM = 1 };

// acc[row, col] = sum over sources s, k: w[row, koff_s + k] * act_s[col, k]
struct SkinnyParams {
  // weights as packed for the tensor-core kernels: packed 128-row tiles, K in blocks of 64 elements (128 bytes); element
  // (tile t, row r, k-block b) starts at t * w_tile_bytes + r * w_row_bytes + b * w_kb_bytes
  const void* w_hi;
  const void* w_lo;  // SK_F16X2: the scaled lo parts
  long long w_tile_bytes;
  int w_row_bytes, w_kb_bytes;
  int nsrc;
  int n_early;          // leading sources that were complete when the predecessor kernel passed its own wait
  const void* a_hi[3];  // [cols][lda] operand rows
  const void* a_lo[3];
  int a_kb0[3];         // first k-block of the source inside the weights' K axis
  int lda;
  int K;  // valid elements per source (a multiple of 4)
  int M;  // batch columns
  int N;  // STORE: output rows; LSTM: hidden size (tiles of 32 hidden units x 4 gates)
  const float* bias;    // STORE: [N] or null; LSTM: [4][N]
  const int* mask;      // [M] or null
  int act, act_rows;    // STORE: tanh for rows < act_rows (0 = all) when act == 1
  float* C;             // fp32 out, column m at C + m * ldc (may be null for LSTM)
  int ldc;
  void* op_hi;          // optional operand-form copy (row m at + m * ld_op): bf16, or fp16 hi + scaled fp16 lo
  void* op_lo;
  int ld_op;
  const float* c_prev;  // LSTM
  float* c_out;
};
struct SkinnyBatch {
  enum { MAX = 8 };
  SkinnyParams p[MAX];
};
// about how long launch_skinny takes for n problems of `rows` weight rows x K elements (all sources) and `cols` columns, on the scale of
// plan_chain's estimate; early: some sources are early and no other stream's launches run beside
float skinny_us(int mode, int epi, int rows, int K, int cols, int n, bool early);
// the fp16 split takes this kernel up to here in any case, because its accumulators absorb fewer products (skinny_gemm.cu)
bool skinny_more_exact(int epi, int rows, int cells, int nsrc, int H, int n_early, int cols);
// n independent problems of the same shape class (mode, epilogue, N, K, M) in one launch
cudaError_t launch_skinny(const SkinnyBatch& b, int n, int mode, int epi, cudaStream_t st);

}  // namespace zrnn
