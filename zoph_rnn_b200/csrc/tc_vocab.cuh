// The vocabulary projection for few batch columns (a beam step, a short sentence): a stream of the weights past a handful of
// columns.  See tc_vocab.cu; for more columns launch_tc_gemm_persistent (tc_gemm.cuh).
#pragma once
#include "tc_gemm.cuh"

namespace zrnn {

constexpr int kVocabMaxCols = 144;
// Beyond 128 columns the split modes have room for one accumulator only, so a tile's epilogue is not hidden.  Against the kernel of
// many columns, which fetches the weights twice, that pays for one more group of 16 columns and from K = 768 on (kb k-blocks of 128
// bytes).  us per beam step of a 2-layer model, here / there, at 144, 152 and 168 columns:
//   fp16 split, K = 1000, 50000 words 173 / 178, 185 / 181, 189 / 182;  K = 768, 50000 words 143 / 146, 157 / 147, 159 / 147
//   3xTF32,     K = 1000, 50000 words 278 / 297, 288 / 301, 303 / 304;  K = 640, 40000 words 191 / 190, 203 / 191, 213 / 192
// (252 columns, K = 1000: 220 / 192 and 342 / 316.)
inline int vocab_max_cols(int mode, int kb) { return (mode == TC_F16X2 && kb >= 12) || (mode == TC_TF32X3 && kb >= 24) ? 144 : 128; }

// z[v, m] = W[v] . h[m] + bias[v] for v < N, m < M
struct VocabParams {
  CUtensorMap w;       // make_rows_map: 128 weight rows, all parts, kbs k-blocks
  CUtensorMap h;       // make_rows_map: nb rows, all parts, kbs k-blocks
  int M, N, nb;        // columns, vocabulary rows, columns rounded up to a multiple of 16
  int kb, kbs;         // k-blocks, k-blocks per ring stage: vocab_kbs(mode)
  const float* bias;
  float* C;            // STORE: z[v, m] at C + m * ldc + v
  long long ldc;
  const int* target;   // LSE: z[target[m] - target_offset, m] goes to tgt_logit[m]
  int target_offset;
  float* tgt_logit;
  float* part_max;     // per part_rows vocabulary rows and column: maximum of z and (part_sum, optional) sum exp(z - max)
  float* part_sum;     //   [n_parts x M]
  int part_rows;       // 64 or 128
  int n_parts;         // parts beyond the vocabulary are left as (-inf, 0)
  int* err;
};
inline int vocab_columns(int M) { return (M + 15) / 16 * 16; }
inline int vocab_kbs(int mode) { return mode == TC_TF32X3 || mode == TC_F16X2 ? 1 : 2; }
cudaError_t launch_tc_vocab(const VocabParams& p, int mode, int epi, cudaStream_t st);

}  // namespace zrnn
