// The vocabulary projection.  Few batch columns (a beam step of a sentence or two): a stream of the weights past a handful of columns,
// tc_vocab.cu.  More columns: pairs of CTAs, tc_vocab_pair.cu.
#pragma once
#include "tc_gemm.cuh"

namespace zrnn {

// Up to here a CTA of the few-columns kernel fits half an SM and asks for its first weights while the kernel before it runs; beyond, pairs
// of CTAs are faster.  us, few columns / pairs, fp16 split, K = 1000, 50000 words: 64 columns 43.5 / 40.2 (14.0 / 14.8 at K = 512,
// 20000 words; without the overlap, which a beam step has), 96 columns 45.7 / 42.3 (20.6 / 17.9), 128 columns 49.7 / 44.0 (25.2 / 16.8);
// bf16, 128 columns 37.3 / 25.3.
constexpr int kVocabFewCols = 64;

// z[v, m] = W[v] . h[m] + bias[v] for v < N, m < M
struct VocabParams {
  CUtensorMap w;       // make_rows_map: 128 weight rows, all parts, kbs k-blocks
  CUtensorMap h;       // make_rows_map: nb rows, all parts, kbs k-blocks
  int M, N, nb;        // columns, vocabulary rows, columns rounded up to a multiple of 16 (pairs: columns of a tile, a multiple of 32)
  int n_ct;            // pairs: column tiles
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

// Pairs of CTAs: n_ct column tiles of nb columns; the box of h has nb / 2 rows.
struct VocabTiles {
  int n_ct, nb;
};
VocabTiles vocab_pair_tiles(int M, int N);
// short products (k-blocks times products per k-step): their log-sum-exp always runs in tiles of one CTA, which read no padding of the rows
inline bool vocab_short(int mode, int kb) { return kb * (mode == TC_TF32X3 || mode == TC_F16X2 ? 3 : 1) <= 16; }
// the log-sum-exp of M columns (more than kVocabFewCols) over N words takes less time in tiles of one CTA (launch_tc_gemm_persistent)
bool vocab_lse_single(int mode, int kb, int M, int N);
cudaError_t launch_tc_vocab_pair(const VocabParams& p, int mode, int epi, cudaStream_t st);

}  // namespace zrnn
