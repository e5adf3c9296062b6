// Tensor-core products on the chain between two time steps: LSTM cells, the attention layer's projections and the tanh
// combiner.  One launch is one link of a chain of dependent launches, so what counts is its latency.  See tc_link.cu (tiles of up
// to 64 weight rows) and tc_chain.cu (wider ones).
#pragma once
#include "tc_gemm.cuh"

namespace zrnn {

// acc[M x N] = sum_s A_s[M x K] * W[N x Kcat]^T, both operands K-major; M: batch columns, N: weight rows
struct ChainParams {
  CUtensorMap a[3];           // activation rows: make_rows_map with a_rows rows, all parts, kbs k-blocks
  CUtensorMap w;              // STORE: make_rows_map with BN rows; LSTM: make_gate_map with BN / 4 units
  int w_first;                // LSTM: the weights' lines leave the L2 first (tiles of 128 rows; the other kernels do not look at it)
  int w_kbtot, w_tiles;       // LSTM: k-blocks per packed tile, packed tiles
  int nsrc, kb;               // sources, k-blocks per source
  int n_early;                // leading sources that were complete when the predecessor kernel passed its own wait
  int kbs;                    // k-blocks per box: chain_kbs
  int wkb0[3];                // first k-block of each source on the weights' K axis
  int a_row0[3];              // first row of each source's map that belongs to this problem
  int a_rows;                 // rows per activation box: a multiple of 8, at most 128
  int M, N;                   // N: STORE output rows; LSTM hidden size
  const float* bias;          // STORE [N] or null; LSTM [4][N] gate-major (i,f,g,o)
  const int* mask;            // [M] or null
  float* C;                   // fp32 out, row m at C + m * ldc
  int ldc;
  int act, act_rows;          // STORE: tanh for n < act_rows (0 = all) when act == 1
  __nv_bfloat16* op_b16;      // operand-form copies of the output for the next product (row m at + m * ld_op)
  float* op_hi;
  float* op_lo;
  __half* op_h_hi;
  __half* op_h_lo;
  int ld_op;
  const float* c_prev;        // LSTM
  float* c_out;
  int* err;
  long long* prof;            // developer stamps, as TcParams
  int prof_slot;
};
struct ChainBatch {
  enum { MAX = 8 };
  ChainParams p[MAX];
};
// n independent problems (same BN, mode, epilogue, N; M <= 128 each when n > 1) in one launch.
// BN: 32, 64, 128 for LSTM; 16, 32, 64, 128 for STORE.
// split == 2 (n == 1, BN <= 64) or 4 (n == 1, BN == 32, STORE, split modes): CTAs per tile, each over its part of the K axis.
// whole (BN == 32 or 64, split modes): a CTA takes an SM, not half of one.
cudaError_t launch_tc_chain(const ChainBatch& b, int n, int BN, int mode, int epi, int split, bool whole, cudaStream_t st);
cudaError_t launch_tc_link(const ChainBatch& b, int n, int BN, int mode, int epi, int split, bool whole, cudaStream_t st);
// k-blocks per ring stage and TMA box: one instruction and one hand-over for several where the ring still holds a few stages
int chain_kbs(int mode, int BN, int a_rows, int kb, int split);
int link_kbs(int mode, int BN, int a_rows, int kb, int split);
// Pairs of CTAs (tc_cell_pair.cu): a_rows = nb / 2, kbs = cell_pair_kbs; weight boxes of 128 rows (STORE) or 32 units (LSTM).
cudaError_t launch_tc_cell_pair(const ChainBatch& b, int n, int mode, int epi, cudaStream_t st);
int cell_pair_kbs(int mode);
// Tile width and K split of a launch, and about how long it takes.
struct ChainPlan {
  int BN, split;
  float us;
  bool whole;
  int nb;  // > 0: pairs of CTAs with tiles of nb columns; the other fields do not count
};
// rows: weight rows (LSTM: 4 H); cells: problems in the launch; kb: 128-byte k-blocks per source; M: columns; beside: links of other
// streams run at the same time
ChainPlan plan_chain(int mode, int epi, int rows, int cells, int nsrc, int kb, int n_early, int M, bool beside);

// K-major rows as 4-D boxes (k within a 128-byte block, row, part, k-block): box_rows rows of all parts of box_kb k-blocks.
// parts == 2: the lo rows lie part_bytes behind the hi rows.
bool make_rows_map(CUtensorMap* out, const void* base, int elem_bytes, long long row_bytes, long long rows, int parts,
                   long long part_bytes, int kblocks, int box_rows, int box_kb);
// Weights of an LSTM layer, packed in tiles of 32 hidden units x 4 gates, every (tile, 128-byte k-block) one 16 KB chunk:
// 5-D boxes (k within a block, hidden unit, gate, part, tile * k-blocks per tile + k-block)
bool make_gate_map(CUtensorMap* out, const void* base, int elem_bytes, int parts, long long part_bytes, int chunks, int box_units,
                   int box_parts, int box_kb);

}  // namespace zrnn
