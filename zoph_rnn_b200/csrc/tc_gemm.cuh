// Blackwell tensor-core GEMM family (tcgen05.mma with TMEM accumulators, TMA-fed shared-memory ring):
//   acc[M x N] = A[M x K] * B[N x K]^T        (both operands K-major)
// M indexes batch columns (the reference's H x B activations are already "B rows of K contiguous values"),
// N indexes weight rows, so every epilogue thread owns one batch column and sees all N outputs of its row: the softmax's
// max / sum-exp and the bias are thread-local.  The recurrent cells and the attention products are in tc_chain.cuh.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace zrnn {

enum { TC_BF16 = 0, TC_TF32 = 1, TC_TF32X3 = 2, TC_F16X2 = 3 };
enum { TC_EPI_STORE = 0, TC_EPI_LSTM = 1, TC_EPI_LSE = 2 };

struct TcParams {
  CUtensorMap a;     // activations (split modes: their hi part)
  CUtensorMap a_lo;  // split modes: the lo part
  CUtensorMap b;     // weights, a row per output
  CUtensorMap b_lo;
  int kblocks;        // 128-byte k-blocks
  int M;              // batch columns
  int N;              // output rows
  const float* bias;  // [N]
  // per (N tile, m) max and sum exp(z - max) of z = acc + bias, plus the logit of target[m]
  const int* target;
  int target_offset;
  float* part_max;  // [n_tiles x M]
  float* part_sum;
  float* tgt_logit;  // [M]
  int* err;          // device error word (0 = ok); set when a bounded wait gives up
  long long* prof;   // optional: 8 globaltimer stamps per CTA (developer profiling)
  int prof_slot;     // >= 0: only CTA (0,0,0) stamps, into prof[prof_slot*8 ..] (timeline of many launches)
};

// One CTA per SM walks over the tiles, log-sum-exp epilogue.  The B tensor map must use
// 256-row boxes for TC_BF16 / TC_TF32 and 128-row boxes for the split modes.  Two epilogue warps share each output
// row of a tile, one per half of its columns, so the (max, sum) partials are indexed
// [(n_tile * kPersistentParts + half) x M] and each covers tile width / kPersistentParts consecutive columns.
constexpr int kPersistentParts = 2;
cudaError_t launch_tc_gemm_persistent(const TcParams& p, int mode, cudaStream_t st);
// One warp waits (bounded by limit_cycles SM cycles) on a barrier that never completes and reports `code` in *err.
cudaError_t launch_wait_probe(int* err, long long limit_cycles, int code, cudaStream_t st);

// Host helpers -------------------------------------------------------------------------------------------
// multiprocessors of the current device (148 where there is none to ask)
int device_sms();
// 2-D K-major tensor map: `rows` rows of `k` elements, row stride ld (elements); box = (128-byte k-block) x box_rows
// elem_bytes 2 (bf16) or 4 (fp32).  Returns false when the driver entry point is unavailable or arguments are
// not encodable (base not 16-byte aligned, ld*elem_bytes not a multiple of 16).
bool make_kmajor_map(CUtensorMap* out, const void* base, int elem_bytes, long long k, long long rows, long long ld,
                     int box_rows);

// round fp32 to the nearest value representable in tf32 (10 mantissa bits), ties away from zero on the bit pattern
inline float tf32_round_host(float x) {
  unsigned u;
  memcpy(&u, &x, 4);
  if ((u & 0x7f800000u) == 0x7f800000u) return x;
  u = (u + 0x1000u) & 0xffffe000u;
  float r;
  memcpy(&r, &u, 4);
  return r;
}

}  // namespace zrnn
