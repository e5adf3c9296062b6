// Vocabulary projection for up to 64 batch columns on tcgen05, bound by the stream of the weights from HBM (f32: 4 bytes a value).
//
// The weights are the M side of the MMA (128 vocabulary rows) and the columns its N side, padded to a multiple of 16 only: with
// the columns as the M side (tc_gemm.cu) a step of 12 columns multiplied 128 padded rows, 19 us of MMAs for 160 MB of weights, and
// ran its epilogue on them.  The split modes multiply W_hi by the stacked [h_hi ; h_lo], one MMA for two products, and W_lo by
// h_hi.  An accumulator row is a vocabulary row, so a warp stores 32 consecutive logits of a column at once; maxima and sums
// over the rows are reductions across the warp that halve the number of columns per lane as they go.
//
// Persistent CTAs walk over the vocabulary, the accumulators are double-buffered in TMEM and the loads run ahead across tiles.  A CTA
// takes half an SM (113 KB, 256 TMEM columns), so that it is resident, and streams its first weights, while the kernel before it
// runs.  us per launch, with the columns as the M side -> now, f32: 12 columns x 40000 words x 1000: 48 -> 31 (HBM: 25).  Marking the
// weights to leave the L2 first changes nothing.
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "kernels.cuh"
#include "tc_chain_device.cuh"
#include "tc_vocab.cuh"

namespace zrnn {
namespace {

constexpr int kEpiWarps = 8, kHWarp = 8, kWWarp = 9, kMmaWarp = 10, kThreads = 352;
constexpr int kHalfSm = 113 * 1024, kMaxStages = 8;
struct VocabCtrl {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort;
};

// behind it, per column: maxima and sums of the four lane quadrants, target
__host__ __device__ constexpr int column_bytes(int nb) { return nb * (4 * 4 + 4 * 4 + 4); }

// eight values per lane -> the reduction over the warp of value lane >> 2: each exchange halves the values that a lane carries
template <class Op>
__device__ __forceinline__ float reduce8(const float* v, int lane, Op op) {
  float a[4], b[2], c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool up = lane & 16;
    const float mine = up ? v[4 + i] : v[i], other = up ? v[i] : v[4 + i];
    a[i] = op(mine, __shfl_xor_sync(0xffffffffu, other, 16));
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool up = lane & 8;
    const float mine = up ? a[2 + i] : a[i], other = up ? a[i] : a[2 + i];
    b[i] = op(mine, __shfl_xor_sync(0xffffffffu, other, 8));
  }
  const bool up = lane & 4;
  c = op(up ? b[1] : b[0], __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 4));
  c = op(c, __shfl_xor_sync(0xffffffffu, c, 2));
  return op(c, __shfl_xor_sync(0xffffffffu, c, 1));
}

template <int MODE, int EPI>
__global__ void __launch_bounds__(kThreads, 2) tc_vocab_kernel(const __grid_constant__ VocabParams p, int stages, int n_tiles,
                                                               int tmem_cols) {
  constexpr bool SPLIT_MODE = mode_split(MODE);
  constexpr int PARTS = SPLIT_MODE ? 2 : 1;
  extern __shared__ __align__(1024) uint8_t vocab_smem[];
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int nb = p.nb, KBS = p.kbs, hkb = nb * 128;
  const int w_bytes = PARTS * KBS * 128 * 128, h_bytes = PARTS * KBS * hkb, stage_bytes = w_bytes + h_bytes;
  uint8_t* tiles = vocab_smem;
  VocabCtrl& ct = *reinterpret_cast<VocabCtrl*>(tiles + (size_t)stages * stage_bytes);
  float* red_max = reinterpret_cast<float*>(&ct + 1);
  float* red_sum = red_max + 4 * nb;
  int* s_target = reinterpret_cast<int*>(red_sum + 4 * nb);
  const int k_its = (p.kb + KBS - 1) / KBS;
  const int acc_cols = PARTS * nb;  // columns of one accumulator buffer
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ct.full[s], 2);
      mbar_init(&ct.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ct.acc_full[b], 1);
      mbar_init(&ct.acc_empty[b], kEpiWarps);
    }
    ct.abort = (smem_u32(vocab_smem) & 1023) ? 1 : 0;  // (the swizzled tiles need the alignment that the declaration asks for)
    if (ct.abort && p.err) atomicExch(p.err, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ct.tmem_base)),
                 "r"((uint32_t)tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ct.tmem_base;
  const bool sound = __all_sync(0xffffffffu, ct.abort == 0);

  if (warp == kWWarp || warp == kHWarp) {
    // ------------------------------------------------------------ loads; the weights do not depend on the predecessor
    {
      const bool one = elect_one();
      if (warp == kHWarp) {
        pdl_wait();
        pdl_trigger();
      }
      bool ok = sound;
      int st = 0, it = 0;
      uint32_t ph = 0;
      for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
        for (int k = 0; k < k_its; ++k, ++it) {
          if (it >= stages && !mbar_wait_warp(&ct.empty[st], ph ^ 1u, &ct.abort, p.err, 1)) { ok = false; break; }
          uint8_t* dst = tiles + (size_t)st * stage_bytes;
          if (one) {
            if (warp == kWWarp) {
              mbar_expect_tx(&ct.full[st], (uint32_t)w_bytes);
              tma_load_4d(dst, &p.w, &ct.full[st], tile * 128, k * KBS);
            } else {
              mbar_expect_tx(&ct.full[st], (uint32_t)h_bytes);
              tma_load_4d(dst + w_bytes, &p.h, &ct.full[st], 0, k * KBS);
            }
          }
          __syncwarp();
          if (++st == stages) { st = 0; ph ^= 1u; }
        }
      }
      if (sound && !ok) settle_copies();
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer
    if (sound) {
      const bool one = elect_one();
      const uint32_t idesc = make_idesc(mode_fmt(MODE), (uint32_t)nb), idesc2 = make_idesc(mode_fmt(MODE), (uint32_t)(PARTS * nb));
      int st = 0, ti = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++ti) {
        const int buf = ti & 1, use = ti >> 1;
        if (!mbar_wait_warp(&ct.acc_empty[buf], (uint32_t)((use & 1) ^ 1), &ct.abort, p.err, 4)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)(buf * acc_cols);
        for (int k = 0; k < k_its; ++k) {
          if (!mbar_wait_warp(&ct.full[st], ph, &ct.abort, p.err, 2)) { ok = false; break; }
          tc_fence_after();
          const uint32_t w_addr = smem_u32(tiles + (size_t)st * stage_bytes), h_addr = w_addr + w_bytes;
          if (one) {
            for (int b = 0; b < KBS; ++b) {
              const uint64_t dw = make_smem_desc(w_addr + b * PARTS * 16384), dwl = make_smem_desc(w_addr + (b * PARTS + 1) * 16384);
              const uint64_t dh = make_smem_desc(h_addr + b * PARTS * hkb);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint32_t acc = (k > 0 || b > 0 || i > 0) ? 1u : 0u;
                umma<mode_kind_tf32(MODE)>(d, dw + 2 * i, dh + 2 * i, idesc2, acc);
                if (SPLIT_MODE) umma<mode_kind_tf32(MODE)>(d + nb, dwl + 2 * i, dh + 2 * i, idesc, 1u);
              }
            }
            umma_commit(&ct.empty[st]);
          }
          __syncwarp();
          if (++st == stages) { st = 0; ph ^= 1u; }
        }
        if (ok && one) umma_commit(&ct.acc_full[buf]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: rows 32 quad .. +31, every other group of 8 columns
    const int quad = warp & 3, half = warp >> 2;
    const bool want_max = p.part_max != nullptr, want_sum = want_max && p.part_sum != nullptr;
    pdl_wait();
    if (EPI == TC_EPI_LSE)
      for (int m = threadIdx.x; m < p.M; m += kEpiWarps * 32) s_target[m] = p.target[m] - p.target_offset;
    asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
    int ti = 0;
    bool ready = sound;
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++ti) {  // (to the end even after a wait that gave up: barriers)
      const int buf = ti & 1, use = ti >> 1, v = tile * 128 + quad * 32 + lane;
      const bool in = v < p.N;
      const float bias = in && p.bias ? __ldg(p.bias + v) : 0.f;
      ready = ready && __all_sync(0xffffffffu, mbar_wait(&ct.acc_full[buf], (uint32_t)(use & 1), &ct.abort, p.err, 3));
      tc_fence_after();
      if (ready) {
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * acc_cols);
        for (int c0 = 8 * half; c0 < p.M; c0 += 16) {
          float z[8], x[8];
          tmem_ld8(taddr + c0, z);
          if (SPLIT_MODE) tmem_ld8(taddr + nb + c0, x);
          tmem_wait_ld();
#pragma unroll
          for (int u = 0; u < 8; ++u) z[u] = (SPLIT_MODE ? fmaf(x[u], mode_cross_scale(MODE), z[u]) : z[u]) + bias;
          if constexpr (EPI == TC_EPI_STORE) {
            if (in) {
#pragma unroll
              for (int u = 0; u < 8; ++u)  // streaming: the consumer reads a few tiles of the logits once, the weights should stay in L2
                if (c0 + u < p.M) __stcs(p.C + (size_t)(c0 + u) * p.ldc + v, z[u]);
            }
          } else {
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (c0 + u < p.M && s_target[c0 + u] == v && in) p.tgt_logit[c0 + u] = z[u];
          }
          if (want_max) {
            if (!in) {
#pragma unroll
              for (int u = 0; u < 8; ++u) z[u] = -INFINITY;
            }
            const float mx = reduce8(z, lane, [](float a, float b) { return fmaxf(a, b); });
            float sm = 0.f;
            if (want_sum) {
              float e[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const float m8 = __shfl_sync(0xffffffffu, mx, u * 4);
                e[u] = m8 == -INFINITY ? 0.f : expf(z[u] - m8);
              }
              sm = reduce8(e, lane, [](float a, float b) { return a + b; });
            }
            if ((lane & 3) == 0) {
              red_max[quad * nb + c0 + (lane >> 2)] = mx;
              red_sum[quad * nb + c0 + (lane >> 2)] = sm;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ct.acc_empty[buf]);
      if (want_max) {
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
        const int per = 128 / p.part_rows, qs = 4 / per;  // parts per tile, lane quadrants per part
        for (int i = threadIdx.x; ready && i < per * p.M; i += kEpiWarps * 32) {
          const int part = i / p.M, m = i - part * p.M, at = tile * per + part;
          if (at >= p.n_parts) continue;
          float M = -INFINITY, S = 0.f;
          for (int q = part * qs; q < (part + 1) * qs; ++q) M = fmaxf(M, red_max[q * nb + m]);
          if (want_sum && M != -INFINITY)
            for (int q = part * qs; q < (part + 1) * qs; ++q) S += red_sum[q * nb + m] * expf(red_max[q * nb + m] - M);
          p.part_max[(size_t)at * p.M + m] = M;
          if (want_sum) p.part_sum[(size_t)at * p.M + m] = S;
        }
        if (tile == n_tiles - 1)  // parts of a packed tile beyond the last row
          for (int i = n_tiles * per * p.M + threadIdx.x; i < p.n_parts * p.M; i += kEpiWarps * 32) {
            p.part_max[i] = -INFINITY;
            if (want_sum) p.part_sum[i] = 0.f;
          }
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)tmem_cols) : "memory");
  }
}

const bool g_pdl_on = std::getenv("ZRNN_NO_PDL") == nullptr;

template <int MODE, int EPI>
cudaError_t launch_t(const VocabParams& p, cudaStream_t st) {
  constexpr int PARTS = mode_split(MODE) ? 2 : 1;
  const int stage = PARTS * p.kbs * (128 + p.nb) * 128;
  const int fixed = (int)sizeof(VocabCtrl) + column_bytes(p.nb);
  const int stages = std::min((kHalfSm - fixed) / stage, (int)kMaxStages);
  if (stages < 2) return cudaErrorInvalidValue;
  const size_t smem = (size_t)stages * stage + fixed;
  int tmem = 32;
  while (tmem < 2 * PARTS * p.nb) tmem *= 2;
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(tc_vocab_kernel<MODE, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHalfSm);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int n_tiles = (p.N + 127) / 128;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(std::min(n_tiles, 2 * device_sms()));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_pdl_on ? 1 : 0;
  count_launch();
  return cudaLaunchKernelEx(&cfg, tc_vocab_kernel<MODE, EPI>, p, stages, n_tiles, tmem);
}
template <int MODE>
cudaError_t launch_mode(const VocabParams& p, int epi, cudaStream_t st) {
  if (epi == TC_EPI_STORE) return launch_t<MODE, TC_EPI_STORE>(p, st);
  if (epi == TC_EPI_LSE) return launch_t<MODE, TC_EPI_LSE>(p, st);
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_tc_vocab(const VocabParams& p, int mode, int epi, cudaStream_t st) {
  if (p.M < 1 || p.M > kVocabFewCols || p.N < 1 || p.nb != vocab_columns(p.M) || p.kb < 1 || p.kbs != vocab_kbs(mode) ||
      (p.part_rows != 64 && p.part_rows != 128))
    return cudaErrorInvalidValue;
  switch (mode) {
    case TC_BF16: return launch_mode<TC_BF16>(p, epi, st);
    case TC_TF32: return launch_mode<TC_TF32>(p, epi, st);
    case TC_TF32X3: return launch_mode<TC_TF32X3>(p, epi, st);
    case TC_F16X2: return launch_mode<TC_F16X2>(p, epi, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace zrnn
