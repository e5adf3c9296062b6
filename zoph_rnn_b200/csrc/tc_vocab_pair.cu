// Vocabulary projection for more than a few batch columns, on pairs of CTAs: a pair computes 256 vocabulary rows x up to 256 columns.
//
// A product of this shape is bound by the tensor cores, if shared memory lets it: an MMA of 128 x 128 reads 8 KB of operands in the 64
// cycles that it takes, all that shared memory delivers, and the split modes' three products per k-step leave no room for the loads
// (128 x 128 x 64 in fp16 halves, measured: 968 cycles where the MMAs take 768).  Here each CTA holds 128 weight rows and half of the
// columns: an MMA of 256 x 256 takes 128 cycles and reads 8 KB in each CTA (1539 cycles for MMAs of 1536), one of 256 x 128 64 cycles
// and 6 KB (771 / 768).
//
// In the split modes the two accumulators of such a tile fill the tensor memory, so they are not double-buffered: the sixteen epilogue
// warps read a tile into registers, main accumulator first, and the next tile's hi * hi products start while the cross products
// are read; everything else of the epilogue runs beside them.  The weights are the M side (tc_vocab.cu: a warp stores 32
// consecutive logits of a column at once), the columns come in tiles of a multiple of 32, as equal as they can be.  Maxima and sums
// are taken over eight rows of a column per lane: the values change hands in shared memory, eight columns at a time (halving exchanges
// across the warp instead took 51 instructions per value and 13 us per tile, more than the MMAs).
//
// us per launch, tiles of one CTA (tc_gemm.cu) -> pairs, K = 1000, 50000 words, fp16 split, logits: 160 columns 70.9 -> 48.1, 312
// 94.4 -> 77, 512 133 -> 111, 768 191 -> 157; log-sum-exp of 6400 columns 1393 -> 1199 (1.60 PFLOP/s of products; cuBLAS in bf16
// 1.65), of 16384 columns x 200000 words, K = 2048 in bf16 within a scoring pass 9.77 -> 8.1 ms: fewer operand reads, less power.
//
// A CTA asks for all of an SM's shared memory, so that no other kernel's CTAs share its SM: the pair's TMEM allocation waits for
// nobody that could wait for it in turn.
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "kernels.cuh"
#include "tc_pair_device.cuh"
#include "tc_vocab.cuh"

namespace zrnn {
namespace {

constexpr int kEpiWarps = 16, kHWarp = 16, kWWarp = 17, kMmaWarp = 18, kThreads = 608;
constexpr int kSmem = 227 * 1024, kMaxStages = 8, kGroups = 8;  // kGroups: groups of 8 columns per epilogue warp
static_assert(fills_sm(kSmem), "both CTAs of a pair hold all of the tensor memory");
struct alignas(16) PairCtrl {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t acc_full[2], main_empty[2], cross_empty[2];
  uint32_t tmem_base;
  int abort;
};
// behind it, per column: maxima and sums of the four lane quadrants, target
__host__ __device__ constexpr int column_bytes(int nb) { return nb * (4 * 4 + 4 * 4 + 4); }
constexpr int kXposeLd = 36, kXposeBytes = kEpiWarps * 8 * kXposeLd * 4;  // 8 columns x 32 rows per epilogue warp, rows spread over the banks

template <int MODE, int EPI>
__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(2, 1, 1)
    tc_vocab_pair_kernel(const __grid_constant__ VocabParams p, int stages, int v_tiles, int bufs) {
  constexpr bool SPLIT_MODE = mode_split(MODE);
  constexpr int PARTS = SPLIT_MODE ? 2 : 1, TMEM_COLS = 512;
  extern __shared__ __align__(1024) uint8_t pair_smem[];
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int nb = p.nb, KBS = p.kbs, hkb = nb / 2 * 128;
  const int w_bytes = PARTS * KBS * 128 * 128, h_bytes = PARTS * KBS * hkb, stage_bytes = w_bytes + h_bytes;
  uint8_t* tiles = pair_smem;
  PairCtrl& ct = *reinterpret_cast<PairCtrl*>(tiles + (size_t)stages * stage_bytes);
  float* xp = reinterpret_cast<float*>(&ct + 1) + warp * (8 * kXposeLd);
  float* red_max = reinterpret_cast<float*>(&ct + 1) + kXposeBytes / 4;
  float* red_sum = red_max + 4 * nb;
  int* s_target = reinterpret_cast<int*>(red_sum + 4 * nb);
  const int k_its = (p.kb + KBS - 1) / KBS;
  const int acc_cols = PARTS * nb, n_tiles = v_tiles * p.n_ct;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ct.full[s], 2);  // (the leader's: its weight and its activation producer, for the bytes of both CTAs)
      mbar_init(&ct.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ct.acc_full[b], 1);
      mbar_init(&ct.main_empty[b], 2 * kEpiWarps);
      mbar_init(&ct.cross_empty[b], 2 * kEpiWarps);
    }
    ct.abort = (smem_u32(pair_smem) & 1023) ? 1 : 0;  // (the swizzled tiles need the alignment that the declaration asks for)
    if (ct.abort && p.err) atomicExch(p.err, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) tmem_alloc_pair(&ct.tmem_base, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the barriers of both CTAs are ready
  tc_fence_after();
  const uint32_t tmem_base = ct.tmem_base;
  const bool sound = __all_sync(0xffffffffu, ct.abort == 0);

  if (warp == kWWarp || warp == kHWarp) {
    // ------------------------------------------------------------ loads; the weights do not depend on the predecessor
    {
      const bool one = elect_one();
      if (warp == kHWarp) pdl_wait();
      bool ok = sound;
      int st = 0, it = 0;
      uint32_t ph = 0;
      for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
        const int col = tile % p.n_ct * nb, row = tile / p.n_ct * 256;
        for (int k = 0; k < k_its; ++k, ++it) {
          if (it >= stages && !mbar_wait_warp(&ct.empty[st], ph ^ 1u, &ct.abort, p.err, 1)) { ok = false; break; }
          uint8_t* dst = tiles + (size_t)st * stage_bytes;
          const uint32_t bar = cluster_map(smem_u32(&ct.full[st]), 0);
          if (one) {
            if (warp == kWWarp) {
              if (rank == 0) mbar_expect_tx(&ct.full[st], (uint32_t)(2 * w_bytes));
              tma_load_4d_pair(dst, &p.w, bar, row + rank * 128, k * KBS);
            } else {
              if (rank == 0) mbar_expect_tx(&ct.full[st], (uint32_t)(2 * h_bytes));
              tma_load_4d_pair(dst + w_bytes, &p.h, bar, col + rank * (nb / 2), k * KBS);
            }
          }
          __syncwarp();
          if (++st == stages) { st = 0; ph ^= 1u; }
        }
      }
      if (sound && !ok) settle_copies();
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer of the pair
    if (rank == 0 && sound) {
      const bool one = elect_one();
      const uint32_t idesc = make_idesc_pair(mode_fmt(MODE), (uint32_t)nb);
      int st = 0, ti = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++ti) {
        const int buf = bufs == 2 ? ti & 1 : 0, use = bufs == 2 ? ti >> 1 : ti;
        const uint32_t free_ph = (uint32_t)((use & 1) ^ 1);
        if (!mbar_wait_warp(&ct.main_empty[buf], free_ph, &ct.abort, p.err, 4)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)(buf * acc_cols);
        for (int k = 0; k < k_its; ++k) {
          if (!mbar_wait_warp(&ct.full[st], ph, &ct.abort, p.err, 2)) { ok = false; break; }
          tc_fence_after();
          const uint32_t w_addr = smem_u32(tiles + (size_t)st * stage_bytes), h_addr = w_addr + w_bytes;
          for (int b = 0; b < KBS; ++b) {
            const uint64_t dw = make_smem_desc(w_addr + b * PARTS * 16384), dwl = make_smem_desc(w_addr + (b * PARTS + 1) * 16384);
            const uint64_t dh = make_smem_desc(h_addr + b * PARTS * hkb), dhl = make_smem_desc(h_addr + (b * PARTS + 1) * hkb);
            if (one) {
#pragma unroll
              for (int i = 0; i < 4; ++i) umma_pair<mode_kind_tf32(MODE)>(d, dw + 2 * i, dh + 2 * i, idesc, (k > 0 || b > 0 || i > 0) ? 1u : 0u);
            }
            if (SPLIT_MODE) {
              if (k == 0 && b == 0) {
                if (!mbar_wait_warp(&ct.cross_empty[buf], free_ph, &ct.abort, p.err, 5)) { ok = false; break; }
                tc_fence_after();
              }
              if (one) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  umma_pair<mode_kind_tf32(MODE)>(d + nb, dwl + 2 * i, dh + 2 * i, idesc, (k > 0 || b > 0 || i > 0) ? 1u : 0u);
                  umma_pair<mode_kind_tf32(MODE)>(d + nb, dw + 2 * i, dhl + 2 * i, idesc, 1u);
                }
              }
            }
          }
          if (!ok) break;
          if (one) umma_commit_pair(&ct.empty[st]);
          __syncwarp();
          if (++st == stages) { st = 0; ph ^= 1u; }
        }
        if (ok && one) umma_commit_pair(&ct.acc_full[buf]);
      }
      if (!ok) settle_copies();
    }
  } else {
    // ------------------------------------------------------------ epilogue: rows 32 quad .. +31, every fourth group of 8 columns
    const int quad = warp & 3, cg = warp >> 2;
    const bool want_max = p.part_max != nullptr, want_sum = want_max && p.part_sum != nullptr;
    const int per = 128 / p.part_rows, qs = 4 / per;  // parts per CTA's rows, lane quadrants per part
    pdl_wait();
    int ti = 0;
    bool ready = sound;
    // the bias of this lane's row and the target of column threadIdx.x, requested a tile ahead
    auto fetch = [&](int tile, float* b, int* t) {
      if (tile >= n_tiles) return;
      const int v = (tile / p.n_ct * 2 + rank) * 128 + quad * 32 + lane, m = tile % p.n_ct * nb + threadIdx.x;
      *b = v < p.N ? (p.bias ? __ldg(p.bias + v) : 0.f) : -INFINITY;
      if (EPI == TC_EPI_LSE) *t = (int)threadIdx.x < nb && m < p.M ? p.target[m] - p.target_offset : -1;
    };
    float next_bias = 0.f;
    int next_target = -1;
    fetch(pair, &next_bias, &next_target);
    for (int tile = pair; tile < n_tiles; tile += n_pairs, ++ti) {  // (to the end even after a wait that gave up: barriers)
      const int buf = bufs == 2 ? ti & 1 : 0, use = bufs == 2 ? ti >> 1 : ti;
      const int col = tile % p.n_ct * nb, cols = min(nb, p.M - col), block = tile / p.n_ct * 2 + rank;
      const int v = block * 128 + quad * 32 + lane;
      const bool in = v < p.N;
      const float bias = next_bias;
      if (EPI == TC_EPI_LSE) {
        if ((int)threadIdx.x < nb) s_target[threadIdx.x] = next_target;
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
      }
      fetch(tile + n_pairs, &next_bias, &next_target);
      ready = ready && __all_sync(0xffffffffu, mbar_wait(&ct.acc_full[buf], (uint32_t)(use & 1), &ct.abort, p.err, 3));
      tc_fence_after();
      float z[kGroups][8];
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * acc_cols + 8 * cg);
      if (ready) {
#pragma unroll
        for (int j = 0; j < kGroups; ++j)
          if (32 * j < nb) tmem_ld8(taddr + 32 * j, z[j]);
        tmem_wait_ld();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(&ct.main_empty[buf]);
      if (SPLIT_MODE) {
        if (ready) {
#pragma unroll
          for (int j = 0; j < kGroups; j += 2) {
            if (32 * j < nb) {
              float x[2][8];
              tmem_ld8(taddr + nb + 32 * j, x[0]);
              if (32 * j + 32 < nb) tmem_ld8(taddr + nb + 32 * j + 32, x[1]);
              tmem_wait_ld();
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                z[j][u] = fmaf(x[0][u], mode_cross_scale(MODE), z[j][u]);
                if (32 * j + 32 < nb) z[j + 1][u] = fmaf(x[1][u], mode_cross_scale(MODE), z[j + 1][u]);
              }
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(&ct.cross_empty[buf]);
      }
      if (ready) {
#pragma unroll
        for (int j = 0; j < kGroups; ++j) {
          const int c0 = 32 * j + 8 * cg;
          if (c0 < cols) {
#pragma unroll
            for (int u = 0; u < 8; ++u) z[j][u] += bias;
            if constexpr (EPI == TC_EPI_STORE) {
              if (in) {  // streaming: the consumer reads a few tiles of the logits once
                float* out = p.C + (size_t)(col + c0) * p.ldc + v;
#pragma unroll
                for (int u = 0; u < 8; ++u, out += p.ldc)
                  if (c0 + u < cols) __stcs(out, z[j][u]);
              }
            }
            if (EPI == TC_EPI_LSE || want_max) {
              // the group's 32 x 8 values change hands: from a row per lane to eight rows of column c0 + lane / 4
#pragma unroll
              for (int u = 0; u < 8; ++u) xp[u * kXposeLd + lane] = z[j][u];
              __syncwarp();
              const float4 lo = *reinterpret_cast<const float4*>(xp + (lane >> 2) * kXposeLd + (lane & 3) * 8);
              const float4 hi = *reinterpret_cast<const float4*>(xp + (lane >> 2) * kXposeLd + (lane & 3) * 8 + 4);
              __syncwarp();
              const float y[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
              const int c = c0 + (lane >> 2);
              if constexpr (EPI == TC_EPI_LSE) {
                const int rel = s_target[c] - (block * 128 + quad * 32 + (lane & 3) * 8);
                if ((unsigned)rel < 8u && rel + block * 128 + quad * 32 + (lane & 3) * 8 < p.N) {  // once per column at most
                  float t = 0.f;
#pragma unroll
                  for (int u = 0; u < 8; ++u)
                    if (u == rel) t = y[u];
                  p.tgt_logit[col + c] = t;
                }
              }
              float mx = fmaxf(fmaxf(fmaxf(y[0], y[1]), fmaxf(y[2], y[3])), fmaxf(fmaxf(y[4], y[5]), fmaxf(y[6], y[7])));
              mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
              mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
              float sm = 0.f;
              if (want_sum) {
                const float ref = mx == -INFINITY ? 0.f : mx;  // (rows beyond the vocabulary: exp(-inf) = 0)
                sm = ((expf(y[0] - ref) + expf(y[1] - ref)) + (expf(y[2] - ref) + expf(y[3] - ref))) +
                     ((expf(y[4] - ref) + expf(y[5] - ref)) + (expf(y[6] - ref) + expf(y[7] - ref)));
                sm += __shfl_xor_sync(0xffffffffu, sm, 1);
                sm += __shfl_xor_sync(0xffffffffu, sm, 2);
              }
              if ((lane & 3) == 0) {
                red_max[quad * nb + c] = mx;
                red_sum[quad * nb + c] = sm;
              }
            }
          }
        }
      }
      if (want_max) {
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
        for (int i = threadIdx.x; ready && i < per * cols; i += kEpiWarps * 32) {
          const int part = i / cols, m = i - part * cols, at = block * per + part;
          if (at >= p.n_parts) continue;
          float M = -INFINITY, S = 0.f;
          for (int q = part * qs; q < (part + 1) * qs; ++q) M = fmaxf(M, red_max[q * nb + m]);
          if (want_sum && M != -INFINITY)
            for (int q = part * qs; q < (part + 1) * qs; ++q) S += red_sum[q * nb + m] * expf(red_max[q * nb + m] - M);
          p.part_max[(size_t)at * p.M + col + m] = M;
          if (want_sum) p.part_sum[(size_t)at * p.M + col + m] = S;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA ends while the other one's MMAs read its tiles or its arrivals come in
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_free_pair(tmem_base, TMEM_COLS);
  }
}

const bool g_pdl_on = std::getenv("ZRNN_NO_PDL") == nullptr;

template <int MODE, int EPI>
cudaError_t launch_t(const VocabParams& p, cudaStream_t st) {
  constexpr int PARTS = mode_split(MODE) ? 2 : 1;
  const int stage = PARTS * p.kbs * (128 + p.nb / 2) * 128;
  const int fixed = (int)sizeof(PairCtrl) + kXposeBytes + column_bytes(p.nb);
  const int stages = std::min((kSmem - fixed) / stage, (int)kMaxStages);
  if (stages < 2) return cudaErrorInvalidValue;
  const int bufs = 2 * PARTS * p.nb <= 512 ? 2 : 1;
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(tc_vocab_pair_kernel<MODE, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int v_tiles = (p.N + 255) / 256;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(2 * std::min(v_tiles * p.n_ct, device_sms() / 2));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_pdl_on ? 1 : 0;
  count_launch();
  return cudaLaunchKernelEx(&cfg, tc_vocab_pair_kernel<MODE, EPI>, p, stages, v_tiles, bufs);
}
template <int MODE>
cudaError_t launch_mode(const VocabParams& p, int epi, cudaStream_t st) {
  if (epi == TC_EPI_STORE) return launch_t<MODE, TC_EPI_STORE>(p, st);
  if (epi == TC_EPI_LSE) return launch_t<MODE, TC_EPI_LSE>(p, st);
  return cudaErrorInvalidValue;
}

}  // namespace

// The time of a launch is the tiles of the busiest pair times the columns of a tile, a tile's fixed part counting as 48 more: 0.3 % more than
// the best tiles take (700 - 40000 words, K = 64 - 1000, 65 - 2400 columns, all widths forced).  Few words are cut into many
// narrow tiles: 700 words, K = 1000, 1200 columns, fp16 split 18.5 us in tiles of 160 columns, 12.8 of 64.
VocabTiles vocab_pair_tiles(int M, int N) {
  const int pairs = device_sms() / 2, v_tiles = (N + 255) / 256;
  VocabTiles best{0, 0};
  long long best_cost = 0;
  for (int w = 256; w >= 32; w -= 32) {
    const int n_ct = (M - 1) / w + 1, nb = ((M - 1) / n_ct + 32) / 32 * 32;
    if ((long long)nb * (n_ct - 1) >= M) continue;  // the last tile would be empty
    const long long cost = (((long long)v_tiles * n_ct + pairs - 1) / pairs) * (nb + 48);
    if (best.n_ct == 0 || cost < best_cost) {
      best = VocabTiles{n_ct, nb};
      best_cost = cost;
    }
  }
  return best;
}

// Tiles of one CTA (tc_gemm.cu) are faster for the log-sum-exp epilogue of short products, which takes longer than their MMAs: it has a column
// per lane, so no value changes hands.  us, single CTAs / pairs, 160, 512 and 6400 columns: fp16 split, K = 100, 10000 words 9.2 / 10.0,
// 11.5 / 14.3, 69 / 86; K = 512, 20000 words 19.1 / 18.8, 30.5 / 30.1, 277 / 246; bf16, 50000 words, K = 1000 26.0 / 22.0 at 160
// columns, 43.6 / 49.7, 405 / 420; K = 1536 41.5 / 36.6, 67 / 64, 598 / 582.  (65 - 144 columns of K = 100 - 1024: 6 - 22 us, the few-columns
// kernel 10 - 41.)  In the split modes they are faster for longer products, too, where these have few tiles for 74 pairs (K = 504, 3000 words,
// 768 columns 9.8 / 12.1): the estimates are fitted to products of 700 - 40000 words, K = 64 - 1000, 65 - 2400 columns (6.5 % rms).
bool vocab_lse_single(int mode, int kb, int M, int N) {
  if (vocab_short(mode, kb)) return true;
  if (!mode_split(mode)) return false;
  const int pairs = device_sms() / 2;
  const VocabTiles t = vocab_pair_tiles(M, N);
  const long long waves = ((long long)((N + 255) / 256) * t.n_ct + pairs - 1) / pairs;
  if (waves > 3) return false;
  const long long waves1 = ((long long)((N + 127) / 128) * ((M + 127) / 128) + 2 * pairs - 1) / (2 * pairs);
  const float loop = 0.0042f * kb * std::max(75, t.nb), epi = 0.8f + 0.0177f * t.nb, loop1 = 0.62f * kb, epi1 = 2.35f;
  return 2.6f + waves1 * std::max(loop1, epi1) + 0.77f * std::min(loop1, epi1) <
         5.2f + waves * std::max(loop, epi) + 0.38f * std::min(loop, epi) * (t.nb > 128 ? waves : 1);
}

cudaError_t launch_tc_vocab_pair(const VocabParams& p, int mode, int epi, cudaStream_t st) {
  if (p.M < 1 || p.N < 1 || p.nb < 32 || p.nb > 256 || (p.nb & 31) || p.n_ct < 1 || p.nb * p.n_ct < p.M || p.nb * (p.n_ct - 1) >= p.M ||
      p.kb < 1 || p.kbs != vocab_kbs(mode) || (p.part_rows != 64 && p.part_rows != 128))
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
