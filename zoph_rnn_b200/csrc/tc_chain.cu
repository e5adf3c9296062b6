// tcgen05 kernel for the links of the recurrent chain with tiles of 128 batch rows x 128 weight rows (a few hundred columns, or several
// cells in a launch), and the rule that picks a link's kernel and tile.  Narrow tiles: tc_link.cu; many columns: tc_cell_pair.cu.
//
// A CTA works over the WHOLE K axis: no CTA waits for another one's partial tile, so a launch is: activations in (one TMA latency),
// K loop, epilogue.
//
// Warps: 16 epilogue warps (warp w reads TMEM lane quadrant w % 4 and takes column group w / 4 of the tile), one for the
// activation loads, one for the weight loads, two that issue MMAs.  The weights do not depend on the predecessor kernel, so
// their loads start before griddepcontrol.wait.
#include "tc_chain.cuh"

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "kernels.cuh"
#include "tc_chain_device.cuh"

namespace zrnn {
namespace {

constexpr int kEpiWarps = 16;
// Two warps issue MMAs, so that the wait for a stage and the commit of one overlap the other's MMAs.  They take alternate stages, each
// into accumulators of its own; in the split modes there is no room for that: one warp issues the hi * hi products of every stage and
// the other the two cross products.
constexpr int kMmaWarps = 2;
constexpr int kThreads = (kEpiWarps + 2 + kMmaWarps) * 32;
// The tensor core's fp32 accumulator truncates, so in the split modes it is not asked to absorb more than round_kb k-blocks in a row:
// the K axis is walked in rounds, each into a fresh accumulator set, and the epilogue warps, idle until the end otherwise, add every
// finished round to sums of their own in registers (round to nearest) while the next round runs.  As many k-steps per round as the
// accumulators of the narrow tiles absorb (tc_link.cu: 4 up to 512 elements per source, else 8), so that the choice of a tile
// is none of precision.
__host__ __device__ constexpr int round_kb(int mode, int kb) { return kb <= (mode == TC_TF32X3 ? 16 : 8) ? 1 : 2; }
// accumulator sets.  Split modes: main accumulators, with one cross accumulator behind them.  bf16: one per MMA warp, tf32: two (tc_link.cu).
__host__ __device__ constexpr int chain_sets(int mode) { return mode_split(mode) ? 3 : (mode == TC_TF32 ? 2 : 1) * kMmaWarps; }
__host__ __device__ constexpr int chain_tmem(int BN, int mode) {
  const int need = (chain_sets(mode) + (mode_split(mode) ? 1 : 0)) * BN;
  int c = 32;
  while (c < need) c *= 2;
  return c;
}
constexpr int kChainRingBytes = 224 * 1024, kMaxStages = 8;

template <int BN, int MODE, int EPI>
__device__ __forceinline__ void chain_body(const ChainParams& p, const int m_block, const int stages) {
  constexpr int EW = kEpiWarps, kAWarp = EW, kWWarp = EW + 1, kMmaWarp = EW + 2;
  // (the modes that walk in rounds are those whose MMA warps share the work by product)
  constexpr bool SPLIT_MODE = mode_split(MODE);
  constexpr int STEP = SPLIT_MODE ? 1 : kMmaWarps;  // stages from one of an MMA warp to its next
  constexpr int PARTS = SPLIT_MODE ? 2 : 1;
  constexpr int WKB = BN * 128;  // bytes of one k-block of one weight part
  constexpr uint32_t IDESC = make_idesc(mode_fmt(MODE), BN);
  constexpr int NSET = chain_sets(MODE), TMEM_COLS = chain_tmem(BN, MODE);
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t full_bar[kMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kMaxStages];
  __shared__ __align__(8) uint64_t accum_bar;  // everything accumulated (rounds: the cross products)
  __shared__ __align__(8) uint64_t set_full[chain_sets(MODE)], set_empty[chain_sets(MODE)];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  __shared__ float s_bias[BN];

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  const int m0 = m_block * 128, n_tile = blockIdx.y;
  const int akb = p.a_rows * 128;  // bytes of one k-block of one activation part
  // k-blocks per ring stage: one TMA instruction and one hand-over for the activations (the weights) of several blocks where the ring
  // still holds a few stages
  const int KBS = p.kbs;
  // KBS x [A hi][A lo], KBS x [W hi][W lo]; every piece is a multiple of 1024 bytes
  const int stage_bytes = PARTS * KBS * (akb + WKB);
  const int src_it = (p.kb + KBS - 1) / KBS, n_it = p.nsrc * src_it;
  const int round_its = KBS < round_kb(MODE, p.kb) ? round_kb(MODE, p.kb) / KBS : 1;  // stages per round
  ZR_STAMP(0);
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 2);  // the activation and the weight producer
      mbar_init(&empty_bar[s], SPLIT_MODE ? kMmaWarps : 1);
    }
    mbar_init(&accum_bar, SPLIT_MODE ? 1 : kMmaWarps);
    for (int i = 0; i < NSET; ++i) {
      mbar_init(&set_full[i], 1);
      mbar_init(&set_empty[i], EW);
    }
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {  // (the first MMA warp owns the TMEM allocation)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  ZR_STAMP(1);

  if (warp == kWWarp) {
    // ------------------------------------------------------------ weights: nothing here depends on the predecessor
    {
      const bool one = elect_one();
      bool ok = true;
      int it = 0, st = 0;
      uint32_t ph = 0;
      int s = 0, c = 0;
      for (; it < n_it; ++it) {
        if (it >= stages && !mbar_wait_warp(&empty_bar[st], ph ^ 1u, &abort_s, p.err, 1)) { ok = false; break; }
        uint8_t* w = tiles + (size_t)st * stage_bytes + PARTS * KBS * akb;
        const int wkb = p.wkb0[s] + c * KBS;
        if (one) {
          mbar_expect_tx(&full_bar[st], (uint32_t)(PARTS * KBS * WKB));
          if constexpr (EPI == TC_EPI_LSTM) {
            constexpr int TH = BN / 4;
            const int chunk = (n_tile * TH / 32) * p.w_kbtot + wkb;
            if (p.w_first) tma_load_5d_first(w, &p.w, &full_bar[st], n_tile * TH % 32, 0, chunk);
            else tma_load_5d(w, &p.w, &full_bar[st], n_tile * TH % 32, 0, chunk);
          } else {
            tma_load_4d(w, &p.w, &full_bar[st], n_tile * BN, wkb);
          }
        }
        __syncwarp();
        if (++st == stages) { st = 0; ph ^= 1u; }
        if (++c == src_it) { c = 0; ++s; }
      }
      if (!ok) settle_copies();
    }
    __syncwarp();
    pdl_wait();
  } else {
    pdl_wait();
    if (warp == kAWarp) {
      // ------------------------------------------------------------ activations
      {
        const bool one = elect_one();
        if (one) pdl_trigger();  // after the wait: the successor may read what this kernel's predecessor left (tc_link.cu)
        bool ok = true;
        int it = 0, st = 0;
        uint32_t ph = 0;
        int s = 0, c = 0;
        for (; it < n_it; ++it) {
          if (it >= stages && !mbar_wait_warp(&empty_bar[st], ph ^ 1u, &abort_s, p.err, 7)) { ok = false; break; }
          uint8_t* a = tiles + (size_t)st * stage_bytes;
          if (one) {
            mbar_expect_tx(&full_bar[st], (uint32_t)(PARTS * KBS * akb));
            tma_load_4d(a, &p.a[s], &full_bar[st], p.a_row0[s] + m0, c * KBS);
          }
          __syncwarp();
          if (++st == stages) { st = 0; ph ^= 1u; }
          if (++c == src_it) { c = 0; ++s; }
        }
        if (!ok) settle_copies();
      }
    } else if (warp >= kMmaWarp) {
      // ------------------------------------------------------------ MMA issuers
      {
        const bool one = elect_one();
        const int mw = warp - kMmaWarp;
        bool ok = true;
        const bool rounds = SPLIT_MODE && mw == 0;
        int st = SPLIT_MODE ? 0 : mw, set = st, in_round = 0, round = 0;
        uint32_t ph = 0;
        for (int it = st; it < n_it; it += STEP) {
          if (rounds && in_round == 0) {
            set = round % NSET;
            if (round >= NSET && !mbar_wait_warp(&set_empty[set], (uint32_t)((round / NSET) & 1) ^ 1u, &abort_s, p.err, 4)) { ok = false; break; }
            tc_fence_after();
          }
          if (!SPLIT_MODE) set = it % NSET;
          if (!mbar_wait_warp(&full_bar[st], ph, &abort_s, p.err, 2)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(tiles + (size_t)st * stage_bytes), w_addr = a_addr + PARTS * KBS * akb;
          const uint32_t d = tmem_base + (uint32_t)(set * BN), d_cross = tmem_base + (uint32_t)(NSET * BN);
          const bool fresh = rounds ? in_round == 0 : it < (SPLIT_MODE ? STEP : NSET);  // the accumulator starts with this stage
          if (one) {
            for (int b = 0; b < KBS; ++b) {
              const uint64_t da = make_smem_desc(a_addr + b * PARTS * akb), dal = make_smem_desc(a_addr + (b * PARTS + 1) * akb);
              const uint64_t dw = make_smem_desc(w_addr + b * PARTS * WKB), dwl = make_smem_desc(w_addr + (b * PARTS + 1) * WKB);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const uint32_t acc = (!fresh || b > 0 || k > 0) ? 1u : 0u;
                if (!SPLIT_MODE || mw == 0) umma<mode_kind_tf32(MODE)>(d, da + 2 * k, dw + 2 * k, IDESC, acc);
                if (SPLIT_MODE && mw == 1) {
                  umma<mode_kind_tf32(MODE)>(d_cross, dal + 2 * k, dw + 2 * k, IDESC, acc);
                  umma<mode_kind_tf32(MODE)>(d_cross, da + 2 * k, dwl + 2 * k, IDESC, 1u);
                }
              }
            }
            umma_commit(&empty_bar[st]);
          }
          __syncwarp();
          if (rounds && (++in_round == round_its || it + STEP >= n_it)) {
            if (one) umma_commit(&set_full[set]);
            in_round = 0;
            ++round;
          }
          st += STEP;
          if (st >= stages) { st -= stages; ph ^= 1u; }
        }
        if (ok && !rounds && one) umma_commit(&accum_bar);
      }
    }
  }
  __syncwarp();
  // ------------------------------------------------------------ epilogue
  const bool epi_warp = warp < EW;
  if (epi_warp) {  // the tile's bias values: fetched beside the main loop, for the epilogue warps alone
    for (int i = threadIdx.x; i < BN; i += EW * 32) {
      float bv = 0.f;
      if (EPI == TC_EPI_LSTM) {
        constexpr int TH = BN / 4;
        const int hid = n_tile * TH + (i % TH);
        if (hid < p.N) bv = p.bias[(i / TH) * p.N + hid];
      } else {
        const int n = n_tile * BN + i;
        if (n < p.N && p.bias) bv = p.bias[n];
      }
      s_bias[i] = bv;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(EW * 32) : "memory");
  }
  const int quad = warp & 3, cg = warp >> 2;
  const int row = m0 + quad * 32 + lane;
  const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
  constexpr int GROUPS = EW / 4;
  constexpr int PER = EPI == TC_EPI_LSTM ? BN / 4 / GROUPS : BN / GROUPS;  // outputs per row and column group
  constexpr int W = 8;                                    // outputs handled at a time (registers)
  // the cell's other inputs do not depend on the accumulators: fetch the first ones while the main loop runs
  float pre_c[W];
  float mk = 1.0f;
  if (epi_warp && row < p.M) {
    if (p.mask) mk = (float)p.mask[row];
    if constexpr (EPI == TC_EPI_LSTM) {
      const int hb = n_tile * (BN / 4) + cg * PER;
#pragma unroll
      for (int u = 0; u < W; ++u) pre_c[u] = hb + u < p.N ? p.c_prev[(size_t)row * p.N + hb + u] : 0.f;
    }
  }
  const bool live = m0 + quad * 32 < p.M;  // whole warps: the TMEM loads are warp-wide
  bool ready = epi_warp;
  // running sums (rounds): chunk ch of W outputs; LSTM: one chunk per gate
  constexpr int NCH = EPI == TC_EPI_LSTM ? 4 : PER / W;
  auto chunk_col = [&](int ch) { return EPI == TC_EPI_LSTM ? ch * (BN / 4) + cg * PER : cg * PER + ch * W; };
  float sum[SPLIT_MODE ? NCH : 1][W];
  if constexpr (SPLIT_MODE) {
    static_assert(EPI != TC_EPI_LSTM || PER == W, "one chunk per gate");
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch)
#pragma unroll
      for (int u = 0; u < W; ++u) sum[ch][u] = 0.f;
    for (int r = 0; ready && r * round_its < n_it; ++r) {
      const int set = r % NSET;
      ready = __all_sync(0xffffffffu, mbar_wait(&set_full[set], (uint32_t)((r / NSET) & 1), &abort_s, p.err, 3));
      tc_fence_after();
      if (ready && live) {
        float t[NCH][W];
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) tmem_ldw<W>(taddr + set * BN + chunk_col(ch), t[ch]);
        tmem_wait_ld();
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch)
#pragma unroll
          for (int u = 0; u < W; ++u) sum[ch][u] += t[ch][u];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&set_empty[set]);
    }
  }
  if (ready) {
    ready = __all_sync(0xffffffffu, mbar_wait(&accum_bar, 0, &abort_s, p.err, 3));
    tc_fence_after();
  }
  ZR_STAMP(2);
  const int n_sets = n_it < NSET ? n_it : NSET;  // sets that were written (without rounds)
  // the W finished accumulator columns of chunk ch, which start at tile column `col`
  auto load_acc = [&](int ch, int col, float* v) {
    if constexpr (SPLIT_MODE) {
      float x[W];
      tmem_ldw<W>(taddr + NSET * BN + col, x);
      tmem_wait_ld();
#pragma unroll
      for (int u = 0; u < W; ++u) v[u] = fmaf(x[u], mode_cross_scale(MODE), sum[ch][u]);
    } else {
      float t[NSET][W];
#pragma unroll
      for (int a = 0; a < NSET; ++a)
        if (a == 0 || a < n_sets) tmem_ldw<W>(taddr + a * BN + col, t[a]);
      tmem_wait_ld();
#pragma unroll
      for (int u = 0; u < W; ++u) v[u] = t[0][u];
#pragma unroll
      for (int a = 1; a < NSET; ++a)
        if (a < n_sets) {
#pragma unroll
          for (int u = 0; u < W; ++u) v[u] += t[a][u];
        }
    }
  };
  if (ready && live) {
    if constexpr (EPI == TC_EPI_LSTM) {
      constexpr int TH = BN / 4, THP = TH < 32 ? TH : 32;  // hidden units per gate block of the accumulator
      const int H = p.N;
#pragma unroll
      for (int j8 = 0; j8 < PER; j8 += W) {
        const int j0 = cg * PER + j8;
        float g[4][W];
#pragma unroll
        for (int q = 0; q < 4; ++q) load_acc(q, (j0 / THP) * (4 * THP) + q * THP + (j0 % THP), g[q]);
        const int hb = n_tile * TH + j0;
        if (row < p.M && hb < H) {
          float hv[W], cv[W];
          if (j8 > 0) {
#pragma unroll
            for (int u = 0; u < W; ++u) pre_c[u] = hb + u < H ? p.c_prev[(size_t)row * H + hb + u] : 0.f;
          }
#pragma unroll
          for (int u = 0; u < W; ++u) {
            const float* sb = s_bias + j0 + u;
            const float gi = act_sigmoid<MODE>(g[0][u] + sb[0]);
            const float gf = act_sigmoid<MODE>(g[1][u] + sb[TH]);
            const float gg = act_tanh<MODE>(g[2][u] + sb[2 * TH]);
            const float go = act_sigmoid<MODE>(g[3][u] + sb[3 * TH]);
            const float c = gf * pre_c[u] + gi * gg;
            hv[u] = go * act_tanh<MODE>(c) * mk;
            cv[u] = c * mk;
          }
          const int nvalid = H - hb >= W ? W : H - hb;
          store_f32<W>(p.c_out, (size_t)row * H + hb, cv, nvalid);
          if (p.C) store_f32<W>(p.C, (size_t)row * p.ldc + hb, hv, nvalid);
          store_operand<W>(p, (size_t)row * p.ld_op + hb, hv, nvalid);
        }
      }
    } else {
#pragma unroll
      for (int c8 = 0; c8 < PER; c8 += W) {
        const int c0 = cg * PER + c8, n = n_tile * BN + c0, left = p.N - n;
        float v[W];
        load_acc(c8 / W, c0, v);
        if (row < p.M && left > 0) {
#pragma unroll
          for (int u = 0; u < W; ++u) {
            float t = v[u] + s_bias[c0 + u];
            if (p.act == 1 && (p.act_rows == 0 || n + u < p.act_rows)) t = act_tanh<MODE>(t);
            v[u] = t * mk;
          }
          const int nvalid = left >= W ? W : left;
          if (p.C) store_f32<W>(p.C, (size_t)row * p.ldc + n, v, nvalid);
          store_operand<W>(p, (size_t)row * p.ld_op + n, v, nvalid);
        }
      }
    }
  }
  // the operand rows' padding up to a whole k-block is read by the next product: the last row tile keeps it at zero
  if (epi_warp && n_tile == (int)gridDim.y - 1 && row < p.M && cg == 0) zero_operand_pad(p, (size_t)row * p.ld_op, p.N, p.ld_op);
  ZR_STAMP(6);
  tc_fence_before();
  __syncthreads();
  ZR_STAMP(7);
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS)
                 : "memory");
  }
}

template <int BN, int MODE, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
    tc_chain_kernel(const __grid_constant__ ChainParams p, int stages) {
  chain_body<BN, MODE, EPI>(p, (int)blockIdx.x, stages);
}
// Several independent problems of one row block each (M <= 128): blockIdx.x selects the problem.  The cells of one
// anti-diagonal of a stack (layer l at step t, layer l - 1 at step t + 1, ...) do not depend on one another.
template <int BN, int MODE, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
    tc_chain_multi_kernel(const __grid_constant__ ChainBatch pb, int stages) {
  chain_body<BN, MODE, EPI>(pb.p[blockIdx.x], 0, stages);
}

const bool g_pdl_on = std::getenv("ZRNN_NO_PDL") == nullptr;

template <int BN, int MODE, int EPI>
cudaError_t launch_t(const ChainBatch& b, int n, cudaStream_t st) {
  const ChainParams& p = b.p[0];
  constexpr int PARTS = mode_split(MODE) ? 2 : 1;
  const int stage = PARTS * p.kbs * (p.a_rows * 128 + BN * 128);
  // the MMA reads 128 rows of activations, the last stage's reads may run past a narrower box
  const int slack = 1024 + (128 - p.a_rows) * 128;
  int stages = (kChainRingBytes - slack) / stage;
  stages = stages > kMaxStages ? kMaxStages : (stages < 2 ? 2 : stages);
  const int its = p.nsrc * ((p.kb + p.kbs - 1) / p.kbs);
  if (stages > its) stages = its;
  // a whole number of stages per MMA warp: each waits on barriers of its own only.  (A barrier shared by two waiters would let
  // one that is a round ahead mistake "the round before last is complete" for its own round.)
  if (!mode_split(MODE)) stages = stages < kMmaWarps ? kMmaWarps : stages / kMmaWarps * kMmaWarps;
  const size_t smem = (size_t)stages * stage + slack;
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(tc_chain_kernel<BN, MODE, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
    if (e != cudaSuccess) return e;
    if constexpr (EPI == TC_EPI_LSTM) {
      e = cudaFuncSetAttribute(tc_chain_multi_kernel<BN, MODE, TC_EPI_LSTM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
      if (e != cudaSuccess) return e;
    }
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  const int rows = EPI == TC_EPI_LSTM ? p.N * 4 : p.N;
  cfg.gridDim = dim3(n > 1 ? n : (p.M + 127) / 128, (rows + BN - 1) / BN);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_pdl_on ? 1 : 0;
  count_launch();
  if constexpr (EPI == TC_EPI_LSTM) {
    if (n > 1) return cudaLaunchKernelEx(&cfg, tc_chain_multi_kernel<BN, MODE, EPI>, b, stages);
  }
  return cudaLaunchKernelEx(&cfg, tc_chain_kernel<BN, MODE, EPI>, p, stages);
}
template <int MODE>
cudaError_t launch_mode(const ChainBatch& b, int n, int BN, int epi, cudaStream_t st) {
  if (epi == TC_EPI_LSTM && BN == 128) return launch_t<128, MODE, TC_EPI_LSTM>(b, n, st);
  if (epi == TC_EPI_STORE && n == 1 && BN == 128) return launch_t<128, MODE, TC_EPI_STORE>(b, n, st);
  return cudaErrorInvalidValue;
}

}  // namespace

// Which tile: a launch takes, per wave of CTAs and k-block, the longer of the bytes a CTA fetches, at the 130 KB/us that an SM takes in
// from L2, and the MMAs, of which each takes 60 cycles at least (the split modes at 128 rows, a warp per product and one cross
// accumulator: 1.6 times their cycles, 1.4 times in a launch of several cells; products in rounds with one accumulator set, on half an SM: 0.15
// us more); then a fixed part per wave, the exchange of a K split and an epilogue that grows with the outputs per CTA.  Of the early sources
// of links on half an SM a half (bf16, tf32: a third) is counted off: that much runs beside the predecessor.  Cells on whole SMs that leave
// the next launch no room beside them take up to 0.5 us more.  The exchange, these two and the factor of several cells are fitted to passes up to 256 columns (skinny_us, skinny_gemm.cu), the rest to launches: us, estimated / measured,
// fp16 split, 1000 units, 384 columns in tiles of 128 rows 25.6 / 25.6; 500 units, 768 columns 15.1 / 15.9; bf16, 1000 units, 384 columns
// 11.7 / 11.4.
// Four CTAs per tile in the split modes only: in bf16 they are worth 0.4 % of a scoring pass (4 x 1000 units, 128 columns 3108 -> 3097 us),
// and the other order of the sums turns results that are rounded to bf16 at every step (6e-4 between the log-probabilities, 1.08e-3 from
// float64 either way).
ChainPlan plan_chain(int mode, int epi, int rows, int cells, int nsrc, int kb, int n_early, int M, bool beside) {
  const bool two = mode_split(mode);
  const int sms = device_sms(), parts = two ? 2 : 1, mt = cells * ((M + 127) / 128), a_rows = M >= 128 ? 128 : (M + 7) / 8 * 8;
  const float two_ctas = epi == TC_EPI_LSTM ? (two ? 1.08f : 0.62f) : (two ? 0.4f : 1.0f);
  ChainPlan best{0, 1, 1e30f, false, 0};
  for (int BN = epi == TC_EPI_LSTM ? 32 : 16; BN <= 128; BN *= 2) {
    for (int split = 1; split <= 4; split *= 2) {
      if (split == 4 && (!two || epi == TC_EPI_LSTM || BN != 32)) continue;
      if (split > 1 && (cells > 1 || BN > 64 || kb < 2 * split)) continue;
      const int ctas = mt * ((rows + BN - 1) / BN) * split, waves = (ctas + sms - 1) / sms;
      const bool whole = two && BN <= 64 && BN >= 32 && !beside;
      const float crowd = whole && epi == TC_EPI_LSTM ? 0.5f * std::min(1.f, std::max(0.f, 2.f * ctas / sms - 1.f)) : 0.f;
      const float cyc = 4.f * (!two ? std::max(60.f, BN / 2.f) : (BN <= 64 ? std::max(60.f, (float)BN) + 60.f : (cells > 1 ? 1.38f : 1.6f) * 3.f * BN / 2.f));
      const float kb_us = std::max(parts * 128.f * (a_rows + BN) / 130e3f, cyc / 1850.f) + (two && epi == TC_EPI_STORE && BN <= 64 && !whole ? 0.15f : 0.f);
      const float kbs = kb * (nsrc - (BN <= 64 && !whole ? (two ? 0.5f : 0.33f) * n_early : 0.f)) / split;
      const float us = (whole ? 3.6f : 3.2f) + 3.f * (waves - 1) + waves * (kb_us * kbs + (two ? 0.01f : 0.005f) * BN / split) + (split == 2 ? two_ctas : split == 4 ? 0.9f : 0.f) + crowd;
      if (us < best.us) best = ChainPlan{BN, split, us, whole, 0};
    }
  }
  // Pairs of CTAs: a k-block's twelve MMAs (four) take 64 cycles each at least, and half a cycle per column and more; a wave's
  // set-up, first loads and end 7 us (5), all of an SM being needed.  (Fitted to cells of 256 - 2048 units, 300 - 3000 columns, tiles of 96 - 256
  // columns forced: 6 % rms; the choices cost 0.4 % more than the best ones.)  More than 160 columns per tile have one accumulator for the whole K axis in the split
  // modes, whose error is several times that of rounds (1000 units 1.74e-6 from float64 against 1.8e-7).  That is paid only where it buys most: in fp16,
  // where tiles of 128 rows and columns take more than 1.6 times the waves of CTAs that tiles of 256 rows would (1000 units 513 - 1152 columns: two
  // waves against one), and tiles of 64 rows, over all or half of the K axis, more than twice the time even if half of the early sources is
  // free to them (1000 units, three sources, two of them early: 6 of 6 k-axes at 513 - 896 columns, 6 of 8 beyond).
  const auto waves_of = [&](int w, int split) { return ((long long)mt * ((rows + w - 1) / w) * split + sms - 1) / sms; };
  const float narrow = (nsrc - 0.5f * n_early) * std::min((float)waves_of(64, 1), 0.5f * waves_of(64, 2));
  const bool one_acc = !two || (mode == TC_F16X2 && 8 * waves_of(256, 1) < 5 * waves_of(128, 1) && 2.f * nsrc * waves_of(256, 1) < narrow);
  const int row_tiles = (rows + 255) / 256;
  for (int w = one_acc ? 256 : 160; M > 256 && cells == 1 && w >= 32; w -= 32) {  // (a width's time grows with the number of column tiles)
    const int n_ct = (M - 1) / w + 1, nb = ((M - 1) / n_ct + 32) / 32 * 32;
    if (n_ct > 65535) break;  // (a grid's second axis)
    const long long waves = ((long long)row_tiles * n_ct + sms / 2 - 1) / (sms / 2);
    const float cyc = two ? std::max(919.f, 7.94f * nb) : std::max(317.f, 2.92f * nb);
    const float us = (two ? 2.7f : 2.05f) + waves * ((two ? 6.9f + 0.01f * nb : 4.9f + 0.016f * nb) + nsrc * kb * cyc / 1850.f);
    if (us < best.us) best = ChainPlan{128, 1, us, false, nb};
  }
  return best;
}

int chain_kbs(int mode, int BN, int a_rows, int kb, int split) {
  if (BN <= 64) return link_kbs(mode, BN, a_rows, kb, split);
  const int parts = mode_split(mode) ? 2 : 1;
  int k = 4;  // as many as leave the ring four stages
  while (k > 1 && 4 * parts * k * (a_rows + BN) * 128 > kChainRingBytes - (128 - a_rows) * 128 - 1024) k /= 2;
  return k;
}

cudaError_t launch_tc_chain(const ChainBatch& b, int n, int BN, int mode, int epi, int split, bool whole, cudaStream_t st) {
  if (n < 1 || n > ChainBatch::MAX) return cudaErrorInvalidValue;
  for (int i = 0; i < n; ++i) {
    const ChainParams& p = b.p[i];
    if (p.M < 1 || (n > 1 && p.M > 128) || p.N != b.p[0].N || p.a_rows < 8 || p.a_rows > 128 || (p.a_rows & 7) ||
        p.a_rows != b.p[0].a_rows || (p.M > 128 && p.a_rows != 128) || p.a_rows < (p.M < 128 ? p.M : 128) || p.kb < 1 || p.nsrc < 1 ||
        p.nsrc * p.kb != b.p[0].nsrc * b.p[0].kb || p.kbs != b.p[0].kbs || p.kbs != chain_kbs(mode, BN, p.a_rows, p.kb, split) ||
        p.n_early < 0 || p.n_early >= p.nsrc)
      return cudaErrorInvalidValue;
  }
  if (BN <= 64) return launch_tc_link(b, n, BN, mode, epi, split, whole, st);
  if (split != 1) return cudaErrorInvalidValue;
  switch (mode) {
    case TC_BF16: return launch_mode<TC_BF16>(b, n, BN, epi, st);
    case TC_TF32: return launch_mode<TC_TF32>(b, n, BN, epi, st);
    case TC_TF32X3: return launch_mode<TC_TF32X3>(b, n, BN, epi, st);
    case TC_F16X2: return launch_mode<TC_F16X2>(b, n, BN, epi, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace zrnn
