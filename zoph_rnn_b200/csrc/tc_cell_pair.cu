// LSTM cells and attention products of many columns on pairs of CTAs (tc_pair_device.cuh): a pair computes 256 weight rows x nb <= 256
// batch columns over the whole K axis.
//
// The weights are the M side: each CTA loads its own 128 weight rows and half of the columns' rows, so a k-block of 256 x 128 in the
// split modes brings 48 KB into an SM, not 64, and its MMAs read 6 KB of shared memory in the 64 cycles that they take, not 8
// (tc_vocab_pair.cu): 0.42 us per k-block in a cell's loop, 0.65 with tiles of one CTA.
//
// An accumulator row is a gate's row (packed tiles of 4 gates x 32 hidden units: a lane quadrant of tensor memory is a gate, a lane a
// unit).  Each epilogue warp applies its gate's function to its share of the columns; the four gates meet in shared memory, in the
// place of the operand tiles, and a warp finishes 32 units of a column at a time: loads and stores of whole lines.
//
// Split modes, up to 160 columns: the K axis is walked in rounds into fresh accumulators, which the epilogue warps add up in
// registers (tc_link.cu); three accumulators take turns up to 128 columns, two up to 160, and beyond there is room for one only.  bf16
// takes two accumulators in turn, stage by stage, and adds them up at the end; tf32 walks the K axis in four rounds with two: the tensor core
// truncates as it accumulates (tf32, 1000 and 2048 units: 0.2 - 0.3 % farther from float64 with one for all of it).
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "kernels.cuh"
#include "tc_chain.cuh"
#include "tc_pair_device.cuh"

namespace zrnn {
namespace {

constexpr int kEpiWarps = 16, kAWarp = 16, kWWarp = 17, kMmaWarp = 18, kThreads = 608;
constexpr int kSmem = 227 * 1024, kMaxStages = 8, kGroups = 8;  // kGroups: groups of 8 columns per epilogue warp
// k-blocks per round: as many k-steps as an accumulator of the links absorbs (tc_link.cu)
__host__ __device__ constexpr int round_kb(int mode, int kb) { return kb <= (mode == TC_TF32X3 ? 16 : 8) ? 1 : 2; }
__host__ __device__ constexpr int acc_sets(int nb) { return nb <= 128 ? 3 : (nb <= 160 ? 2 : 1); }  // (split modes: and one for the cross products)
static_assert(fills_sm(kSmem), "both CTAs of a pair hold all of the tensor memory");
struct alignas(16) PairCtrl {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t set_full[3], set_empty[3], accum;
  uint32_t tmem_base;
  int abort;
};

// one value of the output's operand-form copy
template <int MODE>
__device__ __forceinline__ void store_op(const ChainParams& p, size_t at, float v) {
  if constexpr (MODE == TC_BF16) {
    if (p.op_b16) p.op_b16[at] = __float2bfloat16(v);
  } else if constexpr (MODE == TC_F16X2) {
    if (p.op_h_hi) {
      const __half h = __float2half_rn(v);
      p.op_h_hi[at] = h;
      p.op_h_lo[at] = __float2half_rn((v - __half2float(h)) * 2048.0f);
    }
  } else {
    if (p.op_hi) {
      const float h = tf32_round_dev(v);
      p.op_hi[at] = h;
      if (p.op_lo) p.op_lo[at] = v - h;
    }
  }
}

template <int MODE, int EPI>
__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(2, 1, 1)
    tc_cell_pair_kernel(const __grid_constant__ ChainBatch pb, int stages) {
  constexpr bool SPLIT_MODE = mode_split(MODE);
  constexpr int PARTS = SPLIT_MODE ? 2 : 1, TMEM_COLS = 512;
  extern __shared__ __align__(1024) uint8_t cell_smem[];
  const ChainParams& p = pb.p[blockIdx.z];
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1, tile = blockIdx.x, nb = 2 * p.a_rows, col0 = blockIdx.y * nb;  // tile: 128 weight rows
  const int KBS = p.kbs, akb = p.a_rows * 128;
  const int w_bytes = PARTS * KBS * 128 * 128, a_bytes = PARTS * KBS * akb, stage_bytes = w_bytes + a_bytes;
  uint8_t* tiles = cell_smem;
  PairCtrl& ct = *reinterpret_cast<PairCtrl*>(tiles + (size_t)stages * stage_bytes);
  const int src_it = (p.kb + KBS - 1) / KBS, n_it = p.nsrc * src_it;
  const int nsets = SPLIT_MODE ? acc_sets(nb) : 2;
  const bool rounds = MODE == TC_TF32 || (SPLIT_MODE && nsets > 1);
  const int R = MODE == TC_TF32 ? (n_it + 3) / 4 : round_kb(MODE, p.kb);  // stages per round (split modes: a k-block per stage)
  ZR_STAMP(0);
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ct.full[s], 2);  // (the leader's: its weight and its activation producer, for the bytes of both CTAs)
      mbar_init(&ct.empty[s], 1);
    }
    for (int i = 0; i < 3; ++i) {
      mbar_init(&ct.set_full[i], 1);
      mbar_init(&ct.set_empty[i], 2 * kEpiWarps);
    }
    mbar_init(&ct.accum, 1);
    ct.abort = (smem_u32(cell_smem) & 1023) ? 1 : 0;  // (the swizzled tiles need the alignment that the declaration asks for)
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
  ZR_STAMP(1);

  if (warp == kWWarp || warp == kAWarp) {
    // ------------------------------------------------------------ loads; the weights do not depend on the predecessor
    const bool one = elect_one();
    if (warp == kAWarp) {
      pdl_wait();
      pdl_trigger();  // after the wait: the successor may read what this kernel's predecessor left (tc_link.cu)
    }
    bool ok = sound;
    int st = 0, s = 0, c = 0;
    uint32_t ph = 0;
    for (int it = 0; it < n_it && ok; ++it) {
      if (it >= stages && !mbar_wait_warp(&ct.empty[st], ph ^ 1u, &ct.abort, p.err, 1)) { ok = false; break; }
      uint8_t* dst = tiles + (size_t)st * stage_bytes;
      const uint32_t bar = cluster_map(smem_u32(&ct.full[st]), 0);
      if (one) {
        if (warp == kWWarp) {
          if (rank == 0) mbar_expect_tx(&ct.full[st], (uint32_t)(2 * w_bytes));
          const int wkb = p.wkb0[s] + c * KBS;
          if constexpr (EPI == TC_EPI_LSTM)  // (the units of a tile beyond the last are dropped)
            tma_load_5d_pair(dst, &p.w, bar, 0, 0, min(tile, p.w_tiles - 1) * p.w_kbtot + wkb);
          else
            tma_load_4d_pair(dst, &p.w, bar, tile * 128, wkb);
        } else {
          if (rank == 0) mbar_expect_tx(&ct.full[st], (uint32_t)(2 * a_bytes));
          tma_load_4d_pair(dst + w_bytes, &p.a[s], bar, p.a_row0[s] + col0 + rank * p.a_rows, c * KBS);
        }
      }
      __syncwarp();
      if (++st == stages) { st = 0; ph ^= 1u; }
      if (++c == src_it) { c = 0; ++s; }
    }
    if (sound && !ok) settle_copies();
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer of the pair
    if (rank == 0 && sound) {
      const bool one = elect_one();
      const uint32_t idesc = make_idesc_pair(mode_fmt(MODE), (uint32_t)nb);
      const uint32_t d_cross = tmem_base + (uint32_t)(nsets * nb);
      int st = 0, set = 0, in_round = 0, round = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int it = 0; it < n_it; ++it) {
        if (rounds && in_round == 0) {
          set = round % nsets;
          if (round >= nsets && !mbar_wait_warp(&ct.set_empty[set], (uint32_t)((round / nsets) & 1) ^ 1u, &ct.abort, p.err, 4)) { ok = false; break; }
          tc_fence_after();
        }
        if (!mbar_wait_warp(&ct.full[st], ph, &ct.abort, p.err, 2)) { ok = false; break; }
        tc_fence_after();
        const uint32_t w_addr = smem_u32(tiles + (size_t)st * stage_bytes), a_addr = w_addr + w_bytes;
        if (MODE == TC_BF16) set = it & 1;
        const uint32_t d = tmem_base + (uint32_t)(set * nb);
        const bool fresh = rounds ? in_round == 0 : it < (SPLIT_MODE ? 1 : 2);
        if (one) {
          for (int b = 0; b < KBS; ++b) {
            const uint64_t dw = make_smem_desc(w_addr + b * PARTS * 16384), dwl = make_smem_desc(w_addr + (b * PARTS + 1) * 16384);
            const uint64_t da = make_smem_desc(a_addr + b * PARTS * akb), dal = make_smem_desc(a_addr + (b * PARTS + 1) * akb);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              umma_pair<mode_kind_tf32(MODE)>(d, dw + 2 * k, da + 2 * k, idesc, (!fresh || b > 0 || k > 0) ? 1u : 0u);
              if (SPLIT_MODE) {
                umma_pair<mode_kind_tf32(MODE)>(d_cross, dwl + 2 * k, da + 2 * k, idesc, (it > 0 || b > 0 || k > 0) ? 1u : 0u);
                umma_pair<mode_kind_tf32(MODE)>(d_cross, dw + 2 * k, dal + 2 * k, idesc, 1u);
              }
            }
          }
          umma_commit_pair(&ct.empty[st]);
        }
        __syncwarp();
        if (rounds && (++in_round == R || it + 1 == n_it)) {
          if (one) umma_commit_pair(&ct.set_full[set]);
          in_round = 0;
          ++round;
        }
        if (++st == stages) { st = 0; ph ^= 1u; }
      }
      if (ok && one) umma_commit_pair(&ct.accum);
      if (!ok) settle_copies();
    }
  } else {
    // ------------------------------------------------------------ epilogue: rows 32 quad .. +31, a quarter of the columns
    const int quad = warp & 3, cg = warp >> 2, per = nb / 4, c0 = cg * per;  // first column of this warp inside the tile
    const int cols = min(nb, p.M - col0);
    const bool live = c0 < cols;  // whole warps
    const int out = EPI == TC_EPI_LSTM ? tile * 32 + lane : tile * 128 + quad * 32 + lane;  // hidden unit / output row of this lane
    float bias = 0.f;
    if (out < p.N && p.bias) bias = EPI == TC_EPI_LSTM ? p.bias[quad * p.N + out] : p.bias[out];
    float sum[kGroups][8];
#pragma unroll
    for (int j = 0; j < kGroups; ++j)
#pragma unroll
      for (int u = 0; u < 8; ++u) sum[j][u] = 0.f;
    const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0;
    auto drain = [&](uint32_t at, float scale) {  // adds an accumulator's columns to the sums
#pragma unroll
      for (int j = 0; j < kGroups; j += 2) {
        if (8 * j < per) {
          float t[2][8];
          tmem_ld8(at + 8 * j, t[0]);
          if (8 * j + 8 < per) tmem_ld8(at + 8 * j + 8, t[1]);
          tmem_wait_ld();
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            sum[j][u] = fmaf(t[0][u], scale, sum[j][u]);
            if (8 * j + 8 < per) sum[j + 1][u] = fmaf(t[1][u], scale, sum[j + 1][u]);
          }
        }
      }
    };
    bool ready = sound;
    if (rounds) {
      for (int r = 0; ready && r * R < n_it; ++r) {
        const int set = r % nsets;
        ready = __all_sync(0xffffffffu, mbar_wait(&ct.set_full[set], (uint32_t)((r / nsets) & 1), &ct.abort, p.err, 3));
        tc_fence_after();
        if (ready && live) drain(taddr + (uint32_t)(set * nb), 1.0f);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader(&ct.set_empty[set]);
      }
    }
    ready = ready && __all_sync(0xffffffffu, mbar_wait(&ct.accum, 0, &ct.abort, p.err, 3));
    tc_fence_after();
    ZR_STAMP(2);
    if (ready && live) {
      if (!rounds) drain(taddr, 1.0f);
      if (MODE == TC_BF16 && n_it > 1) drain(taddr + (uint32_t)nb, 1.0f);
      if (SPLIT_MODE) drain(taddr + (uint32_t)(nsets * nb), mode_cross_scale(MODE));
    }
    pdl_wait();
    if constexpr (EPI == TC_EPI_LSTM) {
      // all MMAs of the pair are complete: the gates take the place of the operand tiles, [gate][column][unit]
      float* ex = reinterpret_cast<float*>(tiles);
      float* mine = ex + (quad * nb + c0) * 32 + lane;
      auto gates = [&](auto f) {
#pragma unroll
        for (int j = 0; j < kGroups; ++j)
          if (8 * j < per) {
#pragma unroll
            for (int u = 0; u < 8; ++u) mine[(8 * j + u) * 32] = f(sum[j][u] + bias);
          }
      };
      if (ready && live) {
        if (quad == 2) gates([](float x) { return act_tanh<MODE>(x); });
        else gates([](float x) { return act_sigmoid<MODE>(x); });
      }
      float pre_c[kGroups * 2];  // columns c0 + quad, c0 + quad + 4, ...
#pragma unroll
      for (int i = 0; i < kGroups * 2; ++i) {
        const int c = 4 * i + quad;
        pre_c[i] = c < per && c0 + c < cols && out < p.N ? __ldcg(p.c_prev + (size_t)(col0 + c0 + c) * p.N + out) : 0.f;
      }
      asm volatile("bar.sync %0, 128;" ::"r"(2 + cg) : "memory");  // the four warps of these columns
      if (ready) {
#pragma unroll
        for (int i = 0; i < kGroups * 2; ++i) {
          const int c = 4 * i + quad;
          if (c < per && c0 + c < cols) {
            const size_t col = col0 + c0 + c;
            const float mk = p.mask ? (float)p.mask[col] : 1.0f;
            const float* g = ex + (c0 + c) * 32 + lane;
            const float cn = g[nb * 32] * pre_c[i] + g[0] * g[2 * nb * 32];
            const float h = g[3 * nb * 32] * act_tanh<MODE>(cn) * mk;
            if (out < p.N) {
              p.c_out[col * p.N + out] = cn * mk;
              if (p.C) p.C[col * p.ldc + out] = h;
              store_op<MODE>(p, col * p.ld_op + out, h);
            } else if (out < p.ld_op) {
              store_op<MODE>(p, col * p.ld_op + out, 0.f);  // the padding up to a whole k-block is read by the next product
            }
          }
        }
      }
    } else {
      if (ready && live) {
        const bool act = p.act == 1 && (p.act_rows == 0 || out < p.act_rows);
#pragma unroll
        for (int j = 0; j < kGroups; ++j)
          if (8 * j < per) {
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (c0 + 8 * j + u < cols) {
                const size_t col = col0 + c0 + 8 * j + u;
                float v = sum[j][u] + bias;
                if (act) v = act_tanh<MODE>(v);
                if (p.mask) v *= (float)p.mask[col];
                if (out < p.N) {
                  if (p.C) p.C[col * p.ldc + out] = v;
                  store_op<MODE>(p, col * p.ld_op + out, v);
                } else if (out < p.ld_op) {
                  store_op<MODE>(p, col * p.ld_op + out, 0.f);
                }
              }
          }
      }
    }
  }
  ZR_STAMP(6);
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA ends while the other one's MMAs read its tiles or its arrivals come in
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_free_pair(tmem_base, TMEM_COLS);
  }
  ZR_STAMP(7);
}

const bool g_pdl_on = std::getenv("ZRNN_NO_PDL") == nullptr;

template <int MODE, int EPI>
cudaError_t launch_t(const ChainBatch& b, int n, cudaStream_t st) {
  const ChainParams& p = b.p[0];
  const int nb = 2 * p.a_rows, stage = (mode_split(MODE) ? 2 : 1) * p.kbs * (128 + p.a_rows) * 128;
  const int stages = std::min((kSmem - (int)sizeof(PairCtrl)) / stage, (int)kMaxStages);
  if (stages < 2 || (EPI == TC_EPI_LSTM && stages * stage < 512 * nb)) return cudaErrorInvalidValue;  // (the gates' place)
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(tc_cell_pair_kernel<MODE, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int rows = EPI == TC_EPI_LSTM ? (p.N + 31) / 32 * 128 : p.N;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((rows + 255) / 256 * 2, (p.M + nb - 1) / nb, n);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;  // all of it: no other kernel's CTAs share the SM (tc_vocab_pair.cu)
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_pdl_on ? 1 : 0;
  count_launch();
  return cudaLaunchKernelEx(&cfg, tc_cell_pair_kernel<MODE, EPI>, b, stages);
}

}  // namespace

int cell_pair_kbs(int mode) { return mode_split(mode) ? 1 : 2; }

cudaError_t launch_tc_cell_pair(const ChainBatch& b, int n, int mode, int epi, cudaStream_t st) {
  if (epi == TC_EPI_LSTM) {
    if (mode == TC_BF16) return launch_t<TC_BF16, TC_EPI_LSTM>(b, n, st);
    if (mode == TC_TF32) return launch_t<TC_TF32, TC_EPI_LSTM>(b, n, st);
    if (mode == TC_TF32X3) return launch_t<TC_TF32X3, TC_EPI_LSTM>(b, n, st);
    if (mode == TC_F16X2) return launch_t<TC_F16X2, TC_EPI_LSTM>(b, n, st);
  } else if (epi == TC_EPI_STORE) {
    if (mode == TC_BF16) return launch_t<TC_BF16, TC_EPI_STORE>(b, n, st);
    if (mode == TC_TF32) return launch_t<TC_TF32, TC_EPI_STORE>(b, n, st);
    if (mode == TC_TF32X3) return launch_t<TC_TF32X3, TC_EPI_STORE>(b, n, st);
    if (mode == TC_F16X2) return launch_t<TC_F16X2, TC_EPI_STORE>(b, n, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace zrnn
