// tcgen05 kernel for the links of the recurrent chain whose tiles are narrow: 128 batch rows x BN = 16 .. 64 weight rows, the K
// axis over SPLIT = 1, 2 or (attention products of the split modes) 4 CTAs of a cluster (LSTM cells, attention projections, combiner; wide tiles: tc_chain.cu).
//
// A link spends 4 - 5 us on launch, barrier and TMEM set-up, the first loads, exchange and epilogue, and the rest on its MMAs: one
// takes some 60 cycles to issue and to run, however few its rows, so a k-block of 128 x 64 in the split modes (8 MMAs) 512 at best.
//
// Half an SM per CTA - 113 KB of shared memory, 256 TMEM columns, 384 threads x 80 registers: the next link's CTAs are resident while
// this one runs, and a link multiplies what it already can before its predecessor has finished: the weights against the sources
// that were complete earlier (n_early: the recurrent input of a cell, the hidden state in the combiner), which are half of the work.
// Only the rest, the exchange and the epilogue are left for the time after the predecessor's end.  Kernels on the chain let their
// successor start only after their own griddepcontrol.wait has returned: everything up to the predecessor's predecessor is then complete.
//
// A whole SM per CTA (WHOLE: cells of the split modes, and launches of several cells): with all 512 TMEM columns each MMA warp has two
// accumulator sets, so that it need not wait for a round to be added up, and a CTA's MMAs have the tensor core to themselves: 0.36 us
// per k-block against 0.51.  That is worth more than the overlap (us per link in a scoring pass, 2 x 1000 units, 64 columns 13.7 ->
// 10.2; 4 x 1000, 128 columns 13.4 -> 11.2; a pass 4693 -> 4378 and 6921 -> 6662), unless other streams' links run beside (two models
// of an ensemble: a search 3806 -> 4008), and it is worth nothing in bf16, which adds up no rounds (3138 / 3150).
//
// Warps: 0 - 7 epilogue (warp w reads TMEM lane quadrant w % 4 and takes column group w / 4 of the tile), 8 activation loads,
// 9 weight loads, 10 and 11 issue MMAs, each into accumulators of its own, so that the wait for a stage and the commit of one overlap
// the other's MMAs.
//
// Not better: the successor's start put off to the end of this link's loads (f32 cells 13.9 -> 16.5); one MMA warp with two sets in turn
// (3 x 500, 50 columns 1036 -> 1336 us a pass).  Four CTAs per tile (STORE): half the k-blocks of the narrower tile that two CTAs
// would need for as many CTAs, for an exchange of 12 KB instead of 4 KB; combiner of 1000 units, 64 columns 6.6 -> 5.2 us, 128 columns
// 8.3 -> 7.1.
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "kernels.cuh"
#include "tc_chain.cuh"
#include "tc_chain_device.cuh"

namespace zrnn {
namespace {

constexpr int kEpiWarps = 8, kAWarp = 8, kWWarp = 9, kMmaWarp = 10, kMmaWarps = 2, kThreads = 384;
constexpr int kHalfSm = 113 * 1024;  // two CTAs per SM: (228 KB - 2 x 1 KB) / 2
constexpr int kWholeSm = 224 * 1024;
static_assert(fills_sm(kWholeSm), "CTAs of split tiles with all of the tensor memory are alone on their SMs");
constexpr int kMaxStages = 8;
// The tensor core's fp32 accumulator truncates, so in the split modes it is not asked to absorb many products in a row: the K axis
// is walked in rounds of round_kb k-blocks (half of them each MMA warp's), and the epilogue warps add each finished round to sums
// of their own in registers (round to nearest).  Up to 512 elements per source (8 k-blocks of fp16, 16 of tf32) an accumulator absorbs
// 4 k-steps, beyond that 8.  Hidden states of a scoring pass against float64 (uniform weights +-0.08, fp16 split), 16 / 8 / 4 k-steps:
// 2 layers x 512, 100 columns 5.5 / 3.2 / 2.1e-7, 1 x 1024, 30 columns 6.1 / 3.4 / 2.3e-7, 4 x 1000, 64 columns 15 / 9.6 / 7.5e-7.
// Every round costs a commit, a wait and a drain: a launch of three cells of 500 units and 50 columns takes 1.2 us longer in 4 k-steps
// than in 16, a target step of 2 x 1000, 64 columns in 8 k-steps 2 % longer than in 16.
__host__ __device__ constexpr int round_kb(int mode, int kb) { return kb <= (mode == TC_TF32X3 ? 16 : 8) ? 2 : 4; }
// Split modes multiply A_hi by the stacked [W_hi ; W_lo] rows, one MMA of twice the columns for two products (an MMA of 128 rows takes some 60
// cycles to issue and to run up to 64 columns, 64 at 128), and A_lo by W_hi: two MMAs per k-step instead of three.
__host__ __device__ constexpr int set_cols(int BN, int mode) { return mode_split(mode) ? 2 * BN : BN; }  // one accumulator set per MMA warp
// sets that an MMA warp takes in turn, one being added up while the next fills: where the CTA's columns hold them (half an SM: 256).  tf32 adds up
// no rounds, but a tile of one CTA has four accumulators, a quarter of the K axis each, like the two CTAs of a split one (256 and 320
// units, 64 - 500 columns: with two 0.03 % farther from float64; in bf16 the sixth digit of that distance is the same).
__host__ __device__ constexpr int set_bufs(int BN, int mode, bool whole_sm, int split) {
  return (mode_split(mode) && (BN <= 32 || whole_sm)) || (mode == TC_TF32 && split == 1) ? 2 : 1;
}
__host__ __device__ constexpr int link_tmem(int BN, int mode, bool whole_sm, int split) {
  int c = 32;
  while (c < kMmaWarps * set_bufs(BN, mode, whole_sm, split) * set_cols(BN, mode)) c *= 2;
  return c;
}
// outputs per row and epilogue warp (LSTM: hidden units); a CTA finishes 1 / SPLIT of them
__host__ __device__ constexpr int per_warp(int BN, int epi) { return epi == TC_EPI_LSTM ? BN / 8 : BN / 2; }
__host__ __device__ constexpr int slot_bytes(int BN, int epi, int split) {  // what the other CTAs of the cluster send
  return split == 1 ? 0 : (split - 1) * kEpiWarps * 32 * (per_warp(BN, epi) / split) * (epi == TC_EPI_LSTM ? 4 : 1) * 4;
}
// Of the first n stages that go round a ring of `stages` slots, how many lie in the slots of MMA warp mw: the even or the odd ones.
// Every slot's barriers have one waiter only: with two, one that is a round ahead could mistake "the round before last is
// complete" for its own round.
__device__ __forceinline__ int own_stages(int mw, int n, int stages) {
  return n / stages * ((stages + 1 - mw) / 2) + (n % stages + 1 - mw) / 2;
}
struct LinkCtrl {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t accum;                               // everything accumulated (modes without rounds)
  uint64_t set_full[2 * kMmaWarps], set_empty[2 * kMmaWarps];
  uint64_t xchg[kEpiWarps];                     // the other CTAs' shares for this warp have arrived
  uint32_t tmem_base;
  int abort;
  float bias[64];
};

template <int BN, int MODE, int EPI, int SPLIT, bool WHOLE>
__device__ __forceinline__ void link_body(const ChainParams& p, const int m_block, const int stages) {
  constexpr bool SPLIT_MODE = mode_split(MODE), ROUNDS = SPLIT_MODE;
  constexpr int PARTS = SPLIT_MODE ? 2 : 1;
  constexpr int WKB = BN * 128;  // bytes of one k-block of one weight part
  constexpr int SETC = set_cols(BN, MODE), NB = set_bufs(BN, MODE, WHOLE, SPLIT), TMEM_COLS = link_tmem(BN, MODE, WHOLE, SPLIT);
  constexpr uint32_t IDESC = make_idesc(mode_fmt(MODE), BN), IDESC2 = make_idesc(mode_fmt(MODE), SETC);
  extern __shared__ __align__(1024) uint8_t link_smem[];
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int m0 = m_block * 128, n_tile = blockIdx.y;
  const int akb = p.a_rows * 128;  // bytes of one k-block of one activation part
  const int KBS = p.kbs;
  const int stage_bytes = PARTS * KBS * (akb + WKB);  // KBS x [A hi][A lo], KBS x [W hi][W lo]
  uint8_t* tiles = link_smem;
  uint8_t* slots = tiles + (size_t)stages * stage_bytes + (128 - p.a_rows) * 128;
  LinkCtrl& ct = *reinterpret_cast<LinkCtrl*>(slots + slot_bytes(BN, EPI, SPLIT));
  const int rank = SPLIT > 1 ? (int)blockIdx.z : 0;
  // this CTA's stages: the same part of every source's K axis, source after source
  const int src_it = (p.kb + KBS - 1) / KBS, c_lo = src_it * rank / SPLIT, n_src = src_it * (rank + 1) / SPLIT - c_lo;
  const int n_it = p.nsrc * n_src, n_early = p.n_early * n_src;
  ZR_STAMP(0);
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ct.full[s], 2);  // the activation and the weight producer
      mbar_init(&ct.empty[s], 1);
    }
    mbar_init(&ct.accum, kMmaWarps);
    for (int i = 0; i < kMmaWarps * NB; ++i) {
      mbar_init(&ct.set_full[i], 1);
      mbar_init(&ct.set_empty[i], kEpiWarps);
    }
    if (SPLIT > 1)
      for (int i = 0; i < kEpiWarps; ++i) {
        mbar_init(&ct.xchg[i], 1);
        mbar_expect_tx(&ct.xchg[i], (uint32_t)(slot_bytes(BN, EPI, SPLIT) / kEpiWarps));
      }
    ct.abort = (smem_u32(link_smem) & 1023) ? 1 : 0;  // (the swizzled tiles need the alignment that the declaration asks for)
    if (ct.abort && p.err) atomicExch(p.err, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ct.tmem_base)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (SPLIT > 1) cluster_arrive();  // (the barriers above are ready; waited for before the first remote store)
  const uint32_t tmem_base = ct.tmem_base;
  const bool sound = __all_sync(0xffffffffu, ct.abort == 0);
  ZR_STAMP(1);

  if (warp == kWWarp) {
    // ------------------------------------------------------------ weights: nothing here depends on the predecessor
    if (sound) {
      const bool one = elect_one();
      bool ok = true;
      int st = 0, s = 0, c = 0;
      uint32_t ph = 0;
      for (int it = 0; it < n_it; ++it) {
        if (it >= stages && !mbar_wait_warp(&ct.empty[st], ph ^ 1u, &ct.abort, p.err, 1)) { ok = false; break; }
        uint8_t* w = tiles + (size_t)st * stage_bytes + PARTS * KBS * akb;
        const int wkb = p.wkb0[s] + (c_lo + c) * KBS;
        if (one) {
          mbar_expect_tx(&ct.full[st], (uint32_t)(PARTS * KBS * WKB));
          if constexpr (EPI == TC_EPI_LSTM) {
            constexpr int TH = BN / 4;
            tma_load_5d(w, &p.w, &ct.full[st], n_tile * TH % 32, 0, (n_tile * TH / 32) * p.w_kbtot + wkb);
          } else {
            tma_load_4d(w, &p.w, &ct.full[st], n_tile * BN, wkb);
          }
        }
        __syncwarp();
        if (++st == stages) { st = 0; ph ^= 1u; }
        if (++c == n_src) { c = 0; ++s; }
      }
      if (!ok) settle_copies();
    }
  } else if (warp == kAWarp) {
    // ------------------------------------------------------------ activations: the early sources before the predecessor's end
    {
      const bool one = elect_one();
      bool ok = sound;
      int st = 0, s = 0, c = 0;
      uint32_t ph = 0;
      for (int it = 0; it < n_it && ok; ++it) {
        if (it == n_early) {
          pdl_wait();
          pdl_trigger();
        }
        if (it >= stages && !mbar_wait_warp(&ct.empty[st], ph ^ 1u, &ct.abort, p.err, 7)) { ok = false; break; }
        if (one) {
          mbar_expect_tx(&ct.full[st], (uint32_t)(PARTS * KBS * akb));
          tma_load_4d(tiles + (size_t)st * stage_bytes, &p.a[s], &ct.full[st], p.a_row0[s] + m0, (c_lo + c) * KBS);
        }
        __syncwarp();
        if (++st == stages) { st = 0; ph ^= 1u; }
        if (++c == n_src) { c = 0; ++s; }
      }
      if (sound && !ok) settle_copies();
    }
  } else if (warp >= kMmaWarp) {
    // ------------------------------------------------------------ MMA issuers
    if (sound) {
      const bool one = elect_one();
      const int mw = warp - kMmaWarp, R = round_kb(MODE, p.kb) / KBS;
      int set = mw * NB;
      int st = mw, it = mw, round_end = 0, round = 0, own = 0;
      uint32_t ph = 0;
      bool ok = true, fresh = true;
      while (it < n_it) {
        if (ROUNDS && it >= round_end) {  // first stage of this warp in a round
          set = mw * NB + round % NB;
          if (round >= NB && !mbar_wait_warp(&ct.set_empty[set], (uint32_t)(round / NB & 1) ^ 1u, &ct.abort, p.err, 4)) { ok = false; break; }
          tc_fence_after();
          fresh = true;
          round_end = (it / R + 1) * R;
          ++round;
        }
        if (!ROUNDS && NB > 1) {
          set = mw * NB + own % NB;
          fresh = own++ < NB;
        }
        if (!mbar_wait_warp(&ct.full[st], ph, &ct.abort, p.err, 2)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(tiles + (size_t)st * stage_bytes), w_addr = a_addr + PARTS * KBS * akb;
        const uint32_t d = tmem_base + (uint32_t)(set * SETC);
        if (one) {
          for (int b = 0; b < KBS; ++b) {
            const uint64_t da = make_smem_desc(a_addr + b * PARTS * akb), dal = make_smem_desc(a_addr + (b * PARTS + 1) * akb);
            const uint64_t dw = make_smem_desc(w_addr + b * PARTS * WKB);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              umma<mode_kind_tf32(MODE)>(d, da + 2 * k, dw + 2 * k, IDESC2, (!fresh || b > 0 || k > 0) ? 1u : 0u);
              if (SPLIT_MODE) umma<mode_kind_tf32(MODE)>(d + BN, dal + 2 * k, dw + 2 * k, IDESC, 1u);
            }
          }
          umma_commit(&ct.empty[st]);
        }
        __syncwarp();
        fresh = false;
        if (st + kMmaWarps < stages) {
          st += kMmaWarps;
          it += kMmaWarps;
        } else {
          it += stages - st + mw;
          st = mw;
          ph ^= 1u;
        }
        if (ROUNDS && (it >= round_end || it >= n_it) && one) umma_commit(&ct.set_full[set]);
      }
      if (ok && !ROUNDS && one) umma_commit(&ct.accum);
    }
  }
  __syncwarp();
  // ------------------------------------------------------------ epilogue
  constexpr int G = EPI == TC_EPI_LSTM ? 4 : 1;             // gates
  constexpr int PER = per_warp(BN, EPI), NF = PER / SPLIT;  // outputs per row and warp; those finished here
  constexpr int GS = EPI == TC_EPI_LSTM ? BN / 4 : 0;       // accumulator columns from one gate to the next
  if (warp < kEpiWarps) {
    const int quad = warp & 3, cg = warp >> 2;
    const int row = m0 + quad * 32 + lane;
    const int out0 = n_tile * (EPI == TC_EPI_LSTM ? BN / 4 : BN) + cg * PER + rank * NF;  // first output finished here
    float sum[G][PER], pre_c[NF];
    float mk = 1.0f;
    bool ready = sound, waited = false;
    const bool live = m0 + quad * 32 < p.M;  // whole warps: the TMEM loads are warp-wide
    const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(cg * PER);
    for (int i = threadIdx.x; i < BN; i += kEpiWarps * 32) {
      float bv = 0.f;
      if (EPI == TC_EPI_LSTM) {
        constexpr int TH = BN / 4;
        const int hid = n_tile * TH + (i % TH);
        if (hid < p.N) bv = p.bias[(i / TH) * p.N + hid];
      } else {
        const int n = n_tile * BN + i;
        if (n < p.N && p.bias) bv = p.bias[n];
      }
      ct.bias[i] = bv;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int u = 0; u < PER; ++u) sum[g][u] = 0.f;
    auto fetch_inputs = [&]() {  // the predecessor has finished: the cell's other inputs
      if (waited) return;
      waited = true;
      pdl_wait();
      if (row < p.M) {
        if (p.mask) mk = (float)p.mask[row];
        if constexpr (EPI == TC_EPI_LSTM) {
#pragma unroll
          for (int u = 0; u < NF; ++u) pre_c[u] = out0 + u < p.N ? __ldcg(p.c_prev + (size_t)row * p.N + out0 + u) : 0.f;
        }
      }
    };
    constexpr int PC = PER < 8 ? PER : 8;                        // columns per TMEM load
    constexpr int GB = SPLIT_MODE && G * PC > 16 ? 16 / PC : G;  // gates in flight (registers)
    auto drain = [&](int set) {  // adds accumulator set `set` to the sums
#pragma unroll
      for (int g0 = 0; g0 < G; g0 += GB)
#pragma unroll
        for (int u0 = 0; u0 < PER; u0 += PC) {
          float t[GB][PC], x[GB][PC];
#pragma unroll
          for (int g = 0; g < GB; ++g) {
            tmem_ldw<PC>(taddr + set * SETC + (g0 + g) * GS + u0, t[g]);
            if (SPLIT_MODE) tmem_ldw<PC>(taddr + set * SETC + BN + (g0 + g) * GS + u0, x[g]);
          }
          tmem_wait_ld();
#pragma unroll
          for (int g = 0; g < GB; ++g)
#pragma unroll
            for (int u = 0; u < PC; ++u) sum[g0 + g][u0 + u] += SPLIT_MODE ? fmaf(x[g][u], mode_cross_scale(MODE), t[g][u]) : t[g][u];
        }
    };
    if constexpr (ROUNDS) {
      const int R = round_kb(MODE, p.kb) / KBS;
      int seen[2] = {0, 0};  // rounds of each MMA warp so far (one in which it has no stage is none of its rounds)
      for (int lo = 0; ready && lo < n_it; lo += R) {
        if (lo + R > n_early) fetch_inputs();
        const int hi = lo + R < n_it ? lo + R : n_it;
#pragma unroll
        for (int mw = 0; mw < kMmaWarps; ++mw) {
          if (!ready || own_stages(mw, hi, stages) == own_stages(mw, lo, stages)) continue;
          const int set = mw * NB + seen[mw] % NB;
          ready = __all_sync(0xffffffffu, mbar_wait(&ct.set_full[set], (uint32_t)(seen[mw] / NB & 1), &ct.abort, p.err, 3));
          ++seen[mw];
          tc_fence_after();
          if (ready && live) drain(set);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ct.set_empty[set]);
        }
      }
      fetch_inputs();
    } else {
      fetch_inputs();
      if (ready) {
        ready = __all_sync(0xffffffffu, mbar_wait(&ct.accum, 0, &ct.abort, p.err, 3));
        tc_fence_after();
        if (ready && live) {
#pragma unroll
          for (int mw = 0; mw < kMmaWarps; ++mw)
#pragma unroll
            for (int b = 0; b < NB; ++b)
              if (own_stages(mw, n_it, stages) > b) drain(mw * NB + b);
        }
      }
    }
    ZR_STAMP(2);
    float fin[G][NF];
    if constexpr (SPLIT > 1) {
      __syncwarp();
      cluster_wait();
      constexpr int V4 = G * NF / 4;
      static_assert(G * NF % 4 == 0, "16-byte pieces of the exchange");
      // float4 units [sender's place among the others][warp][V4][lane]
      const uint32_t slot0 = smem_u32(slots) + (uint32_t)((warp * V4 * 32 + lane) * 16);
      constexpr uint32_t SENDER = kEpiWarps * V4 * 32 * 16;
      if (ready && live) {
#pragma unroll
        for (int q = 0; q < SPLIT; ++q) {
          float f[G * NF];
#pragma unroll
          for (int g = 0; g < G; ++g)
#pragma unroll
            for (int u = 0; u < NF; ++u) f[g * NF + u] = sum[g][q * NF + u];
          if (q == rank) {
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
              for (int u = 0; u < NF; ++u) fin[g][u] = f[g * NF + u];
          } else {
            // the bytes themselves complete the receiver's barrier: no release, whose fence cost as much as the transfer
            const uint32_t peer = cluster_map(slot0 + (uint32_t)(rank < q ? rank : rank - 1) * SENDER, (uint32_t)q);
            const uint32_t bar = cluster_map(smem_u32(&ct.xchg[warp]), (uint32_t)q);
#pragma unroll
            for (int i = 0; i < V4; ++i) st_async_v4(peer + i * 512, bar, f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
          }
        }
        ready = __all_sync(0xffffffffu, mbar_wait_cluster(&ct.xchg[warp], 0, &ct.abort, p.err, 6));
        if (ready) {
#pragma unroll
          for (int q = 0; q < SPLIT - 1; ++q)
#pragma unroll
            for (int i = 0; i < V4; ++i) {
              const float4 o = *reinterpret_cast<const float4*>(slots + q * SENDER + ((warp * V4 + i) * 32 + lane) * 16);
              const float oo[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) fin[(4 * i + e) / NF][(4 * i + e) % NF] += oo[e];
            }
        }
      }
    } else {
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int u = 0; u < NF; ++u) fin[g][u] = sum[g][u];
    }
    const int left = p.N - out0;
    if (ready && live && row < p.M && left > 0) {
      const int nvalid = left >= NF ? NF : left;
      const float* sb = ct.bias + cg * PER + rank * NF;
      float hv[NF];
      if constexpr (EPI == TC_EPI_LSTM) {
        constexpr int TH = BN / 4;
        float cv[NF];
#pragma unroll
        for (int u = 0; u < NF; ++u) {
          const float gi = act_sigmoid<MODE>(fin[0][u] + sb[u]);
          const float gf = act_sigmoid<MODE>(fin[1][u] + sb[TH + u]);
          const float gg = act_tanh<MODE>(fin[2][u] + sb[2 * TH + u]);
          const float go = act_sigmoid<MODE>(fin[3][u] + sb[3 * TH + u]);
          const float c = gf * pre_c[u] + gi * gg;
          hv[u] = go * act_tanh<MODE>(c) * mk;
          cv[u] = c * mk;
        }
        store_f32<NF>(p.c_out, (size_t)row * p.N + out0, cv, nvalid);
      } else {
#pragma unroll
        for (int u = 0; u < NF; ++u) {
          float t = fin[0][u] + sb[u];
          if (p.act == 1 && (p.act_rows == 0 || out0 + u < p.act_rows)) t = act_tanh<MODE>(t);
          hv[u] = t * mk;
        }
      }
      if (p.C) store_f32<NF>(p.C, (size_t)row * p.ldc + out0, hv, nvalid);
      store_operand<NF>(p, (size_t)row * p.ld_op + out0, hv, nvalid);
    }
    // the operand rows' padding up to a whole k-block is read by the next product: the last row tile keeps it at zero
    if (n_tile == (int)gridDim.y - 1 && row < p.M && cg == 0 && rank == 0) zero_operand_pad(p, (size_t)row * p.ld_op, p.N, p.ld_op);
    ZR_STAMP(6);
  } else if (SPLIT > 1) {
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  ZR_STAMP(7);
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS)
                 : "memory");
  }
  // In an orderly run a CTA ends after the other one's bytes have come.  One that gave up waiting (ct.abort, set by every wait that
  // gives up) may still be written to: it stays until the other one's threads have ended, or wait here as well, and what they sent
  // has landed.  (Such a barrier on every run costs 0.4 us a link.)
  if (SPLIT > 1 && ct.abort) {
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    settle_copies();
  }
}

template <int BN, int MODE, int EPI, int SPLIT>
__global__ void __launch_bounds__(kThreads, 2) tc_link_kernel(const __grid_constant__ ChainParams p, int stages) {
  link_body<BN, MODE, EPI, SPLIT, false>(p, (int)blockIdx.x, stages);
}
template <int BN, int MODE, int EPI, int SPLIT>
__global__ void __launch_bounds__(kThreads, 1) tc_link_whole_kernel(const __grid_constant__ ChainParams p, int stages) {
  link_body<BN, MODE, EPI, SPLIT, true>(p, (int)blockIdx.x, stages);
}
// Several independent problems of one row block each (M <= 128): blockIdx.x selects the problem.  The cells of one
// anti-diagonal of a stack (layer l at step t, layer l - 1 at step t + 1, ...) do not depend on one another.
template <int BN, int MODE>
__global__ void __launch_bounds__(kThreads, 1) tc_link_multi_kernel(const __grid_constant__ ChainBatch pb, int stages) {
  link_body<BN, MODE, TC_EPI_LSTM, 1, true>(pb.p[blockIdx.x], 0, stages);
}

const bool g_pdl_on = std::getenv("ZRNN_NO_PDL") == nullptr;

template <int BN, int MODE, int EPI, int SPLIT, bool WHOLE>
auto link_kernel() {
  if constexpr (WHOLE) return &tc_link_whole_kernel<BN, MODE, EPI, SPLIT>;
  else return &tc_link_kernel<BN, MODE, EPI, SPLIT>;
}
template <int BN, int MODE, int EPI, int SPLIT, bool WHOLE>
cudaError_t launch_t(const ChainBatch& b, int n, cudaStream_t st) {
  const ChainParams& p = b.p[0];
  const int stage = (mode_split(MODE) ? 2 : 1) * p.kbs * (p.a_rows + BN) * 128;
  // the MMA reads 128 rows of activations, the last stage's reads may run past a narrower box
  const int fixed = (128 - p.a_rows) * 128 + slot_bytes(BN, EPI, SPLIT) + (int)sizeof(LinkCtrl);
  const int its = (p.kb + p.kbs - 1) / p.kbs;
  if (its < SPLIT) return cudaErrorInvalidValue;
  // (a launch of several cells has no early sources: it takes the whole SM, 3 x 500, 50 columns 9.7 us a launch against 11)
  int stages = ((WHOLE ? kWholeSm : kHalfSm) - fixed) / stage;
  stages = std::min(std::min(stages, (int)kMaxStages), p.nsrc * ((its + SPLIT - 1) / SPLIT));
  if (stages < kMmaWarps) stages = kMmaWarps;  // (both MMA warps own a stage)
  // an even ring gives the MMA warps stages in turn: in an odd one a round's k-blocks may all fall to one of them, whose accumulator then
  // absorbs twice as many (500 units, 128 columns: 1.44e-7 from float64 against 1.35e-7)
  if (WHOLE && mode_split(MODE)) stages &= ~1;
  // On a whole SM a CTA of a split tile holds all of the tensor memory while it waits for its cluster partner: it asks for all of the shared
  // memory too, so that no CTA of another stream is there that holds tensor memory, and waits for some, in its turn.  (Without partners
  // it takes what it needs: the next launch's set-up beside it is worth 1.4 % of a pass of 3 x 500 units, 50 columns.)
  if ((size_t)stages * stage + fixed > kWholeSm) return cudaErrorInvalidValue;
  const size_t smem = WHOLE && SPLIT > 1 ? (size_t)kWholeSm : (size_t)stages * stage + fixed;
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(link_kernel<BN, MODE, EPI, SPLIT, WHOLE>(), cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeSm);
    if (e != cudaSuccess) return e;
    if constexpr (EPI == TC_EPI_LSTM && SPLIT == 1 && WHOLE) {
      e = cudaFuncSetAttribute(tc_link_multi_kernel<BN, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeSm);
      if (e != cudaSuccess) return e;
    }
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  const int rows = EPI == TC_EPI_LSTM ? p.N * 4 : p.N;
  cfg.gridDim = dim3(n > 1 ? n : (p.M + 127) / 128, (rows + BN - 1) / BN, SPLIT);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (SPLIT > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = SPLIT;
    ++na;
  }
  if (g_pdl_on) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  count_launch();
  if constexpr (EPI == TC_EPI_LSTM && SPLIT == 1 && WHOLE) {
    if (n > 1) return cudaLaunchKernelEx(&cfg, tc_link_multi_kernel<BN, MODE>, b, stages);
  }
  return cudaLaunchKernelEx(&cfg, link_kernel<BN, MODE, EPI, SPLIT, WHOLE>(), p, stages);
}
template <int MODE, int EPI, int SPLIT>
cudaError_t launch_bn(const ChainBatch& b, int n, int BN, bool whole, cudaStream_t st) {
  if constexpr (mode_split(MODE) || (EPI == TC_EPI_LSTM && SPLIT == 1)) {
    if (n > 1 || whole) {
      if (BN == 32) return launch_t<32, MODE, EPI, SPLIT, true>(b, n, st);
      if (BN == 64) return launch_t<64, MODE, EPI, SPLIT, true>(b, n, st);
      return cudaErrorInvalidValue;
    }
  }
  if (BN == 32) return launch_t<32, MODE, EPI, SPLIT, false>(b, n, st);
  if (BN == 64) return launch_t<64, MODE, EPI, SPLIT, false>(b, n, st);
  if constexpr (EPI == TC_EPI_STORE) {
    if constexpr (SPLIT < 4) if (BN == 16) return launch_t<16, MODE, EPI, SPLIT, false>(b, n, st);
  }
  return cudaErrorInvalidValue;
}
template <int MODE>
cudaError_t launch_mode(const ChainBatch& b, int n, int BN, int epi, int split, bool whole, cudaStream_t st) {
  if (n > 1 && split > 1) return cudaErrorInvalidValue;
  if (epi == TC_EPI_LSTM) {
    if (split == 1) return launch_bn<MODE, TC_EPI_LSTM, 1>(b, n, BN, whole, st);
    if (split == 2) return launch_bn<MODE, TC_EPI_LSTM, 2>(b, n, BN, whole, st);
  } else if (n == 1) {
    if (split == 1) return launch_bn<MODE, TC_EPI_STORE, 1>(b, n, BN, whole, st);
    if (split == 2) return launch_bn<MODE, TC_EPI_STORE, 2>(b, n, BN, whole, st);
    if constexpr (mode_split(MODE))
      if (split == 4) return launch_bn<MODE, TC_EPI_STORE, 4>(b, n, BN, whole, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

int link_kbs(int mode, int BN, int a_rows, int kb, int split) {
  const int kb_bytes = (mode_split(mode) ? 2 : 1) * (a_rows + BN) * 128;
  // k-blocks per stage: as many as leave the ring four stages and every CTA two stages of a source; a round has two stages at least,
  // one for each MMA warp
  int k = mode_split(mode) ? round_kb(mode, kb) / 2 : 4;
  const int least = mode == TC_TF32 ? 4 : 2 * split;  // (tf32: a stage for each of the four accumulators)
  while (k > 1 && (4 * k * kb_bytes > kHalfSm - 20 * 1024 - (128 - a_rows) * 128 || (kb + k - 1) / k < least)) k /= 2;
  return k;
}

cudaError_t launch_tc_link(const ChainBatch& b, int n, int BN, int mode, int epi, int split, bool whole, cudaStream_t st) {
  switch (mode) {
    case TC_BF16: return launch_mode<TC_BF16>(b, n, BN, epi, split, whole, st);
    case TC_TF32: return launch_mode<TC_TF32>(b, n, BN, epi, split, whole, st);
    case TC_TF32X3: return launch_mode<TC_TF32X3>(b, n, BN, epi, split, whole, st);
    case TC_F16X2: return launch_mode<TC_F16X2>(b, n, BN, epi, split, whole, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace zrnn
