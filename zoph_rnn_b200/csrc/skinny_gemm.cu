// Matrix products with few batch columns on warp-level tensor-core instructions.
//
// The tcgen05 kernels (tc_gemm.cu) work on 128-row weight tiles and split K over a thread-block cluster to fill the SMs; with
// few columns their time is the fixed cost of that: pipeline fill through one 64 KB stage after another, two cluster
// barriers, the exchange of partial tiles.  Here a CTA takes MT tiles of 16 weight rows over the whole K axis: H = 1000
// gives 125 CTAs of 32 rows without splitting K between CTAs.  Its eight warps split the K axis among themselves (warp w
// takes the 32-element chunks w, w + 8, ...), each warp streams its weights and activations through a private ring in
// shared memory with 16-byte asynchronous copies, and the eight partial tiles meet in shared memory once, at the end.
// Every lane copies exactly the 16-byte pieces that it will feed to its own mma fragments, so the ring needs no barrier:
// K may be permuted inside a chunk as long as both operands agree, so lane (g, q) takes the contiguous elements
// 8q .. 8q+7 of row (column) g.  The weights of the first stages are requested before the predecessor kernel has
// finished (they do not depend on it).
//
// SK_F16X2 keeps the split engines' arithmetic: hi * hi plus 2^-11 (lo * hi + hi * lo) with fp32 accumulation.  The products
// of a chunk (two k16 steps) are summed by the tensor core and then added to the running sums with ordinary fp32 adds,
// so the tensor core's truncating accumulator never absorbs more than four products in a row.
#include "skinny_gemm.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "att_device.cuh"
#include "kernels.cuh"
#include "tc_gemm.cuh"

namespace zrnn {
namespace {

constexpr int kWarps = 8;

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
template <int MODE>
__device__ __forceinline__ void mma16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (MODE == SK_BF16)
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the two k16 steps of a 32-element chunk: row g from u, row g + 8 from v, columns from b
template <int MODE>
__device__ __forceinline__ void mma_chunk(float* c, const uint4& u, const uint4& v, const uint4& b) {
  mma16816<MODE>(c, u.x, v.x, u.y, v.y, b.x, b.y);
  mma16816<MODE>(c, u.z, v.z, u.w, v.w, b.z, b.w);
}
template <int MODE>
__device__ __forceinline__ float sk_tanh(float x) {
  if (MODE == SK_F16X2) return tanh_f32(x);
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <int MODE>
__device__ __forceinline__ float sk_sigmoid(float x) {
  if (MODE == SK_F16X2) return sigmoid_f32(x);
  return fmaf(0.5f, sk_tanh<MODE>(0.5f * x), 0.5f);
}
template <int MODE>
__device__ __forceinline__ void sk_store_op(const SkinnyParams& p, size_t at, float v) {
  if (!p.op_hi) return;
  if (MODE == SK_BF16) {
    reinterpret_cast<__nv_bfloat16*>(p.op_hi)[at] = __float2bfloat16(v);
  } else {
    const __half h = __float2half_rn(v);
    reinterpret_cast<__half*>(p.op_hi)[at] = h;
    reinterpret_cast<__half*>(p.op_lo)[at] = __float2half_rn((v - __half2float(h)) * 2048.0f);
  }
}

// zeros in elements [n, ld_op) of operand row `row`
__device__ __forceinline__ void sk_zero_pad(const SkinnyParams& p, int row, int n) {
  if (!p.op_hi) return;
  for (int i = n; i < p.ld_op; i += 4) {
    const size_t at = (size_t)row * p.ld_op + i;
    *reinterpret_cast<uint2*>((char*)p.op_hi + 2 * at) = make_uint2(0u, 0u);
    if (p.op_lo) *reinterpret_cast<uint2*>((char*)p.op_lo + 2 * at) = make_uint2(0u, 0u);
  }
}

// floats between two rows of a partial tile: 8-byte stores of the accumulator fragments and the epilogue's reads (four rows
// of one gate at a time) both spread over the banks when it is an odd multiple of 8
__host__ __device__ constexpr int part_ld(int NT) { return (NT & 1) ? 8 * NT : 8 * NT + 8; }
__host__ __device__ constexpr int parts_of(int mode) { return mode == SK_F16X2 ? 2 : 1; }
// bytes of one warp's ring stage: its weight and activation pieces of one chunk
__host__ __device__ constexpr int warp_stage(int MT, int NT, int mode) {
  return (2 * MT + NT) * parts_of(mode) * 512;
}
__host__ __device__ constexpr int warp_part_bytes(int MT, int NT) { return MT * 16 * part_ld(NT) * 4; }
__device__ __forceinline__ void cp16z(uint32_t dst, const void* src, int bytes) {  // the rest of the 16 bytes is zeroed
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <int MT, int NT, int MODE, int EPI>
__global__ void __launch_bounds__(kWarps * 32, (MT * NT <= 4) ? 2 : 1)
    skinny_kernel(const __grid_constant__ SkinnyBatch pb, int PD) {
  constexpr int P = parts_of(MODE);
  constexpr int STAGE = warp_stage(MT, NT, MODE);
  constexpr int LD = part_ld(NT), NC = 8 * NT;
  extern __shared__ __align__(16) unsigned char sk_smem[];
  const SkinnyParams& p = pb.p[blockIdx.z];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int n_tiles = EPI == SK_EPI_LSTM ? (p.N + 3) >> 2 : (p.N + 15) >> 4;
  const int tile0 = blockIdx.x * MT, col0 = blockIdx.y * NC;
  const int region = PD * STAGE > warp_part_bytes(MT, NT) ? PD * STAGE : warp_part_bytes(MT, NT);
  unsigned char* mine = sk_smem + (size_t)warp * region;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(mine) + lane * 16;

  // byte offset of this lane's row g inside the weights, per tile (row g + 8 lies `row8` bytes further)
  size_t wrow[MT];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    int t = tile0 + mt;
    if (t >= n_tiles) t = n_tiles - 1;  // computed and dropped
    int pt, r;
    if (EPI == SK_EPI_LSTM) {
      pt = t >> 3;
      r = (g >> 2) * 32 + (t & 7) * 4 + (g & 3);
    } else {
      pt = t >> 3;
      r = (t & 7) * 16 + g;
    }
    wrow[mt] = (size_t)pt * p.w_tile_bytes + (size_t)r * p.w_row_bytes + q * 16;
  }
  const size_t row8 = (size_t)(EPI == SK_EPI_LSTM ? 64 : 8) * p.w_row_bytes;
  const int cps = (p.K + 31) >> 5, chunks = p.nsrc * cps;
  const int n_my = chunks > warp ? (chunks - warp + kWarps - 1) / kWarps : 0;

  auto load_w = [&](int i, int slot) {
    const int c = warp + i * kWarps;
    const int s = c >= 2 * cps ? 2 : (c >= cps ? 1 : 0), cc = c - s * cps;
    const size_t koff = (size_t)(p.a_kb0[s] + (cc >> 1)) * p.w_kb_bytes + (cc & 1) * 64;
    uint32_t d = ring + slot * STAGE;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const size_t o = wrow[mt] + koff;
      cp16(d, (const char*)p.w_hi + o);
      if (P == 2) cp16(d + 512, (const char*)p.w_lo + o);
      cp16(d + P * 512, (const char*)p.w_hi + o + row8);
      if (P == 2) cp16(d + P * 512 + 512, (const char*)p.w_lo + o + row8);
      d += 2 * P * 512;
    }
  };
  auto load_a = [&](int i, int slot) {
    const int c = warp + i * kWarps;
    const int s = c >= 2 * cps ? 2 : (c >= cps ? 1 : 0), cc = c - s * cps;
    const int k = cc * 32 + q * 8;
    uint32_t d = ring + slot * STAGE + 2 * MT * P * 512;
    const int left = p.K - k;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int col = col0 + nt * 8 + g;
      const bool in = col < p.M;  // missing columns are zeros: reading a stand-in would make every SM poll the same few lines
      // what an operand row holds beyond K may be anything
      const int bytes = !in ? 0 : (left >= 8 ? 16 : (left > 0 ? 2 * left : 0));
      const size_t o = bytes ? ((size_t)col * p.lda + k) * 2 : 0;
      cp16z(d, (const char*)p.a_hi[s] + o, bytes);
      if (P == 2) cp16z(d + 512, (const char*)p.a_lo[s] + o, bytes);
      d += P * 512;
    }
  };

  // The weights of the first stages do not depend on the predecessor kernel, and the chunks of the early sources were complete
  // when it passed its own wait: this warp works on them (its first n_e) until it needs the predecessor's results.  The successor
  // may start after that, so that what it reads early is complete in its turn.
  const int early = p.n_early * cps, n_e = early > warp ? (early - warp + kWarps - 1) / kWarps : 0;
  bool waited = false;
  auto wait_for = [&](int i) {
    if (waited || i < n_e) return;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    waited = true;
  };
  const int pre = n_my < PD ? n_my : PD;
  for (int i = 0; i < pre; ++i) load_w(i, i);
  for (int i = 0; i < PD; ++i) {
    if (i < n_my) {
      wait_for(i);
      load_a(i, i);
    }
    cp_commit();
  }
  float acc[MT][NT][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[mt][nt][e] = 0.f;

  int slot = 0;
  for (int i = 0; i < n_my; ++i) {
    // the groups complete in order: all but the PD - 1 youngest covers chunk i
    switch (PD) {
      case 1: cp_wait<0>(); break;
      case 2: cp_wait<1>(); break;
      case 3: cp_wait<2>(); break;
      case 4: cp_wait<3>(); break;
      case 5: cp_wait<4>(); break;
      default: cp_wait<5>(); break;
    }
    const uint32_t d = ring + slot * STAGE;
    uint4 w[MT][2][P];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int x = 0; x < P; ++x) w[mt][h][x] = lds128(d + ((mt * 2 + h) * P + x) * 512);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const uint32_t da = d + (2 * MT + nt) * P * 512;
      const uint4 b_hi = lds128(da), b_lo = P == 2 ? lds128(da + 512) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        if (MODE == SK_BF16) {
          mma_chunk<MODE>(acc[mt][nt], w[mt][0][0], w[mt][1][0], b_hi);
        } else {
          float m4[4] = {0.f, 0.f, 0.f, 0.f}, x4[4] = {0.f, 0.f, 0.f, 0.f};
          mma_chunk<MODE>(m4, w[mt][0][0], w[mt][1][0], b_hi);
          mma_chunk<MODE>(x4, w[mt][0][P - 1], w[mt][1][P - 1], b_hi);
          mma_chunk<MODE>(x4, w[mt][0][0], w[mt][1][0], b_lo);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[mt][nt][e] += fmaf(x4[e], 1.0f / 2048.0f, m4[e]);
        }
      }
    }
    if (i + PD < n_my) {
      load_w(i + PD, slot);
      wait_for(i + PD);
      load_a(i + PD, slot);
    }
    cp_commit();
    if (++slot == PD) slot = 0;
  }

  wait_for(n_e);
  // the cell's other inputs, requested while the partial tiles are put down
  constexpr int OUT = EPI == SK_EPI_LSTM ? MT * 4 * NC : MT * 16 * NC;
  constexpr int EPT = (OUT + kWarps * 32 - 1) / (kWarps * 32);
  float pre_c[EPT], pre_m[EPT];
#pragma unroll
  for (int u = 0; u < EPT; ++u) {
    const int e = tid + u * kWarps * 32;
    pre_c[u] = 0.f;
    pre_m[u] = 1.f;
    if (e < OUT) {
      constexpr int R = EPI == SK_EPI_LSTM ? MT * 4 : MT * 16;
      const int row = (EPI == SK_EPI_LSTM ? tile0 * 4 : tile0 * 16) + e % R, col = col0 + e / R;
      if (row < p.N && col < p.M) {
        if (EPI == SK_EPI_LSTM) pre_c[u] = p.c_prev[(size_t)col * p.N + row];
        if (p.mask) pre_m[u] = (float)p.mask[col];
      }
    }
  }
  float* part = reinterpret_cast<float*>(mine);
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      float* d = part + (mt * 16 + g) * LD + nt * 8 + 2 * q;
      *reinterpret_cast<float2*>(d) = make_float2(acc[mt][nt][0], acc[mt][nt][1]);
      *reinterpret_cast<float2*>(d + 8 * LD) = make_float2(acc[mt][nt][2], acc[mt][nt][3]);
    }
  __syncthreads();
  const size_t rstep = (size_t)region / 4;
  const float* base = reinterpret_cast<const float*>(sk_smem);
  auto total = [&](int r, int c) {  // the eight warps' shares in a fixed order
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v += base[w * rstep + r * LD + c];
    return v;
  };
  // the operand rows' padding is read by the next product: the last row group keeps it at zero
  if (blockIdx.x == gridDim.x - 1 && tid < NC && col0 + tid < p.M) sk_zero_pad(p, col0 + tid, p.N);
#pragma unroll
  for (int u = 0; u < EPT; ++u) {
    const int e = tid + u * kWarps * 32;
    if (e >= OUT) break;
    if (EPI == SK_EPI_LSTM) {
      const int hl = e % (MT * 4), c = e / (MT * 4), hid = tile0 * 4 + hl, col = col0 + c;
      if (hid >= p.N || col >= p.M) continue;
      const int r = (hl >> 2) * 16 + (hl & 3);
      const float gi = sk_sigmoid<MODE>(total(r, c) + p.bias[hid]);
      const float gf = sk_sigmoid<MODE>(total(r + 4, c) + p.bias[p.N + hid]);
      const float gg = sk_tanh<MODE>(total(r + 8, c) + p.bias[2 * p.N + hid]);
      const float go = sk_sigmoid<MODE>(total(r + 12, c) + p.bias[3 * p.N + hid]);
      const float cn = gf * pre_c[u] + gi * gg;
      const float h = go * sk_tanh<MODE>(cn) * pre_m[u];
      p.c_out[(size_t)col * p.N + hid] = cn * pre_m[u];
      if (p.C) p.C[(size_t)col * p.ldc + hid] = h;
      sk_store_op<MODE>(p, (size_t)col * p.ld_op + hid, h);
    } else {
      const int rl = e % (MT * 16), c = e / (MT * 16), row = tile0 * 16 + rl, col = col0 + c;
      if (row >= p.N || col >= p.M) continue;
      float v = total(rl, c) + (p.bias ? p.bias[row] : 0.f);
      if (p.act == 1 && (p.act_rows == 0 || row < p.act_rows)) v = sk_tanh<MODE>(v);
      v *= pre_m[u];
      if (p.C) p.C[(size_t)col * p.ldc + row] = v;
      sk_store_op<MODE>(p, (size_t)col * p.ld_op + row, v);
    }
  }
}

const bool g_pdl = std::getenv("ZRNN_NO_PDL") == nullptr;

template <int MT, int NT, int MODE, int EPI>
cudaError_t launch_t(const SkinnyBatch& b, int n, cudaStream_t st) {
  constexpr int STAGE = warp_stage(MT, NT, MODE);
  const SkinnyParams& p = b.p[0];
  const int tiles = EPI == SK_EPI_LSTM ? (p.N + 3) / 4 : (p.N + 15) / 16;
  const int chunks = p.nsrc * ((p.K + 31) / 32), per_warp = (chunks + kWarps - 1) / kWarps;
  // ring depth: two CTAs per SM where two stages each fit half of the shared memory, else one CTA with what fits.  A cell without
  // early operands (the first of a beam step) has nothing to do beside its predecessor, so it takes the SM for a deeper ring
  // (3 x 1000 x 4000 weights, 12 columns: 16.0 -> 11.5 us; the next cell, which then starts later, 8.7 -> 12.6, a step 2 us less)
  const bool shared = 2 * kWarps * STAGE <= 110 * 1024 && MT * NT <= 4 && !(EPI == SK_EPI_LSTM && p.n_early == 0);
  const int budget = shared ? 110 * 1024 : 220 * 1024;
  int PD = budget / (kWarps * STAGE);
  PD = PD > 6 ? 6 : PD;
  PD = PD > per_warp ? per_warp : PD;
  if (PD < 1) PD = 1;
  const int region = PD * STAGE > warp_part_bytes(MT, NT) ? PD * STAGE : warp_part_bytes(MT, NT);
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(skinny_kernel<MT, NT, MODE, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         227 * 1024);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((tiles + MT - 1) / MT, (p.M + 8 * NT - 1) / (8 * NT), n);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.dynamicSmemBytes = (size_t)kWarps * region;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_pdl ? 1 : 0;
  count_launch();
  return cudaLaunchKernelEx(&cfg, skinny_kernel<MT, NT, MODE, EPI>, b, PD);
}
template <int NT, int MODE, int EPI>
cudaError_t launch_mt(const SkinnyBatch& b, int n, int mt, cudaStream_t st) {
  if (mt <= 1) return launch_t<1, NT, MODE, EPI>(b, n, st);
  if (mt == 2) return launch_t<2, NT, MODE, EPI>(b, n, st);
  return launch_t<4, NT, MODE, EPI>(b, n, st);
}
template <int MODE, int EPI>
cudaError_t launch_nt(const SkinnyBatch& b, int n, int mt, int nt, cudaStream_t st) {
  switch (nt) {
    case 1: return launch_mt<1, MODE, EPI>(b, n, mt, st);
    case 2: return launch_mt<2, MODE, EPI>(b, n, mt, st);
    case 3: return launch_mt<3, MODE, EPI>(b, n, mt, st);
    case 4: return launch_mt<4, MODE, EPI>(b, n, mt, st);
    case 5: case 6: return launch_mt<6, MODE, EPI>(b, n, mt, st);
  }
  return launch_mt<8, MODE, EPI>(b, n, mt, st);
}

}  // namespace

// Fitted, with the constants of plan_chain, to scoring passes in which every kernel and tile was taken for one kind of link after the other
// (1 - 4 x 256 - 1000 units, 1 - 256 columns, f32, bf16 and 3xTF32): the choices cost 0.15 us per launch more than the best ones.
// A cell with early operands starts beside its predecessor, but then holds up the next one's start (1.65 and 0.5 us); products of the attention
// take 0.9 and 0.5 us more.  (From two column groups on every weight is read twice: not offered.)
float skinny_us(int mode, int epi, int rows, int K, int cols, int n, bool early) {
  const float mw = (float)rows * K * n * 1e-6f, nt = (float)((cols + 7) / 8);
  const bool cell = epi == SK_EPI_LSTM;
  if (mode == SK_F16X2) return 3.1f + (cell ? (early ? 1.65f : 0.f) : 0.9f) + mw * (0.105f + nt * (0.195f + 0.025f * nt));
  return 3.15f + (cell ? (early ? 0.5f : 0.f) : 0.5f) + mw * (0.09f + 0.105f * nt);
}

// An accumulator of this kernel absorbs 2 k-steps, one of the links 4 or 8, and a cell of 600 units is 1.30e-7 from float64 here and 1.65e-7 there;
// log-probabilities of 1 x 1024 units, 30 columns 1.36e-6 with the combiner here and 1.54e-6 with it there.  Time alone does not decide, then: the
// links take over from the number of columns on at which this kernel's time reaches what a link took while one thread issued its MMAs
// (this estimate), up to 2 us more than one takes now.
bool skinny_more_exact(int epi, int rows, int cells, int nsrc, int H, int n_early, int cols) {
  const float mw = (float)rows * H * nsrc * cells * 1e-6f, nt = (float)((cols + 7) / 8);
  const float here = 4.0f + mw * (0.285f + nt * (0.144f + 0.0114f * nt));
  const int kb = (H + 63) / 64, a_rows = (cols + 7) / 8 * 8, sms = device_sms();
  for (int BN = epi == SK_EPI_LSTM ? 32 : 16; BN <= 128; BN *= 2)
    for (int split = 1; split <= 2; ++split) {
      if (split > 1 && (cells > 1 || BN > 64 || kb < 2 * split)) continue;
      const int waves = (cells * ((rows + BN - 1) / BN) * split + sms - 1) / sms;
      const float mma = BN <= 64 ? 4.f * (std::max(45, BN) + 45) : 6.f * BN, reads = BN <= 64 ? 4.f * (8192 + 96 * BN) : 12.f * (4096 + 32 * BN);
      const float writes = 256.f * (a_rows + BN), kb_us = std::max(writes / 77e3f, std::max(mma, (reads + writes) / 128.f) / 1900.f);
      const float kbs = kb * (nsrc - (BN <= 64 ? 0.5f * n_early : 0.f)) / split;
      if (here >= 3.2f + waves * (kb_us * kbs + 0.01f * BN / split) + (split == 2 ? 1.3f : 0.f)) return false;
    }
  return true;
}

cudaError_t launch_skinny(const SkinnyBatch& b, int n, int mode, int epi, cudaStream_t st) {
  const SkinnyParams& p = b.p[0];
  if (n < 1 || n > SkinnyBatch::MAX || p.M < 1 || p.N < 1 || p.nsrc < 1 || p.nsrc > 3 || p.n_early < 0 || p.n_early >= p.nsrc || (p.K & 3)) return cudaErrorInvalidValue;
  for (int i = 1; i < n; ++i)
    if (b.p[i].N != p.N || b.p[i].K != p.K || b.p[i].M != p.M || b.p[i].nsrc != p.nsrc) return cudaErrorInvalidValue;
  const int tiles = n * (epi == SK_EPI_LSTM ? (p.N + 3) / 4 : (p.N + 15) / 16);
  const int groups = (p.M + 63) / 64, nt = (p.M + groups * 8 - 1) / (groups * 8);
  // as few row tiles per CTA as keep the launch at one CTA per SM: the activations are read once per CTA
  const int mt = tiles <= 148 ? 1 : (tiles <= 296 ? 2 : 4);
  if (mode == SK_F16X2)
    return epi == SK_EPI_LSTM ? launch_nt<SK_F16X2, SK_EPI_LSTM>(b, n, mt, nt, st) : launch_nt<SK_F16X2, SK_EPI_STORE>(b, n, mt, nt, st);
  if (mode == SK_BF16)
    return epi == SK_EPI_LSTM ? launch_nt<SK_BF16, SK_EPI_LSTM>(b, n, mt, nt, st) : launch_nt<SK_BF16, SK_EPI_STORE>(b, n, mt, nt, st);
  return cudaErrorInvalidValue;
}

}  // namespace zrnn
