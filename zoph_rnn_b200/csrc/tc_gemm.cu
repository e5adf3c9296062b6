// tcgen05 / TMEM / TMA product of the scoring softmax for short K (others: tc_vocab_pair.cu) and the tensor-map helpers.  See tc_gemm.cuh for the
// operand convention.  A ring of shared-memory stages is guarded by full/empty mbarriers; every wait is bounded (about a
// second of SM clock) and reports through p.err instead of spinning forever.
#include "tc_gemm.cuh"

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "kernels.cuh"
#include "tc_chain.cuh"
#include "tc_device.cuh"

namespace zrnn {
namespace {

// ------------------------------------------------------------------ persistent variant for large GEMMs
// One CTA per SM walks over output tiles (M tile fastest, so concurrently running CTAs share the same rows of B in
// L2).  The TMA producer runs ahead across tile boundaries and the accumulator is double-buffered in TMEM, so the
// epilogue of tile i overlaps the main loop of tile i+1 and the load pipe never drains.
// Warp roles: warps 0-7 run the epilogue (warp w reads TMEM lanes 32 (w % 4) .. +31, the only ones it may access, and
// the column half w / 4 of the tile), warp 8 is the TMA producer, warp 9 issues the MMAs and owns the TMEM allocation.
// Every tile therefore leaves kPersistentParts = 2 (max, sum) partials per output row, one per column half.
__host__ __device__ constexpr int persistent_stages(int BN, int mode) {
  return 192 * 1024 / stage_bytes(BN, mode);
}

template <int BN, int MODE>
__global__ void __launch_bounds__(320, 1) tc_gemm_persistent_kernel(const __grid_constant__ TcParams p, int m_tiles,
                                                                     int n_tiles) {
  constexpr int ST = persistent_stages(BN, MODE);
  constexpr int STAGE = stage_bytes(BN, MODE);
  constexpr int BBYTES = BN * 128;
  constexpr uint32_t IDESC = make_idesc(mode_fmt(MODE), BN);
  constexpr int ACC_COLS = (mode_split(MODE) ? 2 : 1) * BN;  // main accumulator (+ cross-term accumulator)
  constexpr int TMEM_COLS = 2 * ACC_COLS;                       // double-buffered
  constexpr int HC = BN / kPersistentParts;                     // columns per epilogue warp
  static_assert(ST >= 2, "need at least a double-buffered ring");
  static_assert(TMEM_COLS <= 512 && (TMEM_COLS & (TMEM_COLS - 1)) == 0, "TMEM budget");
  static_assert(HC % 32 == 0, "the epilogue works on chunks of 32 columns");
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t full_bar[ST];
  __shared__ __align__(8) uint64_t empty_bar[ST];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  // bias values of the tile whose epilogue is running (two named barriers per tile order its refill)
  __shared__ __align__(16) float s_bias[BN];

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  const int total_tiles = m_tiles * n_tiles;
  ZR_STAMP(0);
  const int kb_per_tile = p.kblocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 8);  // one arrival per epilogue warp
    }
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  pdl_wait();  // (no early trigger: with the combine's CTAs waiting beside, the smallest scoring call takes 0.8 us longer)

  if (warp == 8) {
    // ------------------------------------------------------------ TMA producer (runs ahead across tiles)
    if (kb_per_tile > 0) {
      const bool one = elect_one();
      int st = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        const int m0 = (tile % m_tiles) * 128, n0 = (tile / m_tiles) * BN;
        for (int kb = 0; kb < kb_per_tile; ++kb) {
          if (!mbar_wait_warp(&empty_bar[st], ph ^ 1u, &abort_s, p.err, 1)) { ok = false; break; }
          uint8_t* base = tiles + (size_t)st * STAGE;
          const int kx = kb * mode_epk(MODE);
          if (one) {
            mbar_expect_tx(&full_bar[st], (uint32_t)STAGE);
            tma_load_2d(base, &p.a, &full_bar[st], kx, m0);
            tma_load_2d(base + kABytes, &p.b, &full_bar[st], kx, n0);
            if (mode_split(MODE)) {
              tma_load_2d(base + kABytes + BBYTES, &p.a_lo, &full_bar[st], kx, m0);
              tma_load_2d(base + 2 * kABytes + BBYTES, &p.b_lo, &full_bar[st], kx, n0);
            }
          }
          __syncwarp();
          if (++st == ST) { st = 0; ph ^= 1u; }
        }
      }
      if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 20000000LL) {}
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------ MMA issuer
    if (kb_per_tile > 0) {
      const bool one = elect_one();
      int st = 0, ti = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++ti) {
        const int buf = ti & 1;
        // wait until the epilogue has drained this accumulator buffer (passes at once on its first use)
        if (!mbar_wait_warp(&acc_empty[buf], (uint32_t)(((ti >> 1) & 1) ^ 1), &abort_s, p.err, 4)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_main = tmem_base + (uint32_t)(buf * ACC_COLS);
        for (int kk = 0; kk < kb_per_tile; ++kk) {
          if (!mbar_wait_warp(&full_bar[st], ph, &abort_s, p.err, 2)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(tiles + (size_t)st * STAGE);
          const uint32_t b_addr = a_addr + kABytes;
          const uint64_t da = make_smem_desc(a_addr), db = make_smem_desc(b_addr);
          if (one) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t acc = (kk > 0 || k > 0) ? 1u : 0u;
              umma<mode_kind_tf32(MODE)>(d_main, da + 2 * k, db + 2 * k, IDESC, acc);
              if (mode_split(MODE)) {
                const uint64_t dal = make_smem_desc(b_addr + BBYTES), dbl = make_smem_desc(b_addr + BBYTES + kABytes);
                umma<mode_kind_tf32(MODE)>(d_main + BN, dal + 2 * k, db + 2 * k, IDESC, acc);
                umma<mode_kind_tf32(MODE)>(d_main + BN, da + 2 * k, dbl + 2 * k, IDESC, 1u);
              }
            }
            umma_commit(&empty_bar[st]);
          }
          __syncwarp();
          if (++st == ST) { st = 0; ph ^= 1u; }
        }
        if (ok && one) umma_commit(&acc_full[buf]);
      }
    }
  } else if (kb_per_tile > 0) {
    // ------------------------------------------------------------ epilogue warps 0-7
    const int q = warp & 3, half = warp >> 2;
    int ti = 0;
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++ti) {
      const int buf = ti & 1;
      const int m_tile = tile % m_tiles, n_tile = tile / m_tiles;
      const int row = m_tile * 128 + q * 32 + lane;
      const bool row_ok = row < p.M;
      asm volatile("bar.sync 1, 256;" ::: "memory");  // all epilogue threads have finished with the previous bias
      for (int i = threadIdx.x; i < BN; i += 256) {
        const int n = n_tile * BN + i;
        s_bias[i] = n < p.N ? (p.bias ? __ldg(p.bias + n) : 0.f) : -INFINITY;
      }
      if (!mbar_wait(&acc_full[buf], (uint32_t)((ti >> 1) & 1), &abort_s, p.err, 3)) break;
      tc_fence_after();
      asm volatile("bar.sync 1, 256;" ::: "memory");  // the new bias values are visible
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * ACC_COLS + half * HC);
      const int n0 = n_tile * BN + half * HC;  // first output column of this warp
      const float* sb = s_bias + half * HC;
      const size_t pi = (size_t)(n_tile * kPersistentParts + half) * p.M + row;
      const int tg = (p.target && row_ok) ? p.target[row] - p.target_offset : -1;
      float mx = -INFINITY, sm = 0.f;
      for (int c0 = 0; c0 < HC; c0 += 32) {
        float v[32];
        tmem_ld32(taddr + c0, v);
        if (mode_split(MODE)) {
          float t[32];
          tmem_ld32(taddr + BN + c0, t);
          tmem_wait_ld();
#pragma unroll
          for (int u = 0; u < 32; ++u) v[u] = fmaf(t[u], mode_cross_scale(MODE), v[u]);
        }
        tmem_wait_ld();
        float cm = -INFINITY;
#pragma unroll
        for (int u = 0; u < 32; u += 4) {
          const float4 b4 = *reinterpret_cast<const float4*>(sb + c0 + u);
          v[u] += b4.x; v[u + 1] += b4.y; v[u + 2] += b4.z; v[u + 3] += b4.w;
          cm = fmaxf(fmaxf(cm, fmaxf(v[u], v[u + 1])), fmaxf(v[u + 2], v[u + 3]));
        }
        const int rel = tg - (n0 + c0);
        if ((unsigned)rel < 32u && tg < p.N) {  // the target's logit lies in this chunk (once per row at most)
          float t = 0.f;
#pragma unroll
          for (int u = 0; u < 32; ++u)
            if (u == rel) t = v[u];
          p.tgt_logit[row] = t;
        }
        if (cm > mx) {
          sm *= expf(mx - cm);
          mx = cm;
        }
        if (mx != -INFINITY) {
          float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
          for (int u = 0; u < 32; u += 4) {
            s0 += expf(v[u] - mx); s1 += expf(v[u + 1] - mx); s2 += expf(v[u + 2] - mx); s3 += expf(v[u + 3] - mx);
          }
          sm += (s0 + s1) + (s2 + s3);
        }
      }
      if (row_ok) {
        p.part_max[pi] = mx;
        p.part_sum[pi] = sm;
      }
      // this warp's TMEM reads are complete: hand the buffer back to the MMA warp
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  ZR_STAMP(7);
  if (warp == 9) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS)
                 : "memory");
  }
}

constexpr int kMaxDevices = 64;
static int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) dev = 0;
  return dev;
}
template <int BN, int MODE>
cudaError_t launch_persistent_t(const TcParams& p, cudaStream_t st) {
  const size_t smem = (size_t)persistent_stages(BN, MODE) * stage_bytes(BN, MODE) + 1024;
  static bool configured[kMaxDevices] = {false};  // the attribute is per device
  const int dev = current_device();
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_persistent_kernel<BN, MODE>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int m_tiles = (p.M + 127) / 128, n_tiles = (p.N + BN - 1) / BN;
  const int total = m_tiles * n_tiles;
  if (total == 0) return cudaSuccess;
  const int grid = total < device_sms() ? total : device_sms();
  static const bool pdl = std::getenv("ZRNN_NO_PDL") == nullptr;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(320);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  count_launch();
  return cudaLaunchKernelEx(&cfg, tc_gemm_persistent_kernel<BN, MODE>, p, m_tiles, n_tiles);
}

}  // namespace

int device_sms() {
  static std::atomic<int> count[kMaxDevices];  // (asked by several threads at a time)
  std::atomic<int>& c = count[current_device()];
  int n = c.load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, current_device()) != cudaSuccess || n < 2) n = 148;
    c.store(n, std::memory_order_relaxed);
  }
  return n;
}

cudaError_t launch_tc_gemm_persistent(const TcParams& p, int mode, cudaStream_t st) {
  // tile widths: 256 columns for bf16 / tf32, 128 for the split modes (their second, cross-term accumulator doubles the TMEM need)
  if (mode == TC_BF16) return launch_persistent_t<256, TC_BF16>(p, st);
  if (mode == TC_TF32) return launch_persistent_t<256, TC_TF32>(p, st);
  if (mode == TC_TF32X3) return launch_persistent_t<128, TC_TF32X3>(p, st);
  if (mode == TC_F16X2) return launch_persistent_t<128, TC_F16X2>(p, st);
  return cudaErrorInvalidValue;
}

// ------------------------------------------------------------------ tensor maps
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)ptr;
  }
  return fn;
}

bool make_kmajor_map(CUtensorMap* out, const void* base, int elem_bytes, long long k, long long rows, long long ld,
                     int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn || !base || k <= 0 || rows <= 0 || box_rows <= 0 || box_rows > 256) return false;
  if (((uintptr_t)base & 15) != 0 || ((ld * elem_bytes) & 15) != 0) return false;
  cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld * elem_bytes)};
  cuuint32_t box[2] = {(cuuint32_t)(128 / elem_bytes), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  const CUtensorMapDataType dt = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  CUresult r = fn(out, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

static bool encode_map(CUtensorMap* out, const void* base, int elem_bytes, int rank, const cuuint64_t* dims,
                       const cuuint64_t* strides, const cuuint32_t* box) {
  EncodeTiledFn fn = encode_fn();
  if (!fn || !base || ((uintptr_t)base & 15) != 0) return false;
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUtensorMapDataType dt = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  return fn(out, dt, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool make_rows_map(CUtensorMap* out, const void* base, int elem_bytes, long long row_bytes, long long rows, int parts,
                   long long part_bytes, int kblocks, int box_rows, int box_kb) {
  const cuuint64_t dims[4] = {(cuuint64_t)(128 / elem_bytes), (cuuint64_t)rows, (cuuint64_t)parts, (cuuint64_t)kblocks};
  const cuuint64_t strides[3] = {(cuuint64_t)row_bytes, (cuuint64_t)(parts > 1 ? part_bytes : row_bytes), 128};
  const cuuint32_t box[4] = {(cuuint32_t)(128 / elem_bytes), (cuuint32_t)box_rows, (cuuint32_t)parts, (cuuint32_t)box_kb};
  return encode_map(out, base, elem_bytes, 4, dims, strides, box);
}
bool make_gate_map(CUtensorMap* out, const void* base, int elem_bytes, int parts, long long part_bytes, int chunks, int box_units,
                   int box_parts, int box_kb) {
  const cuuint64_t dims[5] = {(cuuint64_t)(128 / elem_bytes), 32, 4, (cuuint64_t)parts, (cuuint64_t)chunks};
  const cuuint64_t strides[4] = {128, 32 * 128, (cuuint64_t)(parts > 1 ? part_bytes : 128 * 128), 128 * 128};
  const cuuint32_t box[5] = {(cuuint32_t)(128 / elem_bytes), (cuuint32_t)box_units, 4, (cuuint32_t)box_parts, (cuuint32_t)box_kb};
  return encode_map(out, base, elem_bytes, 5, dims, strides, box);
}

// ------------------------------------------------------------------------------------------
// Exercise of the bounded wait: one warp waits on a barrier that nothing ever completes, with a short limit, and
// must come back with the error word set and the context intact.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(32) wait_probe_kernel(int* err, long long limit_cycles, int code) {
  __shared__ uint64_t bar;
  __shared__ int abort_s;
  if (threadIdx.x == 0) {
    abort_s = 0;
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_wait(&bar, 0, &abort_s, err, code, limit_cycles);
}
cudaError_t launch_wait_probe(int* err, long long limit_cycles, int code, cudaStream_t st) {
  wait_probe_kernel<<<1, 32, 0, st>>>(err, limit_cycles, code);
  count_launch();
  return cudaGetLastError();
}

}  // namespace zrnn
