// What the two kernels for links of the recurrent chain (tc_link.cu, tc_chain.cu) share on the device.
#pragma once
#include "tc_device.cuh"

namespace zrnn {
namespace {

// rows y.. of k-blocks kb.., all parts (make_rows_map)
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int y, int kb) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %5}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(y), "r"(kb)
      : "memory");
}
// hidden units y.. of all gates from part `part` and k-block kb on (make_gate_map)
__device__ __forceinline__ void tma_load_5d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int y, int part, int kb) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(y), "r"(part), "r"(kb)
      : "memory");
}
// ... whose lines leave the L2 first
__device__ __forceinline__ void tma_load_5d_first(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int y, int part, int kb) {
  asm volatile(
      "{\n\t.reg .b64 pol;\n\tcreatepolicy.fractional.L2::evict_first.b64 pol, 1.0;\n\t"
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %3, %5, %6}], [%2], pol;\n\t}"
      :
      : "r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(0), "r"(y), "r"(part), "r"(kb)
      : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float* v) {
  uint32_t r0, r1, r2, r3;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(taddr));
  v[0] = __uint_as_float(r0); v[1] = __uint_as_float(r1); v[2] = __uint_as_float(r2); v[3] = __uint_as_float(r3);
}
template <int W>
__device__ __forceinline__ void tmem_ldw(uint32_t taddr, float* v) {
  if constexpr (W == 4) tmem_ld4(taddr, v);
  else tmem_ld8(taddr, v);
}
// 16 bytes into the shared memory of another CTA of the cluster, counted on a transaction barrier there
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t bar, float a, float b, float c, float d) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];" ::"r"(addr), "r"(bar),
               "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(__float_as_uint(d))
               : "memory");
}
// after a wait that gave up: copies in flight land before the CTA may retire
__device__ __forceinline__ void settle_copies() {
  const long long t0 = clock64();
  while (clock64() - t0 < 20000000LL) {}
}

}  // namespace
}  // namespace zrnn
