// Device helpers shared by the tiled kernels: bounded mbarrier waits, TMA tile
// loads, and packed FP32 arithmetic.
#pragma once

#include <cuda.h>

#include "ernn_common.cuh"

namespace ernn {
namespace {

__device__ __forceinline__ uint32_t s32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Fetch a tensor map (a __grid_constant__ kernel parameter) into the
// descriptor cache ahead of its first copy.
__device__ __forceinline__ void prefetch_map(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

__device__ __forceinline__ void bar_init(uint64_t* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s32(b)) : "memory");
}

__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(b)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(s32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait (about a second); on timeout records ERNN_ERR_TIMEOUT and
// returns so that the CTA's barriers stay matched.
__device__ __forceinline__ void bar_wait(uint64_t* b, uint32_t parity, int* err) {
  if (bar_try(b, parity)) return;
  if (*(volatile int*)err != 0) return;
  const long long t0 = clock64();
  for (;;) {
    for (int k = 0; k < 64; ++k)  // the clock is read once per 64 polls
      if (bar_try(b, parity)) return;
    if (clock64() - t0 > kWaitLimitCycles) {
      atomicExch(err, kDeviceTimeout);
      return;
    }
  }
}

// Error path of a tile pipeline.  A wait that gives up (its own time limit,
// or an error another CTA of the launch already recorded) marks the CTA
// failed: from then on no further tile loads are issued (the launch's
// outputs are invalid anyway), and before the CTA exits one thread waits,
// again with a time limit, for the loads it had already issued, so no copy
// is still writing into the shared memory of a CTA that has ended.
struct PipeGuard {
  int failed;  // a wait of this CTA gave up
  int issued;  // tiles 0 .. issued-1 of this CTA had their loads issued
};

__device__ __forceinline__ void pipe_init(PipeGuard* g) {
  g->failed = 0;
  g->issued = 0;
}
__device__ __forceinline__ bool pipe_failed(const PipeGuard* g) {
  return *reinterpret_cast<const volatile int*>(&g->failed) != 0;
}
__device__ __forceinline__ void pipe_issued(PipeGuard* g, int k) { atomicMax(&g->issued, k + 1); }

// bar_wait that reports whether the phase completed (false: timed out, or an
// error of the launch was already recorded); a false marks the CTA failed.
// The error word is read once per 64 polls: reading it first would hold a
// wait whose copies are about to land for a trip to global memory.
__device__ __forceinline__ bool bar_wait_ok(uint64_t* b, uint32_t parity, int* err, PipeGuard* g) {
  const long long t0 = clock64();
  for (;;) {
    for (int k = 0; k < 64; ++k)
      if (bar_try(b, parity)) return true;
    if (*(volatile int*)err != 0) break;
    if (clock64() - t0 > kWaitLimitCycles) {
      atomicExch(err, kDeviceTimeout);
      break;
    }
  }
  *reinterpret_cast<volatile int*>(&g->failed) = 1;
  __threadfence_block();
  return false;
}

// After a failed CTA's tile loop (one thread): wait, each with a time limit,
// for the phases of the last `ns` issued tiles (tile k: stage k % ns, phase
// parity (k / ns) & 1).  A phase that already completed returns at once.
__device__ __forceinline__ void pipe_drain(uint64_t* bar, int ns, const PipeGuard* g) {
  const int issued = *reinterpret_cast<const volatile int*>(&g->issued);
  for (int k = issued - ns < 0 ? 0 : issued - ns; k < issued; ++k) {
    const long long t0 = clock64();
    while (!bar_try(&bar[k % ns], (uint32_t)(k / ns) & 1u))
      if (clock64() - t0 > kWaitLimitCycles) break;
  }
}

// 3D tile load (columns, rows, component planes) into shared memory.
__device__ __forceinline__ void tma_load3(void* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                          uint64_t* b) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(s32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(s32(b))
      : "memory");
}

// TMA destinations start on 128-byte boundaries: the dynamic shared block is
// allocated 128 bytes longer and its start rounded up.
// (pointer arithmetic on the __shared__ array, so the compiler keeps the
// shared state space and emits shared-memory loads)
__device__ __forceinline__ float* aligned128(float* p) {
  const uint32_t a = s32(p);
  return p + ((((a + 127u) & ~127u) - a) >> 2);
}

__device__ __forceinline__ void fence_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

struct Coefs {
  float k11, k22, kq12, k16, k26, k66, k16h, k26h;
};

__device__ __forceinline__ Coefs coefs(const Coef* c) {
  return Coefs{c->k11, c->k22, c->kq12, c->k16, c->k26, c->k66, c->k16h, c->k26h};
}

// Packed FP32 (sm_100 family): one instruction applies the same operation to
// two cells of a quad, each lane rounded as the scalar operation would be,
// which halves the arithmetic instructions of a quad.  Sums whose operands
// are column neighbours (not register pairs of the window) are formed by
// scalar adds first, so every value keeps the association and rounding of
// the scalar formulas.
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 pair(const float v[4], int p) { return make_float2(v[2 * p], v[2 * p + 1]); }
__device__ __forceinline__ float2 pair4(const float4& v, int p) {
  return p == 0 ? make_float2(v.x, v.y) : make_float2(v.z, v.w);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ void put(float v[4], int p, float2 a) {
  v[2 * p] = a.x;
  v[2 * p + 1] = a.y;
}

// 2D tile load (columns, rows) into shared memory: the degradation plane.
__device__ __forceinline__ void tma_load2(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* b) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(s32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(s32(b))
      : "memory");
}

__device__ __forceinline__ float4 one_minus(const float4 d) {
  return make_float4(1.f - d.x, 1.f - d.y, 1.f - d.z, 1.f - d.w);
}

}  // namespace
}  // namespace ernn
