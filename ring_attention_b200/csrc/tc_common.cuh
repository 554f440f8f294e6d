// Device-side building blocks shared by the tcgen05 step kernels (step_tc.cu: fp16 / bf16,
// step_f32.cu: fp32 through split fp16 operands): mbarrier / TMA / tcgen05 wrappers with bounded
// waits, shared-memory and instruction descriptors, the visible key-tile range of a query
// block, the kernel argument block and the host-side tensor-map encoder.
#pragma once

#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"

namespace rab {
namespace tcgen {

constexpr int kBM = 128;           // query rows per tile
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRowSumLimit = 32768.f;  // a tile's row sum of P above this moves the reference
constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // default limit of every wait: 2 s

// ---- PTX wrappers -------------------------------------------------------------------
__device__ inline unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ inline void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ inline void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ inline void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ inline bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same with acquire semantics at cluster scope: for a barrier that threads of the peer CTA of
// a pair arrive on.
__device__ inline bool mbar_try_wait_cluster(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Non-blocking form: has the phase with this parity completed?
__device__ inline bool mbar_test_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// One lane of a converged warp (the same lane every time for a full mask).
__device__ inline bool elect_one() {
  unsigned pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ inline unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait. Returns false when the block is aborting (own limit reached or another
// role flagged it). `which` identifies the wait in the status word.
template <bool kClusterScope = false>
__device__ inline bool mbar_wait(unsigned bar, unsigned parity, volatile int* abort_flag,
                                 int* status, int which, int tile, unsigned long long limit_ns) {
  auto try_wait = [&]() {
    return kClusterScope ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity);
  };
  if (try_wait()) return true;
  const unsigned long long t0 = global_ns();
  unsigned spins = 0;
  while (true) {
    if (try_wait()) return true;
    if ((++spins & 255u) == 0) {
      if (*abort_flag) return false;
      if (global_ns() - t0 > limit_ns) {
        *abort_flag = 1;
        if (atomicCAS(&status[0], 0, RA_ERR_DEVICE_WAIT) == 0) {
          status[1] = which;
          status[2] = static_cast<int>(blockIdx.x + blockIdx.y * gridDim.x);
          status[3] = tile;
        }
        return false;
      }
    }
  }
}

__device__ inline void tma_load_3d(unsigned dst, const CUtensorMap* map, unsigned bar, int c0,
                                   int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%3, %4, %5}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// `bytes` (a multiple of 16) of contiguous memory, both ends 16-byte aligned.
__device__ inline void bulk_load(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(src)), "r"(bytes), "r"(bar)
      : "memory");
}

__device__ inline void tma_load_5d(unsigned dst, const CUtensorMap* map, unsigned bar, int c0, int c1, int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%3, %4, %5, %6, %7}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}

__device__ inline void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<unsigned long long>(map)) : "memory");
}
__device__ inline void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ inline void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ inline void tc_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]
__device__ inline void mma_ss(unsigned d_tmem, unsigned long long a_desc,
                              unsigned long long b_desc, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ inline void mma_ts(unsigned d_tmem, unsigned a_tmem, unsigned long long b_desc,
                              unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}


// The same with descriptors as their low words (addresses, in 16-byte units) and a common high word: an instruction of 32
// clk leaves its issuer no time for sums of 64 bits.
__device__ inline void mma_ss_lo(unsigned d_tmem, unsigned a_lo, unsigned b_lo, unsigned hi, unsigned idesc,
                                 unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ inline void mma_ts_lo(unsigned d_tmem, unsigned a_tmem, unsigned b_lo, unsigned hi, unsigned idesc,
                                 unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// ---- CTA pairs (cta_group::2): one instruction drives the tensor cores of two CTAs of a cluster,
// M = 256 (128 rows from each CTA's A operand and into each CTA's tensor memory), each CTA
// holding half of the B operand's N columns in its own shared memory at the same offset.
__device__ inline unsigned cluster_ctarank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ inline void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
// The same for threads of warps that may be diverged: every thread of the cluster arrives.
__device__ inline void cluster_sync_threads() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// Shared memory of CTA `rank` of the cluster at this CTA's address `saddr`.
__device__ inline unsigned cluster_addr(unsigned saddr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ inline float2 ld_cluster_f2(unsigned addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}
__device__ inline float4 ld_cluster_f4(unsigned addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}
// Arrive on the barrier at the same shared-memory offset in CTA `rank` of the cluster.
__device__ inline void mbar_arrive_cluster(unsigned bar, unsigned rank) {
  asm volatile(
      "{\n\t.reg .b32 r;\n\t"
      "mapa.shared::cluster.u32 r, %0, %1;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [r];\n\t}" ::"r"(bar),
      "r"(rank)
      : "memory");
}
// The barrier at this offset in BOTH CTAs of the pair gets the arrival.
__device__ inline void tc_commit_pair(unsigned bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(bar),
      "h"(static_cast<unsigned short>(3))
      : "memory");
}
__device__ inline void mma_ss_pair(unsigned d_tmem, unsigned long long a_desc,
                                   unsigned long long b_desc, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ inline void mma_ts_pair(unsigned d_tmem, unsigned a_tmem, unsigned long long b_desc,
                                   unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ inline void tmem_ld32(unsigned taddr, float (&r)[32]) {
  unsigned u[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"  // same statement: no use of the registers can move above it
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]),
        "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]),
        "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]),
        "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]), "=r"(u[25]),
        "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) r[i] = __uint_as_float(u[i]);
}
// All 128 columns of a row: four 32-column loads in flight and one wait, in a single asm
// statement so that no use of the registers can be scheduled above the wait.
__device__ inline void tmem_ld128(unsigned taddr, float (&r)[128]) {
  unsigned u[128];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%128];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%129];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%64, %65, %66, %67, %68, %69, %70, %71, %72, %73, %74, %75, %76, %77, %78, %79, %80, %81, %82, %83, %84, %85, %86, %87, %88, %89, %90, %91, %92, %93, %94, %95}, [%130];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%96, %97, %98, %99, %100, %101, %102, %103, %104, %105, %106, %107, %108, %109, %110, %111, %112, %113, %114, %115, %116, %117, %118, %119, %120, %121, %122, %123, %124, %125, %126, %127}, [%131];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
        "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]),
        "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]),
        "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31]),
        "=r"(u[32]), "=r"(u[33]), "=r"(u[34]), "=r"(u[35]), "=r"(u[36]), "=r"(u[37]), "=r"(u[38]), "=r"(u[39]),
        "=r"(u[40]), "=r"(u[41]), "=r"(u[42]), "=r"(u[43]), "=r"(u[44]), "=r"(u[45]), "=r"(u[46]), "=r"(u[47]),
        "=r"(u[48]), "=r"(u[49]), "=r"(u[50]), "=r"(u[51]), "=r"(u[52]), "=r"(u[53]), "=r"(u[54]), "=r"(u[55]),
        "=r"(u[56]), "=r"(u[57]), "=r"(u[58]), "=r"(u[59]), "=r"(u[60]), "=r"(u[61]), "=r"(u[62]), "=r"(u[63]),
        "=r"(u[64]), "=r"(u[65]), "=r"(u[66]), "=r"(u[67]), "=r"(u[68]), "=r"(u[69]), "=r"(u[70]), "=r"(u[71]),
        "=r"(u[72]), "=r"(u[73]), "=r"(u[74]), "=r"(u[75]), "=r"(u[76]), "=r"(u[77]), "=r"(u[78]), "=r"(u[79]),
        "=r"(u[80]), "=r"(u[81]), "=r"(u[82]), "=r"(u[83]), "=r"(u[84]), "=r"(u[85]), "=r"(u[86]), "=r"(u[87]),
        "=r"(u[88]), "=r"(u[89]), "=r"(u[90]), "=r"(u[91]), "=r"(u[92]), "=r"(u[93]), "=r"(u[94]), "=r"(u[95]),
        "=r"(u[96]), "=r"(u[97]), "=r"(u[98]), "=r"(u[99]), "=r"(u[100]), "=r"(u[101]), "=r"(u[102]), "=r"(u[103]),
        "=r"(u[104]), "=r"(u[105]), "=r"(u[106]), "=r"(u[107]), "=r"(u[108]), "=r"(u[109]), "=r"(u[110]), "=r"(u[111]),
        "=r"(u[112]), "=r"(u[113]), "=r"(u[114]), "=r"(u[115]), "=r"(u[116]), "=r"(u[117]), "=r"(u[118]), "=r"(u[119]),
        "=r"(u[120]), "=r"(u[121]), "=r"(u[122]), "=r"(u[123]), "=r"(u[124]), "=r"(u[125]), "=r"(u[126]), "=r"(u[127])
      : "r"(taddr), "r"(taddr + 32), "r"(taddr + 64), "r"(taddr + 96)
      : "memory");
#pragma unroll
  for (int i = 0; i < 128; ++i) r[i] = __uint_as_float(u[i]);
}
// 64 columns of a row: two loads in flight and one wait.
__device__ inline void tmem_ld64(unsigned taddr, float (&r)[64]) {
  unsigned u[64];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%64];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%65];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
        "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]),
        "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]),
        "=r"(u[22]), "=r"(u[23]), "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]),
        "=r"(u[29]), "=r"(u[30]), "=r"(u[31]), "=r"(u[32]), "=r"(u[33]), "=r"(u[34]), "=r"(u[35]),
        "=r"(u[36]), "=r"(u[37]), "=r"(u[38]), "=r"(u[39]), "=r"(u[40]), "=r"(u[41]), "=r"(u[42]),
        "=r"(u[43]), "=r"(u[44]), "=r"(u[45]), "=r"(u[46]), "=r"(u[47]), "=r"(u[48]), "=r"(u[49]),
        "=r"(u[50]), "=r"(u[51]), "=r"(u[52]), "=r"(u[53]), "=r"(u[54]), "=r"(u[55]), "=r"(u[56]),
        "=r"(u[57]), "=r"(u[58]), "=r"(u[59]), "=r"(u[60]), "=r"(u[61]), "=r"(u[62]), "=r"(u[63])
      : "r"(taddr), "r"(taddr + 32)
      : "memory");
#pragma unroll
  for (int i = 0; i < 64; ++i) r[i] = __uint_as_float(u[i]);
}
__device__ inline void tmem_st32(unsigned taddr, const float (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(
          taddr),
      "r"(__float_as_uint(r[0])), "r"(__float_as_uint(r[1])), "r"(__float_as_uint(r[2])),
      "r"(__float_as_uint(r[3])), "r"(__float_as_uint(r[4])), "r"(__float_as_uint(r[5])),
      "r"(__float_as_uint(r[6])), "r"(__float_as_uint(r[7])), "r"(__float_as_uint(r[8])),
      "r"(__float_as_uint(r[9])), "r"(__float_as_uint(r[10])), "r"(__float_as_uint(r[11])),
      "r"(__float_as_uint(r[12])), "r"(__float_as_uint(r[13])), "r"(__float_as_uint(r[14])),
      "r"(__float_as_uint(r[15])), "r"(__float_as_uint(r[16])), "r"(__float_as_uint(r[17])),
      "r"(__float_as_uint(r[18])), "r"(__float_as_uint(r[19])), "r"(__float_as_uint(r[20])),
      "r"(__float_as_uint(r[21])), "r"(__float_as_uint(r[22])), "r"(__float_as_uint(r[23])),
      "r"(__float_as_uint(r[24])), "r"(__float_as_uint(r[25])), "r"(__float_as_uint(r[26])),
      "r"(__float_as_uint(r[27])), "r"(__float_as_uint(r[28])), "r"(__float_as_uint(r[29])),
      "r"(__float_as_uint(r[30])), "r"(__float_as_uint(r[31]))
      : "memory");
}
__device__ inline void tmem_ld8(unsigned taddr, float (&r)[8]) {
  unsigned u[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = __uint_as_float(u[i]);
}
__device__ inline void tmem_st8(unsigned taddr, const float (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
               "r"(__float_as_uint(r[0])), "r"(__float_as_uint(r[1])), "r"(__float_as_uint(r[2])),
               "r"(__float_as_uint(r[3])), "r"(__float_as_uint(r[4])), "r"(__float_as_uint(r[5])),
               "r"(__float_as_uint(r[6])), "r"(__float_as_uint(r[7]))
               : "memory");
}
__device__ inline void tmem_st16(unsigned taddr, const unsigned (&u)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]),
      "r"(u[8]), "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15])
      : "memory");
}
// 32 packed columns from an array slice
__device__ inline void tmem_st32u(unsigned taddr, const unsigned* u) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(
          taddr),
      "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]),
      "r"(u[8]), "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]),
      "r"(u[15]), "r"(u[16]), "r"(u[17]), "r"(u[18]), "r"(u[19]), "r"(u[20]), "r"(u[21]),
      "r"(u[22]), "r"(u[23]), "r"(u[24]), "r"(u[25]), "r"(u[26]), "r"(u[27]), "r"(u[28]),
      "r"(u[29]), "r"(u[30]), "r"(u[31])
      : "memory");
}
__device__ inline float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ inline float min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// packed fp32x2 arithmetic: one instruction for two lanes of a float2
__device__ inline float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return d;
}
__device__ inline float2 fadd2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)));
  return d;
}
__device__ inline void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ inline float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Shared-memory matrix descriptors for 128B-swizzled tiles (8-row groups 1024 B apart).
// K-major operand (rows = M or N index, 64 contiguous 16-bit elements of the contraction
// dimension per 128-byte row); the leading byte offset is unused for swizzled K-major.
constexpr unsigned kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO, version 1, SWIZZLE_128B
__device__ inline unsigned long long desc_kmajor(unsigned saddr) {
  const unsigned lo = ((saddr & 0x3FFFFu) >> 4) | (1u << 16);
  const unsigned hi = kDescHi;
  return (static_cast<unsigned long long>(hi) << 32) | lo;
}
// MN-major operand (rows = contraction index, 64 contiguous elements of N per 128-byte row):
// leading byte offset = distance between 64-element N blocks (one 128-row box, 16 KiB),
// stride = between 8-row groups (1 KiB); one MMA (16 rows) advances the start by 2 KiB.
__device__ inline unsigned long long desc_mnmajor(unsigned saddr, unsigned lbo_bytes,
                                               unsigned sbo_bytes) {
  const unsigned lo = ((saddr & 0x3FFFFu) >> 4) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
  const unsigned hi = ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
  return (static_cast<unsigned long long>(hi) << 32) | lo;
}

// Instruction descriptor, kind::f16: fp32 accumulate, A/B format (0 fp16, 1 bf16), A K-major,
// B K-major (b_mn = 0) or MN-major (1), N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr unsigned make_idesc(unsigned fmt, unsigned b_mn, unsigned n,
                                                  unsigned m) {
  return (1u << 4) | (fmt << 7) | (fmt << 10) | (b_mn << 16) | ((n >> 3) << 17) |
         ((m >> 4) << 24);
}

struct TileRange {
  int lo, hi;  // key tiles [lo, hi) of a segment that some row of the block can see
};

// Visible key-tile range of key segment `sk` for a query block whose rows span positions
// [qmin, qmax] (both ends are positions of real rows).
template <int kTileKeys>
__host__ __device__ inline TileRange tile_range(const PosMap& kmap, int sk, int stride, bool causal,
                                       long long doc_len, int qmin, int qmax) {
  const int L = kmap.seg_len;
  const long long kb = kmap.base[sk];
  long long j_lo = 0, j_hi = L - 1;  // visible local key indices, inclusive
  if (causal) {
    const long long d = static_cast<long long>(qmax) - kb;
    if (d < 0) return {0, 0};
    j_hi = min(j_hi, d / stride);
  }
  if (doc_len > 0) {
    const long long p_lo = (static_cast<long long>(qmin) / doc_len) * doc_len;
    const long long p_hi = (static_cast<long long>(qmax) / doc_len + 1) * doc_len - 1;
    if (p_hi < kb) return {0, 0};
    j_hi = min(j_hi, (p_hi - kb) / stride);
    if (p_lo > kb) j_lo = (p_lo - kb + stride - 1) / stride;
  }
  if (j_hi < j_lo) return {0, 0};
  return {static_cast<int>(j_lo / kTileKeys), static_cast<int>(j_hi / kTileKeys) + 1};
}

// Query tile i of a KV head in the spread form: by position, then by query head of the group; or, with `pack` heads to a
// tile, all rows of heads i * pack and on, one head behind the other.
struct SpreadTile {
  int head, seg, row0;  // (first) head inside the group, query segment, first row inside it
};
__host__ __device__ inline SpreadTile spread_tile(int i, int group, int per_seg, int pack) {
  if (pack > 1) return {i * pack, 0, 0};
  const int pos = i / group;
  return {i - pos * group, pos / per_seg, (pos % per_seg) * kBM};
}
// Positions [qmin, qmax] that the rows of tiles [i0, i1) span.
__host__ __device__ inline void spread_span(const PosMap& qmap, int stride, int group, int per_seg, int pack, int i0, int i1,
                                            int* qmin, int* qmax) {
  *qmin = 0x7fffffff;
  *qmax = -0x7fffffff;
  for (int i = i0; i < i1; ++i) {
    const SpreadTile t = spread_tile(i, group, per_seg, pack);
    const int rows = qmap.seg_len - t.row0 < kBM ? qmap.seg_len - t.row0 : kBM;
    const int first = qmap.base[t.seg] + t.row0 * stride, last = first + (rows - 1) * stride;
    *qmin = first < *qmin ? first : *qmin;
    *qmax = last > *qmax ? last : *qmax;
  }
}

// A block's share of its query block's tile list when the list is cut across the blocks of a
// cluster: list entries [beg, end). clip() is called once per key segment, in order.
struct TileShare {
  int beg, end, seen;
  __device__ TileRange clip(TileRange r) {
    const int n = r.hi - r.lo;
    const int lo = max(0, beg - seen), hi = min(n, end - seen);
    seen += n;
    return {r.lo + lo, r.lo + max(lo, hi)};
  }
};

// Spread form: the key tiles of every query block of a KV head are cut into shares, a block each, whose partial
// states go to a workspace (see plan_spread).
constexpr int kMaxSpread = 160;  // blocks of one KV head, at most (a B200 has 148 SMs)
struct Spread {
  int total;                             // blocks of one KV head
  int pack;                              // heads whose rows share a query tile (1: a tile is rows of one head)
  unsigned char beg[kMaxSpread + 1];     // first block of query block j; beg[number of query blocks] = total
};

struct TcArgs {
  float* out;
  float* m;
  float* l;
  int H, kvH, Sq;
  int n_qblocks_per_seg;
  PosMap qmap, kmap;
  int kseg_head[RA_MAX_SEG];  // key segment -> head-coordinate offset and first row in K / V
  int kseg_row[RA_MAX_SEG];
  int stride;
  unsigned flags;
  long long doc_len;
  int* status;
  unsigned long long wait_ns;  // limit of every device-side wait
  int stall_after;             // test hook: the producer stops after this many ring items (< 0: off)
  int kv_per_wave;             // block order: waves of this many KV heads (0: heads fastest)
  int key_split;               // blocks of a cluster that share one query block's key tiles
  Spread spread;               // spread form: the shares, and where their partial states go
  float* part_o;
  float2* part_ml;
};

// What a block does whose rows see no key: nothing, or the state of `rows` rows from row0 on is written empty
// or normalised. Without tensor memory, barriers or a meeting of the cluster, whose blocks take every n-th piece:
// such a block had held its SM for 5 us, and a call that has as many of them as of others, as the ring steps of a zig-zag
// shard do, waited for them: 16 heads, 64 blocks of 256 rows with keys and 64 without, us per step 31.4 -> 27.8, the one
// that normalises 36.7 -> 31.2.
template <int DR>
__device__ inline void rows_without_keys(const TcArgs& a, size_t row0, int rows, unsigned rank, int n, bool fresh,
                                         bool finalize) {
  if (!(fresh || finalize) || *reinterpret_cast<volatile int*>(a.status) != 0) return;
  constexpr int kVec = DR / 4;
  for (int i = static_cast<int>(rank * blockDim.x + threadIdx.x); i < rows * kVec; i += n * static_cast<int>(blockDim.x)) {
    const size_t row = row0 + i / kVec;
    float4* const dst = reinterpret_cast<float4*>(a.out) + row0 * kVec + i;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!fresh) {
      const bool empty = a.m[row] == -INFINITY;
      const float l = empty ? 0.f : a.l[row];
      const float inv = l > 0.f ? 1.f / l : 0.f;
      v = *dst;
      v = make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv);
      if (empty && i % kVec == 0) a.l[row] = 0.f;
    } else if (i % kVec == 0) {
      a.m[row] = -INFINITY;
      a.l[row] = 0.f;
    }
    *dst = v;
  }
}

// End of a block of the key-split form, run by the softmax threads (one per row; the other threads
// of the cluster only join the three barriers): the partial (O, m, l) of the cluster's blocks are
// merged and folded into the state as one step. Every block scales its O to the common reference
// point (o_unit: what one unit of the accumulator is worth) and stages it in its own shared memory,
// then each block sums its slice of the elements over all blocks and writes it. 128 KB of staged O per
// block at head_dim 128 cross the cluster once (about 2 us); no workspace and no second launch. A row
// that some block of the cluster gave up on (a wait ran out) keeps its state, as without a split.
template <class C, int DR>
__device__ inline void merge_key_split(const TcArgs& a, unsigned char* smem, unsigned s_base,
                                       unsigned t_o, int w, int row, bool row_valid, size_t grow0, bool gave_up,
                                       bool worked, float m_ref, float l_run, float o_unit, unsigned rank,
                                       bool fresh, bool finalize) {
  constexpr int kRows = C::kTiles * kBM;
  constexpr int kStride = DR + 4;  // floats: rows 16 bytes apart modulo 128, so float4 stores do not collide
  constexpr int kOffFac = kRows * kStride * 4;
  float* const o_stage = reinterpret_cast<float*>(smem);
  float2* const fac = reinterpret_cast<float2*>(smem + kOffFac);
  float2* const ml = reinterpret_cast<float2*>(smem + C::kOffMl);
  const int rb = w * kBM + row;
  const int n = a.key_split;
  const bool have = worked && row_valid && m_ref > -INFINITY;
  ml[rb] = have ? make_float2(m_ref, l_run) : make_float2(-INFINITY, gave_up ? -1.f : 0.f);
  cluster_sync_threads();  // all (m, l) are there, no block reads its Q or ring any more
  const unsigned ml_addr = s_base + C::kOffMl + rb * 8;
  float m_all = -INFINITY, l_all = 0.f;
  for (int r = 0; r < n; ++r) m_all = fmaxf(m_all, ld_cluster_f2(cluster_addr(ml_addr, r)).x);
  bool lost = false;  // (a sum is never negative)
  for (int r = 0; r < n; ++r) {
    const float2 p = ld_cluster_f2(cluster_addr(ml_addr, r));
    if (p.x > -INFINITY) l_all += p.y * ex2(p.x - m_all);
    else lost = lost || p.y == -1.f;
  }
  const size_t grow = grow0 + (row_valid ? rb : 0);
  const bool any = row_valid && m_all > -INFINITY;
  float m_old = -INFINITY, l_old = 0.f;
  if (!fresh && row_valid) {
    m_old = a.m[grow];
    l_old = a.l[grow];
  }
  const float m_new = any ? m_all * kLn2 : -INFINITY;
  const float m_fin = fmaxf(m_old, m_new);
  const float ca = (m_old == -INFINITY) ? 0.f : expf(m_old - m_fin);
  const float cb = any ? expf(m_new - m_fin) : 0.f;
  const float l_fin = ca * l_old + cb * l_all;
  const float inv = finalize ? (l_fin > 0.f ? 1.f / l_fin : 0.f) : 1.f;
  const bool touch = row_valid && !lost && (any || fresh || finalize);
  fac[rb] = touch ? make_float2(ca * inv, cb * inv) : make_float2(-1.f, 0.f);  // factors are never negative
  const float scale = have ? ex2(m_ref - m_all) : 0.f;
#pragma unroll 1
  for (int c = 0; c < DR / 32; ++c) {
    float o[32];
    if (worked) {  // warp-uniform: the tensor-memory load is warp-collective
      tmem_ld32(t_o + c * 32, o);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) o[i] = 0.f;
    }
    float4* dst = reinterpret_cast<float4*>(o_stage + rb * kStride + c * 32);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      dst[i] = have ? make_float4(o[4 * i] * o_unit * scale, o[4 * i + 1] * o_unit * scale,
                                  o[4 * i + 2] * o_unit * scale, o[4 * i + 3] * o_unit * scale)
                    : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  cluster_sync_threads();  // every block's O is staged, every old (m, l) has been read
  constexpr int kVec = DR / 4;
  for (int idx = static_cast<int>(rank) * kRows + rb; idx < kRows * kVec; idx += n * kRows) {
    const int r_out = idx / kVec, col = (idx % kVec) * 4;
    const float2 f = fac[r_out];
    if (f.x == -1.f) continue;
    const unsigned addr = s_base + (r_out * kStride + col) * 4;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int r = 0; r < n; ++r) {
      const float4 o = ld_cluster_f4(cluster_addr(addr, r));
      acc.x += o.x;
      acc.y += o.y;
      acc.z += o.z;
      acc.w += o.w;
    }
    float4* dst = reinterpret_cast<float4*>(a.out + (grow0 + r_out) * DR + col);
    float4 old = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!fresh) old = *dst;
    *dst = make_float4(f.x * old.x + f.y * acc.x, f.x * old.y + f.y * acc.y, f.x * old.z + f.y * acc.z,
                       f.x * old.w + f.y * acc.w);
  }
  if (rank == 0 && touch) {
    a.m[grow] = m_fin;
    a.l[grow] = l_fin;
  }
  cluster_sync_threads();  // nobody leaves while its shared memory is still read
}

// One row's part of a block's result: o * unit * f_new (nothing if !have) plus f_old times the state.
struct RowOut {
  bool touch, have;
  float f_old, f_new, unit;
};

// The end of a block that merges with nobody: 32 rows of O from tensor memory into the state, run by one
// warp (lane = row). A row per lane would touch 32 rows with every load and store, 16 bytes each; so the
// rows go through shared memory (`stage`: kStageBytes of this warp, swizzled 16-byte chunks, at most 64
// columns at a time, 128 take half again as long) and the state is read and written in pieces of 128 bytes and more. The old state
// does not depend on the MMAs still running: its first loads are issued before wait_o(), which returns whether O is
// there, and row_out() says what becomes of this lane's row. us per call with one key tile, 128 blocks of 256 rows, a
// row per lane -> so: head_dim 64 into a new state 8.6 -> 7.8, into an old one 11.5 -> 8.0; head_dim 128 12.0 -> 9.5,
// 17.0 -> 10.0; head_dim 256 (128 rows) 12.4 -> 10.1, 17.8 -> 11.1. With few rows the stores of a row per lane are few too:
// fp32 head_dim 128, 20 rows into a new state 8.6 -> 9.6, 128 rows 12.5 -> 11.9.
template <int DR>
struct RowStore {
  static constexpr int kCols = DR > 64 ? 64 : 32;       // columns of a pass
  static constexpr int kChunks = kCols / 4;             // 16-byte chunks of a row
  static constexpr int kRowsPer = 32 / kChunks;         // rows that one access of the warp covers
  static constexpr int kStageBytes = 32 * kCols * 4;
  template <typename Wait, typename Row>
  __device__ static inline bool run(int lane, float* out, size_t grow0, unsigned valid_rows, unsigned stage, unsigned t_o,
                                    bool worked, bool fresh, Wait wait_o, Row row_out) {
    const int sub = lane / kChunks, chunk = lane % kChunks;
    float4 old[kChunks];
    auto row_of = [&](int i) { return i * kRowsPer + sub; };
    // (one address and offsets known at compile time: an address from every row's index took calls with an old state
    // 0.4 us more at head_dim 128)
    float4* const mine = reinterpret_cast<float4*>(out + (grow0 + sub) * DR + chunk * 4);
    auto at = [&](int pass, int i) { return mine + i * (kRowsPer * DR / 4) + pass * (kCols / 4); };
    auto load_old = [&](int pass) {
#pragma unroll
      for (int i = 0; i < kChunks; ++i)
        old[i] = !fresh && (valid_rows >> row_of(i) & 1u) ? *at(pass, i) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    load_old(0);
    if (!wait_o()) return false;
    const RowOut ro = row_out();
    const unsigned touched = __ballot_sync(0xffffffffu, ro.touch);
    if (touched == 0) return true;
#pragma unroll 1
    for (int pass = 0; pass < DR / kCols; ++pass) {
      if (pass > 0) load_old(pass);
#pragma unroll
      for (int c = 0; c < kCols / 32; ++c) {
        float o[32];
        if (worked) {  // warp-uniform: the tensor-memory load is warp-collective
          tmem_ld32(t_o + pass * kCols + c * 32, o);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = ro.have ? o[i] * ro.unit * ro.f_new : 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const unsigned dst = stage + lane * (kCols * 4) + (((c * 8 + i) ^ (lane & 7)) << 4);
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "f"(o[4 * i]), "f"(o[4 * i + 1]),
                       "f"(o[4 * i + 2]), "f"(o[4 * i + 3])
                       : "memory");
        }
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < kChunks; ++i) {
        const int r = row_of(i);
        const float f = __shfl_sync(0xffffffffu, ro.f_old, r);
        float4 v;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                     : "r"(stage + r * (kCols * 4) + ((chunk ^ (r & 7)) << 4)));
        if (!fresh) {
          v.x += f * old[i].x;
          v.y += f * old[i].y;
          v.z += f * old[i].z;
          v.w += f * old[i].w;
        }
        if (touched >> r & 1u) *at(pass, i) = v;
      }
      __syncwarp();
    }
    return true;
  }
};

// ---- host side ----------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// (D, rows, heads) tensor of 16-bit (RA_F16 / RA_BF16) or 32-bit (RA_F32) elements, box = one
// 128-byte row piece (64 or 32 elements) x box_rows rows x 1, 128B swizzle. With a box wider than
// the tensor (head_dim 32 in 16 bits) the upper elements of every row are out of bounds and
// arrive as zeros, which is exactly a head_dim 64 tile whose upper half is zero.
inline int make_map(CUtensorMap* map, int dtype, const void* base, int D, long long rows,
                    long long heads, long long head_stride_elems, int box_rows = 128) {
  EncodeTiledFn fn = encode_fn();
  RAB_REQUIRE(fn != nullptr, RA_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t es = dtype == RA_F32 ? 4 : 2;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(rows),
                              static_cast<cuuint64_t>(heads)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(D) * es,
                                 static_cast<cuuint64_t>(head_stride_elems) * es};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(128 / es), static_cast<cuuint32_t>(box_rows), 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUtensorMapDataType type = dtype == RA_F32    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                   : dtype == RA_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                      : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const CUresult r = fn(map, type, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  RAB_REQUIRE(r == CUDA_SUCCESS, RA_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d",
              static_cast<int>(r));
  return RA_OK;
}

// 16-bit queries as (D, rows, kv heads, heads that share one, batch), box = one 128-byte row piece x box_rows x 1 x box_heads x
// 1: the box lands as box_heads times box_rows rows, swizzled as one tile of them.
inline int make_query_map(CUtensorMap* map, int dtype, const StepArgs& a, int box_rows, int box_heads) {
  EncodeTiledFn fn = encode_fn();
  RAB_REQUIRE(fn != nullptr, RA_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t row = static_cast<cuuint64_t>(a.D) * 2, head = row * a.Sq;
  const cuuint64_t dims[5] = {static_cast<cuuint64_t>(a.D), static_cast<cuuint64_t>(a.Sq), static_cast<cuuint64_t>(a.kvH),
                              static_cast<cuuint64_t>(a.H / a.kvH), static_cast<cuuint64_t>(a.B)};
  const cuuint64_t strides[4] = {row, head, head * a.kvH, head * a.H};
  const cuuint32_t box[5] = {64, static_cast<cuuint32_t>(box_rows), 1, static_cast<cuuint32_t>(box_heads), 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUresult r = fn(map, dtype == RA_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5,
                        const_cast<void*>(a.q), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  RAB_REQUIRE(r == CUDA_SUCCESS, RA_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", static_cast<int>(r));
  return RA_OK;
}

// How many blocks the current device holds at once when they come in clusters of n, n = 1..8: asked for
// once per device, with whichever key-split kernel comes first (all of them hold one block per SM, so the
// answers are the same; a cluster lives inside one GPC: 148, 148, 135, 132, 130, 132, 126, 120 on a B200).
struct ClusterSlots {
  std::once_flag once;
  int blocks[9];
};
ClusterSlots& cluster_slots_of(int device);

template <class Kern>
inline int cluster_slots(Kern kern, int threads, int smem_bytes, const int** out) {
  int dev = 0;
  RAB_CUDA(cudaGetDevice(&dev));
  RAB_REQUIRE(dev >= 0 && dev < 64, RA_ERR_INVALID, "device index %d out of range", dev);
  ClusterSlots& t = cluster_slots_of(dev);
  std::call_once(t.once, [&]() {
    for (int n = 0; n <= 8; ++n) t.blocks[n] = 0;
    if (cudaDeviceGetAttribute(&t.blocks[1], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess) {
      cudaGetLastError();
      return;  // no split on this device
    }
    for (int n = 2; n <= 8; ++n) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(n);
      cfg.blockDim = dim3(threads);
      cfg.dynamicSmemBytes = smem_bytes;
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = n;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        clusters = 0;
      }
      t.blocks[n] = clusters * n;
    }
  });
  *out = t.blocks;
  return RA_OK;
}

// Key split: how many blocks of a cluster share the key tiles of one query block (1: no split).
// A block walks its key tiles one after the other, so a call with fewer query blocks than SMs
// leaves SMs idle however many keys there are. Cutting the tile list in n shortens the walk to
// 1/n and costs every block its own prologue and the merge (kFixed and merge_tiles, in tiles of
// work; a query block without a visible key costs kEmpty). The estimate is the walk of the longest
// block while the blocks with work fit the SMs that clusters of that size can occupy (`slots`, see
// ClusterSlots), else the total work over them plus half a block for the last wave.
// Measured, us per call at n = 1 / 2 / 4 / 8 (fp16, causal): 384 rows on 40384 keys H32/kvH8 D128
// 542 / 296 / 303 / 410 (735 before the second tile of the last block was left out); 64 rows on
// 65536 keys H8 D128 1077 / 540 / 277 / 146; 1024 x 1024 H8 D64 23 / 19 / 17 / 38; 2048 x 2048 H16
// D64 (128 blocks) 36 / 38 / 59 / 122; 1024 x 1024 H8 D128 29 / 25 / 18.5 / 49, H16 29 / 25 / 33 / 80;
// 1024 x 1024 H8 D256 (64 blocks) 27 / 29 / 39 / 82; 2048 x 2048 H4 D256 41 / 37 / 41 / 86.
// Four tiles at n = 1 / 2 / 4: 512 x 512 H8 D128 20.5 / 20.5 / 16, fp32 200 x 200 H8 D64 18.5 / 19 / 16.5, D128
// 29 / 28 / 22.6 (so a share may be a single tile); three tiles, fp32 D64: 12.6 at n = 1, 14.4 at 3.
// The figures and constants are from before unsplit blocks stored their rows through shared memory and blocks
// without keys left at once; both cost less now than kFixed and kEmpty say. Over 195 steps of zig-zag ranks (H8 to H16,
// 400 to 2048 rows a segment) the choice is 1.2 % off the best of n = 1 to 4 in the mean and 15 % at worst (H16 D64,
// 400 rows, half of the blocks hidden: 16.2 at the chosen 2, 14.1 at 1).
constexpr double kBlockTiles = 3;  // start and end of a block, in tiles of work
template <int kTileKeys>
inline int pick_key_split(const StepArgs& a, int q_block_rows, double merge_tiles, const int* slots,
                          double* estimate = nullptr) {
  const int forced = static_cast<int>((a.flags >> RA_STEP_KEY_SPLIT_SHIFT) & 15u);
  if (forced) return forced > 8 ? 8 : forced;
  constexpr double kFixed = kBlockTiles, kEmpty = 0.7;
  const int per_seg = (a.qmap.seg_len + q_block_rows - 1) / q_block_rows;
  const long long heads = static_cast<long long>(a.B) * a.H;
  if (heads * per_seg * a.qmap.n_seg >= slots[1]) return 1;
  const bool causal = (a.flags & RA_STEP_CAUSAL) != 0;
  long long total = 0;
  int longest = 0, busy = 0, idle = 0;  // per head
  for (int sq = 0; sq < a.qmap.n_seg; ++sq)
    for (int tq = 0; tq < per_seg; ++tq) {
      const int row0 = tq * q_block_rows;
      const int rows = a.qmap.seg_len - row0 < q_block_rows ? a.qmap.seg_len - row0 : q_block_rows;
      const int qmin = a.qmap.base[sq] + row0 * a.stride;
      int tiles = 0;
      for (int sk = 0; sk < a.kmap.n_seg; ++sk) {
        const TileRange r = tile_range<kTileKeys>(a.kmap, sk, a.stride, causal, a.doc_len, qmin,
                                                  qmin + (rows - 1) * a.stride);
        tiles += r.hi - r.lo;
      }
      total += tiles;
      longest = tiles > longest ? tiles : longest;
      tiles > 0 ? ++busy : ++idle;
    }
  if (busy == 0) return 1;
  const double mean = static_cast<double>(total) / busy;
  constexpr int kSizes[7] = {1, 2, 3, 4, 5, 6, 8};
  int best = 1;
  double best_t = 0;
  for (int i = 0; i < 7; ++i) {
    const int n = kSizes[i];
    if (longest < n) break;
    if (slots[n] == 0) continue;
    const double fixed = kFixed + (n > 1 ? merge_tiles : 0);
    const double empties = static_cast<double>(heads * idle) * n * kEmpty / slots[n];
    double t = (longest + n - 1) / n + fixed + empties;
    const double n_blocks = static_cast<double>(heads * busy) * n;
    if (n_blocks > slots[n]) {
      const double spread = (n_blocks / slots[n] + 0.5) * (mean / n + fixed) + empties;
      t = t > spread ? t : spread;
    }
    if (i == 0 || t < best_t) {
      best = n;
      best_t = t;
    }
  }
  if (estimate) *estimate = best_t;
  return best;
}

// Whether to pair a head's query tiles light with heavy (the first with the last, ...) instead of neighbours.
// For causal calls of one wave or less, whose time is that of the block with the most keys: its two tiles walk
// all of them, the first block's next to none. A folded block walks the heavy tile's keys, alone where the light one
// has ended, and a tile alone takes `alone` of the time of two (its MMAs and its softmax have nothing to
// overlap with); so all blocks take about the same time, but all of them together more: a grid of several
// waves keeps neighbours. `tiles`: the estimate of the best other form (0: none; see pick_key_split). us per
// call, neighbours / two blocks a query block / folded, fp16 causal: 2048 rows H16 D64 31.2 / 34.7 / 25.4; 4096 H8 D64
// 53.8 / 45.6 / 42.8, D128 64.4 / 55.9 / 58.6 (not taken); 1531 B2 H12 D64 29.2 / 34.3 / 21.2, D128 30.8 / 42.3 / 27.6; 512
// H64 D64 12.6 / 26.0 / 12.3; 8192 H4 D64 (not taken) 97.6 / 67.2. From these and 1024 and 1536 rows `alone`: 0.77 to 0.82 at
// head_dim 64 (512 rows 0.94), 0.86 to 0.87 at 128. Over 60 random causal calls of one wave the folded ones (15) are 0.2 %
// off the best form in the mean and 2.5 % at worst.
template <int kTileKeys>
inline bool fold_rows(const StepArgs& a, double alone, double tiles) {
  if (tiles <= 0 || (a.flags & RA_STEP_CAUSAL) == 0 || a.doc_len > 0) return false;
  const int per_seg = (a.qmap.seg_len + kBM - 1) / kBM, n = per_seg * a.qmap.n_seg;
  for (int s = 1; s < a.qmap.n_seg; ++s)  // later tiles see what earlier ones do
    if (a.qmap.base[s] < a.qmap.base[s - 1] + (a.qmap.seg_len - 1) * a.stride) return false;
  auto keys = [&](int lin) {
    const int s = lin / per_seg, row0 = (lin - s * per_seg) * kBM;
    const int rows = a.qmap.seg_len - row0 < kBM ? a.qmap.seg_len - row0 : kBM;
    const int qmin = a.qmap.base[s] + row0 * a.stride;
    int sum = 0;
    for (int sk = 0; sk < a.kmap.n_seg; ++sk)
      sum += tile_range<kTileKeys>(a.kmap, sk, a.stride, true, 0, qmin, qmin + (rows - 1) * a.stride).hi;
    return sum;
  };
  double longest = 0;
  for (int i = 0; i <= n - 1 - i; ++i) {
    const int light = n - 1 - i > i ? keys(i) : 0, heavy = keys(n - 1 - i);
    const double t = light + alone * (heavy - light);
    longest = t > longest ? t : longest;
  }
  return longest + kBlockTiles < 0.95 * tiles;
}

// Spread: the same for a call with a workspace, without clusters. All 128-row query tiles of the query heads that share
// a KV head are paired into blocks (by position, then by head, so that the tiles of a block see about the same keys),
// and block j's key tiles are cut into n_j contiguous shares, a thread block each, for the smallest longest share whose
// blocks all fit the SMs at once. Where a head has at most 64 rows, as many heads as fit share a tile. A share writes its partial (O, m, l) to the workspace and a second launch folds the
// shares into the state. Against the key split: no SM is left out because clusters do not fit (135 of 148 in threes), a
// block may have more than eight shares, grouped heads fill up each other's blocks, and blocks may differ in their number of
// shares; against that stand a launch and the way of the partial states through L2 (`fold_tiles`, in tiles of work).
// Chosen where the estimate is 5 %, and four tiles, below that of the best other form (the workspace and the second launch
// cost the host 5 to 7 us, which a call that is waited for shows). Only from kSpreadKeys keys on: shorter
// calls never gain, and a caller need not ask for a workspace. us per call, key split / spread (16 bits, causal, CUDA
// graphs): 384 rows on 40384 keys H32/kvH8 D128 285 / 211, D64 261 / 177; 64 rows on 65536 keys H8 D128 109 / 62; 16 rows on
// 100000 keys H16/kvH2 D128 212 / 36 (90 with a tile for each head); 144 rows on 32376 keys H2 D64 71 / 28; 700 rows on 9000 keys H8/kvH2 D256 86 / 62; 337
// rows on 8336 keys H16/kvH8 D64 39 / 34. Over 104 random calls (16 to 2048 rows on 1000 to 40000 keys more) that gain by
// more than 5 % in the estimate 0.69 in the mean, 1.05 at worst (19.7 / 20.7, a call that the four tiles now keep out);
// over 41 of 16 to 128 rows, with heads that share tiles, 0.47 and 0.77.
constexpr int kSpreadKeys = RA_STEP_SPREAD_KEYS;
template <int kTileKeys>
inline bool plan_spread(const StepArgs& a, int tiles_per_block, double fold_tiles, int sms, double best_other, Spread* out) {
  if (a.Sk < kSpreadKeys || best_other <= 0 || a.H % a.kvH != 0) return false;
  const long long heads = static_cast<long long>(a.B) * a.kvH;
  const int cap = static_cast<int>(heads < sms ? sms / heads : 0) < kMaxSpread ? static_cast<int>(heads < sms ? sms / heads : 0) : kMaxSpread;
  const int group = a.H / a.kvH;
  const int per_seg = (a.qmap.seg_len + kBM - 1) / kBM;
  // (few rows: the tile's place in the tensor core is paid whether rows stand in it or not)
  const int pack = a.qmap.n_seg == 1 && 2 * a.Sq <= kBM ? std::min(group, kBM / a.Sq) : 1;
  const long long tiles = pack > 1 ? (group + pack - 1) / pack : static_cast<long long>(group) * a.qmap.n_seg * per_seg;
  const long long n_blocks = (tiles + tiles_per_block - 1) / tiles_per_block;
  if (n_blocks > cap) return false;
  int keys[kMaxSpread], longest = 1;
  for (int j = 0; j < n_blocks; ++j) {
    int qmin, qmax;
    spread_span(a.qmap, a.stride, group, per_seg, pack, j * tiles_per_block,
                static_cast<int>((j + 1) * tiles_per_block < tiles ? (j + 1) * tiles_per_block : tiles), &qmin, &qmax);
    keys[j] = 0;
    for (int sk = 0; sk < a.kmap.n_seg; ++sk) {
      const TileRange r = tile_range<kTileKeys>(a.kmap, sk, a.stride, (a.flags & RA_STEP_CAUSAL) != 0, a.doc_len, qmin, qmax);
      keys[j] += r.hi - r.lo;
    }
    longest = keys[j] > longest ? keys[j] : longest;
  }
  auto blocks = [&](int share) {
    int n = 0;
    for (int j = 0; j < n_blocks; ++j) n += keys[j] > share ? (keys[j] + share - 1) / share : 1;
    return n;
  };
  int lo = 1, hi = longest;  // the smallest share that fits is in [lo, hi]
  while (lo < hi) {
    const int mid = (lo + hi) / 2;
    if (blocks(mid) <= cap) hi = mid;
    else lo = mid + 1;
  }
  const double gain = best_other - (lo + kBlockTiles + fold_tiles);
  if (gain < 4 || gain < 0.05 * best_other) return false;
  out->total = 0;
  out->pack = pack;
  for (int j = 0; j < n_blocks; ++j) {
    out->beg[j] = static_cast<unsigned char>(out->total);
    out->total += keys[j] > lo ? (keys[j] + lo - 1) / lo : 1;
  }
  for (int j = static_cast<int>(n_blocks); j <= kMaxSpread; ++j) out->beg[j] = static_cast<unsigned char>(out->total);
  return true;
}

// Limits set through the test hooks (step_tc.cu owns them).
unsigned long long tc_wait_limit_ns();
int tc_stall_after();
// What ra_debug_step_form answers on this thread.
void set_step_form(int form);

}  // namespace tcgen
}  // namespace rab
