// Blackwell (sm_100a) building blocks shared by every kernel in this library:
// mbarrier with bounded waits, TMA tile copies, TMEM allocation, tcgen05 MMA
// issue/commit, TMEM loads/stores and the shared-memory operand descriptors.
//
// Conventions
//  * Every wait on an mbarrier is bounded (WAIT_LIMIT_CYCLES). When a wait gives up
//    it records a code in the device status word and returns false; callers
//    leave their loops and fall through to the common tear-down, which frees
//    TMEM. A kernel that timed out therefore returns; the host reads the status.
//  * Shared-memory operand tiles are K-major, rows of 128 B (64 bf16) under the
//    128-byte swizzle, or rows of 64 B (32 bf16) under the 64-byte swizzle. Tiles
//    start on 1024-byte boundaries.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

constexpr long long WAIT_LIMIT_CYCLES = 4000000000ll;  // about 2 s of SM clock per wait

// Status codes written by kernels (0 = fine).
enum : int {
  ST_OK = 0,
  ST_TIMEOUT_PRODUCER = 101,
  ST_TIMEOUT_MMA = 102,
  ST_TIMEOUT_EPILOGUE = 103,
  ST_TIMEOUT_PROLOGUE = 104,
  ST_TIMEOUT_SOFTMAX = 105,
  ST_TIMEOUT_SELFTEST = 110,  // the wait of b200tri_selftest_wait ran out (as it is meant to)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " elect.sync _|p, 0xffffffff;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      // the last operand is the suspend-time hint: the hardware parks the thread until
      // the phase completes (or this many ns pass), so a waiting warp issues almost no
      // instructions instead of competing with the working warps of its sub-partition
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 0x989680;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Has the phase completed? Does not wait.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait. `status` points at the device status word (global memory).
// Gives up after WAIT_LIMIT_CYCLES, or as soon as another thread has recorded a
// failure, so that one stuck role drains the whole CTA quickly.
__device__ __forceinline__ bool mbar_wait_limited(uint64_t* bar, uint32_t parity, int* status, int code,
                                                  long long limit_cycles, uint32_t check_mask) {
  // Fast path: a few plain polls (the hardware parks the thread inside try_wait),
  // no clock reads on the way.
#pragma unroll 1
  for (int i = 0; i < 32; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & check_mask) == 0) {
      if (*reinterpret_cast<volatile int*>(status) != ST_OK) return false;
      if (clock64() - t0 > limit_cycles) {
        atomicCAS(status, ST_OK, code);
        return false;
      }
    }
  }
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, int code) {
  return mbar_wait_limited(bar, parity, status, code, WAIT_LIMIT_CYCLES, 0x3fu);
}

// ---------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(m), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::
          "r"(smem_u32(dst)),
      "l"(m), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z,
                                            int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(smem_u32(dst)),
      "l"(m), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}

__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z,
                                            int w, int v) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], "
      "[%2];" ::"r"(smem_u32(dst)),
      "l"(m), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(v)
      : "memory");
}

// Tiled TMA store, shared memory -> global (bulk async-group completion). The tile must have
// been written with ordinary shared-memory stores followed by fence_proxy_async() and a
// barrier; elements outside the tensor are not written.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* src, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(m),
               "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(m),
               "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(m), "r"(smem_u32(src)),
               "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Until the stores committed so far have READ their shared-memory source (it may be reused).
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// The end of a kernel that stores by TMA. The device status word is asked for while the last stores read their
// tiles (a trip to L2 on its own otherwise, 0.3 us of a launch of one tile per SM); the grid is complete when they
// are written, so nothing waits for that here. Nothing that can give up on a wait follows in the warp.
__device__ __forceinline__ int ask_status(const int* status) {
  int st;
  asm volatile("ld.volatile.global.s32 %0, [%1];" : "=r"(st) : "l"(status) : "memory");
  return st;
}
__device__ __forceinline__ int stores_read_and_status(bool stored, const int* status) {
  const int st = ask_status(status);
  if (stored) tma_store_wait_read();
  return st;
}
// Tear-down of a warp: `status` as it was asked for, or -1. After a timeout (of this warp, or of another: that
// one comes here too, and they meet at a barrier next) give in-flight bulk copies time to land first.
__device__ __forceinline__ void settle(int status, const int* word) {
  if ((status >= 0 ? status : *reinterpret_cast<const volatile int*>(word)) != ST_OK)
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
}

// ---------------------------------------------------------------- TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_in_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_in_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Arrive on `bar` once every tcgen05.mma issued so far by this thread is done.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]^T, bf16 operands, fp32 accumulate.
__device__ __forceinline__ void umma_bf16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Same with the A operand read from TMEM (bf16 pairs packed in 32-bit columns).
__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Instruction descriptor for kind::f16 with bf16 A/B, fp32 D, both operands
// K-major, MMA shape M x N (K = 16 per instruction).
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
  return (1u << 4)                          // D format: fp32
         | (1u << 7)                        // A format: bf16
         | (1u << 10)                       // B format: bf16
         | (static_cast<uint32_t>(N >> 3) << 17)  // N / 8
         | (static_cast<uint32_t>(M >> 4) << 24); // M / 16
}

// Shared-memory matrix descriptor, K-major tile. `row_bytes` is 128 (swizzle
// 128B), 64 (swizzle 64B) or 32 (swizzle 32B); eight rows form one swizzle atom and atoms follow
// one another every 8*row_bytes bytes.
__device__ __forceinline__ uint64_t umma_desc_kmajor(uint32_t saddr, uint32_t row_bytes) {
  const uint64_t swz = (row_bytes == 128) ? 2ull : (row_bytes == 64 ? 4ull : 6ull);
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);        // start address
  d |= static_cast<uint64_t>(((8u * row_bytes) >> 4) & 0x3FFFu) << 32;  // stride between 8-row atoms
  d |= 1ull << 46;                                             // descriptor version (sm_100)
  d |= swz << 61;
  return d;
}
// The same for an MN-major tile under the 128-byte swizzle: smem row = one k, 128 B = 64
// consecutive M (or N) elements, eight k rows per atom. `group_bytes` separates successive
// groups of 64 M/N elements; atoms along K follow one another every 1024 bytes, so stepping
// K by 16 advances the start address by 2048. A linear kernel stored [in][out] is loaded by
// TMA straight into this form: no transposed copy of a weight is ever made.
__device__ __forceinline__ uint64_t umma_desc_mnmajor(uint32_t saddr, uint32_t group_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((group_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((1024u >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}
constexpr uint32_t UMMA_A_MN = 1u << 15, UMMA_B_MN = 1u << 16;  // instruction descriptor: operand is MN-major
// Step the descriptor along K by `bytes` inside the swizzled row.
__device__ __forceinline__ uint64_t umma_desc_advance(uint64_t d, uint32_t bytes) { return d + (bytes >> 4); }

// ------------------------------------------------------------ TMEM <-> regs
// 32 lanes x 32 bit, 32 consecutive columns: thread t of the warp gets lane
// (base lane + t), registers r[0..31] get columns c..c+31.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ------------------------------------------------------------------ helpers
// 32 bytes in one access (address on a 32-byte boundary): a whole sector of L2 instead of two halves.
// For threads that each walk a row of their own, where every access of a warp touches 32 lines.
__device__ __forceinline__ void store_sector(void* dst, const uint4& a, const uint4& b) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
               "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
               : "memory");
}
__device__ __forceinline__ void load_sector(const void* src, uint4& a, uint4& b) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
               : "l"(src)
               : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x = lo (low half), .y = hi
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
// v + a packed pair's two values, rounded once: an instruction each, against two to unpack and half a packed addition.
__device__ __forceinline__ float2 add_bf16x2(float2 v, uint32_t w) {
  float2 r;
  asm("{\n"
      " .reg .b16 lo, hi, one;\n"
      " mov.b32 {lo, hi}, %2;\n"
      " mov.b16 one, 0x3F80;\n"
      " fma.rn.f32.bf16 %0, lo, one, %3;\n"
      " fma.rn.f32.bf16 %1, hi, one, %4;\n"
      "}\n"
      : "=f"(r.x), "=f"(r.y)
      : "r"(w), "f"(v.x), "f"(v.y));
  return r;
}
// The sum of a packed pair's two values.
__device__ __forceinline__ float sum_bf16x2(uint32_t w) {
  float r;
  asm("{\n"
      " .reg .b16 lo, hi, one;\n"
      " mov.b32 {lo, hi}, %1;\n"
      " mov.b16 one, 0x3F80;\n"
      " fma.rn.f32.bf16 %0, lo, one, %2;\n"
      "}\n"
      : "=f"(r)
      : "r"(w), "f"(bf16_hi(w)));
  return r;
}
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Packed bf16 arithmetic (the _rn forms, which the compiler may not contract into
// an fma): one rounding per operation, which is exactly what the
// reference's XLA path does wherever it multiplies or adds two bf16 arrays.
__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, uint32_t b) {
  __nv_bfloat162 r = __hmul2_rn(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf16x2_add(uint32_t a, uint32_t b) {
  __nv_bfloat162 r = __hadd2_rn(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}

// sigmoid in fp32 to ~1e-6 relative: one ex2 and one rcp (the flushing approximate
// forms, a single MUFU operation each with no range fix-up around them), the
// multiply and the add packed two at a time. The gates are rounded to bf16
// afterwards like the reference's; a cheaper tanh-based sigmoid (2^-11) flips
// that rounding often enough to push the mean error past the parity budget.
// Saturation is exact: x -> -inf gives rcp(inf) = 0, x -> +inf gives rcp(1) = 1.
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 sigmoid_f32x2(float2 x) {
  const float2 t = __fmul2_rn(x, make_float2(-1.4426950408889634f, -1.4426950408889634f));
  const float2 d = __fadd2_rn(make_float2(fast_exp2(t.x), fast_exp2(t.y)), make_float2(1.0f, 1.0f));
  return make_float2(fast_rcp(d.x), fast_rcp(d.y));
}

// bf16(sigmoid(bf16(g0))), bf16(sigmoid(bf16(g1))) packed: the reference's
// sigmoid(x @ w) on a bf16 trunk.
__device__ __forceinline__ uint32_t sigmoid_bf16x2(float g0, float g1) {
  const uint32_t g = pack_bf16x2(g0, g1);
  const float2 s = sigmoid_f32x2(make_float2(bf16_lo(g), bf16_hi(g)));
  return pack_bf16x2(s.x, s.y);
}
// max of three (one instruction on sm_100).
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Mask bias of one key: inf * (mask - 1), or the caller's additive bias as it is. A value at or
// below MASKED_SCORE replaces the score (see the attention core). fmaxf drops a NaN operand, so a
// NaN bias would silently become "keep": it is mapped to "drop".
constexpr float MASKED_SCORE = -30000.0f;
__device__ __forceinline__ float mask_bias(float m, float inf, bool additive) {
  const float b = additive ? m : inf * (m - 1.0f);
  return (b == b) ? fmaxf(b, MASKED_SCORE) : MASKED_SCORE;
}
// Byte offset of (row, 16-byte chunk) inside a K-major tile with 128-byte rows
// under the 128-byte swizzle (the layout TMA writes and tcgen05.mma reads).
__device__ __forceinline__ uint32_t sw128_offset(uint32_t row, uint32_t chunk) {
  return row * 128u + (((chunk ^ row) & 7u) << 4);
}

// Programmatic dependent launch. A kernel launched with the attribute may start while its
// predecessor in the stream still runs; pdl_wait() returns once that predecessor has finished
// and its writes are visible. pdl_trigger() lets the successor be scheduled as soon as every
// CTA of this grid has got there. Both do nothing in a plain launch.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Named barrier among `nthreads` threads (id 1..15; 0 is __syncthreads()).
__device__ __forceinline__ void named_barrier(uint32_t id, uint32_t nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// The same barrier with an AND-reduction of a predicate: every thread learns whether ALL of
// them passed `ok`. Used after a bounded wait whose result must be acted on by a whole group
// that later meets at a named barrier: if one thread gave up and left while the others
// proceeded, the next barrier would never complete.
__device__ __forceinline__ bool named_barrier_and(uint32_t id, uint32_t nthreads, bool ok) {
  uint32_t out;
  asm volatile(
      "{\n"
      " .reg .pred p, q;\n"
      " setp.ne.u32 q, %3, 0;\n"
      " bar.red.and.pred p, %1, %2, q;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(out)
      : "r"(id), "r"(nthreads), "r"(static_cast<uint32_t>(ok))
      : "memory");
  return out != 0;
}

}  // namespace b200
