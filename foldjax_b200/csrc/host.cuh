// Host-side plumbing shared by the translation units of libb200tri: error
// reporting, the device status word, TMA descriptor encoding (through the
// driver entry point, so the library does not link libcuda and still loads on
// a machine without a GPU), and the workspace carve-up helper.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/b200tri.h"

namespace b200 {

// Thread-local message behind b200tri_last_error().
void set_error(const char* fmt, ...);
const char* get_error();

// Address of this device's status word (global memory, zero = fine). Kernels
// record a bounded-wait timeout there.
int* device_status_word();

#define B200_CUDA_OK(expr)                                                              \
  do {                                                                                  \
    cudaError_t _e = (expr);                                                            \
    if (_e != cudaSuccess) {                                                            \
      b200::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, \
                      __LINE__);                                                        \
      return B200TRI_ERR_CUDA;                                                          \
    }                                                                                   \
  } while (0)

#define B200_REQUIRE(cond, code, ...) \
  do {                                \
    if (!(cond)) {                    \
      b200::set_error(__VA_ARGS__);   \
      return (code);                  \
    }                                 \
  } while (0)

enum class Swz { None, B32, B64, B128 };

// Encode a tiled tensor map over `rank` dimensions (innermost first).
// strides_bytes[i] is the byte stride of dimension i+1 (dimension 0 is dense).
int make_tmap(CUtensorMap* out, const void* base, CUtensorMapDataType dtype, int rank, const uint64_t* dims,
              const uint64_t* strides_bytes, const uint32_t* box, Swz swz);

// Carves aligned pieces out of a caller-provided workspace.
struct Carver {
  uint8_t* base;
  size_t off = 0;
  explicit Carver(void* p) : base(static_cast<uint8_t*>(p)) {}
  template <typename T>
  T* take(size_t count, size_t align = 1024) {
    off = (off + align - 1) / align * align;
    T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
    off += count * sizeof(T);
    return p;
  }
  size_t total() const { return (off + 1023) / 1024 * 1024; }
};

inline int round_up(int x, int m) { return (x + m - 1) / m * m; }

// Division by a number that a launch knows and its kernel does not: a high product, an addition and two shifts
// (Granlund and Montgomery, Division by Invariant Integers using Multiplication, 1994, figure 4.1) for every 32-bit
// dividend. An integer division by an argument is some 20 instructions, and a warp of a small tile's epilogue made several
// (four updates of a 100-token template, with masks multiplied only where there are any, 98.3 -> 95.8 us; float32, 100 tokens,
// 243 -> 240; a 150-token refiner 489 -> 484).
struct Divisor {
  uint32_t d, m;
  uint8_t first, second;
  Divisor() = default;
  explicit Divisor(uint32_t by) : d(by) {  // by > 0
    int log2up = 0;
    while ((1ull << log2up) < by) ++log2up;
    m = static_cast<uint32_t>((((1ull << log2up) - by) << 32) / by + 1);
    first = log2up < 1 ? log2up : 1;
    second = log2up < 1 ? 0 : log2up - 1;
  }
  __host__ __device__ __forceinline__ uint32_t quotient(uint32_t x) const {
#ifdef __CUDA_ARCH__
    const uint32_t high = __umulhi(m, x);
#else
    const uint32_t high = static_cast<uint32_t>(static_cast<uint64_t>(m) * x >> 32);
#endif
    return (high + ((x - high) >> first)) >> second;
  }
};

// SMs the persistent kernels of the current device may use (its SM count, or the limit
// set for that device with b200tri_set_sm_limit).
int sm_count();
// While one of these lives, sm_count() on this host thread returns `keep` SMs fewer than before
// (one inside another adds to it): the context-parallel ops leave room beside a persistent kernel
// for the small NCCL kernels that carry their tokens (a kernel that fills every SM would hold them
// back until it ends), and a stack of blocks keeps its pair bias to the SMs that are left over.
struct SmReserve {
  int before;
  explicit SmReserve(int keep);
  ~SmReserve();
};

// Raises a kernel's dynamic shared-memory limit, once per (kernel, device); safe to call
// from several host threads (one per device under XLA).
int ensure_smem_limit(const void* kernel, int bytes);

void count_launch(int n = 1);

// Launches a kernel, counted. `pdl` lets it start before its predecessor in the stream has
// drained (programmatic dependent launch): only for a kernel that calls pdl_wait() before it
// touches anything the predecessor reads or writes.
template <typename... KArgs, typename... Args>
int launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pdl, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  count_launch();
  B200_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...));
  return B200TRI_OK;
}

// While one of these lives, the library's launches on this host thread are chained: the kernel
// before the next one in the stream was launched by the same call. A chained kernel may start
// early (launch with pdl) and may read the caller's weights before pdl_wait(): every kernel of
// the library triggers its successor only after its own pdl_wait(), so whatever wrote the
// weights has finished by then.
struct PdlChain {
  bool before;
  explicit PdlChain(bool on = true);
  void set();
  ~PdlChain();
};
bool pdl_chained();

// A second stream for work of one call that does not depend on what the caller's stream does
// meanwhile. Taken from a per-device pool for the duration of the call (several host threads
// each get their own) and given back with the call's work enqueued: everything put on it is
// ordered by events, so the next user may follow at once. `stream` is null when there is none to
// be had or the caller's stream is being captured (a stream of the pool must not stay part of
// somebody's capture), and the call stays on one stream.
struct SideStream {
  cudaStream_t main, stream = nullptr;
  cudaEvent_t to_side = nullptr, to_main = nullptr, early = nullptr;
  bool joined = true;
  explicit SideStream(cudaStream_t main);
  ~SideStream();  // joins if need be
  SideStream(const SideStream&) = delete;
  SideStream& operator=(const SideStream&) = delete;
  int fork();  // what follows on the side stream comes after what is on the main stream now
  int mark();  // `join` waits for what is on the side stream now
  int join();  // what follows on the main stream comes after the last mark
  // A mark and a join of their own for something the main stream needs sooner than the rest.
  int mark_early();
  int join_early();
};

// A weight as TMA needs it: `w` itself when it is 16-byte aligned, else a copy in `scratch`.
int aligned_weight(const void* w, size_t bytes, void* scratch, cudaStream_t stream, const void** out);

// Tensor map over a [k][n] bf16 linear kernel as stored (row pitch n), read in boxes of 64
// columns x `box_k` rows: MN-major operand tiles under the 128-byte swizzle.
int make_weight_map(CUtensorMap* out, const void* w, int k, int n, int box_k);

// TMA clips the rows of a bf16 output at a multiple of 16 bytes. `pad_is_scratch`: what lies between a
// row's end and the next multiple of 8 elements may be written, so an output may leave by TMA whatever
// its width.

// The projection stage of the multiplicative update.
int mul_project_launch(const b200tri_trimul_project_args* a, bool pad_is_scratch, cudaStream_t stream);

// A contraction over `channels` channel planes. `terms` (if any) replaces the sources by a list
// of operand-plane pairs accumulated one after the other in the same float32 accumulator: the
// piece products of split operands, smallest first, so that only the leading one is summed at
// full magnitude.
struct ContractTerms {
  int n;
  uint8_t a[8], b[8];
};
int contract_launch(const b200tri_trimul_contract_args* a, int channels, const ContractTerms& terms, bool pad_is_scratch,
                    cudaStream_t stream);

// The mask-bias rows of the attention core, written by the projection stage of the same call.
struct MaskBiasOut {
  const float* mask;  // null = all ones
  long long ms_outer, ms_inner;
  float inf;
  float* out;  // [n_outer][ld]
  int ld;
};
int att_project_launch(const b200tri_triatt_project_args* a, const MaskBiasOut* mb, cudaStream_t stream);
// The core with its mask-bias rows already in the workspace.
// `strides` (null: q, k and o are [row][token][head][32]): where a token, a head and a row of q / o
// (head_j, row_j) and of k (head_k, row_k) start, in elements and in multiples of 8.
struct CoreStrides {
  long long token, head_j, head_k, row_j, row_k;
};
int att_core_launch_premasked(const b200tri_triatt_core_args* a, const CoreStrides* strides, cudaStream_t stream);

// The two module-level ops for every shape / element type outside the tensor-core
// specialisation (generic.cu): other channel and head counts, float32 trunks.
size_t trimul_workspace_bytes_generic(int32_t n, int32_t c_z, int32_t c_hidden, int32_t dtype);
size_t triatt_workspace_bytes_generic(int32_t n, int32_t c_z, int32_t heads, int32_t head_dim, int32_t dtype);
int trimul_forward_generic(const b200tri_trimul_args* a, int c_z, int c_hidden, cudaStream_t stream);
int triatt_forward_generic(const b200tri_triatt_args* a, int c_z, cudaStream_t stream);

// Launch accounting and optional per-kernel event timing.
enum KernelId { K_TRIMUL_PROJECT = 0, K_TRIMUL_CONTRACT, K_TRIMUL_FINISH, K_TRIATT_PROJECT, K_TRIATT_CORE,
                K_TRIATT_FINISH, K_PAIR_TRANSITION, K_PAIR_BIAS, K_CP_EXCHANGE, K_CP_READY, K_CP_COPY, K_COUNT };
bool timing_enabled();
struct TimedLaunch {  // brackets the launches made during its lifetime
  int id;
  cudaStream_t stream;
  cudaEvent_t start = nullptr;
  TimedLaunch(int id, cudaStream_t stream, bool may_time = true);
  ~TimedLaunch();
};

}  // namespace b200
