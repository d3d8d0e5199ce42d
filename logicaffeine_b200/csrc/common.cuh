// Shared internals of liblogos_b200: status/error plumbing, the handle
// registry, and small device helpers.  Nothing here is part of the C ABI.
#pragma once
#include <utility>

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <string>

#include "../../include/logos_b200.h"

namespace logos {

// ---------------------------------------------------------------- errors
// Per-thread message store, read through logos_b200_last_error(); same contract as
// the reference's thread-keyed store (crates/logicaffeine_compile/src/codegen/ffi.rs:214-251).
void set_last_error(const std::string& msg);
const char* last_error_text();  // null when the calling thread has no pending message
void clear_last_error();
logos_status_t fail(logos_status_t code, const char* fmt, ...);
logos_status_t cuda_fail(cudaError_t e, const char* what);

#define LOGOS_CUDA_TRY(expr)                                            \
  do {                                                                  \
    cudaError_t _e = (expr);                                            \
    if (_e != cudaSuccess) return ::logos::cuda_fail(_e, #expr);        \
  } while (0)

#define LOGOS_TRY(expr)                                                 \
  do {                                                                  \
    logos_status_t _s = (expr);                                         \
    if (_s != LOGOS_OK) return _s;                                      \
  } while (0)

// Every extern "C" body runs inside this guard: a C++ exception never crosses
// the ABI (the reference wraps each export in catch_unwind, ffi.rs:329-345).
template <class F>
logos_status_t guarded(F&& f) {
  try {
    return f();
  } catch (const std::bad_alloc&) {
    return fail(LOGOS_MEMORY_EXHAUSTED, "host allocation failed");
  } catch (const std::exception& e) {
    return fail(LOGOS_THREAD_PANIC, "internal exception: %s", e.what());
  } catch (...) {
    return fail(LOGOS_THREAD_PANIC, "internal exception");
  }
}

// ---------------------------------------------------------------- handles
enum class ObjKind : uint32_t { DevBuf = 1, Model = 2 };

struct DevBuf {
  void*   ptr = nullptr;
  int64_t bytes = 0;
  int32_t device = 0;
};

// Registers an object and returns its id (never 0).  The id packs a slot
// counter; a freed id is never reused, so stale handles stay invalid.
logos_handle_t registry_put(ObjKind kind, void* obj);
// Looks an id up; nullptr when unknown or of another kind.
void* registry_get(logos_handle_t h, ObjKind kind);
// Removes the id and returns the object, nullptr when unknown.
void* registry_take(logos_handle_t h, ObjKind kind);

// Resolves a device buffer handle, checking that [offset, offset+need) fits.
logos_status_t buf_resolve(logos_handle_t h, int64_t offset, int64_t need, const char* name, DevBuf** out);

template <class T>
logos_status_t buf_ptr(logos_handle_t h, int64_t elems, const char* name, T** out, int32_t* device = nullptr) {
  DevBuf* b = nullptr;
  LOGOS_TRY(buf_resolve(h, 0, elems * (int64_t)sizeof(T), name, &b));
  *out = reinterpret_cast<T*>(b->ptr);
  if (device) *device = b->device;
  return LOGOS_OK;
}

// Per-device scratch the library owns, for the stand-alone operators (activation planes and
// split-K partials of logos_q8_gemm*).  One block
// per (device, slot), shared by every caller on that device: calls that use it must be ordered
// on the GPU (one stream, or the caller's own events).  Grows on demand, outside any stream
// capture; outgrown blocks are kept until the process exits.  A model never uses it: what a
// captured decode step points at is owned by the model.
logos_status_t scratch_get(int32_t device, int slot, int64_t bytes, void** out);
// The same for a caller that can do without: false, and no error, if the block would have to grow while `st` is being
// captured, or there is no memory left for it.
bool scratch_try(int32_t device, int slot, int64_t bytes, cudaStream_t st, void** out);

// Whether `st` is being captured, as far as can be told: nothing may be allocated then.
bool stream_capturing(cudaStream_t st);

// Arrival counters of the attention calls that advance the lengths, one block per device (every call asks for the same
// size), zeroed when it is allocated; the kernels leave them at zero.  Ordered like scratch_get's blocks.
logos_status_t counters_get(int32_t device, int64_t bytes, void** out);
// A kernel that gave up may leave them in the middle of a count: zeroes them once such a failure has been read.
logos_status_t counters_reset(int32_t device);

// cudaFuncAttributeMaxDynamicSharedMemorySize of `kernel` on the current device, raised to `bytes` once instead of
// on every launch; never lowered, whichever threads call.
logos_status_t allow_smem(const void* kernel, int device, int bytes);

int sm_count(int device);

// Per-device status word in device memory: kernels store a non-zero code when
// a bounded wait gives up.  0 = fine.  Allocated when first asked for; without may_allocate null until then.
int* kernel_status_ptr(int device, bool may_allocate = true);
constexpr int KERNEL_STATUS_WORDS = 8;
logos_status_t kernel_status_read(int device, int* out, bool clear);
// the same for words that the caller has copied to the host already
logos_status_t kernel_status_judge(int device, const int (&words)[KERNEL_STATUS_WORDS], int* out, bool clear);

// ---------------------------------------------------------------- launch helpers
logos_status_t check_launch(const char* kernel);

// Process-wide count of kernel launches by kind (read through logos_launch_counts).
enum LaunchKind : int {
  LK_GEMV = 0, LK_GEMM_TC = 1, LK_GEMM_SIMT = 2, LK_ATTN = 3, LK_ELEMWISE = 5, LK_SYNTH = 6,   // 4 is free
  LK_KINDS = 8
};
void count_launch(int kind, int64_t n = 1);

static inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// ---------------------------------------------------------------- programmatic dependent launch
// Inside a PdlScope (the decode step opens one) kernels are launched so that the next kernel in
// the stream may start while the previous one is still running: its CTAs are scheduled, do the
// work that depends on nothing (barrier set-up, tensor-memory allocation, fetching WEIGHTS, which
// nothing in a decode step writes) and then block in pdl_wait() until the previous kernel has
// completed and its writes are visible.  The contract every kernel of the step keeps:
//   * before pdl_wait() no write, and no read of anything that a kernel still running can write: weights only, and
//     in a decode step the lengths and cached rows, whose writers are over by then (AttnArgs::early_reads);
//   * at least the threads that do such accesses call pdl_wait(), and every path through the
//     kernel has some thread calling it (so "this kernel completed" implies "its predecessor did");
//   * pdl_trigger() after the point where a successor's CTAs may take up SM resources.
// Outside a scope the launch is an ordinary one and both calls are no-ops.
//
// A stand-alone operator outside a scope opens an OrderedScope: its first kernel is launched the same way, but waits
// before it reads or writes anything and triggers only after that, so that its effects are those of an ordinary
// launch: whatever starts early behind it starts when all before it has ended.  What is saved is the gap between two
// kernels of a stream, two to three microseconds with ordinary launches (calls in a row: q8_gemv of 4096 x 4096 8.19 ->
// 5.63 us, a short attention call 8.20 -> 6.46, q8_gemm_f32 of 64 x 3584 x 2368 15.5 -> 13.7).  In a stream that is being
// captured the launch is an ordinary one: what precedes it need not be a kernel.
enum class PdlMode { Off, Early, Ordered };
bool pdl_active();
// in a scope of the first kind: weights may be read before the wait
bool pdl_early();
// LOGOS_B200_PDL=0 in the environment: the library opens no scopes of its own
bool pdl_enabled();
struct PdlScope {
  PdlMode prev;
  explicit PdlScope(bool on);
  ~PdlScope();
};
struct OrderedScope {
  PdlMode prev;
  explicit OrderedScope(cudaStream_t st);
  ~OrderedScope();
};

#if defined(__CUDACC__)
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                 Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_active() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
#endif

}  // namespace logos
