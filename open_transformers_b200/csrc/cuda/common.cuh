// Host-side helpers shared by the .cu files of this library.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <atomic>
#include <type_traits>
#include <utility>

typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled is a driver symbol; fetch it through the runtime so the library
// links against libcudart only (it must also load on machines without a driver, for build checks).
inline PFN_encodeTiled get_encode_tiled() {
  static PFN_encodeTiled fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_encodeTiled>(p);
  }
  return fn;
}

// Encoding a tensor map is a driver call and needs a current context, which the runtime gives a thread only with its first
// runtime call that needs one: a thread whose first device work is a product into memory that it already holds (autograd's
// own thread, say) has none yet and gets CUDA_ERROR_INVALID_CONTEXT. It then takes its device's primary context and repeats.
template <typename F>
inline CUresult otb_encode(F encode) {
  CUresult r = encode();
  int dev = 0;
  if (r == CUDA_ERROR_INVALID_CONTEXT && cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) {
    r = encode();
    if (r == CUDA_ERROR_INVALID_CONTEXT && cudaFree(nullptr) == cudaSuccess) r = encode();
  }
  return r;
}

inline int otb_sm_count() {
  static int sm[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  if (sm[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    sm[dev] = n;
  }
  return sm[dev];
}

// Lets KERN take `bytes` of dynamic shared memory. The attribute belongs to the current device, so it is remembered for each
// device by itself; two threads that come first together both set it. An error is not remembered.
template <auto KERN>
inline int otb_allow_smem(int bytes) {
  static std::atomic<bool> allowed[64];
  int dev = 0;
  if (const cudaError_t e = cudaGetDevice(&dev)) return (int)e;
  const bool kept = dev >= 0 && dev < 64;
  if (kept && allowed[dev].load(std::memory_order_acquire)) return 0;
  if (const cudaError_t e = cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)) return (int)e;
  if (kept) allowed[dev].store(true, std::memory_order_release);
  return 0;
}

// Launches that may begin before the kernel in front of them in the stream has ended: at its end without the pause of an
// ordinary launch, or, where that kernel calls let_successor_begin(), as soon as all its CTAs are there. In front of an ordinary
// launch the order of the stream is the ordinary one.
// Behind a predecessor: the kernel waits for it before it touches any memory. What overlaps is the launch, the CTAs' start and
// their set-up (barriers, tensor memory), which a chain of kernels of 4 to 15 us pays one after the other otherwise. The memory-bound
// kernels and the products are launched that way, and the attention forward where it is small. Which of them lets its successor
// begin is what decides: memory-bound kernels and the attention do where a product follows, whose CTAs take an SM each; a product does
// not, since small CTAs that are placed while it runs pile up on the SMs that happen to have room (what it costs is a product behind a
// product: 333 x 768 x 768 with residual back to back 6.9 ordinary, 6.4 so, 5.9 with the former letting go). us, every launch ordinary / so /
// every small grid early and every kernel letting go at its start: block without gradients, 768 wide, 16 tokens 45.0 / 39.4 / 40.4, 333
// tokens 52.0 / 47.5 / 52.6, 2048 wide, 128 tokens 78.2 / 72.8 / 79.3, 1111 tokens 146 / 142 / 152; feed-forward sublayer forward and
// backward, 2048 wide, 128 tokens 128 / 125 / 132. With the memory-bound kernels launched in the ordinary way a block of 333 tokens takes
// 48.1, and a micro-batch of the two-layer fp32 decoder 2065 instead of 2007.
// A kernel that waits exists while what it reads is still being written. Its inputs, and what it both reads and writes, are
// therefore not __restrict__ and not read by __ldg: either would tell the compiler that nothing changes them while the kernel
// runs, and let it take a load past the wait, whose "memory" clobber covers only what others may write. Buffers that are only
// written may be __restrict__, as what goes into them follows from loads behind the wait.
// Side by side, where two kernels need nothing of each other: the first, launched in the ordinary way, calls
// let_successor_begin(), so that all that ran before it is complete by then; the second touches memory at once and lets one
// thread call wait_for_predecessor() at its end, so that what follows in the stream waits for both. It reads nothing that its
// predecessor writes and may say so.
__device__ __forceinline__ void let_successor_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void after_predecessor() {
  let_successor_begin();
  wait_for_predecessor();
}
// A launch that is refused is tried once in the ordinary way, which is right in either use, and whose error is the one to report.
// The code returned is the only report: nothing is left pending for the next reader of the runtime's last error, and an entry
// point with several launches looks at each, because the retry clears what an earlier one left there.
template <typename... P>
inline int otb_launch_args(bool early, const void* kern, dim3 grid, dim3 block, size_t smem, cudaStream_t s, P... v) {
  void* argv[] = {const_cast<void*>(static_cast<const void*>(&v))...};
  if (early) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelExC(&cfg, kern, argv) == cudaSuccess) return 0;
    (void)cudaGetLastError();
  }
  const int rc = (int)cudaLaunchKernel(kern, grid, block, argv, smem, s);
  if (rc) (void)cudaGetLastError();
  return rc;
}
template <typename... P, typename... A>
inline int otb_launch_if_early(bool early, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  return otb_launch_args<P...>(early, reinterpret_cast<const void*>(kern), grid, block, smem, s, static_cast<P>(args)...);
}
template <typename... P, typename... A>
inline int otb_launch(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  return otb_launch_if_early(false, kern, grid, block, smem, s, args...);
}
template <typename... P, typename... A>
inline int otb_launch_early(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  return otb_launch_if_early(true, kern, grid, block, smem, s, args...);
}

#define OTB_CUDA_CHECK_RET(expr)              \
  do {                                        \
    cudaError_t _e = (expr);                  \
    if (_e != cudaSuccess) return (int)_e;    \
  } while (0)

// OTB_PACKED(entry) adds `entry_p`, which takes the arguments of the C entry point as one array of 8-byte words (integers
// and pointers as 64-bit integers, floats as doubles). Python builds that array with one struct.pack, several times cheaper
// than an object per argument; the hot entry points are called this way.
template <typename T>
inline T otb_packed_arg(const char* word) {
  if constexpr (std::is_pointer<T>::value) {
    uint64_t v;
    memcpy(&v, word, 8);
    return reinterpret_cast<T>(static_cast<uintptr_t>(v));
  } else if constexpr (std::is_floating_point<T>::value) {
    double v;
    memcpy(&v, word, 8);
    return static_cast<T>(v);
  } else {
    int64_t v;
    memcpy(&v, word, 8);
    return static_cast<T>(v);
  }
}
template <typename... A, size_t... I>
inline int otb_packed_call(int (*f)(A...), const char* words, std::index_sequence<I...>) {
  return f(otb_packed_arg<A>(words + 8 * I)...);
}
template <typename... A>
inline int otb_packed(int (*f)(A...), const char* words) {
  return otb_packed_call(f, words, std::index_sequence_for<A...>());
}
#define OTB_PACKED(entry) \
  extern "C" int entry##_p(const char* words) { return otb_packed(entry, words); }
