// Shared host/device helpers of the montjoie_gb300 library.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "montjoie_gb300.h"

namespace mj {

// Largest supported order r (n = r + 1 points per axis).
constexpr int kMaxOrder = 8;
constexpr int kMaxN = kMaxOrder + 1;

// Element count padding of the element-major layout: a multiple of every
// tile size the element kernels use, so any of them covers the mesh with
// whole tiles of empty (zero) padding elements.
constexpr int kElemPad = 240;

// Slots per element: n^3 rounded up to 4, so per-element blocks of int32,
// float and double start on 16-byte boundaries (the bulk-copy rule).
__host__ __device__ constexpr int elem_slots(int n) { return (n * n * n + 3) / 4 * 4; }

void set_error(const std::string& msg);
std::atomic<uint64_t>& launch_counter();

inline void count_launch(uint64_t n = 1) { launch_counter().fetch_add(n, std::memory_order_relaxed); }

// Evaluates a CUDA call; on failure records the error and returns MJ_ERR_CUDA
// (MJ_ERR_NOMEM for allocation failures) from the calling function.
#define MJ_CUDA(call)                                                                       \
  do {                                                                                      \
    cudaError_t mj_err_ = (call);                                                           \
    if (mj_err_ != cudaSuccess) {                                                           \
      ::mj::set_error(std::string(#call) + ": " + cudaGetErrorString(mj_err_));             \
      return mj_err_ == cudaErrorMemoryAllocation ? MJ_ERR_NOMEM : MJ_ERR_CUDA;             \
    }                                                                                       \
  } while (0)

#define MJ_CHECK_ARG(cond, msg)            \
  do {                                     \
    if (!(cond)) {                         \
      ::mj::set_error(msg);                \
      return MJ_ERR_ARG;                   \
    }                                      \
  } while (0)

// Device memory that the library holds, and the most it may hold (a test's
// limit; none by default).
struct DeviceMemory {
  std::atomic<size_t> held{0}, limit{SIZE_MAX};
};
DeviceMemory& device_memory();

// Device buffer owned by the library (cudaMalloc/cudaFree).
struct DevBuf {
  void* ptr = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { release(); }
  void release() {
    if (ptr) {
      cudaFree(ptr);
      device_memory().held -= bytes;
    }
    ptr = nullptr;
    bytes = 0;
  }
  cudaError_t alloc(size_t b) {
    release();
    if (b == 0) return cudaSuccess;
    DeviceMemory& m = device_memory();
    if (m.held + b > m.limit) return cudaErrorMemoryAllocation;
    const cudaError_t e = cudaMalloc(&ptr, b);
    if (e) {
      ptr = nullptr;
      return e;
    }
    bytes = b;
    m.held += b;
    return cudaSuccess;
  }
  template <class T>
  T* as() const { return static_cast<T*>(ptr); }
};

// Page-locked host buffer owned by the library: device-to-host copies into it
// are queued, where a copy into pageable memory makes the host wait for each.
struct PinBuf {
  void* ptr = nullptr;
  size_t bytes = 0;
  PinBuf() = default;
  PinBuf(const PinBuf&) = delete;
  PinBuf& operator=(const PinBuf&) = delete;
  ~PinBuf() {
    if (ptr) cudaFreeHost(ptr);
  }
  cudaError_t alloc(size_t b) {
    if (ptr) cudaFreeHost(ptr);
    ptr = nullptr;
    bytes = b;
    return cudaMallocHost(&ptr, b);
  }
  template <class T>
  T* as() const { return static_cast<T*>(ptr); }
};

// Local numbering NumDofs3D of a Q_r hexahedron, num[(i*n+j)*n+k] = local
// index of the node (i,j,k) (i along x): vertices, the 12 edges, the faces
// x=0, y=0, z=0, z=1, y=1, x=1, then the interior
// (MONTJOIE/src/Quadrature/HexahedronQuadrature.cxx:51-171).
std::vector<int> hex_local_numbering(int r);

// Gauss-Lobatto points and weights on [0,1] (r+1 points) and the derivative
// matrix g[a*n+b] = phi_a'(x_b) (MONTJOIE/src/Quadrature/GaussLobatto.cxx:175-191).
void gauss_lobatto(int r, double* pts, double* wts);
void gl_derivative_matrix(int r, const double* pts, double* g);

int sm_count();

// Lets a kernel be launched with any dynamic shared memory the device has room
// for beside its static one, *limit bytes.  A kernel whose size depends on the
// integrator (the EN steps: on S) takes this and not its own size: the
// attribute belongs to the kernel, and a second integrator of a smaller size
// would lower it under the first one's launches.
template <class... P>
cudaError_t allow_dynamic_smem(void (*kernel)(P...), size_t* limit) {
  int dev = 0, optin = 0;
  cudaFuncAttributes a;
  cudaError_t e = cudaGetDevice(&dev);
  if (!e) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (!e) e = cudaFuncGetAttributes(&a, kernel);
  if (e) return e;
  *limit = (size_t)optin - a.sharedSizeBytes;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*limit);
}

// Reads a kernel's device error flag after the work on `s`; when it is set,
// clears it (so the next call starts clean), records "<what>: <message>" and
// returns MJ_ERR_CUDA.  Synchronises `s`.  host: a page-locked int to read it
// through.
int take_kernel_error(void* dev_flag, cudaStream_t s, const char* what, int* host);

// Launch of a kernel that begins with dependent_wait(): it may be launched
// while the kernel before it on the stream is ending, which hides the launch
// and the start of its CTAs; it reads and writes nothing before that kernel
// has ended and its stores are visible.  A step of two such kernels gains
// about 0.8 us: 2^3 Q4 in FP32 5.5 -> 4.7 us, 32^3 Q4 41.0 -> 40.2, Q8 32^3
// 232.6 -> 230.8; MltAdd of Q4 23x21x19 in FP64 36.9 -> 34.7.  (They do not let the next kernel start any earlier than at
// their end: its waiting CTAs would take the room of other streams' kernels.)
template <class... P, class... A>
void launch_dependent(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
__device__ __forceinline__ void dependent_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Load from an array that the kernel before writes (an element kernel's x, a
// gather's R), in a kernel that begins with dependent_wait().  The read-only
// path (__ldg, or const __restrict__) is for data that nobody writes while the
// kernel is resident, and its loads may be moved: an ordinary load, volatile
// so that it stays behind the wait.  It costs nothing: MltAdd of Q4 48^3 in
// FP32 126.3 -> 126.3 us, in FP64 315.7 -> 315.6; order-4 step of Q8 16^3 69.7
// -> 69.8.
__device__ __forceinline__ float ld_fresh(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_fresh(const double* p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

}  // namespace mj
