// Shared device/host helpers of libblsgpu.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "host_layout.hpp"

namespace bls {

void set_error(const std::string& msg);

#define BLS_CUDA(x)                                                                                     \
  do {                                                                                                  \
    cudaError_t e_ = (x);                                                                               \
    if (e_ != cudaSuccess) throw ::bls::Error(BLS_ECUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Device status word of a plan. `failed` is the lowest failing eliminated block; `einval_r` / `einval_e` the lowest
// non-finite or negative entry of the reset's scaling_r / the reduction's scaling_e; LLONG_MAX means none. Kernels read
// it to skip their work, as the reference throws before writing (src/utils.jl:100-107) and returns before phase 2
// after a failure (src/schur_reduction.jl:499).
struct Status {
  long long failed;
  long long einval_r;
  long long einval_e;
  long long pad;
};

template <class T>
__device__ __forceinline__ T ldg(const T* p) { return __ldg(p); }

#ifdef __CUDACC__
// An asynchronous 16-byte global -> shared copy of `bytes` bytes (the rest zero-filled), both on 16-byte boundaries
__device__ __forceinline__ void run_cp16(void* smem, const void* gmem, int bytes) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void run_cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void run_cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Add six consecutive entries of a column of S (vector reductions where the address allows: red.global.add.v4/.v2
// for FP32, scalar for FP64). v[i] goes to col[i].
__device__ __forceinline__ void red2(float* p, float a, float b) {
  asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};\n" ::"l"(p), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void red4(float* p, float a, float b, float c, float d) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void red_column6(float* col, const float v[6]) {
  switch ((reinterpret_cast<uintptr_t>(col) >> 2) & 3) {   // position of col[0] within its 16-byte line
    case 0: red4(col, v[0], v[1], v[2], v[3]); red2(col + 4, v[4], v[5]); break;
    case 1: atomicAdd(col, v[0]); red2(col + 1, v[1], v[2]); red2(col + 3, v[3], v[4]); atomicAdd(col + 5, v[5]); break;
    case 2: red2(col, v[0], v[1]); red4(col + 2, v[2], v[3], v[4], v[5]); break;
    default: atomicAdd(col, v[0]); red4(col + 1, v[1], v[2], v[3], v[4]); atomicAdd(col + 5, v[5]); break;
  }
}
// Four or eight entries of a column the same way
__device__ __forceinline__ void red_column4(float* col, const float* v) {
  switch ((reinterpret_cast<uintptr_t>(col) >> 2) & 3) {
    case 0: red4(col, v[0], v[1], v[2], v[3]); break;
    case 2: red2(col, v[0], v[1]); red2(col + 2, v[2], v[3]); break;
    default: atomicAdd(col, v[0]); red2(col + 1, v[1], v[2]); atomicAdd(col + 3, v[3]); break;
  }
}
__device__ __forceinline__ void red_column8(float* col, const float* v) {
  switch ((reinterpret_cast<uintptr_t>(col) >> 2) & 3) {
    case 0: red4(col, v[0], v[1], v[2], v[3]); red4(col + 4, v[4], v[5], v[6], v[7]); break;
    case 1: atomicAdd(col, v[0]); red2(col + 1, v[1], v[2]); red4(col + 3, v[3], v[4], v[5], v[6]); atomicAdd(col + 7, v[7]); break;
    case 2: red2(col, v[0], v[1]); red4(col + 2, v[2], v[3], v[4], v[5]); red2(col + 6, v[6], v[7]); break;
    default: atomicAdd(col, v[0]); red4(col + 1, v[1], v[2], v[3], v[4]); red2(col + 5, v[5], v[6]); atomicAdd(col + 7, v[7]); break;
  }
}
__device__ __forceinline__ void red_column6(double* col, const double v[6]) {
#pragma unroll
  for (int i = 0; i < 6; ++i) atomicAdd(col + i, v[i]);
}
#endif

// Allows the launches of `kernel` all the dynamic shared memory that a CTA can have beside the kernel's static part. The
// limit is an attribute of the kernel, process-wide: set to one launch's own size, it could be lowered by another host
// thread's smaller launch before this one's larger launch, which is then refused. So it is set once per device, to the
// most that any launch may ask for.
inline void allow_smem(const void* kernel) {
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  int dev = 0, most = 0;
  BLS_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({kernel, dev})) return;
  cudaFuncAttributes a;
  BLS_CUDA(cudaFuncGetAttributes(&a, kernel));
  BLS_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  BLS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes));
  done.insert({kernel, dev});
}

// The SMs of a device
inline int sm_count(int device) {
  int n = 0;
  BLS_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device));
  return n;
}

inline int grid_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }

// A device buffer that frees itself (unless it is a part of another one, see SmallBufs).
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  bool owned = true;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { if (p && owned) cudaFree(p); }
  void alloc(size_t b) {
    if (p && owned) cudaFree(p);
    p = nullptr;
    owned = true;
    bytes = b;
    if (b) BLS_CUDA(cudaMalloc(&p, b));
  }
  template <class T> T* as() const { return static_cast<T*>(p); }
};

template <class T>
void upload(DevBuf& buf, const std::vector<T>& v, cudaStream_t s) {
  buf.alloc(v.size() * sizeof(T));
  if (!v.empty()) BLS_CUDA(cudaMemcpyAsync(buf.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
}

// A host array that is not initialised (a large std::vector is, by one thread).
template <class T>
struct HostArray {
  std::unique_ptr<T[]> p;
  int64_t n = 0;
  HostArray() = default;
  explicit HostArray(int64_t count) : p(new T[count > 0 ? (size_t)count : 1]), n(count) {}
  T* get() const { return p.get(); }
  T& operator[](int64_t i) const { return p[(size_t)i]; }
};

// Many small device arrays in one allocation and few copies (an allocation takes up to 0.4 ms): add() takes an array's
// contents, reserve() room without contents, and flush() makes the allocation and points the buffers into it; `arena` has to
// outlive them, and this object the copies. Above kSmall bytes a buffer gets its own allocation at once.
class SmallBufs {
 public:
  template <class T>
  void add(DevBuf& b, const T* v, int64_t n, cudaStream_t s) {
    const size_t bytes = (size_t)n * sizeof(T);
    if (bytes > kSmall) {
      b.alloc(bytes);
      BLS_CUDA(cudaMemcpyAsync(b.p, v, bytes, cudaMemcpyHostToDevice, s));
      return;
    }
    b.alloc(0);
    if (!bytes) return;
    if (chunks.empty() || used + bytes > kChunk) {
      chunks.emplace_back(new unsigned char[kChunk]);
      used = 0;
    }
    std::memcpy(chunks.back().get() + used, v, bytes);
    parts.push_back({&b, (chunks.size() - 1) * kChunk + used, bytes, true});
    used = (used + bytes + 255) / 256 * 256;
  }
  template <class T>
  void add(DevBuf& b, const std::vector<T>& v, cudaStream_t s) { add(b, v.data(), (int64_t)v.size(), s); }
  template <class T>
  void add(DevBuf& b, const HostArray<T>& v, cudaStream_t s) { add(b, v.get(), v.n, s); }
  void reserve(DevBuf& b, size_t bytes) {
    if (bytes > kSmall) {
      b.alloc(bytes);
      return;
    }
    b.alloc(0);
    parts.push_back({&b, room, bytes, false});
    room += (bytes + 255) / 256 * 256;
  }
  void flush(DevBuf& arena, cudaStream_t s) {
    const size_t contents = chunks.empty() ? 0 : (chunks.size() - 1) * kChunk + used;
    arena.alloc(contents + room);
    unsigned char* base = arena.as<unsigned char>();
    for (size_t i = 0; i < chunks.size(); ++i)
      BLS_CUDA(cudaMemcpyAsync(base + i * kChunk, chunks[i].get(), i + 1 < chunks.size() ? kChunk : used, cudaMemcpyHostToDevice, s));
    for (const Part& x : parts) {
      x.buf->p = base + (x.contents ? 0 : contents) + x.off;
      x.buf->bytes = x.bytes;
      x.buf->owned = false;
    }
    parts.clear();
  }

 private:
  static constexpr size_t kSmall = 1 << 20, kChunk = 4 << 20;
  struct Part { DevBuf* buf; size_t off, bytes; bool contents; };
  std::vector<Part> parts;
  std::vector<std::unique_ptr<unsigned char[]>> chunks;
  size_t used = 0, room = 0;   // bytes of the last chunk, bytes reserved
};

// One block of symmetrifyfull!: data[src ...] (rd x cd, column-major) to mat's rows rs.. and columns cs.., and
// transposed to rows cs.. and columns rs.. unless diag.
struct SymBlock {
  int64_t src, rs, cs;
  int32_t rd, cd, diag, pad;
};
// Zeroes the m x m matrix and copies the blocks (a host list, copied to the device on stream s).
void launch_symmetrify(cudaStream_t s, int dtype, const void* data, const SymBlock* blocks_host, int64_t nblocks, void* mat,
                       int64_t m);

}  // namespace bls

struct bls_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int* flag = nullptr;   // device scratch word for calls that report a device-side decision (allocated at first use)
};
