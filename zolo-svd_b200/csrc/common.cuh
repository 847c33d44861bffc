// Shared device helpers for the FP64 kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#define ZDEV __device__ __forceinline__

namespace zolo {

// 16-byte async global->shared copy; src_bytes in {0, 8, 16}, the rest is zero-filled.
ZDEV void cp_async16(void* smem, const void* gmem, int src_bytes) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
// 8-byte async global->shared copy; src_bytes in {0, 8}.
ZDEV void cp_async8(void* smem, const void* gmem, int src_bytes) {
  unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
ZDEV void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
ZDEV void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// D(16x8) += A(16x8) * B(8x8), FP64 tensor core (DMMA).
// Fragment layout (PTX ISA, mma.m16n8k8 .f64): g = lane/4, t = lane%4
//   a0=(g,t) a1=(g+8,t) a2=(g,t+4) a3=(g+8,t+4);  b0=(t,g) b1=(t+4,g)
//   c0=(g,2t) c1=(g,2t+1) c2=(g+8,2t) c3=(g+8,2t+1)
ZDEV void dmma_16x8x8(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

ZDEV double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Kernel attributes (cudaFuncSetAttribute) and device properties are per device: these
// helpers apply / compute them once for each device the library launches on.
constexpr int kMaxDevices = 64;
template <class F>
inline cudaError_t once_per_device(std::atomic<int> (&state)[kMaxDevices], F&& set) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return set();
  if (state[dev].load(std::memory_order_acquire) == 1) return cudaSuccess;
  e = set();
  if (e == cudaSuccess) state[dev].store(1, std::memory_order_release);
  return e;
}
// cache[device] holds compute() (a positive value) after the first call on that device.
template <class F>
inline int per_device_value(std::atomic<int> (&cache)[kMaxDevices], F&& compute) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return compute();
  int v = cache[dev].load(std::memory_order_acquire);
  if (v <= 0) {
    v = compute();
    cache[dev].store(v, std::memory_order_release);
  }
  return v;
}

// Programmatic dependent launch: a kernel launched with launch_dependent may become resident while
// the kernel before it in the stream still runs, so it must pass dependency_wait (which holds until
// that kernel has completed and its writes are visible) before it touches global memory.
// Its pointer parameters carry no __restrict__ and it loads nothing through __ldg: what both promise is
// read-only for the kernel's whole lifetime, which here begins while its predecessor still writes.
// release_dependents lets the next such kernel start its launch; placed after the main work, so that
// waiting CTAs do not hold SMs that other streams could use.
// A solve is a chain of about a thousand launches of 4 to 50 us; the launch itself then overlaps the
// end of the kernel before it: QDWH n = 1024 10.7 -> 9.6 ms, Zolo-PD fast n = 4096 94.4 -> 89.4.
ZDEV void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
ZDEV void release_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
inline cudaError_t launch_dependent(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, dim3 cluster,
                                    A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute la[2];
  la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  la[0].val.programmaticStreamSerializationAllowed = 1;
  la[1].id = cudaLaunchAttributeClusterDimension;
  la[1].val.clusterDim.x = cluster.x;
  la[1].val.clusterDim.y = cluster.y;
  la[1].val.clusterDim.z = cluster.z;
  cfg.attrs = la;
  cfg.numAttrs = cluster.x * cluster.y * cluster.z > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

// f(i, j) for this thread's share of the entries of an m x n column-major matrix, all threads of
// the grid's x dimension together in storage order.  One 32-bit division at the start; a 64-bit
// quotient and remainder per entry made these kernels instruction-bound (1.8 TB/s for a copy).
template <class F>
ZDEV void for_entries(int m, int n, F&& f) {
  if (m <= 0) return;
  const unsigned stride = gridDim.x * blockDim.x, e0 = blockIdx.x * blockDim.x + threadIdx.x;
  const int di = static_cast<int>(stride % m), dj = static_cast<int>(stride / m);
  int i = static_cast<int>(e0 % m), j = static_cast<int>(e0 / m);
#pragma unroll 4
  for (; j < n;) {
    f(i, j);
    i += di;
    j += dj;
    if (i >= m) {
      i -= m;
      ++j;
    }
  }
}

// for_entries in batches: v = f(i, j) for up to four entries of this thread, all loads in flight together, then
// store(i, j, v) for them in the same order (after a store the compiler may not move the next load
// up: it could read what was stored).  With __restrict__ and for_entries instead, which dependent kernels
// may not use, 8192^2 took 411 us in combine_kernel (255 here), 147 in frob2_kernel (102), 260 in
// copy_upper_kernel (211), 351 in scale_copy_kernel (358).  A store under a condition or one entry a
// thread is better off with for_entries (shift_lower_kernel of eight 2048^2: 38 us, 49 here).
template <class F, class G>
ZDEV void map_entries(int m, int n, F&& f, G&& store) {
  if (m <= 0) return;
  constexpr int U = 4;
  const unsigned stride = gridDim.x * blockDim.x, e0 = blockIdx.x * blockDim.x + threadIdx.x;
  const int di = static_cast<int>(stride % m), dj = static_cast<int>(stride / m);
  int i = static_cast<int>(e0 % m), j = static_cast<int>(e0 / m);
  while (j < n) {
    int vi[U], vj[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      vi[u] = i;
      vj[u] = j;
      i += di;
      j += dj;
      if (i >= m) {
        i -= m;
        ++j;
      }
    }
    decltype(f(0, 0)) v[U];
    if (vj[U - 1] < n) {  // all of them inside
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = f(vi[u], vj[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) store(vi[u], vj[u], v[u]);
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (vj[u] < n) v[u] = f(vi[u], vj[u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (vj[u] < n) store(vi[u], vj[u], v[u]);
    }
  }
}

// Device status word: kernels record the first error code here (never trap).
ZDEV void set_status(int* status, int code) {
  if (status) atomicCAS(status, 0, code);
}

}  // namespace zolo
