// The part of CUDA that the kernels under test use, on the CPU.
//
// A block runs at a time, a fiber per thread; a thread runs until it meets the
// others of its warp in a collective or those of its block in a barrier, so the
// kernels' index arithmetic, bounds and protocols run as written, with plain
// memory that a test can look at.  emulate.py turns the sources' launches and
// dynamic shared arrays into the calls at the end of this file.
#pragma once

#include <ucontext.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#define __global__
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
#define __restrict__
#define __shared__ static
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))

using std::max;
using std::min;

typedef void *cudaStream_t;
typedef void *cudaEvent_t;
enum cudaError_t { cudaSuccess = 0 };
enum {
  cudaFuncAttributeMaxDynamicSharedMemorySize,
  cudaDevAttrMultiProcessorCount,
  cudaDevAttrCooperativeLaunch,
  cudaMemcpyDeviceToHost
};
struct dim3 {
  unsigned x;
  dim3(unsigned n) : x(n) {}
};
struct int2 {
  int x, y;
};
inline int2 make_int2(int a, int b) { return {a, b}; }

namespace emu {

struct Dim {
  unsigned x = 1;
};
struct Warp {
  unsigned long long buf[2][32];  // the lanes' values of this rendezvous and of the last
  int arrived = 0, gen = 0;
};
struct Fiber {
  ucontext_t ctx;
  bool done = false;
};
struct Block {
  std::vector<Fiber> threads;
  std::vector<Warp> warps;
  int arrived = 0, gen = 0;  // __syncthreads
  unsigned cur = 0;          // the running thread
  ucontext_t main;
};

inline Block *block = nullptr;
inline std::function<void()> *body = nullptr;
inline unsigned long long max_rounds = 100000000ull;  // scheduling rounds before a block is stuck

inline void yield() {
  const unsigned t = block->cur;
  swapcontext(&block->threads[t].ctx, &block->main);
}

// Leaves v for the warp's other lanes and waits for theirs; which half of buf has them.
inline const unsigned long long *meet(unsigned long long v) {
  Warp &w = block->warps[block->cur >> 5];
  const int gen = w.gen;
  w.buf[gen & 1][block->cur & 31] = v;
  if (++w.arrived == 32) {
    w.arrived = 0;
    w.gen++;
  } else {
    while (w.gen == gen) yield();
  }
  return w.buf[gen & 1];
}

template <typename T>
unsigned long long pack(T t) {
  unsigned long long x = 0;
  memcpy(&x, &t, sizeof t);
  return x;
}
template <typename T>
T unpack(unsigned long long x) {
  T t;
  memcpy(&t, &x, sizeof t);
  return t;
}

inline void trampoline() {
  (*body)();
  block->threads[block->cur].done = true;
  yield();
}

inline void run_block(unsigned threads, std::function<void()> f) {
  static std::vector<std::vector<char>> stacks;
  Block b;
  block = &b;
  body = &f;
  b.threads.resize(threads);
  b.warps.resize((threads + 31) / 32);
  while (stacks.size() < threads) stacks.emplace_back(1 << 17);
  for (unsigned i = 0; i < threads; ++i) {
    ucontext_t &c = b.threads[i].ctx;
    getcontext(&c);
    c.uc_stack.ss_sp = stacks[i].data();
    c.uc_stack.ss_size = stacks[i].size();
    c.uc_link = &b.main;
    makecontext(&c, trampoline, 0);
  }
  unsigned long long rounds = 0;
  for (unsigned left = threads; left;) {
    left = 0;
    for (unsigned i = 0; i < threads; ++i) {
      if (b.threads[i].done) continue;
      b.cur = i;
      swapcontext(&b.main, &b.threads[i].ctx);
      left += !b.threads[i].done;
    }
    if (++rounds > max_rounds) {
      fprintf(stderr, "emulated block does not end\n");
      exit(3);
    }
  }
  block = nullptr;
}

struct ThreadIdx {
  struct X {
    operator unsigned() const { return block->cur; }
  } x;
};

}  // namespace emu

inline emu::ThreadIdx threadIdx;
inline emu::Dim blockIdx, blockDim, gridDim;

template <typename T>
T __shfl_sync(unsigned, T v, int src) {
  return emu::unpack<T>(emu::meet(emu::pack(v))[src & 31]);
}
template <typename T>
T __shfl_up_sync(unsigned, T v, int d) {
  const int lane = threadIdx.x & 31;
  return emu::unpack<T>(emu::meet(emu::pack(v))[lane < d ? lane : lane - d]);
}
template <typename T>
T __shfl_down_sync(unsigned, T v, int d) {
  const int lane = threadIdx.x & 31;
  return emu::unpack<T>(emu::meet(emu::pack(v))[lane + d > 31 ? lane : lane + d]);
}
inline unsigned __ballot_sync(unsigned, bool p) {
  const unsigned long long *b = emu::meet(p);
  unsigned r = 0;
  for (int i = 0; i < 32; ++i) r |= b[i] ? 1u << i : 0u;
  return r;
}
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
inline bool __all_sync(unsigned m, bool p) { return __ballot_sync(m, p) == ~0u; }
inline unsigned __reduce_or_sync(unsigned, unsigned v) {
  const unsigned long long *b = emu::meet(v);
  unsigned r = 0;
  for (int i = 0; i < 32; ++i) r |= (unsigned)b[i];
  return r;
}
inline unsigned __reduce_max_sync(unsigned, unsigned v) {
  const unsigned long long *b = emu::meet(v);
  return (unsigned)*std::max_element(b, b + 32);
}
inline unsigned __reduce_min_sync(unsigned, unsigned v) {
  const unsigned long long *b = emu::meet(v);
  return (unsigned)*std::min_element(b, b + 32);
}
inline unsigned __reduce_add_sync(unsigned, unsigned v) {
  const unsigned long long *b = emu::meet(v);
  unsigned r = 0;
  for (int i = 0; i < 32; ++i) r += (unsigned)b[i];
  return r;
}
template <typename T>
unsigned __match_any_sync(unsigned, T v) {
  const unsigned long long *b = emu::meet(emu::pack(v));
  unsigned r = 0;
  for (int i = 0; i < 32; ++i) r |= emu::unpack<T>(b[i]) == v ? 1u << i : 0u;
  return r;
}
inline void __syncwarp() { emu::meet(0); }
inline void __syncthreads() {
  emu::Block &b = *emu::block;
  const int gen = b.gen;
  if (++b.arrived == (int)b.threads.size()) {
    b.arrived = 0;
    b.gen++;
  } else {
    while (b.gen == gen) emu::yield();
  }
}
inline void __threadfence() {}
inline void __nanosleep(unsigned) { emu::yield(); }

inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int __popcll(unsigned long long x) { return __builtin_popcountll(x); }
inline int __ffs(int x) { return __builtin_ffs(x); }
inline int __ffsll(long long x) { return __builtin_ffsll(x); }
inline int __clz(unsigned x) { return x ? __builtin_clz(x) : 32; }
inline long long clock64() { return 0; }
template <typename T>
T __ldcg(const T *p) {
  return *p;
}

template <typename T, typename U>
T atomicAdd(T *p, U v) {
  const T old = *p;
  *p = old + (T)v;
  return old;
}
template <typename T, typename U>
T atomicSub(T *p, U v) {
  const T old = *p;
  *p = old - (T)v;
  return old;
}
template <typename T, typename U>
T atomicOr(T *p, U v) {
  const T old = *p;
  *p = old | (T)v;
  return old;
}
template <typename T, typename U>
T atomicMax(T *p, U v) {
  const T old = *p;
  *p = max(old, (T)v);
  return old;
}
template <typename T, typename U>
T atomicMin(T *p, U v) {
  const T old = *p;
  *p = min(old, (T)v);
  return old;
}
template <typename T, typename U, typename V>
T atomicCAS(T *p, U expected, V v) {
  const T old = *p;
  if (old == (T)expected) *p = (T)v;
  return old;
}

// the runtime calls of the launchers: one SM with one resident block
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
  memset(p, v, n);
  return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, int, cudaStream_t) {
  memcpy(to, from, n);
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
inline cudaError_t cudaDeviceGetAttribute(int *v, int, int) {
  *v = 1;
  return cudaSuccess;
}
inline cudaError_t cudaLaunchCooperativeKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) {
  fprintf(stderr, "no grid barriers here: a block runs at a time\n");
  exit(5);
}
template <typename F>
cudaError_t cudaFuncSetAttribute(F, int, int) {
  return cudaSuccess;
}
template <typename F>
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *blocks, F, int, size_t) {
  *blocks = 1;
  return cudaSuccess;
}

namespace emu {

struct Config {
  unsigned grid, threads;
  size_t smem;
  Config(long long g, long long t, size_t sm = 0, cudaStream_t = nullptr)
      : grid((unsigned)g), threads((unsigned)t), smem(sm) {}
};

// Dynamic shared memory; what lies past a launch's own bytes stays 0xA5 unless
// the kernel writes out of bounds.
constexpr size_t DYNAMIC_MAX = 256 << 10, DYNAMIC_GUARD = 64 << 10;
alignas(128) inline unsigned char dynamic_mem[DYNAMIC_MAX + DYNAMIC_GUARD];
inline void *dynamic() { return dynamic_mem; }

template <typename F>
void launch(const Config &c, F f) {
  memset(dynamic_mem, 0xA5, sizeof(dynamic_mem));
  gridDim.x = c.grid;
  blockDim.x = c.threads;
  for (unsigned b = 0; b < c.grid; ++b) {
    blockIdx.x = b;
    run_block(c.threads, f);
    for (size_t i = c.smem; i < sizeof(dynamic_mem); ++i)
      if (dynamic_mem[i] != 0xA5) {
        fprintf(stderr, "shared memory written at byte %zu of %zu\n", i, c.smem);
        exit(4);
      }
  }
}

}  // namespace emu
