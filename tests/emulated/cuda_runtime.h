// Enough of CUDA to run the cooperative PPE solvers' kernel sources on the CPU, so that what they do
// does not depend on which block is ahead can be checked where the order of the blocks is chosen.
//
// A block is a host thread, of which one at a time holds the turn; a CUDA thread is a fiber of its
// block, which runs on until it meets the others (a block or warp barrier, a shuffle).  A block gives
// the turn away
//  * when it polls the grid barrier in vain: the last one to arrive finds it open and runs on alone, up
//    to its next vain poll, before any other has left the barrier ("ahead"); as the turn goes round,
//    every block is that one in its turn;
//  * with emu::fair, at each of its own barriers too: the blocks then stay within one block barrier
//    of one another, the order in which a missing wait shows least.
#pragma once
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __launch_bounds__(...)
#define __grid_constant__
#define __align__(n) __attribute__((aligned(n)))
#define __shared__ thread_local

struct dim3 {
  unsigned x, y, z;
  dim3(unsigned x_ = 1, unsigned y_ = 1, unsigned z_ = 1) : x(x_), y(y_), z(z_) {}
};
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct double2 { double x, y; };
struct double3 { double x, y, z; };
inline float2 make_float2(float x, float y) { return {x, y}; }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
inline double2 make_double2(double x, double y) { return {x, y}; }
inline double3 make_double3(double x, double y, double z) { return {x, y, z}; }

namespace emu {

inline bool fair = false;
inline int multiprocessors = 1;
inline int device = 0;

// ---- the turn
struct Turn {
  std::mutex mu;
  std::condition_variable cv;
  std::vector<char> live;
  int whose = 0;
  long vain = 0;  // polls without any arrival between them
  void next(int me) {
    for (size_t k = 1; k <= live.size(); ++k) {
      const int b = (me + (int)k) % (int)live.size();
      if (live[b]) { whose = b; break; }
    }
    cv.notify_all();
  }
  void pass(int me) {
    std::unique_lock<std::mutex> l(mu);
    next(me);
    cv.wait(l, [&] { return whose == me; });
  }
};

struct Meeting {  // a barrier among the threads that have not returned
  int alive = 0, arrived = 0;
  unsigned gen = 0;
  bool open() {
    if (arrived == 0 || arrived < alive) return false;
    arrived = 0;
    ++gen;
    return true;
  }
};
struct Fiber {
  ucontext_t ctx;
  std::unique_ptr<char[]> stack;
  bool done = false;
  unsigned shuffles = 0;
};
struct Block {
  int idx;
  dim3 grid, dim;
  Turn* turn;
  const std::function<void()>* kernel;
  ucontext_t main;
  std::vector<Fiber> f;
  std::vector<uint64_t> word;  // two per thread: a thread is one shuffle ahead of its warp at most
  std::vector<Meeting> warp;
  Meeting all;
  int cur = 0, votes = 0, result = 0;
  bool arrived = false;  // at the grid barrier, and has not polled yet
};
inline thread_local Block* B = nullptr;

inline void yield() { swapcontext(&B->f[B->cur].ctx, &B->main); }
inline bool meet(Meeting& m) {  // true for the thread that opens it
  ++m.arrived;
  if (m.open()) return true;
  for (const unsigned g = m.gen; m.gen == g;) yield();
  return false;
}
inline void fiber_main() {
  (*B->kernel)();
  Fiber& me = B->f[B->cur];
  me.done = true;
  for (Meeting* m : {&B->all, &B->warp[B->cur / 32]}) {
    --m->alive;
    m->open();
  }
  yield();
}
inline void run_block(Block& b) {
  {
    std::unique_lock<std::mutex> l(b.turn->mu);
    b.turn->cv.wait(l, [&] { return b.turn->whose == b.idx; });
  }
  B = &b;
  const int n = (int)(b.dim.x * b.dim.y);
  b.f = std::vector<Fiber>(n);
  b.word.assign(2 * n, 0);
  b.warp.resize((n + 31) / 32);
  b.all.alive = n;
  for (int t = 0; t < n; ++t) {
    ++b.warp[t / 32].alive;
    Fiber& f = b.f[t];
    constexpr size_t S = 65536;
    f.stack.reset(new char[S]);
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = f.stack.get();
    f.ctx.uc_stack.ss_size = S;
    f.ctx.uc_link = nullptr;
    makecontext(&f.ctx, fiber_main, 0);
  }
  for (bool any = true; any;) {
    any = false;
    for (b.cur = 0; b.cur < n; ++b.cur)
      if (!b.f[b.cur].done) {
        any = true;
        swapcontext(&b.main, &b.f[b.cur].ctx);
      }
  }
  std::unique_lock<std::mutex> l(b.turn->mu);
  b.turn->live[b.idx] = 0;
  b.turn->next(b.idx);
}
inline void run(dim3 grid, dim3 dim, const std::function<void()>& kernel) {
  Turn turn;
  turn.live.assign(grid.x, 1);
  std::vector<Block> blocks(grid.x);
  std::vector<std::thread> th;
  for (int i = 0; i < (int)grid.x; ++i) {
    Block& b = blocks[i];
    b.idx = i;
    b.grid = grid;
    b.dim = dim;
    b.turn = &turn;
    b.kernel = &kernel;
    th.emplace_back([&b] { run_block(b); });
  }
  for (auto& t : th) t.join();
}

// ---- the grid barrier's words
inline void arrive() {
  B->arrived = true;
  B->turn->vain = 0;
}
inline void poll() {
  const bool first = B->arrived;
  B->arrived = false;
  if (first && !fair) return;
  if (++B->turn->vain > 20000) {
    std::printf("a block waits for one that has left the solve\n");
    std::fflush(stdout);
    std::_Exit(3);
  }
  B->turn->pass(B->idx);
}

template <unsigned (*F)()>
struct Value {
  operator unsigned() const { return F(); }
};
inline unsigned thread_x() { return (unsigned)B->cur % B->dim.x; }
inline unsigned thread_y() { return (unsigned)B->cur / B->dim.x; }
inline unsigned block_x() { return (unsigned)B->idx; }
inline unsigned block_dim() { return B->dim.x; }
inline unsigned grid_dim() { return B->grid.x; }

template <class T>
T shuffle(T v, int from) {  // from: lane of the warp
  Fiber& me = B->f[B->cur];
  uint64_t* w = B->word.data() + (me.shuffles++ & 1) * B->f.size();
  std::memcpy(w + B->cur, &v, sizeof(T));
  meet(B->warp[B->cur / 32]);
  T o;
  std::memcpy(&o, w + (B->cur & ~31) + from, sizeof(T));
  return o;
}
inline int lane() { return B->cur & 31; }

}  // namespace emu

inline struct { emu::Value<emu::thread_x> x; emu::Value<emu::thread_y> y; } threadIdx;
inline struct { emu::Value<emu::block_x> x; } blockIdx;
inline struct { emu::Value<emu::block_dim> x; } blockDim;
inline struct { emu::Value<emu::grid_dim> x; } gridDim;

inline void __syncthreads() {
  if (emu::meet(emu::B->all) && emu::fair) emu::B->turn->pass(emu::B->idx);
}
inline int __syncthreads_or(int v) {
  emu::Block& b = *emu::B;
  b.votes |= v;
  if (emu::meet(b.all)) {
    b.result = b.votes;
    b.votes = 0;
    if (emu::fair) b.turn->pass(b.idx);
  }
  const int r = b.result;
  emu::meet(b.all);  // nobody votes again before all have read
  return r;
}
inline void __syncwarp(unsigned = ~0u) { emu::meet(emu::B->warp[emu::B->cur / 32]); }
template <class T> T __shfl_sync(unsigned, T v, int src, int w = 32) {
  return emu::shuffle(v, (emu::lane() & ~(w - 1)) + (src & (w - 1)));
}
template <class T> T __shfl_xor_sync(unsigned, T v, int m, int = 32) { return emu::shuffle(v, emu::lane() ^ m); }
template <class T> T __shfl_down_sync(unsigned, T v, int d, int w = 32) {
  const int l = emu::lane(), in = (l & (w - 1)) + d;
  return emu::shuffle(v, in < w ? l + d : l);
}
template <class T> T __shfl_up_sync(unsigned, T v, int d) {
  const int l = emu::lane();
  return emu::shuffle(v, l >= d ? l - d : l);
}
inline unsigned __ballot_sync(unsigned, bool p) {
  unsigned b = p ? 1u << emu::lane() : 0u;
  for (int o = 16; o > 0; o >>= 1) b |= emu::shuffle(b, emu::lane() ^ o);
  return b;
}
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0u; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __reduce_max_sync(unsigned, int v) {
  int r = v;
  for (int o = 16; o > 0; o >>= 1) r = std::max(r, emu::shuffle(r, emu::lane() ^ o));
  return r;
}
inline void __nanosleep(unsigned) { emu::poll(); }
inline void __threadfence() {}

template <class T> T atomicAdd(T* a, T v) { T o = *a; *a = o + v; emu::arrive(); return o; }
template <class T> T atomicExch(T* a, T v) { T o = *a; *a = v; return o; }
template <class T> T atomicOr(T* a, T v) { T o = *a; *a = o | v; return o; }
template <class T> T atomicMax(T* a, T v) { T o = *a; *a = std::max(o, v); return o; }
template <class T, class C, class V> T atomicCAS(T* a, C c, V v) { T o = *a; if (o == (T)c) *a = (T)v; return o; }
template <class T> T __ldg(const T* p) { return *p; }
template <class T> T __ldca(const T* p) { return *p; }
template <class T> T __ldcg(const T* p) { return *p; }
using std::isnan;
using std::max;
using std::min;

template <class To, class From> To emu_bits(From f) { To t; std::memcpy(&t, &f, sizeof(To)); return t; }
inline long long __double_as_longlong(double x) { return emu_bits<long long>(x); }
inline double __longlong_as_double(long long x) { return emu_bits<double>(x); }
inline unsigned __float_as_uint(float x) { return emu_bits<unsigned>(x); }
inline float __uint_as_float(unsigned x) { return emu_bits<float>(x); }

// ---- the runtime calls of the solvers' host code
enum cudaError_t { cudaSuccess = 0 };
using cudaStream_t = void*;
using cudaEvent_t = void*;
using cudaGraphExec_t = void*;
enum { cudaLaunchAttributeCooperative, cudaEventRecordExternal, cudaDevAttrMultiProcessorCount,
       cudaDevAttrMaxSharedMemoryPerBlockOptin, cudaFuncAttributeMaxDynamicSharedMemorySize, cudaMemcpyDeviceToHost };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone };
struct cudaLaunchAttribute {
  int id;
  struct { int cooperative; } val;
};
struct cudaLaunchConfig_t {
  dim3 gridDim, blockDim;
  size_t dynamicSmemBytes;
  cudaStream_t stream;
  cudaLaunchAttribute* attrs;
  unsigned numAttrs;
};
template <class... P, class... A>
cudaError_t cudaLaunchKernelEx(const cudaLaunchConfig_t* c, void (*kernel)(P...), A&&... a) {
  emu::run(c->gridDim, c->blockDim, [&] { kernel(a...); });
  return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline const char* cudaGetErrorString(cudaError_t) { return ""; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, int) { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int* d) { *d = emu::device; return cudaSuccess; }
inline cudaError_t cudaDeviceGetAttribute(int* v, int what, int) {
  *v = what == cudaDevAttrMultiProcessorCount ? emu::multiprocessors : 232448;
  return cudaSuccess;
}
template <class T> cudaError_t cudaGetSymbolAddress(void** p, T& symbol) { *p = (void*)&symbol; return cudaSuccess; }
template <class K>
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, K, int, size_t) { *n = 4; return cudaSuccess; }
template <class K> cudaError_t cudaFuncSetAttribute(K, int, int) { return cudaSuccess; }
inline cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
inline cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, int, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
