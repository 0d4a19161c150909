// Runs a CUDA kernel's source on the CPU, one fiber per thread of a CTA, with every buffer between
// two unmapped pages: an access one float outside a buffer is caught and reported, not executed.
// Barriers, ballots and shuffles switch fibers; cp.async copies at once.
#pragma once
#include <math.h>
#include <setjmp.h>
#include <signal.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <ucontext.h>
#include <unistd.h>

#include <functional>
#include <vector>

#include <vector_types.h>
#include <vector_functions.h>
#undef __device__
#undef __host__
#undef __global__
#undef __forceinline__
#undef __launch_bounds__
#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __shared__ static

namespace emu {

struct Index { unsigned x, y, z; };
struct Fiber { ucontext_t ctx; std::vector<char> stack; bool done; };
inline Index tid, bid, bdim, gdim;
inline std::vector<Fiber> fibers;
inline ucontext_t scheduler;
inline int current, warp_count[32], warp_gen[32], block_count, block_gen;
inline unsigned long long exchange[32][32];
inline float* smem;
inline const std::function<void()>* body;
inline sigjmp_buf bail;
inline void* fault_at;

inline void yield() {
  swapcontext(&fibers[current].ctx, &scheduler);
  tid.x = (unsigned)current;
}
inline void sync(int& count, int& gen, int n) {
  const int g = gen;
  if (++count == n) {
    count = 0;
    ++gen;
    return;
  }
  for (long turns = 0; gen == g; ++turns) {
    if (turns > 1000000) { fprintf(stderr, "a barrier that not every thread reaches\n"); abort(); }
    yield();
  }
}
inline void entry() {
  tid.x = (unsigned)current;
  (*body)();
  fibers[current].done = true;
  swapcontext(&fibers[current].ctx, &scheduler);
}
inline void on_fault(int, siginfo_t* info, void*) {
  fault_at = info->si_addr;
  siglongjmp(bail, 1);
}

// A buffer between two unmapped pages: its last byte (or its first) touches one.
struct Guarded {
  char *map, *data;
  size_t total, bytes;
  Guarded(const void* src, size_t n, bool at_end) : bytes(n) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), body = (n + page - 1) / page * page;
    total = body + 2 * page;
    map = (char*)mmap(nullptr, total, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    mprotect(map + page, body, PROT_READ | PROT_WRITE);
    data = at_end ? map + page + body - n : map + page;
    if (src) memcpy(data, src, n);
    else memset(data, 0xff, n);  // NaN
  }
  ~Guarded() { munmap(map, total); }
  Guarded(const Guarded&) = delete;
};

// Runs f as a grid of CTAs one after the other; the address of an access outside every buffer, else null.
inline void* launch(int grid, int block, size_t smem_bytes, const std::function<void()>& f) {
  struct sigaction act = {}, old_segv, old_bus;
  act.sa_sigaction = on_fault;
  act.sa_flags = SA_SIGINFO | SA_NODEFER;
  sigaction(SIGSEGV, &act, &old_segv);
  sigaction(SIGBUS, &act, &old_bus);
  body = &f;
  fault_at = nullptr;
  bdim = {(unsigned)block, 1, 1};
  gdim = {(unsigned)grid, 1, 1};
  if (!sigsetjmp(bail, 1)) {
    for (int b = 0; b < grid; ++b) {
      Guarded shared(nullptr, smem_bytes, true);
      smem = (float*)shared.data;
      bid = {(unsigned)b, 0, 0};
      block_count = block_gen = 0;
      memset(warp_count, 0, sizeof(warp_count));
      memset(warp_gen, 0, sizeof(warp_gen));
      fibers.assign(block, Fiber{});
      for (Fiber& t : fibers) {
        t.stack.resize(256 * 1024);
        getcontext(&t.ctx);
        t.ctx.uc_stack.ss_sp = t.stack.data();
        t.ctx.uc_stack.ss_size = t.stack.size();
        t.ctx.uc_link = nullptr;
        makecontext(&t.ctx, entry, 0);
      }
      for (bool any = true; any;) {
        any = false;
        for (current = 0; current < block; ++current) {
          if (fibers[current].done) continue;
          any = true;
          tid.x = (unsigned)current;
          swapcontext(&scheduler, &fibers[current].ctx);
        }
      }
    }
  }
  sigaction(SIGSEGV, &old_segv, nullptr);
  sigaction(SIGBUS, &old_bus, nullptr);
  return fault_at;
}

template <class T>
inline T trade(T v, int src) {
  const int w = current >> 5, l = current & 31;
  unsigned long long bits = 0;
  memcpy(&bits, &v, sizeof(T));
  exchange[w][l] = bits;
  sync(warp_count[w], warp_gen[w], 32);
  T r;
  memcpy(&r, &exchange[w][src & 31], sizeof(T));
  sync(warp_count[w], warp_gen[w], 32);
  return r;
}

}  // namespace emu

#define threadIdx emu::tid
#define blockIdx emu::bid
#define blockDim emu::bdim
#define gridDim emu::gdim

static inline void __syncthreads() { emu::sync(emu::block_count, emu::block_gen, (int)emu::bdim.x); }
static inline void __syncwarp(unsigned = 0xffffffffu) {
  emu::sync(emu::warp_count[emu::current >> 5], emu::warp_gen[emu::current >> 5], 32);
}
template <class T> static inline T __shfl_sync(unsigned, T v, int src) { return emu::trade(v, src); }
template <class T> static inline T __shfl_xor_sync(unsigned, T v, int x) { return emu::trade(v, (emu::current & 31) ^ x); }
static inline unsigned __reduce_or_sync(unsigned, unsigned v) {
  for (int o = 16; o; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
static inline unsigned __ballot_sync(unsigned, bool v) { return __reduce_or_sync(0xffffffffu, v ? 1u << (emu::current & 31) : 0u); }
static inline bool __any_sync(unsigned, bool v) { return __ballot_sync(0xffffffffu, v) != 0u; }
static inline bool __all_sync(unsigned, bool v) { return __ballot_sync(0xffffffffu, v) == 0xffffffffu; }
static inline int atomicAdd(int* p, int v) { const int r = *p; *p += v; return r; }
static inline int __popcll(unsigned long long v) { return __builtin_popcountll(v); }
static inline int __ffsll(long long v) { return __builtin_ffsll(v); }
static inline int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }
static inline float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }
static inline float rsqrtf(float x) { return 1.f / sqrtf(x); }
static inline double rsqrt(double x) { return 1. / sqrt(x); }
static inline float __fdividef(float a, float b) { return a / b; }
static inline void sincospif(float x, float* s, float* c) { sincosf(x * (float)M_PI, s, c); }
static inline void sincospi(double x, double* s, double* c) { sincos(x * M_PI, s, c); }
template <class T> static inline T __ldg(const T* p) { return *p; }

#include "br_b200.h"
namespace br {
constexpr int kWarp = 32;
inline int round4(int n) { return (n + 3) & ~3; }
inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
template <int N> inline void cp_async(void* d, const void* s) {
  if (((uintptr_t)d | (uintptr_t)s) & (N - 1)) { fprintf(stderr, "misaligned copy of %d bytes\n", N); abort(); }
  memcpy(d, s, N);
}
inline void cp_async16(void* d, const void* s) { cp_async<16>(d, s); }
inline void cp_async4(void* d, const void* s) { cp_async<4>(d, s); }
inline void cp_async_commit() {}
template <int N> inline void cp_async_wait_groups() {}
}  // namespace br
