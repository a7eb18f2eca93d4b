// Backend layer: one kernel source, two ways to run it.
//
//  * default (nvcc, sm_100a): kernels are __global__ functions launched on a CUDA stream.
//  * -DS2C_EMUL (g++, test-only): every CUDA thread of a block becomes a user-level fiber on
//    the host and __syncthreads() becomes a fiber barrier, so the same kernel bodies, index
//    arithmetic, dispatch code and table builders can be checked on a machine without a GPU.
//    The emulation library is built and loaded by the test-suite only; the shipped Python
//    package never loads it.
//
// A kernel is written once as
//
//     S2C_KERNEL(my_kernel, MyParams) { ... ctx.tid / ctx.nthr / ctx.bid / ctx.sync() ... }
//
// and launched with S2C_LAUNCH(my_kernel, grid, block, smem_bytes, stream, params).
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

namespace s2c {

// Thread-local last error text, returned by s2c_last_error().
inline std::string& last_error_ref() {
  static thread_local std::string e;
  return e;
}
inline int fail(int code, const std::string& msg) {
  last_error_ref() = msg;
  return code;
}

enum Status : int {
  S2C_OK = 0,
  S2C_ERR_BAD_ARG = 1,
  S2C_ERR_CUDA = 2,
  S2C_ERR_WORKSPACE = 3,
  S2C_ERR_UNSUPPORTED = 4,
};

}  // namespace s2c

#ifndef S2C_EMUL
// ------------------------------------------------------------------------------------------
// CUDA backend
// ------------------------------------------------------------------------------------------
#include <cuda_runtime.h>

#define S2C_D __device__ __forceinline__
#define S2C_HD __host__ __device__ __forceinline__

namespace s2c {

typedef cudaStream_t stream_t;

struct Ctx {
  int tid, nthr, bid, nblk;
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  // barrier among the 32 threads of a warp (every warp of the block must call it equally often:
  // the emulation build implements it as a block barrier)
  __device__ __forceinline__ void sync_warp() const { __syncwarp(); }
};

inline int cuda_check(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return S2C_OK;
  return fail(S2C_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

inline void* dev_alloc(size_t bytes) {
  void* p = nullptr;
  if (cudaMalloc(&p, bytes ? bytes : 1) != cudaSuccess) return nullptr;
  return p;
}
inline void dev_free(void* p) { cudaFree(p); }
inline int dev_upload(void* dst, const void* src, size_t bytes) {
  return cuda_check(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice), "table upload");
}
inline int dev_current() {
  int d = 0;
  cudaGetDevice(&d);
  return d;
}
inline int dev_memset_async(void* p, int v, size_t bytes, stream_t s) {
  return cuda_check(cudaMemsetAsync(p, v, bytes, s), "memset");
}
// Per-device values the host looks up on every call, remembered after the first (0 = not yet known).
constexpr int kMaxDevices = 64;
inline int dev_sm_count() {
  static std::atomic<int> known[kMaxDevices];
  const int dev = dev_current();
  int n = dev < kMaxDevices ? known[dev].load(std::memory_order_relaxed) : 0;
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
    if (dev < kMaxDevices) known[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}
inline int dev_smem_limit() {
  static std::atomic<int> known[kMaxDevices];
  const int dev = dev_current();
  int v = dev < kMaxDevices ? known[dev].load(std::memory_order_relaxed) : 0;
  if (v == 0) {
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (dev < kMaxDevices) known[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

}  // namespace s2c

// Launches are programmatic (launch_impl): the blocks of a kernel may be placed before the kernel ahead of it in the stream
// has finished, and wait in stream_order_wait, which every __global__ function calls before it reads or writes memory that
// another kernel touches; that returns when the kernel ahead has finished, its writes included.  So the order of the stream
// stands; what goes away is 1 - 2 us between the end of a kernel and the first instruction of the next (two launches at
// b = 22, 45 signals: 24.6 -> 20.8 us; 135 at b = 30, a training step: 2672 -> 2515; five, a rotation: 50.7 -> 39.5).
// Those are calls one after another, whose first kernel also meets the last one of the call before.  Calls that are waited for
// keep the gaps between their own kernels: analysis, synthesis and rotation of 200 signals at b = 12 24.6 -> 22.1, 26.1 -> 24.2
// and 58 -> 49 us, of 2000 at b = 16, many waves each, 192 -> 189, 211 -> 204, 526 -> 515.  None at b = 9 - 64 got slower either way.
// stream_order_next lets the next kernel's blocks in once every block has called it: at a block's end.  Called at the
// beginning, the next kernel's blocks crowd on the SMs that are done first (rotation 46.9 us, S2 transforms of 192 signals
// 77.6 instead of 67.4); the tensor-core products, one block per SM whatever comes next, call it there.
__device__ __forceinline__ void stream_order_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void stream_order_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

#define S2C_KERNEL(name, P)                                                                  \
  struct name##_impl {                                                                       \
    static __device__ __forceinline__ void run(const s2c::Ctx& ctx, const P& p,              \
                                               unsigned char* smem);                         \
  };                                                                                         \
  static __global__ void name(const P p) {                                                        \
    extern __shared__ float4 s2c_dyn_smem[];                                                 \
    s2c::Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};        \
    stream_order_wait();                                                                     \
    name##_impl::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));                \
    stream_order_next();                                                                     \
  }                                                                                          \
  __device__ __forceinline__ void name##_impl::run(const s2c::Ctx& ctx, const P& p,          \
                                                   unsigned char* smem)

#define S2C_KERNEL_BOUNDS(name, P, MAXT, MINB)                                               \
  struct name##_impl {                                                                       \
    static __device__ __forceinline__ void run(const s2c::Ctx& ctx, const P& p,              \
                                               unsigned char* smem);                         \
  };                                                                                         \
  static __global__ void __launch_bounds__(MAXT, MINB) name(const P p) {                            \
    extern __shared__ float4 s2c_dyn_smem[];                                                 \
    s2c::Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};        \
    stream_order_wait();                                                                     \
    name##_impl::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));                \
    stream_order_next();                                                                     \
  }                                                                                          \
  __device__ __forceinline__ void name##_impl::run(const s2c::Ctx& ctx, const P& p,          \
                                                   unsigned char* smem)

namespace s2c {
extern thread_local long g_launch_count;  // kernels launched by this thread (bench counter)

// Optional per-kernel timing (s2c_timing_begin / s2c_timing_end): one CUDA event pair per launch,
// recorded on the launching stream.
struct TimingRec {
  const char* name;
  cudaEvent_t a, b;
};
inline std::atomic<bool>& timing_on() {
  static std::atomic<bool> on{false};
  return on;
}
inline std::mutex& timing_mutex() {
  static std::mutex m;
  return m;
}
inline std::vector<TimingRec>& timing_recs() {   // guarded by timing_mutex()
  static std::vector<TimingRec> r;
  return r;
}

// The kernel is a template argument, so that the shared-memory limit it has been given on each device
// is remembered per kernel: the attribute is set when a launch needs more than any launch before it
// (cudaFuncSetAttribute on every launch was a tenth of the host time of a small call).
template <auto kernel, class P>
inline int launch_impl(const char* kname, long grid, int block, size_t smem, stream_t stream, const P& p, int cluster = 1) {
  if (grid <= 0) return S2C_OK;
  if (grid > 2147483647L) return fail(S2C_ERR_UNSUPPORTED, std::string(kname) + ": grid too large");
  if (smem > 48 * 1024) {
    static std::atomic<int> granted[kMaxDevices];
    const int dev = dev_current();
    if (dev >= kMaxDevices || granted[dev].load(std::memory_order_acquire) < (int)smem) {
      static std::mutex mu;
      std::lock_guard<std::mutex> lock(mu);   // a smaller request must not undo a larger one
      if (dev >= kMaxDevices || granted[dev].load(std::memory_order_relaxed) < (int)smem) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return cuda_check(e, kname);
        if (dev < kMaxDevices) granted[dev].store((int)smem, std::memory_order_release);
      }
    }
  }
  TimingRec rec{kname, nullptr, nullptr};
  const bool timed = timing_on();
  if (timed) {
    cudaEventCreate(&rec.a);
    cudaEventCreate(&rec.b);
    cudaEventRecord(rec.a, stream);
  }
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;     // see stream_order_wait
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;     // clusters of a size chosen at run time (at most 8, a divisor of the grid)
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kernel, p);   // (an error is reported below)
  if (timed) {
    cudaEventRecord(rec.b, stream);
    std::lock_guard<std::mutex> lock(timing_mutex());
    timing_recs().push_back(rec);
  }
  ++g_launch_count;
  return cuda_check(cudaGetLastError(), kname);
}
}  // namespace s2c

#define S2C_LAUNCH(name, grid, block, smem, stream, params) \
  s2c::launch_impl<name>(#name, (long)(grid), (int)(block), (size_t)(smem), stream, params)

namespace s2c {
// ---- asynchronous bulk copy global -> shared (TMA, 1-D) completing on an mbarrier -------------
// dst, src and bytes must be multiples of 16.  One thread initialises the barrier and issues the
// copies; every thread waits with bulk_wait (bounded: returns false if the copy has not landed by then, in
// which case the caller reads the data from global memory instead).  A further copy may only be issued into a phase
// that is over, and while a phase is not over the parity of the next one reads as landed: who issues looks at it
// (bulk_over) first, and once a copy has been given up none is issued or trusted any more.
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void bulk_barrier_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bulk_load_issue(void* dst, const void* src, unsigned bytes,
                                                unsigned long long* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// two independent single-precision operations in one instruction, each rounded as the scalar one
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\t"
      "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
// max(v, 0) with NaN passed on, as torch's relu does (fmaxf and "v > 0 ? v : 0" turn NaN into 0)
__device__ __forceinline__ float relu(float v) {
  float r;
  asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(v));
  return r;
}
// 32-byte global accesses (one full sector per lane and instruction); p must be 32-byte aligned
struct float8 {
  float4 lo, hi;
};
__device__ __forceinline__ float8 ld_global_256(const float* p) {
  float8 r;
  asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(r.lo.x), "=f"(r.lo.y), "=f"(r.lo.z), "=f"(r.lo.w), "=f"(r.hi.x), "=f"(r.hi.y),
                 "=f"(r.hi.z), "=f"(r.hi.w)
               : "l"(p));
  return r;
}
__device__ __forceinline__ void st_global_256(float* p, const float8& v) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v.lo.x), "f"(v.lo.y),
               "f"(v.lo.z), "f"(v.lo.w), "f"(v.hi.x), "f"(v.hi.y), "f"(v.hi.z), "f"(v.hi.w)
               : "memory");
}

// ---- thread-block clusters: block rank, cluster barrier, access to the other blocks' shared memory ------
struct ClCtx {
  int tid, nthr, bid, rank;      // bid: cluster index, rank: block within the cluster
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  __device__ __forceinline__ void sync_cluster() const {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  }
};
typedef unsigned cl_addr;        // shared::cluster address
// where `local` (an address of this block's shared memory) lies in block `rank` of the cluster
__device__ __forceinline__ cl_addr cl_map(const ClCtx&, const float2* local, int rank) {
  cl_addr a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
  return a;
}
__device__ __forceinline__ float2 cl_load(cl_addr base, int off) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(base + 8u * (unsigned)off) : "memory");
  return v;
}
// two complex numbers at a 16-byte boundary (off even)
__device__ __forceinline__ float4 cl_load4(cl_addr base, int off) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(base + 8u * (unsigned)off) : "memory");
  return v;
}
__device__ __forceinline__ void cl_store4(cl_addr base, int off, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(base + 8u * (unsigned)off), "f"(v.x), "f"(v.y),
               "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void cl_store_float(cl_addr base, int off, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(base + 4u * (unsigned)off), "f"(v) : "memory");
}


// is the phase of this parity over?  (one try, of bounded length)
__device__ __forceinline__ bool bulk_over(unsigned long long* bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done;
}
__device__ __forceinline__ bool bulk_wait(const Ctx&, unsigned long long* bar, unsigned parity) {
  for (int spin = 0; spin < (1 << 20); ++spin) {
    if (bulk_over(bar, parity)) return true;
    if (spin > 32) __nanosleep(32);
  }
  return false;
}
// for results that are known to be wrong
__device__ __forceinline__ float bulk_nan() { return __int_as_float(0x7fffffff); }
}  // namespace s2c

#else
// ------------------------------------------------------------------------------------------
// Host emulation backend (test-only)
// ------------------------------------------------------------------------------------------
#include <ucontext.h>

#define S2C_D inline
#define S2C_HD inline

struct float2 {
  float x, y;
};
struct float4 {
  float x, y, z, w;
};
struct int2 {
  int x, y;
};
struct int4 {
  int x, y, z, w;
};
inline int4 make_int4(int x, int y, int z, int w) { return int4{x, y, z, w}; }
inline float2 make_float2(float x, float y) { return float2{x, y}; }
inline float4 make_float4(float x, float y, float z, float w) { return float4{x, y, z, w}; }
inline float __ldg(const float* p) { return *p; }
inline float2 __ldg(const float2* p) { return *p; }
inline int __ldg(const int* p) { return *p; }
inline long long __ldg(const long long* p) { return *p; }
inline unsigned short __ldg(const unsigned short* p) { return *p; }

namespace s2c {

typedef void* stream_t;

struct EmuBlock {
  int nthr = 0;
  std::vector<ucontext_t> th;
  ucontext_t sched;
  std::vector<unsigned char> stacks;
  std::vector<char> done;
  void (*entry)(int tid, void* arg) = nullptr;
  void* arg = nullptr;
  int cur = 0;
};
inline EmuBlock*& emu_cur() {
  static thread_local EmuBlock* b = nullptr;
  return b;
}

struct Ctx {
  int tid, nthr, bid, nblk;
  void sync() const {
    EmuBlock* b = emu_cur();
    if (b->nthr > 1) swapcontext(&b->th[tid], &b->sched);
  }
  void sync_warp() const { sync(); }
};

inline void emu_trampoline() {
  EmuBlock* b = emu_cur();
  int t = b->cur;
  b->entry(t, b->arg);
  b->done[t] = 1;
  swapcontext(&b->th[t], &b->sched);
}

// Run one block: every thread is a fiber; a barrier is "yield to the scheduler"; the scheduler
// resumes the fibers round-robin, which executes the block phase by phase.
inline void emu_run_block(int nthr, void (*entry)(int, void*), void* arg) {
  static thread_local EmuBlock blk;
  const size_t kStack = 128 * 1024;
  blk.nthr = nthr;
  blk.entry = entry;
  blk.arg = arg;
  emu_cur() = &blk;
  if (nthr == 1) {
    entry(0, arg);
    return;
  }
  blk.th.resize(nthr);
  blk.done.assign(nthr, 0);
  if (blk.stacks.size() < kStack * nthr) blk.stacks.resize(kStack * nthr);
  for (int t = 0; t < nthr; ++t) {
    getcontext(&blk.th[t]);
    blk.th[t].uc_stack.ss_sp = blk.stacks.data() + kStack * t;
    blk.th[t].uc_stack.ss_size = kStack;
    blk.th[t].uc_link = &blk.sched;
    makecontext(&blk.th[t], (void (*)())emu_trampoline, 0);
  }
  int remaining = nthr;
  while (remaining > 0) {
    for (int t = 0; t < nthr; ++t) {
      if (blk.done[t]) continue;
      blk.cur = t;
      swapcontext(&blk.sched, &blk.th[t]);
      if (blk.done[t]) --remaining;
    }
  }
}

inline void* dev_alloc(size_t bytes) { return std::malloc(bytes ? bytes : 1); }
inline void dev_free(void* p) { std::free(p); }
inline int dev_upload(void* dst, const void* src, size_t bytes) {
  std::memcpy(dst, src, bytes);
  return S2C_OK;
}
inline int dev_current() { return 0; }
inline int dev_memset_async(void* p, int v, size_t bytes, stream_t) {
  std::memset(p, v, bytes);
  return S2C_OK;
}
inline int dev_smem_limit() { return 227 * 1024; }
inline int dev_sm_count() { return 3; }

extern thread_local long g_launch_count;
void emu_bulk_block_end();     // (see EmuBulk)

template <class Impl, class P>
struct EmuLaunch {
  const P* p;
  int bid, nblk, nthr;
  unsigned char* smem;
  static void entry(int tid, void* a) {
    EmuLaunch* self = (EmuLaunch*)a;
    Ctx ctx{tid, self->nthr, self->bid, self->nblk};
    Impl::run(ctx, *self->p, self->smem);
  }
};

template <class Impl, class P>
inline int emu_launch(const char* kname, long grid, int block, size_t smem, const P& p) {
  if (grid <= 0) return S2C_OK;
  if (smem > (size_t)dev_smem_limit())
    return fail(S2C_ERR_UNSUPPORTED, std::string(kname) + ": shared memory over the limit");
  if (block > 1024) return fail(S2C_ERR_UNSUPPORTED, std::string(kname) + ": block > 1024");
  std::vector<unsigned char> sm(smem + 64);
  EmuLaunch<Impl, P> L;
  L.p = &p;
  L.nblk = (int)grid;
  L.nthr = block;
  L.smem = sm.data() + ((64 - (uintptr_t)sm.data() % 64) % 64);
  for (long b = 0; b < grid; ++b) {
    L.bid = (int)b;
    emu_run_block(block, &EmuLaunch<Impl, P>::entry, &L);
    emu_bulk_block_end();
  }
  ++g_launch_count;
  return S2C_OK;
}

}  // namespace s2c

#define S2C_KERNEL(name, P)                                                                  \
  struct name##_impl {                                                                       \
    static inline void run(const s2c::Ctx& ctx, const P& p, unsigned char* smem);            \
  };                                                                                         \
  inline void name##_impl::run(const s2c::Ctx& ctx, const P& p, unsigned char* smem)

#define S2C_KERNEL_BOUNDS(name, P, MAXT, MINB) S2C_KERNEL(name, P)

namespace s2c {
// Host stand-ins of the bulk-copy helpers.  The wait is a block barrier (every thread of the block calls it at the same
// point).  The copy happens at issue time and ends the barrier's phase (bit 0 of the barrier: its parity), except for one
// that a test holds back: that one lands when one thread asks for it by itself (bulk_over), or never.
struct EmuBulk {
  long hold = 0, issued = 0;                  // hold: the number of the copy to hold back, from 1 (0: none)
  int never = 0;
  long faults = 0;                            // copies into a phase that is not over, and past the end of their block
  void* dst = nullptr;
  const void* src = nullptr;
  unsigned bytes = 0;
  unsigned long long* bar = nullptr;          // the held copy's barrier, until it lands
};
extern EmuBulk g_emu_bulk;
inline void bulk_barrier_init(unsigned long long* bar) { *bar = 0; }
inline void bulk_load_issue(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  EmuBulk& e = g_emu_bulk;
  if (e.bar == bar) ++e.faults;
  if (++e.issued == e.hold) {
    e.dst = dst; e.src = src; e.bytes = bytes; e.bar = bar;
    return;
  }
  std::memcpy(dst, src, bytes);
  *bar ^= 1;
}
// (a thread's own try, behind the waits: the held copy lands now, or never)
inline bool bulk_over(unsigned long long* bar, unsigned parity) {
  EmuBulk& e = g_emu_bulk;
  if (e.bar == bar && !e.never) {
    std::memcpy(e.dst, e.src, e.bytes);
    e.bar = nullptr;
    *bar ^= 1;
  }
  return (*bar & 1) != parity;
}
inline float bulk_nan() { return std::nanf(""); }
inline float2 fma2(float2 a, float2 b, float2 c) { return make_float2(std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)); }
inline float relu(float v) { return v <= 0.f ? 0.f : v; }
struct float8 {
  float4 lo, hi;
};
inline float8 ld_global_256(const float* p) {
  float8 r;
  r.lo = *reinterpret_cast<const float4*>(p);
  r.hi = *reinterpret_cast<const float4*>(p + 4);
  return r;
}
inline void st_global_256(float* p, const float8& v) {
  *reinterpret_cast<float4*>(p) = v.lo;
  *reinterpret_cast<float4*>(p + 4) = v.hi;
}
// A cluster: the fibers of all its blocks run as one group (a block barrier is then a cluster barrier, which
// is stronger), every block with shared memory of its own.
struct EmuCluster {
  unsigned char* smem = nullptr;
  size_t stride = 0;
};
inline EmuCluster& emu_cluster() {
  static thread_local EmuCluster c;
  return c;
}
struct ClCtx {
  int tid, nthr, bid, rank;
  void sync() const {
    EmuBlock* b = emu_cur();
    if (b->nthr > 1) swapcontext(&b->th[rank * nthr + tid], &b->sched);
  }
  void sync_cluster() const { sync(); }
};
typedef unsigned char* cl_addr;
inline cl_addr cl_map(const ClCtx& ctx, const float2* local, int rank) {
  return (cl_addr)local + (long)(rank - ctx.rank) * (long)emu_cluster().stride;
}
inline float2 cl_load(cl_addr base, int off) { return reinterpret_cast<float2*>(base)[off]; }
inline float4 cl_load4(cl_addr base, int off) { return *reinterpret_cast<float4*>(reinterpret_cast<float2*>(base) + off); }
inline void cl_store4(cl_addr base, int off, float4 v) { *reinterpret_cast<float4*>(reinterpret_cast<float2*>(base) + off) = v; }
inline void cl_store_float(cl_addr base, int off, float v) { reinterpret_cast<float*>(base)[off] = v; }

template <class Impl, class P>
struct EmuClusterLaunch {
  const P* p;
  int bid, nthr;
  static void entry(int fiber, void* a) {
    EmuClusterLaunch* self = (EmuClusterLaunch*)a;
    ClCtx ctx{fiber % self->nthr, self->nthr, self->bid, fiber / self->nthr};
    Impl::run(ctx, *self->p, emu_cluster().smem + ctx.rank * emu_cluster().stride);
  }
};
template <class Impl, class P>
inline int emu_launch_cluster(const char* kname, long nclusters, int c, int block, size_t smem, const P& p) {
  if (nclusters <= 0) return S2C_OK;
  if (smem > (size_t)dev_smem_limit())
    return fail(S2C_ERR_UNSUPPORTED, std::string(kname) + ": shared memory over the limit");
  const size_t stride = (smem + 63) / 64 * 64 + 64;   // a guard behind every block's shared memory
  std::vector<unsigned char> sm(stride * c + 64, 0xA5);
  emu_cluster().smem = sm.data() + ((64 - (uintptr_t)sm.data() % 64) % 64);
  emu_cluster().stride = stride;
  EmuClusterLaunch<Impl, P> L;
  L.p = &p;
  L.nthr = block;
  for (long b = 0; b < nclusters; ++b) {
    L.bid = (int)b;
    emu_run_block(c * block, &EmuClusterLaunch<Impl, P>::entry, &L);
    for (int r = 0; r < c; ++r)
      for (size_t i = smem; i < stride; ++i)
        if (emu_cluster().smem[r * stride + i] != 0xA5)
          return fail(S2C_ERR_CUDA, std::string(kname) + ": write past the shared memory of a block");
  }
  ++g_launch_count;
  return S2C_OK;
}
inline bool bulk_wait(const Ctx& ctx, unsigned long long* bar, unsigned parity) {
  ctx.sync();
  return (*bar & 1) != parity;
}
}  // namespace s2c

#define S2C_LAUNCH(name, grid, block, smem, stream, params)                                  \
  s2c::emu_launch<name##_impl>(#name, (long)(grid), (int)(block), (size_t)(smem), params)

#endif  // S2C_EMUL

namespace s2c {
// gradient of relu: v where the activation is positive or NaN, 0 elsewhere (torch's rule)
S2C_HD float relu_grad(float act, float v) { return act <= 0.f ? 0.f : v; }
}  // namespace s2c
