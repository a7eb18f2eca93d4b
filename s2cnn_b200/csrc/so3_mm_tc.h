// so3_mm and its two gradients on the 5th-generation tensor cores (tcgen05.mma, accumulator in
// TMEM), 3xTF32.
//
//   z[l,m,n,i,j] = sum_{p,k} x[l,m,p,i,k] conj(y[l,n,p,k,j])            (s2cnn/so3_mm.py:8-93)
//
// is, for every degree l, ONE real GEMM on the reference's interleaved layouts:
//   C'[(m,i), (n,j,c)] = sum_{(p,k,c')} A'[(m,i),(p,k,c')] * B'[(p,k,c'),(n,j,c)]
// where A' is the x tensor read as plain floats (re, im interleaved along K - no transformation),
// C' is the z tensor written as plain floats, and B' is built from y while staging:
//   B'[(k,0),(j,0)] =  yr   B'[(k,1),(j,0)] = yi      (real part of x * conj(y))
//   B'[(k,0),(j,1)] = -yi   B'[(k,1),(j,1)] = yr      (imaginary part)
// so the complex product costs 8 real flops per complex MAC, the algorithmic count.  The two
// gradient products (s2cnn/so3_mm.py:95-122 and the backward kernels :125-261) have the same
// shape with other row / column / contraction roles; the kernel is instantiated per product.
//
// Precision: TF32 has 10 mantissa bits, not enough for the 1e-4 bar.  Every operand is split in
// float32 into hi = v truncated to TF32 and lo = v - hi and three MMAs (hi*hi, lo*hi, hi*lo)
// accumulate into the same float32 TMEM accumulator.  The tensor core's own accumulation
// truncates - a bias of up to one unit in the last place per MMA, always in the same direction,
// which adds up along the K loop.  The MMAs therefore alternate between two accumulators: every
// kTcFlushBlocks K blocks the issuer switches to the other one, and while the tensor core fills
// it the threads add the finished partial sum, rounding properly, into a third TMEM region.
//
// Tiling: one CTA per (l, 128-row tile, 128-column tile); the K loop walks blocks of at most
// kTcKMax floats (outer contraction index, slice of its run of floats).  The CTA is warp
// specialised (17 warps):
//   * 12 producer warps in three groups of four; a group stages every third K block.  A thread owns one row of
//     the row operand and half the K range of one complex column of the column operand: two pointers and
//     constant offsets, no per-slot geometry.  The row operand goes, split into hi / lo TF32 parts, into
//     TENSOR MEMORY (its thread is its TMEM lane; two stages of 64 columns), the column operand into shared
//     memory in the canonical K-major, no-swizzle UMMA layout (8 rows x 16 bytes core matrices; the real
//     columns of a tile are its rows 0 - 63, the imaginary ones 64 - 127: one load and one split serve both),
//     kTcStages stages deep.  The next block's loads are issued before the barrier waits of the current one; a
//     warp arrives on the stage's "full" mbarrier once its lanes have written their share;
//   * one issuer warp waits for "full", issues the nine tcgen05.mma of the block (hi*hi, lo*hi,
//     hi*lo for each k-step of 8) from one elected lane and commits them to the stage's "empty"
//     mbarrier, which lets the producers overwrite the stage; it alternates between two accumulators
//     in tensor memory every kTcFlushBlocks blocks and commits to an "accumulator done" mbarrier;
//   * 4 collector warps (one per TMEM lane quarter) add each finished accumulator, with proper
//     rounding, into a third tensor-memory region and hand the accumulator back ("accumulator
//     free") - all of it while the tensor core fills the other one.
// With both operands in shared memory a K block moved 48 KB of stores and 72 KB of MMA reads through a
// 128-byte-per-clock pipe (960 clocks) and its producers, every warp taking part in every block, issued
// about 1600 instructions: 1250 clocks per block measured, 480 us for 100 -> 100 channels at nl = 10, batch 32.
// Now 24 KB of stores and 36 KB of reads remain; 820 clocks per block in a lone CTA, 960 on a full chip, where
// nine 128 x 128 x 8 MMAs alone take 750.
// The epilogue (all 16 non-issuer warps) reads the last accumulator and the sum region with
// tcgen05.ld (32 lanes x 16 real and 16 imaginary columns per warp) and stores the result directly in
// its interleaved layout.  Every mbarrier wait is bounded; on a time-out the waiting thread raises a
// block-wide abort flag, every role leaves its loop, the kernel raises the error flag, frees its
// TMEM columns and returns.
#pragma once

#ifndef S2C_EMUL

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "backend.h"
#include "so3_kernels.h"   // align_up

namespace s2c {

// The same kernel runs the forward product and its two gradients; they differ in how the rows
// of the two operands are addressed and in the sign pattern that turns complex into real
// arithmetic (the op code selects both):
//   kTcFwd    z[l,m,n,i,j]  = sum_{p,k} x[l,m,p,i,k] conj(y[l,n,p,k,j])     a = x,  b = y,  c = z
//   kTcGradX  gx[l,m,p,i,k] = sum_{n,j} gz[l,m,n,i,j] y[l,n,p,k,j]          a = gz, b = y,  c = gx
//   kTcGradY  gy[l,n,p,k,j] = sum_{m,i} conj(gz[l,m,n,i,j]) x[l,m,p,i,k]    a = x,  b = gz, c = gy
// (s2cnn/so3_mm.py:8-122).  An output row is (outer, inner) = (m, i) - or (p, k) for kTcGradY - and
// an output column (outer, 2 * inner + re/im).  The contraction index is (outer, run of `run`
// floats): a "contiguous" operand holds the run of a row as consecutive floats (16-byte loads), a
// "strided" one holds it as complex pairs `stride` floats apart (two 8-byte loads per chunk).
//   kTcPlainCC / kTcPlainSC: a plain real product C[r][c] = sum_k A[r][k] B[c][k] on the same
//   pipeline, with explicit strides (rows, pairs of consecutive k, pairs of consecutive c) instead
//   of the spectral geometry: the kernel-grid -> spectrum transforms s2_rft / so3_rft and their
//   transposes (s2cnn/s2_ft.py:22, s2cnn/so3_ft.py:22).  CC: both operands hold k contiguously;
//   SC: the row operand holds k as pairs `a_ps` floats apart.
enum TcOp : int { kTcFwd = 0, kTcGradX = 1, kTcGradY = 2, kTcPlainCC = 3, kTcPlainSC = 4 };

// The forward product takes half of the columns: their number does not shrink with the batch, so that small batches gain, too
// (two signals, 46 -> 93 channels, nl = 10: 150 tiles, one wave and a rest -> 80), and which half is computed - and so the
// rounding - does not depend on it.
enum TcHalf : int { kTcWhole = 0, kTcHalfRows = 1, kTcHalfColumns = 2 };

struct MmTcParams {
  const float* a;   // operand read along the output rows
  const float* b;   // operand read along the output columns
  float* c;         // output
  int nl, nb, fi, fo;
  int half;         // spectra of real signals: rows (kTcHalfRows) or columns (kTcHalfColumns) of outer index l .. 2l only,
                    // the others are their mirrors
  int two;          // without partial sums: the products with a lo part go into the second accumulator
  int twins;        // half products, one CTA per tile: two CTAs compute it, one writes the tile and one its mirror (tc_twins)
  int segs;         // > 1: a tile's K blocks are summed in this many segments, in one CTA or one to a CTA of a cluster (tc_segments)
  int run;          // floats per outer contraction index: 2 fi (fwd), 2 fo (grad x), 2 nb (grad y)
  int kblk;         // floats per K block (multiple of 8, <= kTcKMax)
  int nblk;         // K blocks per run
  int csize, groups;   // a tile's contraction is shared by csize * groups CTAs: `groups` clusters of csize, whose
                    // partial results are added in the order of their K blocks (see tc_pick_share)
  float* part;      // groups > 1: the clusters' sums (kTcTileFloats each, in grid order) and, zero at the launch,
  int* count;       // eight arrival counters per tile
  int* err;         // device flag, set to 1 on a wait time-out
  // plain products only (floats): element (row r, k) of a at r * a_rs + (k / 2) * a_ps + k % 2,
  // element (column c, k) of b likewise, element (r, c) of the result at r * c_rs + (c / 2) * c_ps + c % 2;
  // nb = rows, fi = K / 2, fo = columns / 2, nl = 1
  long a_rs, a_ps, b_rs, b_ps, c_rs, c_ps;
  float scale;      // kTcPlainCC: the row operand is multiplied by this (and rounded) while it is staged;
                    // kTcPlainSC: the result is
};

// row / column geometry of one degree
struct TcGeom {
  int RI;           // inner extent of a row index
  int CW;           // floats per outer column index (2 * inner extent)
};
__host__ __device__ __forceinline__ TcGeom tc_geom(int op, int nb, int fi, int fo) {
  TcGeom g;
  g.RI = op == kTcGradY ? fi : nb;
  g.CW = op == kTcGradX ? 2 * fi : 2 * fo;
  return g;
}

constexpr int kTcBM = 128, kTcBN = 128;
constexpr int kTcKMax = 24;                       // floats per K block
constexpr int kTcStages = 6;                      // of the column operand (shared memory)
constexpr int kTcLBO = kTcBM * 16 + 64;           // bytes between K-adjacent core matrices (padded)
constexpr int kTcSBO = 128;                       // bytes between row-adjacent core matrices
constexpr int kTcBufBytes = (kTcKMax / 4) * kTcLBO;   // one operand buffer (hi or lo)
constexpr int kTcStageBytes = 2 * kTcBufBytes;        // B hi, B lo
constexpr int kTcSmemBytes = kTcStages * kTcStageBytes + 256;   // + mbarriers, TMEM slot, abort flag
constexpr int kTcGroups = 3, kTcGroupWarps = 4;     // producer groups (a group = one warp per TMEM lane quarter)
constexpr int kTcProducerWarps = kTcGroups * kTcGroupWarps, kTcCollectorWarps = 4;
constexpr int kTcFirstProducer = 32 * (1 + kTcCollectorWarps);  // thread index of the first producer
constexpr int kTcThreads = 32 * (1 + kTcCollectorWarps + kTcProducerWarps);
// K blocks accumulated by the tensor core before the partial sum is added, in FP32 with rounding,
// into the sum region (bounds the length of the tensor core's own accumulation chain, whose
// additions truncate): 8 blocks = 72 MMAs per chain.  Half products flush every 7: a coefficient and its mirror are then no
// longer two sums of which the synthesis takes the mean, and the shorter chain makes up for that (relative error of the
// symmetric part, nl = 10, 100 -> 100, batch 32: 1.69e-6 full, 1.75e-6 half with 8, 1.58e-6 with 7).
constexpr int kTcFlushBlocks = 8;
// longest chain (in MMAs) left to the tensor core's own accumulation without partial sums: its truncation bias stays
// below about 1e-5 relative.  The second accumulator is then free; in half products it takes the products with a lo part:
// they are 2^-11 of the others, so their truncations do not count, and a third of the chain's remain (198 MMAs, nl = 6,
// 20 -> 40: relative error 3.3e-6 in one accumulator, 1.2e-6 in two).  Full products stay as they were, to the bit.
constexpr int kTcChainMax = 200;
// tensor-memory columns: two alternating accumulators, the FP32 sum region and two stages of the row operand
// (hi in columns 0 - 23, lo in 32 - 55 of each)
constexpr int kTcTmemCols = 512;
constexpr int kTcSumCol = 2 * kTcBN;
constexpr int kTcACol = 3 * kTcBN, kTcAStages = 2, kTcAPitch = 64, kTcALo = 32;
static_assert(kTcACol + kTcAStages * kTcAPitch == kTcTmemCols && kTcKMax <= kTcALo, "tensor memory");
static_assert(kTcSmemBytes > 114 * 1024, "one CTA per SM: each allocates all of the tensor memory");

__device__ __forceinline__ uint32_t tc_smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t saddr) {
  // K-major, no swizzle: start >> 4 | LBO >> 4 << 16 | SBO >> 4 << 32 | version 1 << 46
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)(kTcLBO >> 4) << 16;
  d |= (uint64_t)(kTcSBO >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

__device__ __forceinline__ float tc_tf32(float v) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}

__device__ __forceinline__ void tc_mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem_u32(bar)), "r"(count));
}

// Bounded wait on an mbarrier phase; returns false on time-out.
__device__ __forceinline__ bool tc_mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = tc_smem_u32(bar);
  for (int spin = 0; spin < (1 << 22); ++spin) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if (spin > 64) __nanosleep(64);
  }
  return false;
}

// row operand in tensor memory, column operand in shared memory
__device__ __forceinline__ void tc_mma_tf32(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// One lane of a converged warp, by elect.sync.  Measured against "lane == 0" as the guard of the issuer's code:
// 820 clocks per K block of a lone CTA instead of 1280.
__device__ __forceinline__ bool tc_elect() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   tc_smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tc_st16(uint32_t taddr, const float (&v)[16]) {
  uint32_t r[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(v[i]);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
        "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
        "r"(r[15])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// CTAs that share a tile form a cluster: each puts its partial result into its own shared memory, and rank r adds
// all of them, in rank order, for its share of the tile's columns.  The result does not depend on which CTA
// finishes when.  (Atomic adds into a cleared output took about the same time, but in the order of arrival:
// gradients then differ from run to run.)  A contraction too long for one cluster is shared by several; the ranks
// of a tile's last cluster to arrive add the clusters' sums, again in a fixed order.
constexpr int kTcTileFloats = kTcBM * kTcBN;
constexpr int kTcMaxCluster = 8;
static_assert(kTcTileFloats * 4 <= kTcStages * kTcStageBytes, "a partial tile lies in the operand stages");
__device__ __forceinline__ void tc_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// Arrival at a counter after this CTA's values have been written; true in the CTA that arrives last of n, whose
// reads then see the others' values.  Called by all threads of the CTA; nobody waits for another CTA.
__device__ __forceinline__ bool tc_last_of(int* counter, int n, int* flag) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *flag = atomicAdd(counter, 1) == n - 1;
  __syncthreads();
  const bool last = *flag != 0;
  __threadfence();
  __syncthreads();       // the flag may be written again
  return last;
}

// 8 columns of a lane's row (completes with tcgen05.wait::st)
__device__ __forceinline__ void tc_st8(uint32_t taddr, const float (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
               "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
               "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
               "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
               : "memory");
}
// v = hi + lo with hi carrying the 10 explicit TF32 mantissa bits (the tensor core ignores the
// lower 13 bits of its inputs, so lo = v - hi needs no further rounding)
__device__ __forceinline__ float tc_hi(float v) { return __uint_as_float(__float_as_uint(v) & 0xFFFFE000u); }

__host__ __device__ __forceinline__ long tc_tiles_for(int op, int half, int nb, int fi, int fo, int l) {
  const TcGeom g = tc_geom(op, nb, fi, fo);
  const long L = 2 * l + 1;
  const long M = (half == kTcHalfRows ? l + 1 : L) * g.RI, N = (half == kTcHalfColumns ? l + 1 : L) * g.CW;
  return ((M + kTcBM - 1) / kTcBM) * ((N + kTcBN - 1) / kTcBN);
}

// FLUSH = false keeps the whole chain in one tensor-memory accumulator and drops the partial-sum
// code; the host selects it while no CTA issues more than kTcChainMax MMAs.
// VEC = true: 16-byte loads and stores (feature counts - for grad y the batch - even); VEC = false:
// 8-byte accesses, any sizes.
template <int OP, bool FLUSH, bool VEC>
__global__ void __launch_bounds__(kTcThreads, 1) so3_mm_tc_kernel(const MmTcParams p) {
  extern __shared__ float4 s2c_dyn_smem[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(s2c_dyn_smem);
  unsigned char* ctl = smem + kTcStages * kTcStageBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(ctl);                 // [stages] producers -> issuer
  uint64_t* empty = full + kTcStages;                                // [stages] tensor core -> producers
  uint64_t* accdone = empty + kTcStages;                             // [2] tensor core -> collectors
  uint64_t* accfree = accdone + 2;                                   // [2] collectors -> issuer
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accfree + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* last_flag = reinterpret_cast<int*>(tmem_slot + 2);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

  // ---- which tile ---------------------------------------------------------------------------
  const int nsplit = p.csize * p.groups, per_tile = p.twins ? 2 : nsplit;
  int l = p.nl - 1;
  long t = blockIdx.x;
  for (;; --l) {
    const long c = tc_tiles_for(OP, p.half, p.nb, p.fi, p.fo, l) * per_tile;
    if (t < c) break;
    t -= c;
  }
  const int L = 2 * l + 1;
  // K blocks handled by this CTA: [it_lo, it_hi) of the L * nblk blocks (outer index, block of its run)
  // (few divisions, of 32 bits: every CTA waits for this)
  int tile_no = (int)t, split = 0, it_lo = 0, it_hi = L * p.nblk, o_lo = 0;
  bool second = false;      // of a pair: writes the mirror
  if (p.twins) {
    second = tile_no & 1;
    tile_no >>= 1;
  } else if (nsplit > 1) {
    const int whole = tile_no / nsplit;
    split = tile_no - whole * nsplit;
    tile_no = whole;
    it_lo = (int)((long)split * L * p.nblk / nsplit);
    it_hi = (int)((long)(split + 1) * L * p.nblk / nsplit);
    o_lo = it_lo / p.nblk;
  }
  const int kb_lo = it_lo - o_lo * p.nblk;
  const TcGeom geo = tc_geom(OP, p.nb, p.fi, p.fo);
  const int RI = geo.RI, CW = geo.CW;
  // outer indices of the first row and column
  const int ro0 = p.half == kTcHalfRows ? l : 0, co0 = p.half == kTcHalfColumns ? l : 0;
  const int M = (L - ro0) * RI, Np = (L - co0) * CW;
  const int tiles_n = (Np + kTcBN - 1) / kTcBN;
  const int row0 = tile_no / tiles_n * kTcBM, col0 = tile_no % tiles_n * kTcBN;
  const long spec0 = (long)l * (4L * l * l - 1) / 3;
  const int fi2 = 2 * p.fi, fo2 = 2 * p.fo;
  const int nit = it_hi - it_lo;                          // K blocks of this CTA (a shared tile: possibly none)
  const bool two_accs = !FLUSH && p.two;
  // accumulator groups (one when the whole chain stays in the tensor core's accumulator)
  const int flush_blocks = p.half ? kTcFlushBlocks - 1 : kTcFlushBlocks;
  const bool segmented = p.segs > 1;
  const int ngroups = !FLUSH ? 1 : segmented ? min(p.segs, nit) : (nit + flush_blocks - 1) / flush_blocks;
  // first block beyond the group that begins at block `it` (segments: floor(r nit / segs), empty ones left out)
  auto group_end = [&](int it) {
    if (!segmented) return it + flush_blocks;
    int r = (it + 1) * p.segs / nit;
    while (r * nit / p.segs <= it) ++r;
    return r * nit / p.segs;
  };

  // ---- set-up: barriers, tensor memory ------------------------------------------------------
  if (tid == 0) {
    for (int i = 0; i < kTcStages; ++i) {
      tc_mbar_init(&full[i], kTcGroupWarps);
      tc_mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc_mbar_init(&accdone[i], 1);
      tc_mbar_init(&accfree[i], kTcCollectorWarps);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // What is above touches no memory of another kernel.  Tensor memory is taken behind the wait: a kernel ahead that lets
  // these CTAs in before it has taken its own could never get it from a CTA that holds all of it and waits.
  stream_order_wait();
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc_smem_u32(tmem_slot)),
                 "r"(kTcTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  stream_order_next();     // (CTAs of 150 KB: none of these beside a waiting one of the next kernel, whose set-up is the longest)

  bool ok = true;
  // a wait that gives up tells every role to leave its loop
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (tc_mbar_wait(bar, parity)) return true;
    *abort_flag = 1;
    ok = false;
    return false;
  };

  if (warp == 0) {
    // ================================ issuer ====================================================
    // instruction descriptor: D = F32, A = B = TF32, both K-major, N = 128, M = 128
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(kTcBN >> 3) << 17) |
                           ((uint32_t)(kTcBM >> 4) << 24);
    // The descriptors of every (stage, buffer, k-step) of the column operand differ from the one of stage 0,
    // hi, k-step 0 only in the 14-bit start-address field (bytes >> 4), so they are obtained by
    // adding constants (the whole staging area is below 256 KB, the field cannot overflow).
    const uint64_t d0 = tc_smem_desc(tc_smem_u32(smem));
    constexpr uint64_t kDBuf = kTcBufBytes >> 4, kDStage = kTcStageBytes >> 4, kDStep = (2u * kTcLBO) >> 4;
    constexpr int kStepsMax = kTcKMax / 8;
    const int steps_full = (p.kblk + 7) / 8;
    const int steps_tail = (p.run - (p.nblk - 1) * p.kblk + 7) / 8;
    int kb = kb_lo, s = 0, g = 0, ing = 0;           // block within its run, stage, group, block within its group
    int g_end = FLUSH && nit > 0 ? group_end(0) : 0;
    uint32_t full_par = 0;                        // parity of the `full` phase of the current round of stages
    for (int it = 0; it < nit; ++it) {
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      if (FLUSH && ing == 0 && g >= 2)            // the collectors are done with this accumulator
        if (!__all_sync(0xffffffffu, wait(&accfree[g & 1], (uint32_t)((g / 2 - 1) & 1)))) break;
      if (!__all_sync(0xffffffffu, wait(&full[s], full_par))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (tc_elect()) {
        const int ksteps = kb + 1 == p.nblk ? steps_tail : steps_full;
        const uint64_t db = d0 + (uint64_t)s * kDStage;
        const uint32_t ta = tmem_base + kTcACol + (uint32_t)(it % kTcAStages) * kTcAPitch;
        const uint32_t acc = tmem_base + (FLUSH ? (uint32_t)((g & 1) * kTcBN) : 0u);
#pragma unroll
        for (int ks = 0; ks < kStepsMax; ++ks) {
          if (ks < ksteps) {
            const uint64_t dbh = db + ks * kDStep, dbl = dbh + kDBuf;
            const uint32_t tah = ta + 8 * ks, tal = tah + kTcALo;
            const uint32_t acc_lo = two_accs ? acc + kTcBN : acc;
            const uint32_t first = ((FLUSH ? ing == 0 : it == 0) && ks == 0) ? 0u : 1u;
            tc_mma_tf32(acc, tah, dbh, idesc, first);
            tc_mma_tf32(acc_lo, tal, dbh, idesc, two_accs ? first : 1u);
            tc_mma_tf32(acc_lo, tah, dbl, idesc, 1u);
          }
        }
        tc_commit(&empty[s]);     // arrives when these MMAs have read the stage
        if ((FLUSH && it + 1 == g_end) || it + 1 == nit) tc_commit(&accdone[g & 1]);
      }
      __syncwarp();
      if (++kb == p.nblk) kb = 0;
      if (++s == kTcStages) { s = 0; full_par ^= 1u; }
      ++ing;
      if (FLUSH && it + 1 == g_end) {
        ing = 0;
        ++g;
        if (it + 1 < nit) g_end = group_end(it + 1);
      }
    }
  } else if (warp <= kTcCollectorWarps) {
    // ================================ collectors ================================================
    // This warp's TMEM lane quarter, all 128 columns: every finished accumulator but the last is
    // added into the sum region while the tensor core fills the other accumulator.
    if (FLUSH) {
      const uint32_t lanes = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16);
      for (int g = 0; g + 1 < ngroups && !*abort_flag; ++g) {
        if (!wait(&accdone[g & 1], (uint32_t)((g / 2) & 1))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int h = 0; h < kTcBN / 16; ++h) {   // 16 columns at a time keeps the registers low
          float v[16];
          tc_ld16(lanes + (uint32_t)((g & 1) * kTcBN + 16 * h), v);
          if (g > 0) {
            float w[16];
            tc_ld16(lanes + (uint32_t)(kTcSumCol + 16 * h), w);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += w[i];
          }
          tc_st16(lanes + (uint32_t)(kTcSumCol + 16 * h), v);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem_u32(&accfree[g & 1]))
                       : "memory");
      }
    }
  } else {
    // ================================ producers =================================================
    // operand addressing (floats): offset of outer contraction index `o`, element `kf` of its run =
    //   contiguous:  o * ko + kf          strided:  o * ko + (kf / 2) * st + (kf % 2)
    constexpr bool plain = OP == kTcPlainCC || OP == kTcPlainSC;
    constexpr bool a_str = OP == kTcGradY || OP == kTcPlainSC, b_str = OP == kTcFwd || OP == kTcGradY;
    long a_ko, b_ko, a_st = 2, b_st = 2;
    if (OP == kTcFwd)        { a_ko = (long)p.nb * fi2;      b_ko = (long)p.fi * fo2;      b_st = fo2; }
    else if (OP == kTcGradX) { a_ko = (long)p.nb * fo2;      b_ko = (long)L * p.fi * fo2; }
    else if (OP == kTcGradY) { a_ko = (long)L * p.nb * fi2;  b_ko = (long)L * p.nb * fo2;  a_st = fi2; b_st = fo2; }
    else                       { a_ko = 0; b_ko = 0; a_st = p.a_ps; b_st = p.b_ps; }   // one outer index
    const int group = (warp - 1 - kTcCollectorWarps) / kTcGroupWarps;
    const int t = tid - kTcFirstProducer - group * 32 * kTcGroupWarps;       // thread of the group
    const int nprs = p.kblk / 2;                                 // complex numbers (pairs of floats) per full block
    const int tail = (p.run - (p.nblk - 1) * p.kblk) / 2;        // pairs of a run's last block (VEC: even)

    // row operand: this thread's row = its TMEM lane
    const float* gA = nullptr;
    {
      const int gr = row0 + 32 * (warp & 3) + lane;
      const int rq = gr / RI, ri = gr - rq * RI, ro = ro0 + rq;
      long base;
      if (OP == kTcFwd)        base = ((spec0 + (long)ro * L) * p.nb + ri) * fi2;
      else if (OP == kTcGradX) base = ((spec0 + (long)ro * L) * p.nb + ri) * fo2;
      else if (OP == kTcGradY) base = (spec0 + ro) * p.nb * fi2 + 2 * ri;
      else                       base = (long)gr * p.a_rs;
      if (gr < M) gA = p.a + base;
    }
    // column operand: complex column t % 64, pairs 6 (t / 64) .. + 5 of the block; plain products: column t, all
    constexpr int kBPairs = plain ? kTcKMax / 2 : kTcKMax / 4;
    const int bcol = plain ? t : (t & 63), bp0 = plain ? 0 : kBPairs * (t >> 6);
    const float* gB = nullptr;
    {
      const int gcol = col0 + (plain ? bcol : 2 * bcol);
      const int cq = gcol / CW, in = (gcol - cq * CW) >> 1, co = co0 + cq;
      long base;
      if (OP == kTcFwd)        base = ((spec0 + (long)co * L) * p.fi * p.fo + in) * 2;
      else if (OP == kTcGradX) base = ((spec0 + co) * p.fi + in) * fo2;
      else if (OP == kTcGradY) base = (spec0 + co) * p.nb * fo2 + 2 * in;
      else                       base = (long)gcol * p.b_rs;
      if (gcol < Np) gB = p.b + base + (long)bp0 * b_st;
    }
    // offsets (floats) from one block of a run to the next
    const long a_stepk = (long)(p.kblk >> 1) * a_st, b_stepk = (long)(p.kblk >> 1) * b_st;

    // A lane reads its own row, so a 16-byte load of a warp touches 32 sectors and uses half of each: 32-byte
    // loads where the rows allow them (with the halves, the plain products - both operands row per lane - were
    // bound by the L1: 154 us for 10000 x 192 by 192 x 2660)
    const bool a_wide = reinterpret_cast<unsigned long long>(p.a) % 32 == 0 && p.run % 8 == 0 && (!plain || p.a_rs % 8 == 0);
    const bool b_wide = reinterpret_cast<unsigned long long>(p.b) % 32 == 0 && p.run % 8 == 0 && p.b_rs % 8 == 0;
    float2 ra[kTcKMax / 2], rb[kBPairs];                         // the block to be staged next
    // `cnt` pairs, `step` floats apart (2: consecutive), zeros beyond; null: a row outside the problem
    auto load_pairs = [&](auto& r, const float* src, bool strided, long step, int cnt, bool wide) {
      constexpr int n = sizeof(r) / sizeof(float2);
      if (VEC && !strided && wide) {
#pragma unroll
        for (int q = 0; q < n; q += 4) {
          float8 v;
          v.lo = v.hi = make_float4(0.f, 0.f, 0.f, 0.f);
          if (src && q < cnt) v = ld_global_256(src + 2 * q);    // cnt is a multiple of 4
          r[q] = make_float2(v.lo.x, v.lo.y); r[q + 1] = make_float2(v.lo.z, v.lo.w);
          r[q + 2] = make_float2(v.hi.x, v.hi.y); r[q + 3] = make_float2(v.hi.z, v.hi.w);
        }
      } else if (VEC && !strided) {                              // cnt is even, 16-byte aligned
#pragma unroll
        for (int q = 0; q < n; q += 2) {
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          if (src && q < cnt) v = __ldg(reinterpret_cast<const float4*>(src + 2 * q));
          r[q] = make_float2(v.x, v.y);
          r[q + 1] = make_float2(v.z, v.w);
        }
      } else {
#pragma unroll
        for (int q = 0; q < n; ++q) {
          r[q] = make_float2(0.f, 0.f);
          if (src && q < cnt) r[q] = __ldg(reinterpret_cast<const float2*>(src + q * step));
        }
      }
    };
    int cur_o = o_lo, cur_kb = kb_lo + group;                    // the block loaded next
    while (cur_kb >= p.nblk) { cur_kb -= p.nblk; ++cur_o; }
    auto prefetch = [&]() {
      const int cnt = cur_kb + 1 == p.nblk ? tail : nprs;
      load_pairs(ra, gA ? gA + cur_o * a_ko + cur_kb * a_stepk : nullptr, a_str, a_st, cnt, a_wide);
      load_pairs(rb, gB ? gB + cur_o * b_ko + cur_kb * b_stepk : nullptr, b_str, b_st, cnt - bp0, plain && b_wide);
      cur_kb += kTcGroups;
      while (cur_kb >= p.nblk) { cur_kb -= p.nblk; ++cur_o; }
    };
    // two adjacent pairs of one row: 16 bytes of the hi and of the lo buffer
    auto store_split = [&](unsigned char* dst, float2 u, float2 w) {
      const float4 hi = make_float4(tc_hi(u.x), tc_hi(u.y), tc_hi(w.x), tc_hi(w.y));
      *reinterpret_cast<float4*>(dst) = hi;
      *reinterpret_cast<float4*>(dst + kTcBufBytes) = make_float4(u.x - hi.x, u.y - hi.y, w.x - hi.z, w.y - hi.w);
    };
    if (group < nit) prefetch();
    // tcgen05.st is executed by whole warps: the exits of this loop are decided by votes
    auto warp_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait(bar, parity)) != 0; };
    for (int it = group; it < nit; it += kTcGroups) {
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      const int s = it % kTcStages;
      if (it >= kTcStages) {   // the MMAs that read this stage kTcStages blocks ago must have finished
        if (!warp_wait(&empty[s], (uint32_t)((it / kTcStages - 1) & 1))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      // ---- column operand.  Real rows per complex number (a, b) of the run:
      //   fwd, grad y (conjugated operand):  real column (a, b)    imaginary column (-b, a)
      //   grad x (plain product):            real column (a, -b)   imaginary column ( b, a)
      unsigned char* stage = smem + (size_t)s * kTcStageBytes + bcol * 16 + (bp0 / 2) * kTcLBO;
#pragma unroll
      for (int q = 0; q < kBPairs; q += 2) {
        if (bp0 + q >= nprs) break;
        const float2 u = rb[q], w = rb[q + 1];
        unsigned char* dst = stage + (q / 2) * kTcLBO;
        if (plain) {
          store_split(dst, u, w);
        } else if (OP == kTcGradX) {
          store_split(dst, make_float2(u.x, -u.y), make_float2(w.x, -w.y));
          store_split(dst + 64 * 16, make_float2(u.y, u.x), make_float2(w.y, w.x));
        } else {
          store_split(dst, u, w);
          store_split(dst + 64 * 16, make_float2(-u.y, u.x), make_float2(-w.y, w.x));
        }
      }
      // make the generic-proxy writes visible to the tensor core (async proxy)
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      // ---- row operand, once the block two before has been read
      if (it >= kTcAStages) {
        const int e = it - kTcAStages;
        if (!warp_wait(&empty[e % kTcStages], (uint32_t)((e / kTcStages) & 1))) break;
      }
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t ta = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + kTcACol + (uint32_t)(it % kTcAStages) * kTcAPitch;
#pragma unroll
      for (int ks = 0; ks < kTcKMax / 8; ++ks) {
        if (4 * ks >= nprs) break;
        float hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float2 v = ra[4 * ks + i];
          if (OP == kTcPlainCC)   // (__fmul_rn: the product must not be contracted into the hi / lo split)
            v = make_float2(__fmul_rn(v.x, p.scale), __fmul_rn(v.y, p.scale));
          hi[2 * i] = tc_hi(v.x); hi[2 * i + 1] = tc_hi(v.y);
          lo[2 * i] = v.x - hi[2 * i]; lo[2 * i + 1] = v.y - hi[2 * i + 1];
        }
        tc_st8(ta + 8 * ks, hi);
        tc_st8(ta + kTcALo + 8 * ks, lo);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)   // hand over: one arrival per producer warp
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem_u32(&full[s])) : "memory");
      if (it + kTcGroups < nit) prefetch();   // (after the hand-over: the loads take a few hundred clocks to issue)
    }
  }

  // ---- every MMA of this CTA has finished once the last accumulator group has been committed ----
  // (waited for by the collectors, which have followed every earlier phase of these barriers; the
  // block barrier below passes the fact on to the other warps)
  __syncwarp();
  if (nit > 0 && warp >= 1 && warp <= kTcCollectorWarps && !*abort_flag) {
    const int glast = ngroups - 1;
    wait(&accdone[glast & 1], (uint32_t)((glast / 2) & 1));
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  ok = __syncthreads_and(ok && !*abort_flag) != 0;  // block-uniform from here on
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  // ---- epilogue: TMEM -> registers -> z -----------------------------------------------------
  // warp w may only touch TMEM lanes 32 (w % 4) .. +31; the four warps sharing a lane quarter
  // split the 128 accumulator columns between them
  constexpr int kColsPerWarp = kTcBN / 4;
  static_assert(kColsPerWarp == 32, "one tcgen05.ld of 32 columns per warp");
  const int q = warp & 3, cg = (warp - 1) >> 2;
  const int r = row0 + 32 * q + lane;
  const int cbase = kColsPerWarp * cg;
  float v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = 0.f;
  if (ok && warp != 0 && nit > 0) {
    const uint32_t last_acc = FLUSH ? (uint32_t)(((ngroups - 1) & 1) * kTcBN) : 0u;
    // 32 result columns of a lane's row; spectral products: real and imaginary columns from the two halves
    auto load_columns = [&](uint32_t region, float (&o)[32]) {
      const uint32_t base = tmem_base + ((uint32_t)(32 * q) << 16) + region;
      if constexpr (OP == kTcPlainCC || OP == kTcPlainSC) {
        tc_ld32(base + (uint32_t)cbase, o);
      } else {
        float re[16], im[16];
        tc_ld16(base + (uint32_t)(cbase / 2), re);
        tc_ld16(base + (uint32_t)(kTcBN / 2 + cbase / 2), im);
#pragma unroll
        for (int i = 0; i < 16; ++i) { o[2 * i] = re[i]; o[2 * i + 1] = im[i]; }
      }
    };
    load_columns(last_acc, v);
    if (two_accs || (FLUSH && ngroups > 1)) {     // the products with a lo part, or the earlier groups' sum
      float w[32];
      load_columns((uint32_t)(FLUSH ? kTcSumCol : kTcBN), w);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] += w[i];
    }
  }
  const int rq = r / RI, ri = r - rq * RI, ro = ro0 + rq;
  // spectral products: coefficient q = ro * sro + co * sco of the degree is c[((spec0 + q) * RI + ri) * CW + rem]; its
  // mirror (-m, -n) is coefficient L * L - 1 - q, (-1)^(m - n) = (-1)^q times the conjugate (L is odd)
  constexpr bool kPlain = OP == kTcPlainCC || OP == kTcPlainSC;
  const int sro = OP == kTcGradY ? 1 : L, sco = OP == kTcGradY ? L : 1;
  const bool mirrors = !kPlain && (second || !p.twins);
  const bool row_mirror = mirrors && p.half == kTcHalfRows && rq > 0, col_half = mirrors && p.half == kTcHalfColumns;
  auto at_coefficient = [&](int q, int rem) { return p.c + ((spec0 + q) * RI + ri) * CW + rem; };
  auto mirrored = [](float4 o, float s) { return make_float4(s * o.x, -s * o.y, s * o.z, -s * o.w); };
  // two columns (one complex number: never straddles an outer column index), four with VEC
  auto store2 = [&](int gcol, float a, float b) {
    if (gcol >= Np) return;
    if constexpr (kPlain) {
      if (OP == kTcPlainSC) { a *= p.scale; b *= p.scale; }
      *reinterpret_cast<float2*>(p.c + (long)r * p.c_rs + (long)(gcol >> 1) * p.c_ps) = make_float2(a, b);
    } else {
      const int cq = gcol / CW, rem = gcol - cq * CW, q = ro * sro + (co0 + cq) * sco;
      if (!second) *reinterpret_cast<float2*>(at_coefficient(q, rem)) = make_float2(a, b);
      if (row_mirror || (col_half && cq > 0)) {
        const float s = (q & 1) ? -1.f : 1.f;
        *reinterpret_cast<float2*>(at_coefficient(L * L - 1 - q, rem)) = make_float2(s * a, -s * b);
      }
    }
  };
  auto store4 = [&](int gcol, float4 o) {
    if constexpr (VEC && !kPlain) {
      if (gcol >= Np) return;     // CW is a multiple of 4, so a group of 4 is all in or all out
      const int cq = gcol / CW, rem = gcol - cq * CW, q = ro * sro + (co0 + cq) * sco;
      if (!second) *reinterpret_cast<float4*>(at_coefficient(q, rem)) = o;
      if (row_mirror || (col_half && cq > 0)) *reinterpret_cast<float4*>(at_coefficient(L * L - 1 - q, rem)) = mirrored(o, (q & 1) ? -1.f : 1.f);
    } else {
      store2(gcol, o.x, o.y);
      store2(gcol + 2, o.z, o.w);
    }
  };
  constexpr bool kShares = OP != kTcPlainCC;
  if (kShares && nsplit > 1) {
    // ---- a shared tile.  16-byte chunk c4 of a thread's 32 columns lies at [c4][warp][lane]; rank r of the cluster
    // takes the chunks 8 r / csize .. of every thread.  (All threads of all CTAs pass the barriers, also after a
    // time-out: what is then added is undefined, and the flag below says so.)
    const int rank = (int)blockIdx.x % p.csize, lo = 8 * rank / p.csize, hi = 8 * (rank + 1) / p.csize;
    const int at = (warp - 1) * 32 + lane;
    float4* const tile = reinterpret_cast<float4*>(smem);
    if (warp != 0) {
#pragma unroll
      for (int c4 = 0; c4 < 8; ++c4) tile[c4 * 512 + at] = make_float4(v[4 * c4], v[4 * c4 + 1], v[4 * c4 + 2], v[4 * c4 + 3]);
    }
    tc_cluster_sync();
    const int cl0 = ((int)blockIdx.x - split) / p.csize;         // first cluster of the tile
    float4* const part = reinterpret_cast<float4*>(p.part);
    const bool mine = warp != 0 && r < M;
    if (mine) {
      for (int c4 = lo; c4 < hi; ++c4) {
        if (col0 + cbase + 4 * c4 >= Np) break;
        float4 t[kTcMaxCluster], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < kTcMaxCluster; ++k)
          if (k < p.csize) t[k] = cl_load4(cl_map(ClCtx(), reinterpret_cast<const float2*>(tile), k), 2 * (c4 * 512 + at));
#pragma unroll
        for (int k = 0; k < kTcMaxCluster; ++k)
          if (k < p.csize) { sum.x += t[k].x; sum.y += t[k].y; sum.z += t[k].z; sum.w += t[k].w; }
        if (p.groups == 1) store4(col0 + cbase + 4 * c4, sum);
        else __stcg(part + (size_t)(blockIdx.x / p.csize) * (kTcTileFloats / 4) + c4 * 512 + at, sum);
      }
    }
    if (p.groups > 1 && tc_last_of(&p.count[(cl0 / p.groups) * kTcMaxCluster + rank], p.groups, last_flag) && mine) {
      for (int c4 = lo; c4 < hi; ++c4) {
        if (col0 + cbase + 4 * c4 >= Np) break;
        const float4* src = part + (size_t)cl0 * (kTcTileFloats / 4) + c4 * 512 + at;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int g = 0; g < p.groups; ++g) {
          const float4 t = __ldcg(src + (size_t)g * (kTcTileFloats / 4));
          sum.x += t.x; sum.y += t.y; sum.z += t.z; sum.w += t.w;
        }
        store4(col0 + cbase + 4 * c4, sum);
      }
    }
    tc_cluster_sync();     // the others have read this CTA's part
  } else if (ok && warp != 0 && r < M) {
    if (VEC && !kPlain && CW % 8 == 0 && reinterpret_cast<unsigned long long>(p.c) % 32 == 0) {
      // a lane owns a row: 32-byte stores write whole sectors (16-byte ones would send every
      // sector to L2 in two halves); CW % 8 == 0 keeps a group of 8 inside one outer column index
#pragma unroll
      for (int c8 = 0; c8 < 4; ++c8) {
        const int gcol = col0 + cbase + 8 * c8;
        if (gcol < Np) {
          const int cq = gcol / CW, rem = gcol - cq * CW, q = ro * sro + (co0 + cq) * sco;
          float8 o;
          o.lo = make_float4(v[8 * c8], v[8 * c8 + 1], v[8 * c8 + 2], v[8 * c8 + 3]);
          o.hi = make_float4(v[8 * c8 + 4], v[8 * c8 + 5], v[8 * c8 + 6], v[8 * c8 + 7]);
          if (!second) st_global_256(at_coefficient(q, rem), o);
          if (row_mirror || (col_half && cq > 0)) {
            const float s = (q & 1) ? -1.f : 1.f;
            o.lo = mirrored(o.lo, s);
            o.hi = mirrored(o.hi, s);
            st_global_256(at_coefficient(L * L - 1 - q, rem), o);
          }
        }
      }
    } else {
#pragma unroll
      for (int c4 = 0; c4 < 8; ++c4)
        store4(col0 + cbase + 4 * c4, make_float4(v[4 * c4], v[4 * c4 + 1], v[4 * c4 + 2], v[4 * c4 + 3]));
    }
  }
  if (!ok && tid == 0) atomicExch(p.err, 1);

  // ---- release tensor memory ------------------------------------------------------------------
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(kTcTmemCols)
                 : "memory");
  }
}

// One product: picks the instantiation (see FLUSH, VEC above).
#if defined(S2C_SPLIT) && !defined(S2C_PART)
template <int OP>
int launch_so3_mm_tc(const char* name, long ctas, bool flush, bool vec, stream_t st, const MmTcParams& p);
#else
template <int OP>
int launch_so3_mm_tc(const char* name, long ctas, bool flush, bool vec, stream_t st, const MmTcParams& p) {
  if (flush)
    return vec ? launch_impl<so3_mm_tc_kernel<OP, true, true>>(name, ctas, kTcThreads, kTcSmemBytes, st, p, p.csize)
               : launch_impl<so3_mm_tc_kernel<OP, true, false>>(name, ctas, kTcThreads, kTcSmemBytes, st, p, p.csize);
  return vec ? launch_impl<so3_mm_tc_kernel<OP, false, true>>(name, ctas, kTcThreads, kTcSmemBytes, st, p, p.csize)
             : launch_impl<so3_mm_tc_kernel<OP, false, false>>(name, ctas, kTcThreads, kTcSmemBytes, st, p, p.csize);
}
#endif

// 16-byte accesses need the run of the contraction index and the column width to be multiples of 4
// floats: fwd and grad x: f_in and f_out even; grad y: batch and f_out even.  Other sizes take the
// 8-byte variant.
inline bool so3_mm_tc_vec16(int op, int nb, int fi, int fo) {
  if (op == kTcGradY) return (nb % 2 == 0) && (fo % 2 == 0);
  return (fi % 2 == 0) && (fo % 2 == 0);
}

inline long so3_mm_tc_tiles(int op, int half, int nl, int nb, int fi, int fo) {
  long t = 0;
  for (int l = 0; l < nl; ++l) t += tc_tiles_for(op, half, nb, fi, fo, l);
  return t;
}
inline size_t tc_count_bytes(long tiles) { return align_up((size_t)tiles * kTcMaxCluster * sizeof(int), 256); }
inline size_t tc_share_bytes(long tiles, int groups) {
  return groups > 1 ? tc_count_bytes(tiles) + (size_t)tiles * groups * kTcTileFloats * sizeof(float) : 0;
}

struct TcShare {
  int csize = 1, groups = 1;
};
// clusters resident on the chip, by size (cudaOccupancyMaxActiveClusters)
constexpr int kTcSlots[kTcMaxCluster + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
// The half forward product of layers whose longest contraction, of `blocks` K blocks, takes up to eight segments of 7.5 on
// average: each segment is one chain of the tensor core, and the segments are added in their order, rounded - in one CTA (as
// groups of partial sums) or, where the tiles are too few for the chip, by a cluster with one segment to a CTA.  The
// number follows from the layer alone, so that a result does not depend on the batch it was computed in.  Whole chain in
// one CTA -> cluster: 20 -> 40, nl = 6, batch 1: 13.7 -> 10.1 us, batch 32: 15.5 -> 12.1; 13 -> 9, nl = 7, batch 5: 17.1 ->
// 9.9; segments in one CTA, for more tiles than clusters: 16 -> 24, nl = 7, batch 32: 17.8 -> 18.6.  0: a layer with too many
// tiles for clusters even at batch 1, or longer contractions: one CTA, the whole chain or groups of seven; or shorter ones,
// whose chain is worth less than a cluster's meeting (24 -> 32, nl = 3, ten blocks, batch 1 and 32: 8.7 and 10.5 in two segments,
// 8.4 and 9.9 in one CTA and its twin; with 14 blocks, 24 -> 24, nl = 4, the clusters are half a microsecond ahead).
inline int tc_segments(int nl, int fi, int fo, int blocks) {
  const int s = (2 * blocks + 14) / 15;
  return blocks >= 12 && s <= kTcMaxCluster && so3_mm_tc_tiles(kTcFwd, kTcHalfColumns, nl, 1, fi, fo) <= kTcSlots[s] ? s : 0;
}

// A half product whose tiles leave half of the chip idle: each is computed twice, by one CTA that writes the tile and one
// that writes its mirror, since a CTA's 64 KB of output take about 1 us on one SM.  The results are the same.  All
// columns / half, one CTA per tile / pairs: 16 -> 24, nl = 7, batch 32: 15.9 / 18.8 / 17.4 us; 24 -> 46, nl = 8, batch 16:
// 22.3 / 25.6 / 23.0; 8 -> 16, nl = 15, batch 7: 15.5 / 17.1 / 15.7.  What is left above the whole product is the adding of
// segments in one CTA (up to 1.9 us), and up to 3 where the pairs no longer run at once (24 -> 46, nl = 8, batch 32: 22.9 /
// 25.7): the price of half of the columns at 49 - 100 tiles, while fewer take clusters (batch 7: 21.5 / 11.4) and more take
// several waves (batch 256: 139.7 / 101.2); the choice may not depend on the batch.
inline bool tc_twins(int half, long tiles, int ns) { return half && ns == 1 && 2 * tiles <= kTcSlots[1]; }

// CTAs per tile.  One CTA fits on an SM; a product with few output tiles and a long contraction (the
// transposed kernel transform of a layer with few channels: one or two tiles of several hundred K
// blocks; the gradients of small batches) leaves most of the 148 SMs idle for the length of the longest
// tile.  Estimate of the makespan in K blocks: where all clusters are resident at once the longest one, else at
// least their average load and a last, short one (the grid starts with the highest degrees).  A CTA costs kCta
// blocks on top of its own (set-up, pipeline fill, epilogue: about 6 us against 0.6 us a block), sharing within a
// cluster another kShare and between clusters another kGather.  The split is taken only where the estimate drops by a tenth, so that large
// products keep one CTA per tile.  One CTA per tile -> shared (us): 100 -> 255 channels, nl 5, batch 32, grad-x 123 -> 86;
// 20 -> 40, nl 6, batch 32, grad-x 29 -> 14, grad-y 22 -> 14; 13 -> 9, nl 7, batch 5, grad-x 14 -> 9; kernel gradients
// (rows x grid x spectrum) 800 x 192 x 286 26 -> 11, 10000 x 192 x 1330 137 -> 115, 128 x 36 x 4495 (15 clusters) 189 -> 16.
inline TcShare tc_pick_share(int op, int half, int nl, int nb, int fi, int fo, int nblk, bool several_clusters) {
  constexpr double kCta = 8, kShare = 4, kGather = 6;
  const long tiles = so3_mm_tc_tiles(op, half, nl, nb, fi, fo);
  auto estimate = [&](int c, int groups) {
    const int ns = c * groups;
    double load = 0, shortest = 0, longest = 0;
    for (int l = nl - 1; l >= 0; --l) {
      const int blocks = (2 * l + 1) * nblk;
      shortest = (blocks + ns - 1) / ns + kCta + (ns > 1 ? kShare : 0) + (groups > 1 ? kGather : 0);
      longest = std::max(longest, shortest);
      load += (double)tc_tiles_for(op, half, nb, fi, fo, l) * groups * shortest;
    }
    return tiles * groups <= kTcSlots[c] ? longest : std::max(longest, load / kTcSlots[c] + shortest);
  };
  TcShare best;
  double t = 0.9 * estimate(1, 1);
  for (int c = 2; c <= kTcMaxCluster; ++c)
    if (const double e = estimate(c, 1); e < t) { t = e; best.csize = c; }
  for (int g = 2; several_clusters && tiles * g <= kTcSlots[kTcMaxCluster]; ++g)
    if (const double e = estimate(kTcMaxCluster, g); e < t) { t = e; best.csize = kTcMaxCluster; best.groups = g; }
  return best;
}

}  // namespace s2c

#endif  // S2C_EMUL
