// Wigner-d contractions of the large-bandwidth SO(3) path (N = 2b in {64, 128}), between the spectrum and the scratch
// array V of the plane kernels (so3_plane_kernels.h).
//
// Same arithmetic as so3_fwd_wigner / so3_inv_wigner (so3_kernels.h), i.e. the beta / l contraction
// of the reference's so3fft.cu / so3ifft.cu tile loops (s2cnn/soft/so3_fft.py:296-336, :391-431).
//
// Organisation: a warp owns the frequency pair (+m, n) and (-m, n).  Analysis: for four batch elements, a block of 16
// warps sixteen consecutive values of |m|, and one block per SM walks its share of these items.  Synthesis: for eight
// batch elements (four where there are no more), a block of 4 warps.
//   * The table holds only the first half of the beta range (TableCache::half_panels): the
//     SOFT grid maps onto itself under beta -> pi - beta and
//         d^l_{m,n}(pi - beta_j) = (-1)^(l+n) d^l_{-m,n}(beta_j),
//     so the second half of panel (m, n) is the first half of panel (-m, n) up to that sign.  A warp
//     reads row l of both half panels once and uses each for both members of its pair.
//   * The 32 lanes are 8 slices of the half beta range (lane b owns the runs of four 4 b .. and, at N = 128,
//     32 + 4 b ..: 16-byte pieces of a table row) times 4 quarters of the numbers of a beta: one member of the pair
//     and half of the batch elements each.  A lane has 16 (8) betas of its four or eight numbers in registers - V in the analysis,
//     the sums in the synthesis - and pairs of neighbouring betas are the two halves of the packed multiply-adds, so
//     that no table value is duplicated into a register pair.
//   * Panel rows reach a warp through a private ring in shared memory filled by 16-byte asynchronous copies
//     (cp.async), four rows a step.
//   * analysis: an output is the sum over the 8 slices.  In step r of four rows lane b works on row r XOR (b % 4), so
//     that what two lanes exchange sits in the same register of both: 4 shuffles and additions for 4 rows and each of a
//     lane's numbers, no selects; lanes b and b + 4 end up with row b and write it and its mirror.
//   * analysis: V comes as bulk copies, see below; an item's part is fetched while the one before is worked on (its
//     numbers are in registers then).
//   * synthesis: the accumulators stay in registers while the rows stream; they leave as runs of 32 bytes.
//
// Bound by latency and the shared-memory pipe (analysis: a lane loads 16 floats of table for 64 multiply-adds, 16 + 4 (ring)
// + 4 (shuffles) clocks of the pipe per row; issue 49 %, packed multiply-adds 45 % of the time).  64 signals at b = 64:
// analysis 275 us, synthesis 309; with one slice of V per lane of 32, staged through registers (124 instructions of
// sums for 64 multiply-adds, V fetched in 64-byte pieces), in chunks of 8 signals: 407 and 390.  Eight batch elements to a
// warp in the analysis, V in pieces of 32 bytes: 8 warps per SM, 35 instead of 39 us per 8 signals, which the plane
// kernels lost to the shorter pieces.  The synthesis as one walking block of 16 warps and bulk stores: 50 us instead of 46.
#pragma once

#include "backend.h"
#include "fft_reg.h"
#include "so3_kernels.h"

namespace s2c {

// Batch elements per chunk, 256 MB of V.  That is more than L2 holds: long launches weigh more than keeping V in L2, also
// with programmatic launches (64 signals at b = 64, analysis / synthesis: 719 / 789 us in chunks of 4, 597 / 659 of 8 (67 MB),
// 558 / 612 of 16, 561 / 598 of 32; 512 signals at b = 32: 901 / 937 us of 8, 552 / 607 of 32, 508 / 575 of 64, 490 / 574 of
// 128, 490 / 555 of 256).
S2C_HD constexpr int rows_zc(int N) { return N == 128 ? 32 : 256; }
constexpr int kRowsZQ = 4;      // batch elements per item
constexpr int kRowsMG = 16;     // values of |m| per item = warps per block
constexpr int kRowsThreads = 32 * kRowsMG;
constexpr int kRowsStep = 4;    // table rows per ring step
#ifndef S2C_EMUL
constexpr int kRowsSlotsF = 3;  // ring steps per warp: analysis
#else
constexpr int kRowsSlotsF = 2;  // (the exchange buffer needs the room)
#endif
// the synthesis: four values of |m| (warps) and up to ZQ = 8 or 4 batch elements per block
constexpr int kRowsMGI = 4, kRowsThreadsI = 32 * kRowsMGI, kRowsSlotsI = 4;

// V between the plane kernels and these: [n < K][sign of m][|m| / 16][z < zc][beta][|m| % 16], so that the plane kernels
// see lines of 128 bytes and an item's part is one run per sign (a bulk copy).  Within a line the order is XOR-ed with a
// number of four bits: the lanes of a half warp, which hold betas four apart of two halves of the batch elements, then
// touch all banks at once.
S2C_HD constexpr int rows_groups(int N) { return N / (2 * kRowsMG); }      // per sign
S2C_HD constexpr long rows_group_stride(int N, int zc) { return (long)zc * N * kRowsMG; }
S2C_HD constexpr int rows_swizzle(int z, int beta) { return ((beta >> 2) & 7) | (((z >> 1) & 1) << 3); }
// Where the bins of one (n, z, beta) lie that a lane handles in a transform over f: f = j + step q for the frequencies
// m = f in the first half, and m = -(step M - j) in the second; step 8 or 16, j < step.
template <int STEP>
struct RowsBins {
  long gs;
  int pos0, pos1;        // step 8: even / odd q
  long neg0, neg1;       // even / odd M
  S2C_D RowsBins(int N, int zc, int z, int beta, int j) : gs(rows_group_stride(N, zc)) {
    const int at = z * N * kRowsMG, line = beta * kRowsMG, h = rows_swizzle(z, beta);
    pos0 = at + ((line + j) ^ h);
    const long ng = rows_groups(N) * gs + at;
    if (STEP == 16) {
      pos1 = pos0;
      neg0 = neg1 = j == 0 ? ng + (line ^ h) : ng - gs + ((line + 16 - j) ^ h);
    } else {
      pos1 = at + ((line + 8 + j) ^ h);
      neg0 = j == 0 ? ng + (line ^ h) : ng - gs + ((line + 16 - j) ^ h);
      neg1 = ng + (j == 0 ? ((line + 8) ^ h) : ((line + 8 - j) ^ h));
    }
  }
  S2C_D long pos(int q) const { return STEP == 16 ? pos0 + q * gs : (q & 1 ? pos1 : pos0) + (q >> 1) * gs; }
  S2C_D long neg(int M) const { return STEP == 16 ? neg0 + M * gs : (M & 1 ? neg1 : neg0) + (M >> 1) * gs; }
};

struct HalfPanelsDev {
  int nbeta;                // N = 2 b of the beta grid
  int nl, K, npairs;
  const float* data;        // per pair: rows l = lmin .. nl-1, N/2 floats each (beta_j, j < N/2)
  const long long* off;     // npairs + 1 offsets in floats
};

// The pairs (n, sixteen values of |m|) of the analysis' items, those with the longest rows first: 16 n + m / 16.  Item i is
// pair i / nzq and the batch elements from 4 (i % nzq); block b of G walks the items b, 2 G - 1 - b, 2 G + b, 4 G - 1 - b, ...
constexpr int kRowsMaxPairs = 64 * 4;
struct RowsOrder {
  unsigned short pair[kRowsMaxPairs];
};

struct FwdRowsParams {
  const float2* v;      // (see rows_swizzle)
  float2* out;          // spectrum rows of out_zstride complex, already offset to the chunk's z0
  long out_zstride;
  HalfPanelsDev pan;
  int zc, K, nl, mode;  // zc <= rows_zc(N) batch elements; mode: kSo3Real or kSo3AccumI
  RowsOrder order;
};

struct InvRowsParams {
  const float2* x;      // spectrum rows of x_zstride complex, offset to the chunk's z0
  long x_zstride;
  float2* s;            // (see rows_swizzle)
  HalfPanelsDev pan;
  int zc, K, mode;      // mode: kSo3Real or kSo3RotI
};

// Shared memory.  Analysis: the item's part of V, [sign][4 z][N beta][16], and behind it the rings
// [warp][slot][row][A, B][N / 2].  Synthesis: the block's part of V, [sign][ZQ z][N beta][4] (before it the symmetrised
// spectrum rows [8 columns][degree][ZQ z]), and the rings.  (+ in the host-emulation build a per-warp exchange buffer that
// stands in for the shuffles.)
S2C_HD constexpr int rows_tile_floats(int N) { return 2 * kRowsZQ * N * kRowsMG * 2; }
S2C_HD constexpr int rows_ring_floats(int N, int slots) { return slots * kRowsStep * N; }      // per warp
S2C_HD constexpr size_t rows_fwd_smem(int N) {
  size_t b = (rows_tile_floats(N) + kRowsMG * rows_ring_floats(N, kRowsSlotsF)) * sizeof(float) + 32;
#ifdef S2C_EMUL
  b += (size_t)kRowsMG * 32 * 17 * sizeof(float);
#endif
  return b;
}
S2C_HD constexpr int rows_inv_tile_floats(int N, int ZQ) { return 2 * ZQ * N * kRowsMGI * 2; }
S2C_HD constexpr size_t rows_inv_smem(int N, int ZQ) {
  return (rows_inv_tile_floats(N, ZQ) + kRowsMGI * rows_ring_floats(N, kRowsSlotsI)) * sizeof(float);
}

// 16 bytes global -> shared, asynchronously; groups complete in issue order
#ifndef S2C_EMUL
S2C_D void rows_copy16_async(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
S2C_D void rows_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Of this thread's SLOTS copy groups all but the oldest may be pending.
template <int SLOTS>
S2C_D void rows_wait_oldest() { asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS - 1) : "memory"); }
S2C_D float2 rows_mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "mul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
#else
inline void rows_copy16_async(float* dst, const float* src) {
  for (int i = 0; i < 4; ++i) dst[i] = src[i];
}
inline void rows_commit() {}
template <int SLOTS>
inline void rows_wait_oldest() {}
inline float2 rows_mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
#endif

// ---- four rows, summed over the 8 beta slices of a warp ------------------------------------------
// part(r) is this lane's part (two complex numbers) of row r XOR (b % 4), b = lane % 8; returns the sum of row b % 4 over
// the 8 lanes of its quarter.  After the exchange over bit 2 lane b holds rows r XOR (b % 4), r < 2, and so on.
#ifndef S2C_EMUL
S2C_D float4 rows_add_from(float4 v, float4 w, int bit) {
  v.x += __shfl_xor_sync(0xffffffffu, w.x, bit);
  v.y += __shfl_xor_sync(0xffffffffu, w.y, bit);
  v.z += __shfl_xor_sync(0xffffffffu, w.z, bit);
  v.w += __shfl_xor_sync(0xffffffffu, w.w, bit);
  return v;
}
template <class Part>
S2C_D float4 rows_sum4(const Ctx&, Part part, int, float*) {
  float4 v0 = part(std::integral_constant<int, 0>{}), v1 = part(std::integral_constant<int, 1>{});
  v0 = rows_add_from(v0, part(std::integral_constant<int, 2>{}), 2);
  v1 = rows_add_from(v1, part(std::integral_constant<int, 3>{}), 2);
  v0 = rows_add_from(v0, v1, 1);
  return rows_add_from(v0, v0, 4);
}
#else
// every warp of the block calls this equally often (a warp barrier is a block barrier here)
template <class Part>
inline float4 rows_sum4(const Ctx& ctx, Part part, int lane, float* xch) {
  const int b = lane & 3;
  static_for<0, 4>([&](auto r) {
    constexpr int k = decltype(r)::value;
    const float4 v = part(std::integral_constant<int, k>{});
    float* dst = xch + lane * 17 + (k ^ b) * 4;
    dst[0] = v.x; dst[1] = v.y; dst[2] = v.z; dst[3] = v.w;
  });
  ctx.sync_warp();
  float o[4];
  for (int c = 0; c < 4; ++c) {     // the order of the shuffles: bits 2, 1, 4
    auto at = [&](int x) { return xch[(lane ^ x) * 17 + b * 4 + c]; };
    auto two = [&](int x) { return at(x) + at(x ^ 2); };
    auto four = [&](int x) { return two(x) + two(x ^ 1); };
    o[c] = four(0) + four(4);
  }
  ctx.sync_warp();
  return make_float4(o[0], o[1], o[2], o[3]);
}
#endif

struct RowsGeom {
  int n, m0, zbase, nz;      // nz: batch elements there are, up to 4
};
S2C_D RowsGeom rows_geom(const RowsOrder& order, int item, int zc) {
  const int nzq = (zc + kRowsZQ - 1) / kRowsZQ, pair = order.pair[item / nzq];
  RowsGeom g;
  g.n = pair / kRowsMG;
  g.m0 = pair % kRowsMG * kRowsMG;
  g.zbase = item % nzq * kRowsZQ;
  g.nz = zc - g.zbase < kRowsZQ ? zc - g.zbase : kRowsZQ;
  return g;
}
S2C_HD int rows_items(int K, int zc) { return K * ((K + kRowsMG - 1) / kRowsMG) * ((zc + kRowsZQ - 1) / kRowsZQ); }
// an item's part of V for sign s, [z][beta][16]
S2C_D long rows_part(int N, int zc, const RowsGeom& g, int s) {
  return (((long)g.n * 2 + s) * rows_groups(N) + g.m0 / kRowsMG) * rows_group_stride(N, zc) + (long)g.zbase * N * kRowsMG;
}

// half-panel rows of the pair (+m, n) and (-m, n); for n = 0 only m >= 0 is stored and
// d_{-m,0} = (-1)^m d_{m,0}; for m = 0 the two coincide
struct RowsPanels {
  const float* a;      // half panel of (+m, n)
  const float* b;      // half panel of (-m, n) (or of (+m, n) with `bsign`)
  float bsign;
};
S2C_D RowsPanels rows_panels(const HalfPanelsDev& pan, int m, int n) {
  RowsPanels r;
  r.a = pan.data + pan.off[so3_pair_index(m, n, pan.K)];
  if (n == 0 || m == 0) {
    r.b = r.a;
    r.bsign = (n == 0 && (m & 1)) ? -1.f : 1.f;
  } else {
    r.b = pan.data + pan.off[so3_pair_index(-m, n, pan.K)];
    r.bsign = 1.f;
  }
  return r;
}

// A warp's ring: a step is kRowsStep rows of both half panels, [row][A, B][NH] floats, copied 16 bytes per lane.  A lane
// copies the same piece of every row (N = 64: of every other row).
template <int N, int SLOTS>
struct RowsRing {
  static constexpr int NH = N / 2, kPieces = N / 4, kRowsAtOnce = 32 / kPieces;
  float* base;
  const float* src;
  int row0, L, dst, lane_row;
  S2C_D RowsRing(float* ring, const RowsPanels& pn, int lane, int rows) : base(ring), L(rows) {
    const int piece = lane % kPieces, ab = piece / (kPieces / 2), q = piece - ab * (kPieces / 2);
    lane_row = lane / kPieces;
    row0 = lane_row;
    src = (ab ? pn.b : pn.a) + (long)lane_row * NH + 4 * q;
    dst = lane_row * 2 * NH + 4 * piece;
  }
  S2C_D const float* slot(int t) const { return base + (t % SLOTS) * (kRowsStep * 2 * NH); }
  S2C_D void issue(int t) {     // the next step, into slot t
    float* d = base + (t % SLOTS) * (kRowsStep * 2 * NH) + dst;
#pragma unroll
    for (int r = 0; r < kRowsStep; r += kRowsAtOnce)
      if (row0 + r < L) rows_copy16_async(d + r * 2 * NH, src + (long)r * NH);
    row0 += kRowsStep;
    src += kRowsStep * NH;
    rows_commit();   // one group per step, empty or not, so that the wait counts steps
  }
};

// Lane = 8 * quarter + b.  Quarter: the pair's member s (0: +m, 1: -m) and two of the four batch elements, from zp.
// The lane's betas are j = 4 b + 32 p + i (p < N / 64, i < 4) and N - 1 - j.
struct RowsLane {
  int b, s, zp;
  S2C_D explicit RowsLane(int lane) : b(lane & 7), s(lane >> 4), zp(2 * ((lane >> 3) & 1)) {}
};

// ---------------------------------------------------------------------------------------------
// analysis:  X[l, +-m, n][z] = sum_beta W[l][beta] V[z][beta]   (+ Hermitian mirror rows)
// ---------------------------------------------------------------------------------------------
template <int N>
struct so3_fwd_wigner_r_impl {
  static S2C_D void run(const Ctx& ctx, const FwdRowsParams& p, unsigned char* smem) {
    constexpr int NH = N / 2, NP = NH / 32;                       // pieces of a half row per lane
    constexpr int kRing = rows_ring_floats(N, kRowsSlotsF);
    float2* tile = reinterpret_cast<float2*>(smem);               // [sign][z][N * 16]
    const int warp = ctx.tid >> 5, lane = ctx.tid & 31;
    float* rings = reinterpret_cast<float*>(smem) + rows_tile_floats(N);
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(rings + kRowsMG * kRing);     // [sign]
    int* readers = reinterpret_cast<int*>(bar + 2);
    // bit 16 of `readers` is set by the lanes whose wait has given up: no copy is issued or trusted any more (the count is
    // never 15 again), V is read from global memory
    constexpr int kLate = 1 << 16;
    auto late = [&] { return *reinterpret_cast<const volatile int*>(readers) >= kLate; };
    float* xch = reinterpret_cast<float*>(bar + 4) + warp * 32 * 17;
    const int K = p.K, zc = p.zc, items = rows_items(K, zc);
    const RowsLane ln(lane);
    auto next = [&](int turn) { return turn * ctx.nblk + (turn & 1 ? ctx.nblk - 1 - ctx.bid : ctx.bid); };

    // the item's part of V, one copy per sign; issued by one thread once every warp has the part before in registers
    auto fetch = [&](int item) {
      if (item >= items) return;
      const RowsGeom g = rows_geom(p.order, item, zc);
      for (int s = 0; s < 2; ++s)
        bulk_load_issue(tile + s * kRowsZQ * N * kRowsMG, p.v + rows_part(N, zc, g, s),
                        (unsigned)(g.nz * N * kRowsMG * sizeof(float2)), bar + s);
    };
    if (ctx.tid == 0) {
      bulk_barrier_init(bar);
      bulk_barrier_init(bar + 1);
      *readers = 0;
      fetch(next(0));
    }
    ctx.sync();

    for (int turn = 0; next(turn) < items; ++turn) {
      const RowsGeom g = rows_geom(p.order, next(turn), zc);
      const unsigned phase = turn & 1;
      const int n = g.n, m = g.m0 + warp;
      const int lmin = m > n ? m : n;
      const int L = (m < K) ? p.nl - lmin : 0;
#ifdef S2C_EMUL
      const int lmin_blk = g.m0 > n ? g.m0 : n;
      const int Lloop = p.nl - lmin_blk > 0 ? p.nl - lmin_blk : 0;   // uniform over the block
#else
      const int Lloop = L;
#endif
      RowsPanels pn;
      pn.a = pn.b = p.pan.data;
      pn.bsign = 1.f;
      if (L > 0) pn = rows_panels(p.pan, m, n);
      RowsRing<N, kRowsSlotsF> ring(rings + warp * kRing, pn, lane, L);
      for (int t = 0; t < kRowsSlotsF; ++t) ring.issue(t);

      // ---- this lane's numbers: v1 goes with the row of the first half panel, v2 with that of the second ----------------
      //   X_{+m} = sum_j A_j V_{+m}[j] + s B_j V_{+m}[N-1-j];   X_{-m} = s (sum_j A_j V_{-m}[N-1-j] + s B_j V_{-m}[j]),
      // s = (-1)^(l+n).  Index [2 z + re/im][pair of neighbouring betas].
      float2 v1[4][2 * NP], v2[4][2 * NP];
      {
        const bool landed = !late() && bulk_wait(ctx, bar, phase) && bulk_wait(ctx, bar + 1, phase);
#ifndef S2C_EMUL
        if (!landed) atomicOr(readers, kLate);
#else
        if (!landed) *readers |= kLate;
#endif
        const float2* col = landed ? tile + ln.s * kRowsZQ * N * kRowsMG : p.v + rows_part(N, zc, g, ln.s);
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const int zz = ln.zp + z;
          const bool there = landed || zz < g.nz;
          auto number = [&](int beta) {
            return there ? col[zz * N * kRowsMG + ((beta * kRowsMG + warp) ^ rows_swizzle(zz, beta))] : make_float2(0.f, 0.f);
          };
#pragma unroll
          for (int k = 0; k < 2 * NP; ++k) {
            const int j = 4 * ln.b + 32 * (k / 2) + 2 * (k % 2);
            const float2 j0 = number(j), j1 = number(j + 1), q0 = number(N - 1 - j), q1 = number(N - 2 - j);
            const float2 jr = make_float2(j0.x, j1.x), ji = make_float2(j0.y, j1.y);
            const float2 qr = make_float2(q0.x, q1.x), qi = make_float2(q0.y, q1.y);
            v1[2 * z][k] = ln.s ? qr : jr;      v2[2 * z][k] = ln.s ? jr : qr;
            v1[2 * z + 1][k] = ln.s ? qi : ji;  v2[2 * z + 1][k] = ln.s ? ji : qi;
          }
        }
      }
      // the last warp to get here starts the next copy; no warp waits for another
#ifndef S2C_EMUL
      __syncwarp();
      if (lane == 0) {
        __threadfence_block();
        if (atomicAdd(readers, 1) == kRowsMG - 1) {
          *readers = 0;
          __threadfence_block();
          fetch(next(turn + 1));
        }
      }
      __syncwarp();
#else
      ctx.sync();
      if (ctx.tid == 0 && !late()) fetch(next(turn + 1));
#endif

      // output: row li + b % 4 (lanes b < 4) or its mirror (b >= 4), frequency +-m, batch elements from zp
      const int o_mm = ln.s ? -m : m, o_z = g.zbase + ln.zp, o_b = ln.b & 3;
      const float sl = ((lmin + n + o_b) & 1) ? -1.f : 1.f;      // (-1)^(l+n) of row b % 4, and of row r XOR (b % 4), r even
      const bool o_mirror = ln.b >= 4;
      // v = (x, y) of a number becomes (cx x, cy y), or of i times it (cx y, cy x); the mirror is (-1)^(m-n) times the conjugate
      const float o_sign = (ln.s ? sl : 1.f) * (o_mirror && ((o_mm - n) & 1) ? -1.f : 1.f);
      const float o_sx = p.mode == kSo3Real || o_mirror ? o_sign : -o_sign;
      const float o_sy = p.mode == kSo3Real && o_mirror ? -o_sign : o_sign;
      const int o_om = o_mirror ? -o_mm : o_mm, o_on = o_mirror ? -n : n;
      // for n = 0 the mirror (-m, 0) is computed directly; m = 0 is its own partner
      const int o_nz = (m == 0 && ln.s) || (o_mirror && n == 0) ? 0 : zc - o_z;
      const bool o_vec = o_nz >= 2 && p.out_zstride % 2 == 0 && reinterpret_cast<unsigned long long>(p.out + o_z) % 16 == 0;
      const float2 bs_even = make_float2(sl * pn.bsign, sl * pn.bsign), bs_odd = make_float2(-sl * pn.bsign, -sl * pn.bsign);

      for (int li = 0, t = 0; li < Lloop; li += kRowsStep, ++t) {
        rows_wait_oldest<kRowsSlotsF>();
        ctx.sync_warp();              // the other lanes' pieces of this step have landed, too
        const float* slot = ring.slot(t) + 4 * ln.b;
        const float4 sum = rows_sum4(ctx, [&](auto r_) {
          constexpr int r = decltype(r_)::value;
          const float* row = slot + (r ^ o_b) * (2 * NH);
          float2 acc[4];
#pragma unroll
          for (int pp = 0; pp < NP; ++pp) {
            const float4 a4 = *reinterpret_cast<const float4*>(row + 32 * pp);
            const float2 a0 = make_float2(a4.x, a4.y), a1 = make_float2(a4.z, a4.w);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              acc[c] = pp == 0 ? rows_mul2(a0, v1[c][0]) : fma2(a0, v1[c][2 * pp], acc[c]);
              acc[c] = fma2(a1, v1[c][2 * pp + 1], acc[c]);
            }
          }
#pragma unroll
          for (int pp = 0; pp < NP; ++pp) {
            const float4 b4 = *reinterpret_cast<const float4*>(row + NH + 32 * pp);
            const float2 sgn = r & 1 ? bs_odd : bs_even;
            const float2 b0 = rows_mul2(make_float2(b4.x, b4.y), sgn), b1 = rows_mul2(make_float2(b4.z, b4.w), sgn);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              acc[c] = fma2(b0, v2[c][2 * pp], acc[c]);
              acc[c] = fma2(b1, v2[c][2 * pp + 1], acc[c]);
            }
          }
          return make_float4(acc[0].x + acc[0].y, acc[1].x + acc[1].y, acc[2].x + acc[2].y, acc[3].x + acc[3].y);
        }, lane, xch);
        ctx.sync_warp();              // every lane has read the slot
        ring.issue(t);
        if (li + o_b < L && o_nz > 0) {
          float2* o = p.out + so3_row(lmin + li + o_b, o_om, o_on) * p.out_zstride + o_z;
          if (p.mode == kSo3Real) {
            const float4 w = make_float4(o_sx * sum.x, o_sy * sum.y, o_sx * sum.z, o_sy * sum.w);
            if (o_vec) {
              *reinterpret_cast<float4*>(o) = w;
            } else {
              o[0] = make_float2(w.x, w.y);
              if (o_nz > 1) o[1] = make_float2(w.z, w.w);
            }
          } else {   // += i * (re + i im):  re -= im, im += re;   mirror += i * (-1)^(m-n) * conj
            o[0] = make_float2(o[0].x + o_sx * sum.y, o[0].y + o_sy * sum.x);
            if (o_nz > 1) o[1] = make_float2(o[1].x + o_sx * sum.w, o[1].y + o_sy * sum.z);
          }
        }
      }
      ctx.sync_warp();                // the ring is free for the next item
    }
    if (late()) {     // what is still under way gets its time, before the block's shared memory goes to another
      for (int k = 0; k < 4; ++k) {
#ifndef S2C_EMUL
        bulk_wait(ctx, bar + k / 2, k & 1);
#else
        bulk_over(bar + k / 2, k & 1);
#endif
      }
    }
  }
};

// ---------------------------------------------------------------------------------------------
// synthesis:  S[z][beta] = sum_l W[l][beta] Xs[l][z],  Xs = symmetrised spectrum
// ---------------------------------------------------------------------------------------------
template <int N, int ZQ>
struct so3_inv_wigner_r_impl {
  static S2C_D void run(const Ctx& ctx, const InvRowsParams& p, unsigned char* smem) {
    constexpr int MG = kRowsMGI, ZL = ZQ / 2, NC = 2 * ZL;       // batch elements and numbers per lane
    constexpr int NH = N / 2, NP = NH / 32;
    float2* tile = reinterpret_cast<float2*>(smem);              // [sign][z][N * 4], written after the loop
    float2* xs = tile;                                             // before: [2 MG][Lmax][ZQ] symmetrised rows
    const int warp = ctx.tid >> 5, lane = ctx.tid & 31;
    float* ring_base = reinterpret_cast<float*>(smem) + rows_inv_tile_floats(N, ZQ) + warp * rows_ring_floats(N, kRowsSlotsI);
    const int K = p.K, zc = p.zc, nl = p.pan.nl;
    const int ngroups = (K + MG - 1) / MG, nzq = (zc + ZQ - 1) / ZQ, zbase = ctx.bid % nzq * ZQ, nm = ctx.bid / nzq;
    const int n = nm / ngroups, m0 = (nm - n * ngroups) * MG;
    const int lmin_blk = m0 > n ? m0 : n;
    const int Lmax = nl - lmin_blk;                      // rows of the block's longest pair (<= N/2)

    const int m = m0 + warp;
    const int lmin = m > n ? m : n;
    const int L = (m < K) ? nl - lmin : 0;
#ifdef S2C_EMUL
    const int Lloop = Lmax;        // uniform over the block: a warp barrier is a block barrier here
#else
    const int Lloop = L;
#endif
    RowsPanels pn;
    pn.a = pn.b = p.pan.data;
    pn.bsign = 1.f;
    if (L > 0) pn = rows_panels(p.pan, m, n);
    RowsRing<N, kRowsSlotsI> ring(ring_base, pn, lane, L);
    for (int t = 0; t < kRowsSlotsI; ++t) ring.issue(t);

    // ---- symmetrised spectrum rows of the block's columns: xs[c][li][z], li from lmin_blk ------
    // thread = (z, li); the loads of all columns are issued before any is used
    {
      const int z = ctx.tid % ZQ;
      for (int li = ctx.tid / ZQ; li < Lmax; li += kRowsThreadsI / ZQ) {
        const int l = lmin_blk + li;
        float2 a[2 * MG], b[2 * MG];
#pragma unroll
        for (int c = 0; c < 2 * MG; ++c) {
          const int mabs = m0 + (c % MG);
          const int mm = c < MG ? mabs : -mabs;
          const bool ok = zbase + z < zc && mabs < K && l >= mabs && !(c >= MG && mabs == 0);
          a[c] = b[c] = make_float2(0.f, 0.f);
          if (ok) {
            a[c] = p.x[so3_row(l, mm, n) * p.x_zstride + zbase + z];
            b[c] = p.x[so3_row(l, -mm, -n) * p.x_zstride + zbase + z];
          }
        }
#pragma unroll
        for (int c = 0; c < 2 * MG; ++c) {
          const int mabs = m0 + (c % MG);
          float2 u = a[c], w = b[c];
          if (p.mode == kSo3RotI) {  // multiply the spectrum by -i
            u = make_float2(u.y, -u.x);
            w = make_float2(w.y, -w.x);
          }
          const float fudge = ((mabs - n) & 1) ? -1.f : 1.f;
          const float sl = c >= MG && ((l + n) & 1) ? -0.5f : 0.5f;      // (see the loop over the degrees)
          xs[(c * Lmax + li) * ZQ + z] = make_float2(sl * (u.x + fudge * w.x), sl * (u.y - fudge * w.y));
        }
      }
    }
    ctx.sync();

    // Sums of this lane's numbers: u1 with the rows of the first half panel, u2 with those of the second.
    //   S_{+m}[j] += A_j X, S_{+m}[N-1-j] += s B_j X;   S_{-m}[N-1-j] += A_j (s X), S_{-m}[j] += s B_j (s X),   s = (-1)^(l+n),
    // and the spectrum rows of -m are kept times s.  Index [2 z + re/im][pair of neighbouring betas].
    const int b = lane & 7, s = lane >> 4, zp = ZL * ((lane >> 3) & 1);
    float2 u1[NC][2 * NP], u2[NC][2 * NP];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int k = 0; k < 2 * NP; ++k) u1[c][k] = u2[c][k] = make_float2(0.f, 0.f);
    {
      const int lrel = L > 0 ? lmin - lmin_blk : 0;
      const float2* x = xs + ((s * MG + warp) * Lmax + lrel) * ZQ + zp;
      const float s0 = (((lmin + n) & 1) ? -1.f : 1.f) * pn.bsign;
      for (int li = 0, t = 0; li < Lloop; li += kRowsStep, ++t) {
        rows_wait_oldest<kRowsSlotsI>();
        ctx.sync_warp();            // the other lanes' pieces of these rows have landed, too
        const float* slot = ring.slot(t) + 4 * b;
#pragma unroll
        for (int r = 0; r < kRowsStep; ++r) {
          if (li + r >= L) break;
          float2 y[NC];
#pragma unroll
          for (int z = 0; z < ZL; z += 2) {
            const float4 x4 = *reinterpret_cast<const float4*>(x + (li + r) * ZQ + z);
            y[2 * z] = make_float2(x4.x, x4.x);
            y[2 * z + 1] = make_float2(x4.y, x4.y);
            y[2 * z + 2] = make_float2(x4.z, x4.z);
            y[2 * z + 3] = make_float2(x4.w, x4.w);
          }
          const float2 s2 = r & 1 ? make_float2(-s0, -s0) : make_float2(s0, s0);
          const float* row = slot + r * (2 * NH);
#pragma unroll
          for (int pp = 0; pp < NP; ++pp) {
            const float4 a4 = *reinterpret_cast<const float4*>(row + 32 * pp);
            const float2 a0 = make_float2(a4.x, a4.y), a1 = make_float2(a4.z, a4.w);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              u1[c][2 * pp] = fma2(a0, y[c], u1[c][2 * pp]);
              u1[c][2 * pp + 1] = fma2(a1, y[c], u1[c][2 * pp + 1]);
            }
          }
#pragma unroll
          for (int pp = 0; pp < NP; ++pp) {
            const float4 b4 = *reinterpret_cast<const float4*>(row + NH + 32 * pp);
            const float2 b0 = rows_mul2(make_float2(b4.x, b4.y), s2), b1 = rows_mul2(make_float2(b4.z, b4.w), s2);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              u2[c][2 * pp] = fma2(b0, y[c], u2[c][2 * pp]);
              u2[c][2 * pp + 1] = fma2(b1, y[c], u2[c][2 * pp + 1]);
            }
          }
        }
        ctx.sync_warp();            // every lane has read the slot
        ring.issue(t);
      }
    }
    ctx.sync();   // every warp is done with the spectrum rows; the memory becomes the block's part of V

    // [sign][z][beta][4], within a line of 16 numbers in the order that spreads a half warp over all banks; a run of four
    // is in memory's order (rows_swizzle, whose two low bits are these)
    auto swizzle = [](int z, int beta) { return ((beta >> 2) & 7) | ((z / ZL & 1) << 3); };
#pragma unroll
    for (int z = 0; z < ZL; ++z) {
      float2* col = tile + (s * ZQ + zp + z) * N * MG;
      auto number = [&](int beta) -> float2& { return col[(beta * MG + warp) ^ swizzle(zp + z, beta)]; };
#pragma unroll
      for (int k = 0; k < 2 * NP; ++k) {
        const int j = 4 * b + 32 * (k / 2) + 2 * (k % 2);
        const float2 jr = s ? u2[2 * z][k] : u1[2 * z][k], ji = s ? u2[2 * z + 1][k] : u1[2 * z + 1][k];
        const float2 qr = s ? u1[2 * z][k] : u2[2 * z][k], qi = s ? u1[2 * z + 1][k] : u2[2 * z + 1][k];
        number(j) = make_float2(jr.x, ji.x);
        number(j + 1) = make_float2(jr.y, ji.y);
        number(N - 1 - j) = make_float2(qr.x, qi.x);
        number(N - 2 - j) = make_float2(qr.y, qi.y);
      }
    }
    ctx.sync();
    // runs of four numbers, 32 bytes, to their places in the lines of V (numbers of frequencies >= K are never read)
    const long gs = rows_group_stride(N, zc);
    float2* dst = p.s + ((long)n * 2 * rows_groups(N) + m0 / kRowsMG) * gs;
    const int run = m0 / MG % (kRowsMG / MG);
    const bool wide = reinterpret_cast<unsigned long long>(p.s) % 32 == 0;
    // (two numbers at a time, lanes 4 - 7 of eight the second pair first: 32-byte steps would meet in half the banks)
    const int up = ctx.tid >> 2 & 1;
#pragma unroll 4
    for (int i = ctx.tid; i < 2 * ZQ * N; i += kRowsThreadsI) {
      const int beta = i % N, zs = i / N, z = zs % ZQ, sg = zs / ZQ;
      if (zbase + z >= zc) continue;
      const float4* src = reinterpret_cast<const float4*>(tile + zs * N * MG + ((beta * MG) ^ (swizzle(z, beta) & 12)));
      float* out = reinterpret_cast<float*>(dst + sg * rows_groups(N) * gs + (long)(zbase + z) * N * kRowsMG +
                                            ((beta * kRowsMG + run * MG) ^ (rows_swizzle(z, beta) & 12)));
      const float4 first = src[up], second = src[1 - up];
      float8 v;
      v.lo = up ? second : first;
      v.hi = up ? first : second;
      if (wide) {
        st_global_256(out, v);
      } else {
        reinterpret_cast<float4*>(out)[0] = v.lo;
        reinterpret_cast<float4*>(out)[1] = v.hi;
      }
    }
  }
};

#ifndef S2C_EMUL
template <int N>
__global__ void __launch_bounds__(kRowsThreads, 1) so3_fwd_wigner_r(const FwdRowsParams p) {
  extern __shared__ float4 s2c_dyn_smem[];
  Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};
  stream_order_wait();
  so3_fwd_wigner_r_impl<N>::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));
  stream_order_next();
}
template <int N, int ZQ>
__global__ void __launch_bounds__(kRowsThreadsI, 2) so3_inv_wigner_r(const InvRowsParams p) {
  extern __shared__ float4 s2c_dyn_smem[];
  Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};
  stream_order_wait();
  so3_inv_wigner_r_impl<N, ZQ>::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));
  stream_order_next();
}
#define S2C_LAUNCH_FWD_ROWS(N, grid, stream, params)                                                             \
  s2c::launch_impl<so3_fwd_wigner_r<N>>("so3_fwd_wigner_r", (long)(grid), s2c::kRowsThreads, s2c::rows_fwd_smem(N), \
                                        stream, params)
#define S2C_LAUNCH_INV_ROWS(N, ZQ, grid, stream, params)                                                          \
  s2c::launch_impl<so3_inv_wigner_r<N, ZQ>>("so3_inv_wigner_r", (long)(grid), s2c::kRowsThreadsI,                 \
                                            s2c::rows_inv_smem(N, ZQ), stream, params)
#else
#define S2C_LAUNCH_FWD_ROWS(N, grid, stream, params) \
  s2c::emu_launch<so3_fwd_wigner_r_impl<N>>("so3_fwd_wigner_r", (long)(grid), s2c::kRowsThreads, s2c::rows_fwd_smem(N), params)
#define S2C_LAUNCH_INV_ROWS(N, ZQ, grid, stream, params)                                                        \
  s2c::emu_launch<so3_inv_wigner_r_impl<N, ZQ>>("so3_inv_wigner_r", (long)(grid), s2c::kRowsThreadsI,           \
                                                s2c::rows_inv_smem(N, ZQ), params)
#endif

}  // namespace s2c
