// C-ABI entry points of s2cnn_b200 (see include/s2cnn_b200.h) and the host-side dispatch that
// sequences the kernels.  nvcc -gencode arch=compute_100a,code=sm_100a for the product, the kernel
// families with many instantiations compiled beside it from parts.cu (-DS2C_SPLIT); one translation unit
// with g++ -x c++ -DS2C_EMUL for the host-emulation build used by the CPU tests.
#include "../../include/s2cnn_b200.h"

#include <algorithm>
#include <atomic>
#include <complex>
#include <map>
#include <mutex>
#include <tuple>

#include "backend.h"
#include "host_math.h"
#include "tables.h"
#include "fft_device.h"
#include "so3_kernels.h"
#include "so3_plane_kernels.h"
#include "so3_fused_kernels.h"
#include "so3_relay_kernels.h"
#include "so3_cluster_kernels.h"
#include "so3_mid_kernels.h"
#include "s2_kernels.h"
#include "so3_small_kernels.h"
#include "wigner_columns.h"
#include "wigner_tiled.h"
#include "wigner_rows.h"
#include "cgemm_kernels.h"
#include "rotate_kernels.h"
#include "s2_mm_thin.h"
#include "so3_mm_tc.h"
#include "misc_kernels.h"
#include "project_kernels.h"

namespace s2c {
thread_local long g_launch_count = 0;
#ifdef S2C_EMUL
EmuBulk g_emu_bulk;
void emu_bulk_block_end() {
  if (g_emu_bulk.bar && !g_emu_bulk.never) ++g_emu_bulk.faults;
  g_emu_bulk.bar = nullptr;
}
#endif
// test switches (process-wide, race-free; see the "test hooks" section of the header)
static std::atomic<int> g_force_general{0};   // 1 = no single-kernel path, 2 = also no plane kernels
static std::atomic<int> g_cluster{0};         // 2b <= 32: 0 by batch size, 1 cluster, 2 walking, 3 plane kernels
static std::atomic<int> g_plane_chunk{0};     // plane path: signals per chunk (0 = default)

#define S2C_TRY(expr)            \
  do {                           \
    int rc__ = (expr);           \
    if (rc__ != S2C_OK) return rc__; \
  } while (0)

static inline stream_t as_stream(void* s) { return (stream_t)s; }

// Rows (or row pairs) per block of the FFT passes: about 4096 complex numbers of shared memory,
// and a divisor of `period` so that a block never straddles two planes / two (z, n) slabs.
static inline int fft_group(int N, int period) {
  const int cap = std::max(1, std::min(256, 4096 / N));
  int g = 1;
  for (int d = 1; d <= period && d <= cap; ++d)
    if (period % d == 0) g = d;
  return g;
}

static size_t so3_ws_per_z(int N, int K) {
  // two scratch arrays of complex numbers: [z][K][N][N] and [K][2K-1][z][N]
  return ((size_t)K * N * N + (size_t)K * (2 * K - 1) * N) * sizeof(float2);
}
static size_t s2_ws_per_z(int N, int K) { return (size_t)(2 * K - 1) * N * sizeof(float2); }

// Large-bandwidth path for N = 64 and 128: a plane kernel (both row transforms of a (z, beta)
// plane) and a Wigner kernel per direction, through the scratch array V of
// 8 K N^2 bytes per signal (8.4 MB at b = 64), in chunks of at most rows_zc(N) signals.
static size_t so3_v_per_z(int N, int K) { return (size_t)K * N * N * sizeof(float2); }
static bool use_plane_kernels(int N) { return plane_supported(N) && g_force_general < 2; }
static int launch_fwd_plane(int N, long zc, stream_t st, const FwdPlaneParams& f) {
  const long grid = zc * N;
  if (N == 128) return S2C_LAUNCH_PLANE(so3_fwd_plane, 128, grid, st, f);
  return S2C_LAUNCH_PLANE(so3_fwd_plane, 64, grid, st, f);
}
static int launch_inv_plane(int N, long zc, stream_t st, const InvPlaneParams& f) {
  const long grid = zc * N;
  if (N == 128) return S2C_LAUNCH_PLANE(so3_inv_plane, 128, grid, st, f);
  return S2C_LAUNCH_PLANE(so3_inv_plane, 64, grid, st, f);
}
// The order in which the analysis' Wigner kernel takes its items, one block per SM (no second one fits, at either length:
// with two to an SM in the grid of N = 64, 64 signals took 63.2 us for 61.4, 512 485 for 482) walking its share:
// sorted by their table rows and dealt out forwards and backwards in turn, so that the shares are equal to a few percent.
// (In the order of n and m a quarter of the SM time was idle at b = 64: 48 us per 8 signals instead of 39.)
static void rows_order(int nl, int K, RowsOrder* out) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, RowsOrder> known;
  std::lock_guard<std::mutex> g(mu);
  auto it = known.find({nl, K});
  if (it == known.end()) {
    if (known.size() >= 64) known.clear();
    std::vector<std::pair<int, int>> pairs;      // (-rows, pair)
    for (int n = 0; n < K; ++n)
      for (int m0 = 0; m0 < K; m0 += kRowsMG) {
        int rows = 0;
        for (int m = m0; m < std::min(m0 + kRowsMG, K); ++m)
          rows += std::max(0, nl - std::max(m, n) + kRowsStep - 1) / kRowsStep * kRowsStep;
        pairs.push_back({-rows, n * kRowsMG + m0 / kRowsMG});
      }
    std::sort(pairs.begin(), pairs.end());
    RowsOrder o{};
    for (size_t i = 0; i < pairs.size(); ++i) o.pair[i] = (unsigned short)pairs[i].second;
    it = known.emplace(std::make_pair(nl, K), o).first;
  }
  *out = it->second;
}
static int launch_fwd_rows(int N, stream_t st, FwdRowsParams& f) {
  rows_order(f.nl, f.K, &f.order);
  const long grid = std::min<long>(rows_items(f.K, f.zc), (long)dev_sm_count());
  if (N == 128) return S2C_LAUNCH_FWD_ROWS(128, grid, st, f);
  return S2C_LAUNCH_FWD_ROWS(64, grid, st, f);
}
// eight batch elements to a warp (a table value is then loaded once for eight numbers) where there are more than four
static int launch_inv_rows(int N, stream_t st, const InvRowsParams& f) {
  const long grid = (long)f.K * ((f.K + kRowsMGI - 1) / kRowsMGI) * ((f.zc + 7) / 8);     // (one or two fours: the same)
  if (f.zc > 4) {
    if (N == 128) return S2C_LAUNCH_INV_ROWS(128, 8, grid, st, f);
    return S2C_LAUNCH_INV_ROWS(64, 8, grid, st, f);
  }
  if (N == 128) return S2C_LAUNCH_INV_ROWS(128, 4, grid, st, f);
  return S2C_LAUNCH_INV_ROWS(64, 4, grid, st, f);
}

// Runs `first(z0, zc, buffer, stream)` then `second(z0, zc, buffer, stream)` for every chunk of the
// batch, in order on the caller's stream, through one scratch buffer.
template <class F1, class F2>
static int plane_pipeline(long nbatch, int N, int K, void* ws, size_t ws_bytes, stream_t st,
                          F1 first, F2 second) {
  const size_t vz = so3_v_per_z(N, K);
  const int want = g_plane_chunk.load();
  const long fit = (long)(ws_bytes / vz);
  if (fit < 1 || ws == nullptr)
    return fail(S2C_ERR_WORKSPACE, "workspace smaller than one batch element (" + std::to_string(vz) +
                                       " bytes needed)");
  long chunk = (want >= 1 && want <= rows_zc(N)) ? want : rows_zc(N);
  chunk = std::min(std::min(chunk, fit), nbatch);
  if (want < 1) {      // equal chunks, of whole eights: the last one is not a fraction
    const long parts = (nbatch + chunk - 1) / chunk;
    chunk = std::min(chunk, ((nbatch + parts - 1) / parts + 7) / 8 * 8);
  }
  for (long z0 = 0; z0 < nbatch; z0 += chunk) {
    const long zc = std::min(chunk, nbatch - z0);
    S2C_TRY(first(z0, zc, (float2*)ws, st));
    S2C_TRY(second(z0, zc, (float2*)ws, st));
  }
  return S2C_OK;
}

// 32 < N < 64: a plane kernel (so3_mid_kernels.h) and a tiled Wigner kernel per direction through
// V[n][m][z][beta].  Signals per chunk: whole tiles of the Wigner kernel, within the workspace.
// A chunk's V may be larger than L2: fewer, longer launches weigh more than re-reading part of it (2560 signals at
// b = 15, synthesis: 237 us in chunks of 64 MB, 227 of 96, 218 of 128 and 192; 512 signals at b = 30: 816 us in chunks
// of 64 MB, 780 of 128, 757 of 192).  The chunks of a batch are equal, so that the last one is not a fraction.
constexpr size_t kChunkBytes = (size_t)192 << 20;
static long chunk_signals(long nbatch, size_t per_z) {
  const long most = std::max(1L, (long)(kChunkBytes / per_z) / kWigZT) * kWigZT;
  const long parts = (nbatch + most - 1) / most;
  const long even = ((nbatch + parts - 1) / parts + kWigZT - 1) / kWigZT * kWigZT;
  return std::min(nbatch, even);
}
static size_t so3_mid_v_per_z(int N, int K) { return (size_t)K * (2 * K - 1) * N * sizeof(float2); }
static bool use_mid_kernels(int N) { return mid_supported(N) && g_force_general < 2; }
static int mid_chunk(long nbatch, int N, int K, const void* ws, size_t ws_bytes, long* chunk) {
  const size_t vz = so3_mid_v_per_z(N, K);
  const long fit = ws ? (long)(ws_bytes / vz) : 0;
  if (fit < 1)
    return fail(S2C_ERR_WORKSPACE, "workspace smaller than one batch element (" + std::to_string(vz) +
                                       " bytes needed)");
  *chunk = std::min(fit, chunk_signals(nbatch, vz));
  return S2C_OK;
}

// Small bandwidths: whether the batch is small enough for the cluster kernels, by the number of groups of
// kFusedZG batch elements (a walking block, or a cluster of cl_size(N) blocks, each).  A walking kernel takes
// the same time for any batch up to one block per SM and resident block; the clusters' time grows from a third of
// that with the batch, at b = 16 to the same at 55 (analysis) and 95 (synthesis) groups, b = 15 at 80 and 130,
// b = 12 at 53 and 88, b = 10 at 600 and 500, b = 6 at 800 and 500.  The relay of N > 20 keeps several times the
// shared memory of a synthesis per walking block (one block of 8 warps per SM) and is never the faster one.
enum ClKind { kClAnalysis, kClSynthesis, kClRelay };
static bool so3_prefers_cluster(ClKind kind, int N, long nbatch) {
  if (const int forced = g_cluster.load()) return forced == 1;
  const long groups = (nbatch + kFusedZG - 1) / kFusedZG;
  if (N <= 20) return groups <= 500;
  return kind == kClRelay || groups <= (kind == kClAnalysis ? 55 : 95);
}

// Large batches at 18 <= 2 b <= 32: plane kernels (so3_small_kernels.h) and one signal per thread in the Wigner step
// (wigner_columns.h), through a workspace that holds at least one tile of signals.  The lines are where they get
// faster than the cluster kernels, and they stay faster than the walking kernels up to 5120 signals (b = 16: 570 ->
// 438 us analysis, 598 -> 486 synthesis; b = 15: 712 -> 384, 783 -> 424; b = 12: 190 -> 185; b = 10: 113 -> 112,
// 138 -> 124).  A spectrum of few degrees (K <= N / 3) leaves a cluster less to do per block: later lines.  At
// 2 b <= 16 a whole spectrum fits beside the planes three blocks to an SM and the walking kernels are the faster ones.
// With an S2 product as input (six features; one in brackets) the chained layers gain at every length (b = 15, 1280 signals
// 446 -> 214 us, b = 16 270 -> 198, b = 10, 5120 signals 215 -> 180 [154 -> 139]), the synthesis up to 1500 signals where
// walking blocks take four betas at a time (b = 16: 193 -> 164 us, at 3200 signals 382 -> 428 [338 -> 302]; b = 12:
// 77 -> 74, 136 -> 173) and everywhere else (b = 15, 3200 signals: 542 -> 361, b = 10, 5120: 161 -> 157 [134 -> 118]).
// `product` 2, both factors spectra of real signals (s2_mirror; full -> half product): b = 16, six features, 3200 signals:
// walking 440 -> 395, planes 442 -> 355; b = 14, three, 3840: 385 -> 372, 337 -> 301; b = 12, one, 4000: walking 150 -> 147,
// planes 176 -> 165; the relay of b = 10, one, 5120: 148 -> 139.
static bool so3_prefers_planes(ClKind kind, int N, int K, int nl, long nbatch, const void* ws, size_t ws_bytes,
                               int product = 0) {
  const int forced = g_cluster.load();
  if (g_force_general || !small_supported(N) || !ws || forced == 1 || forced == 2) return false;
  if (ws_bytes < so3_mid_v_per_z(N, K) * (size_t)std::min<long>(kWigZT, nbatch) || nl > kColMaxDegrees) return false;
  if (forced == 3) return true;
  const bool full = 3 * K > N, relay = kind == kClRelay;
  if (product) return nbatch >= (N >= 22 ? 256 : 600) && (relay || N < 24 || N % 4 != 0 || nbatch <= 1500 || (product == 2 && N > 24));
  if (N >= 26) return nbatch >= (full ? (relay ? 32 : 48) : 256);
  if (N == 24) return nbatch >= (full ? 64 : relay ? 512 : 256);
  return nbatch >= (N == 22 ? 256 : 600);
}

// 2b >= 66 with 2b mod 4 = 2: the tiled Wigner kernels stage these panels in small pieces and keep few threads busy on
// few signals; below these lines (signals x 2b) the untiled ones are the faster ones.  Analysis, tiled / untiled: 1
// signal b = 45 71 / 53 us, 8 signals b = 39 149 / 139, 32 signals b = 33 259 / 255, b = 39 385 / 386, b = 45
// 358 / 372; synthesis: 1 signal b = 45 55 / 47, 8 signals b = 33 92 / 88, 16 signals b = 33 146 / 146, b = 45 184 / 189.
static bool few_for_tiles(int N, long zc, long line) { return N > 64 && N % 4 == 2 && zc * N <= line; }

// Which kernels a transform takes: one rule for the dispatcher and for the workspace queries.
//   cluster, walking: one kernel, no workspace          planes: so3_small_kernels.h, 18 <= 2b <= 32
//   mid: so3_mid_kernels.h, 32 < 2b < 64                rows: 2b = 64, 128            passes: any other size
enum So3Route { kCluster, kWalking, kPlanes, kMid, kRows, kPasses };
// rows (m, n, l) of the table panels: degrees below nl, |m|, |n| < K, one of each mirror pair
static int panel_rows(int nl, int K) {
  const long all = so3_nspec(K) + (long)(nl - K) * (2 * K - 1) * (2 * K - 1);
  return (int)((all - nl) / 2 + nl);
}
static bool has_smem(size_t bytes) { return bytes <= (size_t)dev_smem_limit() - 1024; }
static So3Route big_route(int N) { return use_plane_kernels(N) ? kRows : use_mid_kernels(N) ? kMid : kPasses; }
static So3Route analysis_route(int N, int K, int nl, long nbatch, const void* ws, size_t ws_bytes) {
  if (so3_prefers_planes(kClAnalysis, N, K, nl, nbatch, ws, ws_bytes)) return kPlanes;
  if (!g_force_general && N <= kFusedMaxN) {
    if (nl <= kFusedMaxDegrees && so3_prefers_cluster(kClAnalysis, N, nbatch)) return kCluster;
    if (has_smem(fwd_fused_smem_bytes(N, panel_rows(nl, K)))) return kWalking;
  }
  return big_route(N);
}
// `one_kernel`: a synthesis that writes no signal (its integral)
static So3Route synthesis_route(int N, int K, long nbatch, const void* ws, size_t ws_bytes, int product = 0,
                                bool one_kernel = false) {
  if (!one_kernel && so3_prefers_planes(kClSynthesis, N, K, K, nbatch, ws, ws_bytes, product)) return kPlanes;
  if (!g_force_general && N <= kFusedMaxN) {
    if (so3_prefers_cluster(kClSynthesis, N, nbatch)) return kCluster;
    if (has_smem(fused_smem_bytes(N, panel_rows(K, K)))) return kWalking;
  }
  return big_route(N);
}
static bool relay_takes_planes(int N, int Kin, int Kout, long nbatch, const void* ws, size_t ws_bytes, int product) {
  return so3_prefers_planes(kClRelay, N, Kin, Kout, nbatch, ws, ws_bytes, product) &&
         ws_bytes >= (so3_mid_v_per_z(N, Kin) + so3_mid_v_per_z(N, Kout)) * (size_t)std::min<long>(kWigZT, nbatch);
}
// a workspace that no route finds too small, for the queries
static const void* const kAnyWorkspace = (const void*)16;
constexpr size_t kAnySize = ~(size_t)0 / 2;
// scratch that a route uses up in full (every transform also works with less, in shorter chunks)
static size_t route_workspace(So3Route r, int N, int K, long nbatch) {
  if (r == kPlanes || r == kMid) return so3_mid_v_per_z(N, K) * (size_t)chunk_signals(nbatch, so3_mid_v_per_z(N, K));
  if (r == kRows) return so3_v_per_z(N, K) * (size_t)std::min<long>(rows_zc(N), nbatch);
  if (r == kPasses) {
    const size_t per_z = so3_ws_per_z(N, K);
    return per_z * (size_t)std::min((long)std::max<size_t>(32, ((size_t)256 << 20) / per_z), nbatch);
  }
  return 0;
}

static int launch_fwd_wigner_col(FwdWignerParams w, stream_t st) {
  w.ZT = std::min(kColZT, (w.nbatch + 31) / 32 * 32);
  w.nzt = (w.nbatch + w.ZT - 1) / w.ZT;
  return S2C_LAUNCH(so3_fwd_wigner_col, (long)w.pan.npairs * w.nzt, w.ZT, wigner_col_smem(w.N, w.nl), st, w);
}
static int launch_inv_wigner_col(InvWignerParams w, stream_t st) {
  w.ZT = std::min(kColZT, (w.nbatch + 31) / 32 * 32);
  w.nzt = (w.nbatch + w.ZT - 1) / w.ZT;
  if (w.xs && w.s2_real)
    return S2C_LAUNCH(so3_inv_wigner_col_s2real, (long)w.pan.npairs * w.nzt, w.ZT, wigner_col_smem(w.N, w.pan.nl), st, w);
  if (w.xs)
    return S2C_LAUNCH(so3_inv_wigner_col_s2, (long)w.pan.npairs * w.nzt, w.ZT, wigner_col_smem(w.N, w.pan.nl), st, w);
  return S2C_LAUNCH(so3_inv_wigner_col, (long)w.pan.npairs * w.nzt, w.ZT, wigner_col_smem(w.N, w.pan.nl), st, w);
}

static int check_b(int b_in, int b_out) {
  if (b_in < 1 || b_out < 1) return fail(S2C_ERR_BAD_ARG, "bandwidths must be >= 1");
  return S2C_OK;
}

// ---------------------------------------------------------------------------------------------
// SO(3) analysis:  real signal (strided) -> spectrum rows [nspec(b_out)][nbatch]
// ---------------------------------------------------------------------------------------------
static int so3_analysis(const float* x, long in_stride, long in_off, float2* out, long nbatch,
                        int b_in, int b_out, bool weighted, int mode, void* ws, size_t ws_bytes,
                        stream_t st, bool relu = false, float* sums = nullptr) {
  const int N = 2 * b_in, K = std::min(b_in, b_out);
  FftDev fft;
  PanelsDev pan;
  S2C_TRY(TableCache::get().fft(N, fft));
  S2C_TRY(TableCache::get().panels(b_in, b_out, K, weighted, false, pan));
  if (b_out > b_in && mode == kSo3Real)  // rows with |m| or |n| >= b_in stay zero (so3_fft.py:44-48)
    S2C_TRY(dev_memset_async(out, 0, (size_t)so3_nspec(b_out) * nbatch * sizeof(float2), st));
  const So3Route route = analysis_route(N, K, b_out, nbatch, ws, ws_bytes);
  const bool small = route == kPlanes, mid = small || route == kMid;
  if (route == kCluster) {
    ClFwdParams f;
    f.x = x; f.in_stride = in_stride; f.in_off = in_off;
    f.out = out; f.out_zstride = nbatch;
    S2C_TRY(TableCache::get().cluster(b_in, b_out, K, weighted, f.tab));
    f.nbatch = (int)nbatch; f.K = K;
    f.mode = mode; f.relu = relu;
    f.wide = in_stride == 1 && in_off == 0 && N % 4 == 0 && (uintptr_t)x % 32 == 0;
    f.sums = sums;
    int rc = S2C_OK;
    S2C_DISPATCH_N(N, rc = S2C_LAUNCH_CL(so3_fwd_cl, kN, (nbatch + kFusedZG - 1) / kFusedZG,
                                         cl_smem_bytes(N, K, 0), st, f));
    return rc;
  }
  if (route == kWalking) {
    FwdFusedParams f;
    f.x = x; f.in_stride = in_stride; f.in_off = in_off;
    f.out = out; f.out_zstride = nbatch;
    f.pan = pan; f.tw = fft.tw;
    f.nbatch = (int)nbatch; f.K = K; f.BG = fused_bg(N); f.KP = fused_kp(N); f.PS = fused_plane_stride(N, K);
    f.nrows = pan.nrows; f.mode = mode; f.relu = relu;
    f.wide = in_stride == 1 && in_off == 0 && N % 4 == 0 && (uintptr_t)x % 32 == 0;
    f.sums = sums;
    int rc = S2C_OK;
    const long grid = (nbatch + kFusedZG - 1) / kFusedZG;
    const size_t sm = fwd_fused_smem_bytes(N, pan.nrows);
    S2C_DISPATCH_N(N, rc = S2C_LAUNCH_N(so3_fwd_fused, kN, grid,
                                        fused_threads(sm, (size_t)dev_smem_limit()), sm, st, f));
    return rc;
  }
  if (relu && !mid) return fail(S2C_ERR_UNSUPPORTED, "fused ReLU input needs 2 b < 64");
  if (sums && (!mid || !ws)) return fail(S2C_ERR_UNSUPPORTED, "per-signal sums need 2 b < 64");
  if (route == kRows) {
    HalfPanelsDev hp;
    hp.nbeta = N; hp.nl = b_out; hp.K = K; hp.npairs = pan.npairs;
    S2C_TRY(TableCache::get().half_panels(b_in, b_out, K, weighted, &hp.data, &hp.off));
    auto planes = [&](long z0, long zc, float2* v, stream_t s) {
      FwdPlaneParams f;
      f.x = x + (size_t)z0 * N * N * N * in_stride;
      f.in_stride = in_stride; f.in_off = in_off;
      f.v = v; f.tw = fft.tw; f.nbatch = (int)zc; f.K = K;
      return launch_fwd_plane(N, zc, s, f);
    };
    auto wigner = [&](long z0, long zc, float2* v, stream_t s) {
      FwdRowsParams r;
      r.v = v; r.out = out + z0; r.out_zstride = nbatch; r.pan = hp;
      r.zc = (int)zc; r.K = K; r.nl = b_out; r.mode = mode;
      return launch_fwd_rows(N, s, r);
    };
    return plane_pipeline(nbatch, N, K, ws, ws_bytes, st, planes, wigner);
  }
  const size_t per_z = so3_ws_per_z(N, K);
  long chunk = (long)std::min<size_t>((size_t)nbatch, ws_bytes / per_z);
  if (mid) {
    S2C_TRY(mid_chunk(nbatch, N, K, ws, ws_bytes, &chunk));
  } else if (chunk < 1 || ws == nullptr) {
    return fail(S2C_ERR_WORKSPACE, "workspace smaller than one batch element (" +
                                       std::to_string(per_z) + " bytes needed)");
  }
  const int G = fft_group(N, N), Gg = fft_group(N, N / 2);  // alpha passes, gamma passes
  const size_t fft_smem = fft_smem_bytes(N, G);
  for (long z0 = 0; z0 < nbatch; z0 += chunk) {
    const long zc = std::min(chunk, nbatch - z0);
    float2* u = (float2*)ws;
    float2* v = mid ? u : u + (size_t)zc * K * N * N;
    if (small) {
      SmallParams g;
      g.x = x + (size_t)z0 * N * N * N * in_stride; g.out = nullptr;
      g.stride = in_stride; g.off = in_off;
      g.v = v; g.v2 = nullptr; g.bias = nullptr; g.nfeat = 1; g.z0 = z0; g.mask = nullptr; g.relu = relu;
      g.nplanes = zc * N; g.nz = (int)zc; g.K = K; g.K2 = 0;
      int rc = S2C_OK;
      S2C_DISPATCH_SMALL(N, rc = S2C_LAUNCH_SMALL(so3_fwd_small, kN, st, g));
      if (rc) return rc;
    } else if (mid) {
      MidParams g;
      g.x = x + (size_t)z0 * N * N * N * in_stride; g.out = nullptr;
      g.stride = in_stride; g.off = in_off;
      g.v = v; g.tw = fft.tw; g.bias = nullptr; g.nfeat = 1; g.z0 = z0;
      g.relu = relu; g.mask = nullptr;
      g.nbatch = (int)zc; g.K = K; g.inv_k = 1.f / (float)K;
      int rc = S2C_OK;
      S2C_DISPATCH_MID(N, rc = S2C_LAUNCH_N(so3_fwd_mid, kN, zc * ((kN + mid_nb(kN) - 1) / mid_nb(kN)),
                                            kMidThreads, mid_smem_bytes(kN), st, g));
      if (rc) return rc;
    } else {
    FwdGammaParams g;
    g.x = x + (size_t)z0 * N * N * N * in_stride;
    g.in_stride = in_stride;
    g.in_off = in_off;
    g.u = u;
    g.N = N; g.b = b_in; g.K = K; g.G = Gg;
    g.npairs = zc * N * b_in;
    g.fft = fft;
    S2C_TRY(S2C_LAUNCH(so3_fwd_gamma, (g.npairs + Gg - 1) / Gg, kThreads, fft_smem_bytes(N, Gg), st, g));
    FwdAlphaParams a;
    a.in = (const float*)u;
    a.in_real = 0;
    a.v = v;
    a.nbatch = (int)zc; a.N = N; a.K = K; a.Kn = K; a.G = G;
    a.nrows = zc * K * N;
    a.fft = fft;
    S2C_TRY(S2C_LAUNCH(so3_fwd_alpha, (a.nrows + G - 1) / G, kThreads, fft_smem, st, a));
    }
    if (sums) {
      MidSumsParams q;
      q.v = v + (size_t)(K - 1) * zc * N; q.sums = sums + z0; q.nbatch = (int)zc; q.N = N;
      q.zs = small ? 1 : N; q.bs = small ? (int)zc : 1;
      S2C_TRY(S2C_LAUNCH(so3_mid_sums, (zc + 31) / 32, 32, 0, st, q));
    }
    FwdWignerParams w;
    w.v = v;
    w.out = out + z0;
    w.out_zstride = nbatch;
    w.pan = pan;
    w.nbatch = (int)zc; w.N = N; w.K = K; w.nl = b_out;
    w.ZT = (int)std::min<long>(32, zc);
    w.nzt = (int)((zc + w.ZT - 1) / w.ZT);
    w.mode = mode;
    if (small) {
      S2C_TRY(launch_fwd_wigner_col(w, st));
      continue;
    }
    if (!few_for_tiles(N, zc, 2240) && fwd_wigner_t_fits(N, b_out, kWigZT, dev_smem_limit())) {
      w.ZT = kWigZT;
      w.nzt = (int)((zc + kWigZT - 1) / kWigZT);
      S2C_TRY(S2C_LAUNCH(so3_fwd_wigner_t, (long)pan.npairs * w.nzt, kThreads,
                         fwd_wigner_t_smem(N, b_out), st, w));
      continue;
    }
    const size_t wsm = align_up((size_t)b_out * (N + 1) * sizeof(float), 16) +
                       (size_t)w.ZT * (N + 1) * sizeof(float2);
    S2C_TRY(S2C_LAUNCH(so3_fwd_wigner, (long)pan.npairs * w.nzt, kThreads, wsm, st, w));
  }
  return S2C_OK;
}

// ---------------------------------------------------------------------------------------------
// SO(3) synthesis:  spectrum rows [nspec(b_in)][nbatch] -> real signal (strided)
// ---------------------------------------------------------------------------------------------
struct S2ProductArgs {
  const float2* xs = nullptr;
  const float2* ys = nullptr;
  int nb = 0, fin = 0, fout = 0;
  int real = 0;      // spectra of real signals
};

static bool so3_synthesis_is_fused(int b_in, int b_out) {
  const int N = 2 * b_out, K = std::min(b_in, b_out);
  if (g_force_general || N > kFusedMaxN) return false;
  return has_smem(fused_smem_bytes(N, panel_rows(K, K)));
}

static int so3_synthesis(const float2* x, float* out, long out_stride, long out_off, long nbatch,
                         int b_in, int b_out, bool weighted, int mode, const float* bias,
                         int nfeat, void* ws, size_t ws_bytes, stream_t st,
                         const S2ProductArgs* prod = nullptr, float* integral = nullptr,
                         const float* mask = nullptr) {
  const int N = 2 * b_out, K = std::min(b_in, b_out);
  FftDev fft;
  PanelsDev pan;
  S2C_TRY(TableCache::get().fft(N, fft));
  S2C_TRY(TableCache::get().panels(b_out, K, K, weighted, false, pan));
  const So3Route route = synthesis_route(N, K, nbatch, ws, ws_bytes, prod ? 1 + prod->real : 0, integral != nullptr);
  const bool small = route == kPlanes, mid = small || route == kMid;
  if (mask && (out_stride != 1 || out_off != 0))
    return fail(S2C_ERR_UNSUPPORTED, "masked synthesis: real output only");
  if (route == kCluster) {
    ClInvParams f;
    f.in.x = x; f.in.x_zstride = nbatch; f.in.mode = mode;
    f.in.xs = f.in.ys = nullptr; f.in.s2_nb = f.in.s2_fin = f.in.s2_fout = f.in.s2_real = 0;
    f.out = out; f.out_stride = out_stride; f.out_off = out_off;
    f.bias = bias; f.nfeat = nfeat > 0 ? nfeat : 1;
    S2C_TRY(TableCache::get().cluster(b_out, K, K, weighted, f.tab));
    f.nbatch = (int)nbatch; f.K = K;
    f.iw = nullptr; f.isum = nullptr;
    f.mask = mask;
    f.wide = out_stride == 1 && out_off == 0 && N % 4 == 0 && out && (uintptr_t)out % 32 == 0 &&
             (uintptr_t)mask % 32 == 0;
    if (integral) {
      S2C_TRY(TableCache::get().quad_weights(b_out, &f.iw));
      f.isum = integral;
    }
    if (prod) {
      f.in.mode = kS2Product;
      f.in.xs = prod->xs; f.in.ys = prod->ys;
      f.in.s2_nb = prod->nb; f.in.s2_fin = prod->fin; f.in.s2_fout = prod->fout; f.in.s2_real = prod->real;
    }
    int rc = S2C_OK;
    S2C_DISPATCH_N(N, rc = S2C_LAUNCH_CL(so3_inv_cl, kN, (nbatch + kFusedZG - 1) / kFusedZG,
                                         cl_smem_bytes(N, K, f.tab.max_rows), st, f));
    return rc;
  }
  if (route == kWalking) {
    InvFusedParams f;
    f.x = x; f.x_zstride = nbatch;
    f.out = out; f.out_stride = out_stride; f.out_off = out_off;
    f.bias = bias; f.nfeat = nfeat > 0 ? nfeat : 1;
    f.pan = pan; f.tw = fft.tw;
    f.nbatch = (int)nbatch; f.K = K; f.BG = fused_bg(N); f.KP = fused_kp(N); f.PS = fused_plane_stride(N, K);
    f.nrows = pan.nrows; f.mode = mode;
    f.xs = nullptr; f.ys = nullptr; f.s2_nb = f.s2_fin = f.s2_fout = f.s2_real = 0;
    f.iw = nullptr; f.isum = nullptr;
    f.mask = mask;
    f.wide = out_stride == 1 && out_off == 0 && N % 4 == 0 && out && (uintptr_t)out % 32 == 0 &&
             (uintptr_t)mask % 32 == 0;
    if (integral) {
      if (N % f.BG != 0 || kFusedZG * f.BG * (N / 2) > 256)
        return fail(S2C_ERR_UNSUPPORTED, "fused integration: unsupported grouping");
      S2C_TRY(TableCache::get().quad_weights(b_out, &f.iw));
      f.isum = integral;
    }
    if (prod) {
      f.mode = kS2Product;
      f.xs = prod->xs; f.ys = prod->ys;
      f.s2_nb = prod->nb; f.s2_fin = prod->fin; f.s2_fout = prod->fout; f.s2_real = prod->real;
    }
    int rc = S2C_OK;
    const long grid = (nbatch + kFusedZG - 1) / kFusedZG;
    const size_t sm = fused_smem_bytes(N, pan.nrows);
    S2C_DISPATCH_N(N, rc = S2C_LAUNCH_N(so3_inv_fused, kN, grid,
                                        fused_threads(sm, (size_t)dev_smem_limit()), sm, st, f));
    return rc;
  }
  if (integral)
    return fail(S2C_ERR_UNSUPPORTED, "fused ReLU + integration needs the small-bandwidth path");
  if (mask && (!mid || !ws)) return fail(S2C_ERR_UNSUPPORTED, "masked synthesis: real output and 2 b < 64");
  if (route == kRows) {
    HalfPanelsDev hp;
    hp.nbeta = N; hp.nl = K; hp.K = K; hp.npairs = pan.npairs;
    S2C_TRY(TableCache::get().half_panels(b_out, K, K, weighted, &hp.data, &hp.off));
    auto wigner = [&](long z0, long zc, float2* s, stream_t sm) {
      InvRowsParams r;
      r.x = x + z0; r.x_zstride = nbatch; r.s = s; r.pan = hp;
      r.zc = (int)zc; r.K = K; r.mode = mode;
      return launch_inv_rows(N, sm, r);
    };
    auto planes = [&](long z0, long zc, float2* s, stream_t sm) {
      InvPlaneParams f;
      f.s = s;
      f.out = out + (size_t)z0 * N * N * N * out_stride;
      f.out_stride = out_stride; f.out_off = out_off;
      f.bias = bias; f.nfeat = nfeat > 0 ? nfeat : 1; f.z0 = z0;
      f.tw = fft.tw; f.nbatch = (int)zc; f.K = K;
      return launch_inv_plane(N, zc, sm, f);
    };
    return plane_pipeline(nbatch, N, K, ws, ws_bytes, st, wigner, planes);
  }
  const size_t per_z = so3_ws_per_z(N, K);
  long chunk = (long)std::min<size_t>((size_t)nbatch, ws_bytes / per_z);
  if (mid) {
    S2C_TRY(mid_chunk(nbatch, N, K, ws, ws_bytes, &chunk));
  } else if (chunk < 1 || ws == nullptr) {
    return fail(S2C_ERR_WORKSPACE, "workspace smaller than one batch element (" +
                                       std::to_string(per_z) + " bytes needed)");
  }
  const int G = fft_group(N, N), Gg = fft_group(N, N / 2);  // alpha passes, gamma passes
  const size_t fft_smem = fft_smem_bytes(N, G);
  for (long z0 = 0; z0 < nbatch; z0 += chunk) {
    const long zc = std::min(chunk, nbatch - z0);
    float2* t = (float2*)ws;                                   // [z][K][N][N]
    float2* s = mid ? t : t + (size_t)zc * K * N * N;          // [K][2K-1][z][N]
    InvWignerParams w;
    w.x = x + z0;
    w.x_zstride = nbatch;
    w.s = s;
    w.pan = pan;
    w.nbatch = (int)zc; w.N = N; w.K = K;
    w.ZT = (int)std::min<long>(32, zc);
    w.nzt = (int)((zc + w.ZT - 1) / w.ZT);
    w.mode = mode;
    if (prod) {
      w.xs = prod->xs; w.ys = prod->ys;
      w.s2_nb = prod->nb; w.s2_fin = prod->fin; w.s2_fout = prod->fout; w.s2_real = prod->real;
      w.z0 = z0;
    }
    if (small) {
      S2C_TRY(launch_inv_wigner_col(w, st));
    } else if (!few_for_tiles(N, zc, 800) && inv_wigner_t_smem(N, K) <= (size_t)dev_smem_limit() - 1024) {
      w.ZT = kWigZT;
      w.nzt = (int)((zc + kWigZT - 1) / kWigZT);
      S2C_TRY(S2C_LAUNCH(so3_inv_wigner_t, (long)pan.npairs * w.nzt, kThreads,
                         inv_wigner_t_smem(N, K), st, w));
    } else {
      const size_t wsm = align_up((size_t)K * N * sizeof(float), 16) + (size_t)K * w.ZT * sizeof(float2);
      S2C_TRY(S2C_LAUNCH(so3_inv_wigner, (long)pan.npairs * w.nzt, kThreads, wsm, st, w));
    }
    if (small) {
      SmallParams g;
      g.x = nullptr; g.out = out + (size_t)z0 * N * N * N * out_stride;
      g.stride = out_stride; g.off = out_off;
      g.v = s; g.v2 = nullptr; g.bias = bias; g.nfeat = nfeat > 0 ? nfeat : 1; g.z0 = z0; g.relu = 0;
      g.mask = mask ? mask + (size_t)z0 * N * N * N : nullptr;
      g.nplanes = zc * N; g.nz = (int)zc; g.K = K; g.K2 = 0;
      int rc = S2C_OK;
      S2C_DISPATCH_SMALL(N, rc = S2C_LAUNCH_SMALL(so3_inv_small, kN, st, g));
      if (rc) return rc;
      continue;
    }
    if (mid) {
      MidParams g;
      g.x = nullptr; g.out = out + (size_t)z0 * N * N * N * out_stride;
      g.stride = out_stride; g.off = out_off;
      g.relu = 0; g.mask = mask ? mask + (size_t)z0 * N * N * N : nullptr;
      g.v = s; g.tw = fft.tw; g.bias = bias; g.nfeat = nfeat > 0 ? nfeat : 1; g.z0 = z0;
      g.nbatch = (int)zc; g.K = K; g.inv_k = 1.f / (float)K;
      int rc = S2C_OK;
      S2C_DISPATCH_MID(N, rc = S2C_LAUNCH_N(so3_inv_mid, kN, zc * ((kN + mid_nb(kN) - 1) / mid_nb(kN)),
                                            kMidThreads, mid_smem_bytes(kN), st, g));
      if (rc) return rc;
      continue;
    }
    InvAlphaParams a;
    a.s = s;
    a.out = (float*)t;
    a.out_real = 0;
    a.herm_n0 = 1;
    a.nbatch = (int)zc; a.N = N; a.K = K; a.Kn = K; a.G = G;
    a.nrows = zc * K * N;
    a.fft = fft;
    S2C_TRY(S2C_LAUNCH(so3_inv_alpha, (a.nrows + G - 1) / G, kThreads, fft_smem, st, a));
    InvGammaParams g;
    g.t = t;
    g.out = out + (size_t)z0 * N * N * N * out_stride;
    g.out_stride = out_stride;
    g.out_off = out_off;
    g.bias = bias;
    g.nfeat = nfeat > 0 ? nfeat : 1;
    g.z0 = z0;
    g.N = N; g.b = b_out; g.K = K; g.G = Gg;
    g.npairs = zc * N * b_out;
    g.fft = fft;
    S2C_TRY(S2C_LAUNCH(so3_inv_gamma, (g.npairs + Gg - 1) / Gg, kThreads, fft_smem_bytes(N, Gg), st, g));
  }
  return S2C_OK;
}

static int mm_dispatch(bool so3, int op, const float* a, const float* b, float* c, int nl, int nb,
                       int fi, int fo, stream_t st) {
  if (nl < 1 || nb < 1 || fi < 1 || fo < 1) return fail(S2C_ERR_BAD_ARG, "sizes must be >= 1");
  CgemmParams p = mm_params(so3, op, nl, nb, fi, fo);
  p.A = (const float2*)a;
  p.B = (const float2*)b;
  p.C = (float2*)c;
  return S2C_LAUNCH(cgemm_grouped, cgemm_total_tiles(p), 256, cgemm_smem_bytes(), st, p);
}

}  // namespace s2c

using namespace s2c;

extern "C" {

const char* s2c_last_error(void) { return last_error_ref().c_str(); }
int s2c_version(void) { return 100; }
long s2c_launch_count(void) { return g_launch_count; }
void s2c_clear_tables(void) { TableCache::get().clear(); }
void s2c_set_table_cache_dir(const char* dir) { TableDiskCache::get().set_dir(dir); }
long s2c_table_cache_hits(void) { return TableDiskCache::get().hits(); }
long s2c_table_cache_stores(void) { return TableDiskCache::get().stores(); }
long s2c_tables_computed(void) { return TableCache::computed_count().load(); }
int s2c_is_cuda_build(void) {
#ifdef S2C_EMUL
  return 0;
#else
  return 1;
#endif
}

#ifdef S2C_EMUL
// test of late bulk copies: holds back the nth copy from now (0: none), for good if `never`; returns the faults so far
long s2c_emul_hold_copy(long nth, int never) {
  const long faults = g_emu_bulk.faults;
  g_emu_bulk = EmuBulk{};
  g_emu_bulk.hold = nth;
  g_emu_bulk.never = never;
  return faults;
}
#endif

void s2c_timing_begin(void) {
#ifndef S2C_EMUL
  {
    std::lock_guard<std::mutex> lock(timing_mutex());
    timing_recs().clear();
  }
  timing_on() = true;
#endif
}

int s2c_timing_end(char* buf, size_t buf_bytes) {
  if (!buf || buf_bytes == 0) return fail(S2C_ERR_BAD_ARG, "s2c_timing_end: no buffer");
  buf[0] = 0;
#ifndef S2C_EMUL
  timing_on() = false;
  std::lock_guard<std::mutex> lock(timing_mutex());
  struct Acc { long n = 0; double ms = 0; };
  std::vector<std::pair<std::string, Acc>> acc;
  for (auto& r : timing_recs()) {
    float ms = 0.f;
    cudaEventSynchronize(r.b);
    cudaEventElapsedTime(&ms, r.a, r.b);
    cudaEventDestroy(r.a);
    cudaEventDestroy(r.b);
    size_t i = 0;
    for (; i < acc.size(); ++i) if (acc[i].first == r.name) break;
    if (i == acc.size()) acc.push_back({r.name, Acc()});
    acc[i].second.n += 1;
    acc[i].second.ms += ms;
  }
  timing_recs().clear();
  std::string out;
  for (auto& kv : acc) {
    char line[256];
    std::snprintf(line, sizeof(line), "%s %ld %.6f\n", kv.first.c_str(), kv.second.n, kv.second.ms);
    out += line;
  }
  if (out.size() + 1 > buf_bytes) return fail(S2C_ERR_BAD_ARG, "s2c_timing_end: buffer too small");
  std::memcpy(buf, out.c_str(), out.size() + 1);
#endif
  return S2C_OK;
}

// ---- host generators ---------------------------------------------------------------------------
int s2c_wigner_d(int l, double beta, double* out) {
  if (l < 0 || !out) return fail(S2C_ERR_BAD_ARG, "s2c_wigner_d: bad argument");
  const int L = 2 * l + 1;
  std::vector<double> col(l + 2);
  for (int m = -l; m <= l; ++m)
    for (int n = -l; n <= l; ++n) {
      const int l0 = wigner_d_degrees(m, n, beta, l + 1, col.data());
      out[(m + l) * L + (n + l)] = col[l - l0];
    }
  return S2C_OK;
}

int s2c_quadrature_weights(int b, double* out) {
  if (b < 1 || !out) return fail(S2C_ERR_BAD_ARG, "s2c_quadrature_weights: bad argument");
  std::vector<double> w;
  quadrature_weights(b, w);
  std::copy(w.begin(), w.end(), out);
  return S2C_OK;
}

int s2c_so3_wigner_table(int b, int nl, int weighted, float* out) {
  if (b < 1 || nl < 1 || !out) return fail(S2C_ERR_BAD_ARG, "s2c_so3_wigner_table: bad argument");
  std::vector<double> beta, w, col(nl + 1);
  soft_betas(b, beta);
  quadrature_weights(b, w);
  const long ns = so3_nspec(nl);
  for (int j = 0; j < 2 * b; ++j)
    for (int m = -(nl - 1); m < nl; ++m)
      for (int n = -(nl - 1); n < nl; ++n) {
        const int l0 = wigner_d_degrees(m, n, beta[j], nl, col.data());
        for (int l = l0; l < nl; ++l)
          out[j * ns + so3_row(l, m, n)] =
              (float)(col[l - l0] * (weighted ? w[j] : (2.0 * l + 1.0)));
      }
  return S2C_OK;
}

int s2c_s2_wigner_table(int b, int nl, int weighted, float* out) {
  if (b < 1 || nl < 1 || !out) return fail(S2C_ERR_BAD_ARG, "s2c_s2_wigner_table: bad argument");
  std::vector<double> beta, w, col(nl + 1);
  soft_betas(b, beta);
  quadrature_weights(b, w);
  for (int j = 0; j < 2 * b; ++j)
    for (int m = -(nl - 1); m < nl; ++m) {
      const int l0 = wigner_d_degrees(m, 0, beta[j], nl, col.data());
      for (int l = l0; l < nl; ++l)
        out[(long)j * nl * nl + l * l + l + m] =
            (float)(col[l - l0] * (weighted ? w[j] * 2.0 * b : (2.0 * l + 1.0)));
    }
  return S2C_OK;
}

// F = conj(D^l_mn(alpha, beta, gamma)) = exp(-i m alpha) d^l_mn(beta) exp(-i n gamma)
int s2c_so3_ft_matrix(int b, const double* grid, int n_grid, float* F) {
  if (b < 1 || n_grid < 1 || !grid || !F) return fail(S2C_ERR_BAD_ARG, "s2c_so3_ft_matrix: bad argument");
  const long ns = so3_nspec(b);
  std::vector<double> col(b + 1);
  for (int i = 0; i < n_grid; ++i) {
    const double beta = grid[3 * i], alpha = grid[3 * i + 1], gamma = grid[3 * i + 2];
    for (int m = -(b - 1); m < b; ++m)
      for (int n = -(b - 1); n < b; ++n) {
        const int l0 = wigner_d_degrees(m, n, beta, b, col.data());
        const std::complex<double> ph = std::exp(std::complex<double>(0.0, -(m * alpha + n * gamma)));
        for (int l = l0; l < b; ++l) {
          const std::complex<double> v = ph * col[l - l0];
          float* dst = F + ((long)i * ns + so3_row(l, m, n)) * 2;
          dst[0] = (float)v.real();
          dst[1] = (float)v.imag();
        }
      }
  }
  return S2C_OK;
}

// F = 2b conj(D^l_m0(alpha, beta, 0))
int s2c_s2_ft_matrix(int b, const double* grid, int n_grid, float* F) {
  if (b < 1 || n_grid < 1 || !grid || !F) return fail(S2C_ERR_BAD_ARG, "s2c_s2_ft_matrix: bad argument");
  std::vector<double> col(b + 1);
  for (int i = 0; i < n_grid; ++i) {
    const double beta = grid[2 * i], alpha = grid[2 * i + 1];
    for (int m = -(b - 1); m < b; ++m) {
      const int l0 = wigner_d_degrees(m, 0, beta, b, col.data());
      const std::complex<double> ph = std::exp(std::complex<double>(0.0, -m * alpha));
      for (int l = l0; l < b; ++l) {
        const std::complex<double> v = (2.0 * b) * ph * col[l - l0];
        float* dst = F + ((long)i * b * b + l * l + l + m) * 2;
        dst[0] = (float)v.real();
        dst[1] = (float)v.imag();
      }
    }
  }
  return S2C_OK;
}

// ---- SO(3) transforms ----------------------------------------------------------------------------
size_t s2c_so3_fft_workspace_min(int b_in, int b_out) {
  if (b_in < 1 || b_out < 1) return 0;
  // the beta grid is b_in's for analysis and b_out's for synthesis; take the larger of the two
  const int K = std::min(b_in, b_out);
  return std::max(so3_ws_per_z(2 * b_in, K), so3_ws_per_z(2 * b_out, K));
}

size_t s2c_so3_fft_workspace(long nbatch, int b_in, int b_out) {
  const size_t per_z = s2c_so3_fft_workspace_min(b_in, b_out);
  if (!per_z) return 0;
  if (plane_supported(2 * b_in) && plane_supported(2 * b_out)) {
    // large-bandwidth path: one chunk of the scratch array V of whichever direction wants more (a chunk's signals and a
    // signal's V go by the length of the grid, b_in's or b_out's); never less than one signal of the three-pass
    // organisation, which the test switches can select instead
    const int K = std::min(b_in, b_out);
    auto v = [&](int N) { return so3_v_per_z(N, K) * (size_t)std::min<long>(rows_zc(N), std::max(1L, nbatch)); };
    return std::max(per_z, std::max(v(2 * b_in), v(2 * b_out)));
  }
  const size_t target = (size_t)256 << 20;
  long chunk = (long)std::max<size_t>(32, target / per_z);
  chunk = std::min(chunk, std::max(1L, nbatch));
  return per_z * (size_t)chunk;
}

size_t s2c_so3_analysis_workspace(long nbatch, int b_in, int b_out) {
  if (nbatch < 1 || b_in < 1 || b_out < 1) return 0;
  const int N = 2 * b_in, K = std::min(b_in, b_out);
  return route_workspace(analysis_route(N, K, b_out, nbatch, kAnyWorkspace, kAnySize), N, K, nbatch);
}
size_t s2c_so3_synthesis_workspace(long nbatch, int b_in, int b_out) {
  if (nbatch < 1 || b_in < 1 || b_out < 1) return 0;
  const int N = 2 * b_out, K = std::min(b_in, b_out);
  return route_workspace(synthesis_route(N, K, nbatch, kAnyWorkspace, kAnySize), N, K, nbatch);
}

int s2c_so3_rfft(const float* x, float* out, long nbatch, int b_in, int b_out, int for_grad,
                 void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || nbatch < 1) return fail(S2C_ERR_BAD_ARG, "s2c_so3_rfft: bad argument");
  return so3_analysis(x, 1, 0, (float2*)out, nbatch, b_in, b_out, !for_grad, kSo3Real, ws,
                      ws_bytes, as_stream(stream));
}

int s2c_so3_rfft_relu(const float* x, float* out, long nbatch, int b_in, int b_out, void* ws,
                      size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || nbatch < 1) return fail(S2C_ERR_BAD_ARG, "s2c_so3_rfft_relu: bad argument");
  return so3_analysis(x, 1, 0, (float2*)out, nbatch, b_in, b_out, true, kSo3Real, ws, ws_bytes,
                      as_stream(stream), true);
}

int s2c_so3_rfft_sums_ws(const float* x, float* out, float* sums, long nbatch, int b_in, int b_out,
                         int for_grad, void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || !sums || nbatch < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_rfft_sums_ws: bad argument");
  return so3_analysis(x, 1, 0, (float2*)out, nbatch, b_in, b_out, !for_grad, kSo3Real, ws, ws_bytes,
                      as_stream(stream), false, sums);
}

int s2c_so3_rfft_sums(const float* x, float* out, float* sums, long nbatch, int b_in, int b_out,
                      int for_grad, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || !sums || nbatch < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_rfft_sums: bad argument");
  return so3_analysis(x, 1, 0, (float2*)out, nbatch, b_in, b_out, !for_grad, kSo3Real, nullptr, 0,
                      as_stream(stream), false, sums);
}

void s2c_debug_force_general_path(int level) { g_force_general = level < 0 ? 0 : level; }
void s2c_debug_cluster(int mode) { g_cluster = mode; }
void s2c_debug_plane_chunk(int signals) { g_plane_chunk = signals < 0 ? 0 : signals; }

int s2c_so3_fft(const float* x, float* out, long nbatch, int b_in, int b_out, int for_grad,
                void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || nbatch < 1) return fail(S2C_ERR_BAD_ARG, "s2c_so3_fft: bad argument");
  // linearity: FT(re + i im) = FT(re) + i FT(im), each a real-input transform
  S2C_TRY(so3_analysis(x, 2, 0, (float2*)out, nbatch, b_in, b_out, !for_grad, kSo3Real, ws,
                       ws_bytes, as_stream(stream)));
  return so3_analysis(x, 2, 1, (float2*)out, nbatch, b_in, b_out, !for_grad, kSo3AccumI, ws,
                      ws_bytes, as_stream(stream));
}

int s2c_so3_rifft(const float* x, float* out, long nbatch, int b_in, int b_out, int for_grad,
                  const float* bias, int nfeature, void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || nbatch < 1) return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft: bad argument");
  if (bias && nfeature < 1) return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft: nfeature must be >= 1 with a bias");
  return so3_synthesis((const float2*)x, out, 1, 0, nbatch, b_in, b_out, for_grad != 0, kSo3Real,
                       bias, nfeature, ws, ws_bytes, as_stream(stream));
}

int s2c_so3_rifft_relu_grad_ws(const float* x, const float* act, float* out, long nbatch, int b_in,
                               int b_out, void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !act || !out || nbatch < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft_relu_grad_ws: bad argument");
  return so3_synthesis((const float2*)x, out, 1, 0, nbatch, b_in, b_out, true, kSo3Real, nullptr, 0,
                       ws, ws_bytes, as_stream(stream), nullptr, nullptr, act);
}

int s2c_so3_rifft_relu_grad(const float* x, const float* act, float* out, long nbatch, int b_in,
                            int b_out, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !act || !out || nbatch < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft_relu_grad: bad argument");
  return so3_synthesis((const float2*)x, out, 1, 0, nbatch, b_in, b_out, true, kSo3Real, nullptr, 0,
                       nullptr, 0, as_stream(stream), nullptr, nullptr, act);
}

int s2c_so3_rifft_relu_integrate(const float* x, float* out, long nbatch, int b_in, int b_out,
                                 const float* bias, int nfeature, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || nbatch < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft_relu_integrate: bad argument");
  if (bias && nfeature < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft_relu_integrate: nfeature must be >= 1 with a bias");
  if (!so3_synthesis_is_fused(b_in, b_out))
    return fail(S2C_ERR_UNSUPPORTED, "s2c_so3_rifft_relu_integrate: needs 2 b_out <= 32");
  return so3_synthesis((const float2*)x, nullptr, 1, 0, nbatch, b_in, b_out, false, kSo3Real, bias,
                       nfeature, nullptr, 0, as_stream(stream), nullptr, out);
}

// Largest beta group (a divisor of N whose row stage fits one pass of the block) that keeps three
// blocks of the relay kernel on an SM; failing that, the largest that fits at all (0: none).
static int relay_bg(int N, int Kin, int nrows_in, int nrows_out) {
  int best3 = 0, best = 0;
  for (int d = 1; d <= N && d <= kMaxBG; ++d) {
    if (N % d != 0 || kFusedZG * d * (N / 2) > 256) continue;
    const size_t sm = relay_smem_bytes(N, Kin, nrows_in, nrows_out, d);
    if (sm <= (size_t)dev_smem_limit() - 1024) best = d;
    if (3 * (sm + 1024) <= (size_t)227 * 1024) best3 = d;
  }
  return best3 ? best3 : best;
}

// relay kernel: synthesis at bandwidth b_mid of a spectrum of bandwidth b_in (plain, or the s2_mm
// product of xs and ys when xs is set), + bias, ReLU, analysis to bandwidth b_next
static int relay_launch(const float2* x, const float2* xs, const float2* ys, int s2_nb, int s2_fin, int s2_real,
                        float* out, long nz, int nfeat, int b_in, int b_mid, int b_next,
                        const float* bias, void* ws, size_t ws_bytes, stream_t st, const char* who) {
  const int N = 2 * b_mid;
  if (N > kFusedMaxN || b_next > b_mid || b_in > b_mid)
    return fail(S2C_ERR_UNSUPPORTED,
                std::string(who) + ": needs 2 b <= 32, b_in <= b and b_next <= b");
  const size_t v1 = so3_mid_v_per_z(N, b_in), v2 = so3_mid_v_per_z(N, b_next);
  if (relay_takes_planes(N, b_in, b_next, nz, ws, ws_bytes, xs ? 1 + s2_real : 0)) {
    PanelsDev pin, pout;
    S2C_TRY(TableCache::get().panels(b_mid, b_in, b_in, false, false, pin));
    S2C_TRY(TableCache::get().panels(b_mid, b_next, b_next, true, false, pout));
    const long chunk = std::min(chunk_signals(nz, v1 + v2), (long)(ws_bytes / (v1 + v2)));
    for (long z0 = 0; z0 < nz; z0 += chunk) {
      const long zc = std::min(chunk, nz - z0);
      float2* v = (float2*)ws;
      float2* vo = v + (size_t)zc * (v1 / sizeof(float2));
      InvWignerParams w;
      w.x = xs ? nullptr : x + z0; w.x_zstride = nz; w.s = v; w.pan = pin;
      w.nbatch = (int)zc; w.N = N; w.K = b_in; w.mode = kSo3Real;
      w.xs = xs; w.ys = ys; w.s2_nb = s2_nb; w.s2_fin = s2_fin; w.s2_fout = nfeat; w.s2_real = s2_real; w.z0 = z0;
      S2C_TRY(launch_inv_wigner_col(w, st));
      SmallParams g;
      g.x = nullptr; g.out = nullptr; g.stride = 1; g.off = 0; g.v = v; g.v2 = vo;
      g.bias = bias; g.nfeat = nfeat > 0 ? nfeat : 1; g.z0 = z0; g.mask = nullptr; g.relu = 1;
      g.nplanes = zc * N; g.nz = (int)zc; g.K = b_in; g.K2 = b_next;
      int rc = S2C_OK;
      S2C_DISPATCH_SMALL(N, rc = S2C_LAUNCH_SMALL(so3_relay_small, kN, st, g));
      if (rc) return rc;
      FwdWignerParams f;
      f.v = vo; f.out = (float2*)out + z0; f.out_zstride = nz; f.pan = pout;
      f.nbatch = (int)zc; f.N = N; f.K = b_next; f.nl = b_next; f.mode = kSo3Real;
      S2C_TRY(launch_fwd_wigner_col(f, st));
    }
    return S2C_OK;
  }
  if (so3_prefers_cluster(kClRelay, N, nz)) {
    ClRelayParams f;
    S2C_TRY(TableCache::get().cluster(b_mid, b_in, b_in, false, f.tin));
    S2C_TRY(TableCache::get().cluster(b_mid, b_next, b_next, true, f.tout));
    f.in.x = x; f.in.x_zstride = nz; f.in.mode = xs ? kS2Product : kSo3Real;
    f.in.xs = xs; f.in.ys = ys;
    f.in.s2_nb = s2_nb; f.in.s2_fin = s2_fin; f.in.s2_fout = nfeat; f.in.s2_real = s2_real;
    f.bias = bias; f.nfeat = nfeat > 0 ? nfeat : 1;
    f.out = (float2*)out; f.out_zstride = nz;
    f.nbatch = (int)nz; f.Kin = b_in; f.Kout = b_next;
    int rc = S2C_OK;
    S2C_DISPATCH_N(N, rc = S2C_LAUNCH_CL(so3_relay_cl, kN, (nz + kFusedZG - 1) / kFusedZG,
                                         cl_smem_bytes(N, std::max(b_in, b_next), f.tin.max_rows), st, f));
    return rc;
  }
  FftDev fft;
  RelayParams f;
  S2C_TRY(TableCache::get().fft(N, fft));
  S2C_TRY(TableCache::get().panels(b_mid, b_in, b_in, false, false, f.pin));
  S2C_TRY(TableCache::get().panels(b_mid, b_next, b_next, true, false, f.pout));
  f.BG = relay_bg(N, b_in, f.pin.nrows, f.pout.nrows);
  if (f.BG < 1) return fail(S2C_ERR_UNSUPPORTED, std::string(who) + ": shared memory");
  S2C_TRY(TableCache::get().grouped(b_mid, b_in, b_in, false, f.BG, &f.win_g, &f.win_stride));
  S2C_TRY(TableCache::get().grouped(b_mid, b_next, b_next, true, f.BG, &f.wout_g, &f.wout_stride));
  f.x = x; f.x_zstride = nz;
  f.xs = xs; f.ys = ys;
  f.s2_nb = s2_nb; f.s2_fin = s2_fin; f.s2_fout = nfeat; f.s2_real = s2_real;
  f.bias = bias; f.nfeat = nfeat > 0 ? nfeat : 1;
  f.out = (float2*)out; f.out_zstride = nz;
  f.tw = fft.tw;
  f.nbatch = (int)nz; f.Kin = b_in; f.Kout = b_next;
  f.KP = fused_kp(N); f.PS = fused_plane_stride(N, b_in);
  int rc = S2C_OK;
  const long grid = (nz + kFusedZG - 1) / kFusedZG;
  const size_t sm = relay_smem_bytes(N, b_in, f.pin.nrows, f.pout.nrows, f.BG);
  S2C_DISPATCH_N20(N, rc = S2C_LAUNCH_N(so3_relay_fused, kN, grid, 256, sm, st, f));
  return rc;
}

static size_t relay_workspace(long nbatch, int b_in, int b_mid, int b_next, int product) {
  const int N = 2 * b_mid;
  if (nbatch < 1 || b_in < 1 || b_next < 1 || N > kFusedMaxN || b_in > b_mid || b_next > b_mid ||
      !relay_takes_planes(N, b_in, b_next, nbatch, kAnyWorkspace, kAnySize, product))
    return 0;
  const size_t v = so3_mid_v_per_z(N, b_in) + so3_mid_v_per_z(N, b_next);
  return v * (size_t)chunk_signals(nbatch, v);
}
size_t s2c_so3_relay_workspace(long nbatch, int b_in, int b_mid, int b_next) {
  return relay_workspace(nbatch, b_in, b_mid, b_next, 0);
}
size_t s2c_s2_conv_relu_so3_rfft_workspace(int nbatch, int f_out, int b, int b_next) {
  return relay_workspace((long)nbatch * f_out, b, b, b_next, 1);
}

static int s2_relay(int real, const float* xs, const float* ys, float* out, int nbatch, int f_in, int f_out, int b, int b_next,
                    const float* bias, void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b, b_next));
  if (!xs || !ys || !out || nbatch < 1 || f_in < 1 || f_out < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_s2_conv_relu_so3_rfft: bad argument");
  return relay_launch(nullptr, (const float2*)xs, (const float2*)ys, nbatch, f_in, real, out,
                      (long)nbatch * f_out, f_out, b, b, b_next, bias, ws, ws_bytes, as_stream(stream),
                      "s2c_s2_conv_relu_so3_rfft");
}

int s2c_s2_conv_relu_so3_rfft_ws(const float* xs, const float* ys, float* out, int nbatch, int f_in,
                                 int f_out, int b, int b_next, const float* bias, void* ws,
                                 size_t ws_bytes, void* stream) {
  return s2_relay(0, xs, ys, out, nbatch, f_in, f_out, b, b_next, bias, ws, ws_bytes, stream);
}
int s2c_s2_conv_real_relu_so3_rfft(const float* xs, const float* ys, float* out, int nbatch, int f_in, int f_out, int b,
                                   int b_next, const float* bias, void* ws, size_t ws_bytes, void* stream) {
  return s2_relay(1, xs, ys, out, nbatch, f_in, f_out, b, b_next, bias, ws, ws_bytes, stream);
}
int s2c_s2_conv_relu_so3_rfft(const float* xs, const float* ys, float* out, int nbatch, int f_in,
                              int f_out, int b, int b_next, const float* bias, void* stream) {
  return s2c_s2_conv_relu_so3_rfft_ws(xs, ys, out, nbatch, f_in, f_out, b, b_next, bias, nullptr, 0, stream);
}

int s2c_so3_rifft_relu_rfft_ws(const float* x, float* out, long nbatch, int b_in, int b_mid, int b_next,
                               const float* bias, int nfeature, void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_mid));
  S2C_TRY(check_b(b_mid, b_next));
  if (!x || !out || nbatch < 1) return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft_relu_rfft: bad argument");
  if (bias && nfeature < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft_relu_rfft: nfeature must be >= 1 with a bias");
  return relay_launch((const float2*)x, nullptr, nullptr, 0, 0, 0, out, nbatch, bias ? nfeature : 0,
                      b_in, b_mid, b_next, bias, ws, ws_bytes, as_stream(stream), "s2c_so3_rifft_relu_rfft");
}

int s2c_so3_rifft_relu_rfft(const float* x, float* out, long nbatch, int b_in, int b_mid, int b_next,
                            const float* bias, int nfeature, void* stream) {
  return s2c_so3_rifft_relu_rfft_ws(x, out, nbatch, b_in, b_mid, b_next, bias, nfeature, nullptr, 0, stream);
}

// 32 < 2 b < 64: the product is evaluated while the tiled Wigner kernel stages the spectrum (b = 30, 256 signals:
// 74 MB less to write and read)
static bool s2_product_in_wigner(int b) {
  return use_mid_kernels(2 * b) && inv_wigner_t_smem(2 * b, b) <= (size_t)dev_smem_limit() - 1024;
}

static size_t s2_synthesis_workspace(int real, int nbatch, int f_out, int b) {
  if (nbatch < 1 || f_out < 1 || b < 1) return 0;
  const long nz = (long)nbatch * f_out;
  const bool product = so3_synthesis_is_fused(b, b) || s2_product_in_wigner(b);
  const size_t z_bytes = product ? 0 : (size_t)so3_nspec(b) * nz * sizeof(float2);
  return z_bytes + route_workspace(synthesis_route(2 * b, b, nz, kAnyWorkspace, kAnySize, product ? 1 + real : 0), 2 * b, b, nz);
}
size_t s2c_s2_conv_synthesis_workspace(int nbatch, int f_out, int b) { return s2_synthesis_workspace(0, nbatch, f_out, b); }
size_t s2c_s2_conv_real_synthesis_workspace(int nbatch, int f_out, int b) { return s2_synthesis_workspace(1, nbatch, f_out, b); }

static int s2_synthesis(int real, const float* xs, const float* ys, float* out, int nbatch, int f_in, int f_out, int b,
                        const float* bias, void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b, b));
  if (!xs || !ys || !out || nbatch < 1 || f_in < 1 || f_out < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_s2_conv_synthesis: bad argument");
  const long nz = (long)nbatch * f_out;
  if (so3_synthesis_is_fused(b, b)) {
    S2ProductArgs pr;
    pr.xs = (const float2*)xs; pr.ys = (const float2*)ys;
    pr.nb = nbatch; pr.fin = f_in; pr.fout = f_out; pr.real = real;
    return so3_synthesis(nullptr, out, 1, 0, nz, b, b, false, kSo3Real, bias, f_out, ws, ws_bytes,
                         as_stream(stream), &pr);
  }
  // larger bandwidths: product into the head of the workspace, then the general synthesis
  if (s2_product_in_wigner(b)) {
    S2ProductArgs pr;
    pr.xs = (const float2*)xs; pr.ys = (const float2*)ys;
    pr.nb = nbatch; pr.fin = f_in; pr.fout = f_out; pr.real = real;
    return so3_synthesis(nullptr, out, 1, 0, nz, b, b, false, kSo3Real, bias, f_out, ws, ws_bytes,
                         as_stream(stream), &pr);
  }
  const size_t z_bytes = (size_t)so3_nspec(b) * nz * sizeof(float2);
  if (!ws || ws_bytes <= z_bytes)
    return fail(S2C_ERR_WORKSPACE, "s2c_s2_conv_synthesis: workspace too small");
  S2C_TRY(mm_dispatch(false, kMmFwd, xs, ys, (float*)ws, b, nbatch, f_in, f_out, as_stream(stream)));
  return so3_synthesis((const float2*)ws, out, 1, 0, nz, b, b, false, kSo3Real, bias, f_out,
                       (unsigned char*)ws + z_bytes, ws_bytes - z_bytes, as_stream(stream));
}
int s2c_s2_conv_synthesis(const float* xs, const float* ys, float* out, int nbatch, int f_in,
                          int f_out, int b, const float* bias, void* ws, size_t ws_bytes,
                          void* stream) {
  return s2_synthesis(0, xs, ys, out, nbatch, f_in, f_out, b, bias, ws, ws_bytes, stream);
}
int s2c_s2_conv_real_synthesis(const float* xs, const float* ys, float* out, int nbatch, int f_in, int f_out, int b,
                               const float* bias, void* ws, size_t ws_bytes, void* stream) {
  return s2_synthesis(1, xs, ys, out, nbatch, f_in, f_out, b, bias, ws, ws_bytes, stream);
}

int s2c_so3_ifft(const float* x, float* out, long nbatch, int b_in, int b_out, int for_grad,
                 void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || nbatch < 1) return fail(S2C_ERR_BAD_ARG, "s2c_so3_ifft: bad argument");
  // Re(A X) and Im(A X) = Re(A (-i X)) for the complex-linear synthesis A
  S2C_TRY(so3_synthesis((const float2*)x, out, 2, 0, nbatch, b_in, b_out, for_grad != 0, kSo3Real,
                        nullptr, 1, ws, ws_bytes, as_stream(stream)));
  return so3_synthesis((const float2*)x, out, 2, 1, nbatch, b_in, b_out, for_grad != 0, kSo3RotI,
                       nullptr, 1, ws, ws_bytes, as_stream(stream));
}

// ---- S2 transforms -------------------------------------------------------------------------------
size_t s2c_s2_fft_workspace(long nbatch, int b_in, int b_out) {
  if (b_in < 1 || b_out < 1) return 0;
  const int K = std::min(b_in, b_out), N = 2 * std::max(b_in, b_out);
  return s2_ws_per_z(N, K) * (size_t)std::max(1L, nbatch);
}

int s2c_s2_fft(const float* x, int x_is_real, float* out, long nbatch, int b_in, int b_out,
               int for_grad, void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || nbatch < 1) return fail(S2C_ERR_BAD_ARG, "s2c_s2_fft: bad argument");
  if (b_out > b_in) return fail(S2C_ERR_BAD_ARG, "s2c_s2_fft: requires b_out <= b_in");
  stream_t st = as_stream(stream);
  const int N = 2 * b_in, K = b_out;
  FftDev fft;
  S2C_TRY(TableCache::get().fft(N, fft));
  // A real signal with few degrees: one kernel, no scratch (a block reads the whole table of K^2 N
  // values for its signal; from K = 33 on the tiled contraction, which shares panels, is the faster one).
  if (!g_force_general && x_is_real && K <= kS2FusedK && s2_length(N) && N < 128) {
    S2FwdFusedParams f;
    f.x = x; f.out = (float2*)out; f.out_zstride = nbatch;
    f.tw = fft.tw; f.K = K;
    S2C_TRY(TableCache::get().s2_transposed(b_in, b_out, !for_grad, &f.wt));
    return s2_dispatch<1, 64>(N, [&](auto nc) {
      constexpr int kN = decltype(nc)::value;
      return S2C_LAUNCH_N(s2_fwd_fused, kN, nbatch, 256, s2_fwd_fused_smem(kN, K), st, f);
    });
  }
  PanelsDev pan;
  S2C_TRY(TableCache::get().panels(b_in, b_out, K, !for_grad, true, pan));
  const size_t per_z = s2_ws_per_z(N, K);
  long chunk = (long)std::min<size_t>((size_t)nbatch, ws_bytes / per_z);
  if (chunk < 1 || !ws) return fail(S2C_ERR_WORKSPACE, "s2c_s2_fft: workspace too small");
  const int G = fft_group(N, N), Gg = fft_group(N, N / 2);  // alpha passes, gamma passes
  for (long z0 = 0; z0 < nbatch; z0 += chunk) {
    const long zc = std::min(chunk, nbatch - z0);
    // A real signal's coefficients of m < 0 mirror those of m > 0.  Up to 32 degrees both are computed, also in calls that
    // would gain from the half: not by speed but because a change of bits there reaches the recorded passes of nearly all
    // layers (see SpectralMm in host_ops.cpp), and this call does not know whether it is recorded.  192 signals, b = 64,
    // analysis and synthesis: 48 -> 35 us and 43 -> 34; 512: 101 -> 65 and 81 -> 62.
    const int ht = wig_s2_zt(K, zc);
    const bool half = x_is_real && K > 32 && !g_force_general && s2_length(N) &&
                      fwd_wigner_t_fits(N, b_out, ht, dev_smem_limit());
    if (!g_force_general && s2_length(N)) {
      S2RowsParams r;
      r.half = half;
      r.x = x + (size_t)z0 * N * N * (x_is_real ? 1 : 2); r.out = nullptr;
      r.complex = !x_is_real; r.v = (float2*)ws; r.tw = fft.tw;
      r.nbatch = (int)zc; r.K = K;
      S2C_TRY((s2_dispatch<1, 64>(N, [&](auto nc) {
        constexpr int kN = decltype(nc)::value;
        return S2C_LAUNCH_N(s2_fwd_rows, kN, zc * s2_rows_groups(kN), 256, s2_fwd_rows_smem(kN), st, r);
      })));
    } else {
    FwdAlphaParams a;
    a.in = x + (size_t)z0 * N * N * (x_is_real ? 1 : 2);
    a.in_real = x_is_real ? 1 : 0;
    a.v = (float2*)ws;
    a.nbatch = (int)zc; a.N = N; a.K = K; a.Kn = 1; a.G = G;
    a.nrows = zc * N;
    a.fft = fft;
    S2C_TRY(S2C_LAUNCH(so3_fwd_alpha, (a.nrows + G - 1) / G, kThreads, fft_smem_bytes(N, G), st, a));
    }
    FwdWignerParams w;
    w.v = (const float2*)ws;
    w.out = (float2*)out + z0;
    w.out_zstride = nbatch;
    w.pan = pan;
    w.nbatch = (int)zc; w.N = N; w.K = K; w.nl = b_out;
    w.ZT = (int)std::min<long>(32, zc);
    w.nzt = (int)((zc + w.ZT - 1) / w.ZT);
    w.mode = kS2;
    if (const int zt = half ? ht : wig_s2_zt(pan.npairs, zc); fwd_wigner_t_fits(N, b_out, zt, dev_smem_limit())) {
      w.ZT = zt;
      w.nzt = (int)((zc + zt - 1) / zt);
      const size_t wsm = fwd_wigner_t_smem(N, b_out, zt);
      if (half) S2C_TRY(S2C_LAUNCH(s2_fwd_wigner_t_half, (long)K * w.nzt, kThreads, wsm, st, w));
      else S2C_TRY(S2C_LAUNCH(so3_fwd_wigner_t, (long)pan.npairs * w.nzt, kThreads, wsm, st, w));
      continue;
    }
    const size_t wsm = align_up((size_t)b_out * (N + 1) * sizeof(float), 16) +
                       (size_t)w.ZT * (N + 1) * sizeof(float2);
    S2C_TRY(S2C_LAUNCH(so3_fwd_wigner, (long)pan.npairs * w.nzt, kThreads, wsm, st, w));
  }
  return S2C_OK;
}

int s2c_s2_ifft(const float* x, float* out, int out_is_real, long nbatch, int b_in, int b_out,
                int for_grad, void* ws, size_t ws_bytes, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || nbatch < 1) return fail(S2C_ERR_BAD_ARG, "s2c_s2_ifft: bad argument");
  if (b_out < b_in) return fail(S2C_ERR_BAD_ARG, "s2c_s2_ifft: requires b_out >= b_in");
  stream_t st = as_stream(stream);
  const int N = 2 * b_out, K = b_in;
  FftDev fft;
  PanelsDev pan;
  S2C_TRY(TableCache::get().fft(N, fft));
  S2C_TRY(TableCache::get().panels(b_out, b_in, K, for_grad != 0, true, pan));
  const size_t per_z = s2_ws_per_z(N, K);
  long chunk = (long)std::min<size_t>((size_t)nbatch, ws_bytes / per_z);
  if (chunk < 1 || !ws) return fail(S2C_ERR_WORKSPACE, "s2c_s2_ifft: workspace too small");
  const int G = fft_group(N, N), Gg = fft_group(N, N / 2);  // alpha passes, gamma passes
  for (long z0 = 0; z0 < nbatch; z0 += chunk) {
    const long zc = std::min(chunk, nbatch - z0);
    InvWignerParams w;
    w.x = (const float2*)x + z0;
    w.x_zstride = nbatch;
    w.s = (float2*)ws;
    w.pan = pan;
    w.nbatch = (int)zc; w.N = N; w.K = K;
    w.ZT = (int)std::min<long>(32, zc);
    w.nzt = (int)((zc + w.ZT - 1) / w.ZT);
    w.mode = kS2;
    // the real part alone: the spectrum is symmetrised while it is staged, and V[-m] = conj V[m]
    const int ht = wig_s2_zt(K, zc);
    const bool half = out_is_real && !g_force_general && s2_length(N) && inv_wigner_t_smem(N, K, ht) <= (size_t)dev_smem_limit() - 1024;
    if (const int zt = half ? ht : wig_s2_zt(pan.npairs, zc); inv_wigner_t_smem(N, K, zt) <= (size_t)dev_smem_limit() - 1024) {
      w.ZT = zt;
      w.nzt = (int)((zc + zt - 1) / zt);
      const size_t wsm = inv_wigner_t_smem(N, K, zt);
      if (half) S2C_TRY(S2C_LAUNCH(s2_inv_wigner_t_half, (long)K * w.nzt, kThreads, wsm, st, w));
      else S2C_TRY(S2C_LAUNCH(so3_inv_wigner_t, (long)pan.npairs * w.nzt, kThreads, wsm, st, w));
    } else {
      const size_t wsm = align_up((size_t)K * N * sizeof(float), 16) + (size_t)K * w.ZT * sizeof(float2);
      S2C_TRY(S2C_LAUNCH(so3_inv_wigner, (long)pan.npairs * w.nzt, kThreads, wsm, st, w));
    }
    if (!g_force_general && s2_length(N)) {
      S2RowsParams r;
      r.half = half;
      r.x = nullptr; r.out = out + (size_t)z0 * N * N * (out_is_real ? 1 : 2);
      r.complex = !out_is_real; r.v = (float2*)ws; r.tw = fft.tw;
      r.nbatch = (int)zc; r.K = K;
      S2C_TRY((s2_dispatch<1, 64>(N, [&](auto nc) {
        constexpr int kN = decltype(nc)::value;
        return S2C_LAUNCH_N(s2_inv_rows, kN, zc * s2_rows_groups(kN), 256, s2_inv_rows_smem(kN), st, r);
      })));
      continue;
    }
    InvAlphaParams a;
    a.s = (const float2*)ws;
    a.out = out + (size_t)z0 * N * N * (out_is_real ? 1 : 2);
    a.out_real = out_is_real ? 1 : 0;
    a.herm_n0 = 0;
    a.nbatch = (int)zc; a.N = N; a.K = K; a.Kn = 1; a.G = G;
    a.nrows = zc * N;
    a.fft = fft;
    S2C_TRY(S2C_LAUNCH(so3_inv_alpha, (a.nrows + G - 1) / G, kThreads, fft_smem_bytes(N, G), st, a));
  }
  return S2C_OK;
}

// ---- spectral products ---------------------------------------------------------------------------
#ifndef S2C_EMUL
static __device__ int g_tc_err_flag;
// its address on the current device, looked up once per device
static int tc_err_flag(int** out) {
  static std::atomic<int*> known[kMaxDevices];
  const int dev = dev_current();
  int* p = dev < kMaxDevices ? known[dev].load(std::memory_order_relaxed) : nullptr;
  if (!p) {
    void* q = nullptr;
    S2C_TRY(cuda_check(cudaGetSymbolAddress(&q, g_tc_err_flag), "tensor-core status flag"));
    p = (int*)q;
    if (dev < kMaxDevices) known[dev].store(p, std::memory_order_relaxed);
  }
  *out = p;
  return S2C_OK;
}
#endif

#ifndef S2C_EMUL
// blocks of the contraction: `run` floats per outer index
static void tc_blocks(MmTcParams& p) {
  if (p.run <= kTcKMax) { p.kblk = (p.run + 7) / 8 * 8; p.nblk = 1; }
  else { p.kblk = kTcKMax; p.nblk = (p.run + kTcKMax - 1) / kTcKMax; }
}
// whether the longest of the ns CTAs of a tile of `blocks` K blocks issues more MMAs than one accumulator may take
static bool tc_flush(const MmTcParams& p, long blocks, int ns) {
  if (ns == 1) return 3 * (blocks / p.nblk) * ((p.run + 7) / 8) > kTcChainMax;
  return 3 * ((blocks + ns - 1) / ns) * (p.kblk / 8) > kTcChainMax;
}
static int tc_run(int op, int nb, int fi, int fo) { return 2 * (op == kTcFwd ? fi : op == kTcGradX ? fo : nb); }
// CTAs per tile; several clusters to a tile only with the workspace they meet in
static int tc_share(MmTcParams& p, int op, long tiles, void* ws, size_t ws_bytes, stream_t st) {
  TcShare s = tc_pick_share(op, p.half, p.nl, p.nb, p.fi, p.fo, p.nblk, true);
  if (s.groups > 1 && (!ws || (uintptr_t)ws % 16 != 0 || ws_bytes < tc_share_bytes(tiles, s.groups)))
    s = tc_pick_share(op, p.half, p.nl, p.nb, p.fi, p.fo, p.nblk, false);
  p.csize = s.csize; p.groups = s.groups;
  if (s.groups == 1) return S2C_OK;
  p.count = (int*)ws;
  p.part = (float*)((unsigned char*)ws + tc_count_bytes(tiles));
  return cuda_check(cudaMemsetAsync(ws, 0, tc_count_bytes(tiles), st), "counters of the shared tiles");
}
static size_t tc_share_workspace(int op, int half, int nl, int nb, int fi, int fo, int run) {
  if (g_force_general) return 0;
  MmTcParams p;
  p.run = run;
  tc_blocks(p);
  return tc_share_bytes(so3_mm_tc_tiles(op, half, nl, nb, fi, fo),
                        tc_pick_share(op, half, nl, nb, fi, fo, p.nblk, true).groups);
}
// so3_mm or one of its gradients on the tensor cores, `half` of it where the operands are spectra of real signals;
// `handled` tells whether the shape qualified.
static int so3_mm_tc_launch(int op, int half, const float* a, const float* b, float* c, int nl, int nb, int fi,
                            int fo, void* ws, size_t ws_bytes, stream_t st, bool* handled) {
  *handled = !g_force_general;
  if (!*handled) return S2C_OK;
  MmTcParams p;
  p.a = a; p.b = b; p.c = c;
  p.nl = nl; p.nb = nb; p.fi = fi; p.fo = fo; p.half = half;
  p.run = tc_run(op, nb, fi, fo);
  tc_blocks(p);
  S2C_TRY(tc_err_flag(&p.err));
  const long tiles = so3_mm_tc_tiles(op, half, nl, nb, fi, fo);
  p.csize = p.groups = 1;
  p.part = nullptr; p.count = nullptr;
  // The rounding of a forward product is the same whatever the batch: one CTA per tile, or segments
  if (op != kTcFwd) S2C_TRY(tc_share(p, op, tiles, ws, ws_bytes, st));
  const int blocks = (2 * nl - 1) * p.nblk;
  p.segs = op == kTcFwd && half ? tc_segments(nl, fi, fo, blocks) : 0;
  if (p.segs > 1 && tiles <= kTcSlots[p.segs]) p.csize = p.segs;
  const int ns = p.csize * p.groups;
  p.twins = tc_twins(half, tiles, ns);
  const long ctas = tiles * (p.twins ? 2 : ns);
  const bool flush = p.segs > 1 ? ns == 1 : tc_flush(p, blocks, ns);
  p.two = half && p.segs <= 1;
  const bool vec = so3_mm_tc_vec16(op, nb, fi, fo);
  if (op == kTcFwd) return launch_so3_mm_tc<kTcFwd>("so3_mm_tc_kernel", ctas, flush, vec, st, p);
  if (op == kTcGradX) return launch_so3_mm_tc<kTcGradX>("so3_mm_tc_gradx", ctas, flush, vec, st, p);
  return launch_so3_mm_tc<kTcGradY>("so3_mm_tc_grady", ctas, flush, vec, st, p);
}

// A plain real product C[r][c] = sum_k A[r][k] B[c][k] (M rows, N columns, K terms; N and K even)
// on the tensor-core pipeline: the kernel-grid -> spectrum transforms and their transposes.
static int plain_tc_launch(bool a_strided, const float* a, const float* b, float* c, long M, long N,
                           long K, long a_rs, long a_ps, long b_rs, long b_ps, long c_rs, long c_ps,
                           float scale, void* ws, size_t ws_bytes, stream_t st) {
  MmTcParams p;
  p.a = a; p.b = b; p.c = c;
  p.nl = 1; p.nb = (int)M; p.fi = (int)(K / 2); p.fo = (int)(N / 2); p.half = p.two = p.segs = p.twins = 0;
  p.run = (int)K;
  tc_blocks(p);
  p.a_rs = a_rs; p.a_ps = a_ps; p.b_rs = b_rs; p.b_ps = b_ps; p.c_rs = c_rs; p.c_ps = c_ps;
  p.scale = scale;
  S2C_TRY(tc_err_flag(&p.err));
  // (one degree, l = 0, with M rows and N columns in the spectral geometry; the forward transform has a
  // short contraction and is not split)
  const long tiles = so3_mm_tc_tiles(kTcPlainSC, 0, 1, (int)M, p.fi, p.fo);
  p.csize = p.groups = 1;
  p.part = nullptr; p.count = nullptr;
  if (a_strided) S2C_TRY(tc_share(p, kTcPlainSC, tiles, ws, ws_bytes, st));
  const int ns = p.csize * p.groups;
  const long ctas = tiles * ns;
  const bool flush = tc_flush(p, p.nblk, ns);
  // 16-byte loads need K a multiple of 4 and 16-byte aligned rows of every contiguous operand
  const bool vec = K % 4 == 0 && b_rs % 4 == 0 && (a_strided || a_rs % 4 == 0);
  if (a_strided) return launch_so3_mm_tc<kTcPlainSC>("rft_tc_backward", ctas, flush, vec, st, p);
  return launch_so3_mm_tc<kTcPlainCC>("rft_tc_forward", ctas, flush, vec, st, p);
}
#endif

int s2c_so3_mm(const float* x, const float* y, float* z, int nl, int nb, int fi, int fo, void* st) {
  if (!x || !y || !z) return fail(S2C_ERR_BAD_ARG, "s2c_so3_mm: null pointer");
  if (nl < 1 || nb < 1 || fi < 1 || fo < 1) return fail(S2C_ERR_BAD_ARG, "sizes must be >= 1");
#ifndef S2C_EMUL
  bool handled = false;
  S2C_TRY(so3_mm_tc_launch(kTcFwd, 0, x, y, z, nl, nb, fi, fo, nullptr, 0, as_stream(st), &handled));
  if (handled) return S2C_OK;
#endif
  return mm_dispatch(true, kMmFwd, x, y, z, nl, nb, fi, fo, as_stream(st));
}

int s2c_so3_mm_tc_status(void) {
#ifndef S2C_EMUL
  // wait for every stream of the device (the products run on the caller's streams, which a plain
  // copy from the symbol would not be ordered after), then read the flag
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc_err_flag, sizeof(int)) != cudaSuccess) return -1;
  return v;
#else
  return 0;
#endif
}
size_t s2c_so3_mm_gradx_workspace(int nl, int nb, int fi, int fo) {
#ifndef S2C_EMUL
  if (nl >= 1 && nb >= 1 && fi >= 1 && fo >= 1)
    return tc_share_workspace(kTcGradX, 0, nl, nb, fi, fo, tc_run(kTcGradX, nb, fi, fo));
#endif
  return 0;
}
int s2c_so3_mm_gradx_ws(const float* gz, const float* y, float* gx, int nl, int nb, int fi, int fo, void* ws,
                        size_t ws_bytes, void* st) {
  if (!gz || !y || !gx) return fail(S2C_ERR_BAD_ARG, "s2c_so3_mm_gradx: null pointer");
  if (nl < 1 || nb < 1 || fi < 1 || fo < 1) return fail(S2C_ERR_BAD_ARG, "sizes must be >= 1");
#ifndef S2C_EMUL
  bool handled = false;
  S2C_TRY(so3_mm_tc_launch(kTcGradX, 0, gz, y, gx, nl, nb, fi, fo, ws, ws_bytes, as_stream(st), &handled));
  if (handled) return S2C_OK;
#endif
  return mm_dispatch(true, kMmGradX, gz, y, gx, nl, nb, fi, fo, as_stream(st));
}
int s2c_so3_mm_gradx(const float* gz, const float* y, float* gx, int nl, int nb, int fi, int fo, void* st) {
  return s2c_so3_mm_gradx_ws(gz, y, gx, nl, nb, fi, fo, nullptr, 0, st);
}
size_t s2c_so3_mm_grady_workspace(int nl, int nb, int fi, int fo) {
#ifndef S2C_EMUL
  if (nl >= 1 && nb >= 1 && fi >= 1 && fo >= 1)
    return tc_share_workspace(kTcGradY, 0, nl, nb, fi, fo, tc_run(kTcGradY, nb, fi, fo));
#endif
  return 0;
}
int s2c_so3_mm_grady_ws(const float* gz, const float* x, float* gy, int nl, int nb, int fi, int fo, void* ws,
                        size_t ws_bytes, void* st) {
  if (!gz || !x || !gy) return fail(S2C_ERR_BAD_ARG, "s2c_so3_mm_grady: null pointer");
  if (nl < 1 || nb < 1 || fi < 1 || fo < 1) return fail(S2C_ERR_BAD_ARG, "sizes must be >= 1");
#ifndef S2C_EMUL
  bool handled = false;
  S2C_TRY(so3_mm_tc_launch(kTcGradY, 0, x, gz, gy, nl, nb, fi, fo, ws, ws_bytes, as_stream(st), &handled));
  if (handled) return S2C_OK;
#endif
  return mm_dispatch(true, kMmGradY, x, gz, gy, nl, nb, fi, fo, as_stream(st));
}
int s2c_so3_mm_grady(const float* gz, const float* x, float* gy, int nl, int nb, int fi, int fo, void* st) {
  return s2c_so3_mm_grady_ws(gz, x, gy, nl, nb, fi, fo, nullptr, 0, st);
}
// Products of spectra of real signals.  X[l,-m,-n] = (-1)^(m-n) conj X[l,m,n] holds for the operands and so for the
// result: the tensor cores compute the columns (z) or rows (gradients) of outer index l .. 2l, half
// of the multiply-adds, and write each coefficient and its mirror.  us on one B200, all rows -> half, for z, gx
// and gy: 100 -> 100 channels, nl = 10, batch 32: 314, 325, 314 -> 199, 211, 203; 16 -> 16, nl = 15, batch 32: 77, 80, 65 -> 49,
// 52, 51; 20 -> 40, nl = 6, batch 256: 42, 50, 52 -> 32, 33, 36; 8 -> 16, nl = 15, batch 32: z 41 -> 28 (half of the rows: 32).
// Calls whose tiles all run at once take the time they took, or up to 3 us more (tc_twins); so do kernel gradients of one to four
// signals (24 -> 46, nl = 8: 13.2 -> 16.5).
size_t s2c_so3_mm_real_workspace(int op, int nl, int nb, int fi, int fo) {
#ifndef S2C_EMUL
  if ((op == kTcGradX || op == kTcGradY) && nl >= 1 && nb >= 1 && fi >= 1 && fo >= 1)
    return tc_share_workspace(op, kTcHalfRows, nl, nb, fi, fo, tc_run(op, nb, fi, fo));
#endif
  return 0;
}
int s2c_so3_mm_real(int op, const float* u, const float* v, float* out, int nl, int nb, int fi, int fo, void* ws,
                    size_t ws_bytes, void* st) {
  if (op < 0 || op > 2) return fail(S2C_ERR_BAD_ARG, "s2c_so3_mm_real: op is 0, 1 or 2");
  if (!u || !v || !out) return fail(S2C_ERR_BAD_ARG, "s2c_so3_mm_real: null pointer");
  if (nl < 1 || nb < 1 || fi < 1 || fo < 1) return fail(S2C_ERR_BAD_ARG, "sizes must be >= 1");
  const float *a = op == 2 ? v : u, *b = op == 2 ? u : v;     // the gradient of y: rows from x
#ifndef S2C_EMUL
  static_assert((int)kTcFwd == 0 && (int)kTcGradX == 1 && (int)kTcGradY == 2, "op codes");
  bool handled = false;
  S2C_TRY(so3_mm_tc_launch(op, op == kTcFwd ? kTcHalfColumns : kTcHalfRows, a, b, out, nl, nb, fi, fo, ws, ws_bytes, as_stream(st), &handled));
  if (handled) return S2C_OK;
#endif
  static_assert(kMmFwd == 0 && kMmGradX == 1 && kMmGradY == 2, "op codes");
  return mm_dispatch(true, op, a, b, out, nl, nb, fi, fo, as_stream(st));
}
int s2c_s2_mm(const float* x, const float* y, float* z, int nl, int nb, int fi, int fo, void* st) {
  if (!x || !y || !z) return fail(S2C_ERR_BAD_ARG, "s2c_s2_mm: null pointer");
  return mm_dispatch(false, kMmFwd, x, y, z, nl, nb, fi, fo, as_stream(st));
}
static int s2_mm_gradx_any(int real, const float* gz, const float* y, float* gx, int nl, int nb, int fi, int fo, void* st) {
  if (!gz || !y || !gx) return fail(S2C_ERR_BAD_ARG, "s2c_s2_mm_gradx: null pointer");
  if (nl < 1 || nb < 1 || fi < 1 || fo < 1) return fail(S2C_ERR_BAD_ARG, "sizes must be >= 1");
  if (!g_force_general && s2_mm_thin_supported(nl, fi, fo)) {
    S2ThinParams p;
    p.gz = (const float2*)gz; p.other = (const float2*)y; p.out = (float2*)gx;
    p.nl = nl; p.nb = nb; p.fi = fi; p.fo = fo; p.real = real;
    const long blocks = (long)thin_rows(nl, real) * ((nb + kThinRows - 1) / kThinRows);
    return S2C_LAUNCH(s2_mm_gradx_thin, blocks, kThinRows * kThinSlices,
                      s2_gradx_thin_smem(nl, fi, fo), as_stream(st), p);
  }
  return mm_dispatch(false, kMmGradX, gz, y, gx, nl, nb, fi, fo, as_stream(st));
}
static int s2_mm_grady_any(int real, const float* gz, const float* x, float* gy, int nl, int nb, int fi, int fo, void* st) {
  if (!gz || !x || !gy) return fail(S2C_ERR_BAD_ARG, "s2c_s2_mm_grady: null pointer");
  if (nl < 1 || nb < 1 || fi < 1 || fo < 1) return fail(S2C_ERR_BAD_ARG, "sizes must be >= 1");
  if (!g_force_general && s2_mm_thin_supported(nl, fi, fo)) {
    S2ThinParams p;
    p.gz = (const float2*)gz; p.other = (const float2*)x; p.out = (float2*)gy;
    p.nl = nl; p.nb = nb; p.fi = fi; p.fo = fo; p.real = real;
    return S2C_LAUNCH(s2_mm_grady_thin, (long)thin_rows(nl, real), s2_grady_thin_threads(fo),
                      s2_grady_thin_smem(fo), as_stream(st), p);
  }
  return mm_dispatch(false, kMmGradY, x, gz, gy, nl, nb, fi, fo, as_stream(st));
}
int s2c_s2_mm_gradx(const float* gz, const float* y, float* gx, int nl, int nb, int fi, int fo, void* st) {
  return s2_mm_gradx_any(0, gz, y, gx, nl, nb, fi, fo, st);
}
int s2c_s2_mm_grady(const float* gz, const float* x, float* gy, int nl, int nb, int fi, int fo, void* st) {
  return s2_mm_grady_any(0, gz, x, gy, nl, nb, fi, fo, st);
}
// Spectra of real signals: half of the result's rows, the others mirrored, and half of gz read.  Gradient of y, all rows ->
// half, 6 -> 100 channels, nl = 16, batch 32: 77 -> 52 us; 1 -> 8, nl = 30, batch 32: 48 -> 27; of x: 278 -> 179, 25 -> 17.
int s2c_s2_mm_real_gradx(const float* gz, const float* y, float* gx, int nl, int nb, int fi, int fo, void* st) {
  return s2_mm_gradx_any(1, gz, y, gx, nl, nb, fi, fo, st);
}
int s2c_s2_mm_real_grady(const float* gz, const float* x, float* gy, int nl, int nb, int fi, int fo, void* st) {
  return s2_mm_grady_any(1, gz, x, gy, nl, nb, fi, fo, st);
}

// ---- kernel-grid -> spectrum -----------------------------------------------------------------------
static int rft_forward_any(const float* x, const float* F, const float* Ft, float* out, int nf, int ng,
                            int ns, float scale, stream_t st) {
#ifndef S2C_EMUL
  if (Ft && ng % 2 == 0)
    // C[f][(s, c)] = sum_a (scale x[f][a]) Ft[(s, c)][a], written to out[s][f][c]
    return plain_tc_launch(false, x, Ft, out, nf, 2L * ns, ng, ng, 2, ng, 2, 2, 2L * nf, scale, nullptr, 0, st);
#endif
  if (!F) return fail(S2C_ERR_UNSUPPORTED, "rft with the transposed matrix: needs the CUDA build and an even n_grid");
  RftFwdParams p;
  p.x = x; p.F = (const float2*)F; p.out = (float2*)out;
  p.nf = nf; p.ng = ng; p.ns = ns; p.scale = scale;
  p.tiles_f = (nf + kRftTF - 1) / kRftTF;
  const long tiles_s = (ns + kRftTS - 1) / kRftTS;
  const size_t sm = kRftTF * (kRftTA + 1) * 4 + kRftTA * kRftTS * 8;
  return S2C_LAUNCH(rft_forward, p.tiles_f * tiles_s, 256, sm, st, p);
}

int s2c_rft_forward(const float* x, const float* F, float* out, int nf, int ng, int ns, void* st) {
  if (!x || !F || !out || nf < 1 || ng < 1 || ns < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_rft_forward: bad argument");
  return rft_forward_any(x, F, nullptr, out, nf, ng, ns, 1.f, as_stream(st));
}

int s2c_rft_forward_t(const float* x, const float* Ft, float* out, int nf, int ng, int ns, void* st) {
  if (!x || !Ft || !out || nf < 1 || ng < 1 || ns < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_rft_forward_t: bad argument");
  return rft_forward_any(x, nullptr, Ft, out, nf, ng, ns, 1.f, as_stream(st));
}

int s2c_rft_forward_scaled(const float* x, const float* F, const float* Ft, float* out, int nf, int ng,
                           int ns, float scale, void* st) {
  if (!x || !F || !out || nf < 1 || ng < 1 || ns < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_rft_forward_scaled: bad argument");
  return rft_forward_any(x, F, Ft, out, nf, ng, ns, scale, as_stream(st));
}

size_t s2c_rft_backward_workspace(int nf, int ng, int ns) {
#ifndef S2C_EMUL
  if (nf >= 1 && ng >= 1 && ns >= 1 && ng % 2 == 0) return tc_share_workspace(kTcPlainSC, 0, 1, nf, ns, ng / 2, 2 * ns);
#endif
  return 0;
}
int s2c_rft_backward_scaled(const float* g, const float* F, float* gx, int nf, int ng, int ns, float scale, void* ws,
                            size_t ws_bytes, void* st) {
  if (!g || !F || !gx || nf < 1 || ng < 1 || ns < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_rft_backward: bad argument");
#ifndef S2C_EMUL
  if (!g_force_general && ng % 2 == 0) {
    // gx[f][a] = scale sum_{(s, c)} g[s][f][c] F[a][(s, c)]: the row operand holds k = (s, c) as pairs
    // 2 nf floats apart
    return plain_tc_launch(true, g, F, gx, nf, ng, 2L * ns, 2, 2L * nf, 2L * ns, 2, ng, 2, scale, ws, ws_bytes,
                           as_stream(st));
  }
#endif
  RftBwdParams p;
  p.g = (const float2*)g; p.F = (const float2*)F; p.gx = gx;
  p.nf = nf; p.ng = ng; p.ns = ns; p.scale = scale;
  p.tiles_f = (nf + kRftTF - 1) / kRftTF;
  const long tiles_a = (ng + kRftTA - 1) / kRftTA;
  const size_t sm = kRftTS * kRftTF * 8 + kRftTA * (kRftTS + 1) * 8;
  return S2C_LAUNCH(rft_backward, p.tiles_f * tiles_a, 256, sm, as_stream(st), p);
}
int s2c_rft_backward(const float* g, const float* F, float* gx, int nf, int ng, int ns, void* st) {
  return s2c_rft_backward_scaled(g, F, gx, nf, ng, ns, 1.f, nullptr, 0, st);
}

// ---- integration ---------------------------------------------------------------------------------
int s2c_so3_integrate(const float* x, float* out, long n, int b, int relu, void* st) {
  if (!x || !out || n < 1 || b < 1) return fail(S2C_ERR_BAD_ARG, "s2c_so3_integrate: bad argument");
  IntegrateParams p;
  p.x = x; p.out = out; p.n = n; p.N = 2 * b; p.relu = relu;
  S2C_TRY(TableCache::get().quad_weights(b, &p.w));
  return S2C_LAUNCH(so3_integrate_fwd, (n + kIntegrateWarps - 1) / kIntegrateWarps,
                    32 * kIntegrateWarps, 32 * kIntegrateWarps * sizeof(float), as_stream(st), p);
}

int s2c_so3_integrate_backward(const float* g, const float* x, float* gx, long n, int b, int relu,
                               void* st) {
  if (!g || !gx || n < 1 || b < 1 || (relu && !x))
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_integrate_backward: bad argument");
  IntegrateBwdParams p;
  p.g = g; p.x = x; p.gx = gx; p.N = 2 * b; p.relu = relu;
  p.total = n * (long)p.N * p.N * p.N;
  S2C_TRY(TableCache::get().quad_weights(b, &p.w));
  const long blocks = std::min<long>((p.total + 255) / 256, 148L * 16);
  return S2C_LAUNCH(so3_integrate_bwd, blocks, 256, 0, as_stream(st), p);
}

int s2c_project_on_sphere(const float* verts, int nv, const int* faces, int nf, const float* grid,
                          int nr, float* out, void* st) {
  if (!verts || !faces || !grid || !out || nv < 1 || nf < 1 || nr < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_project_on_sphere: bad argument");
  ProjectParams p;
  p.verts = verts; p.faces = faces; p.grid = grid; p.out = out;
  p.nv = nv; p.nf = nf; p.nr = nr;
  return S2C_LAUNCH(project_on_sphere, (nr + kProjThreads - 1) / kProjThreads, kProjThreads,
                    kProjTile * 12 * sizeof(float), as_stream(st), p);
}

int s2c_so3_rotation_matrices(int b, double alpha, double beta, double gamma, float* out) {
  if (b < 1 || !out) return fail(S2C_ERR_BAD_ARG, "s2c_so3_rotation_matrices: bad argument");
  std::vector<double> col(b + 1);
  for (int m = -(b - 1); m <= b - 1; ++m)
    for (int n = -(b - 1); n <= b - 1; ++n) {
      const int l0 = wigner_d_degrees(m, n, beta, b, col.data());
      const double ph = m * alpha + n * gamma;
      const double cr = std::cos(ph), ci = std::sin(ph);
      for (int l = l0; l < b; ++l) {
        const long idx = so3_offset(l) + (long)(m + l) * (2 * l + 1) + (n + l);
        out[2 * idx] = (float)(cr * col[l - l0]);
        out[2 * idx + 1] = (float)(ci * col[l - l0]);
      }
    }
  return S2C_OK;
}

int s2c_so3_rotate_spectrum(const float* U, const float* x, float* z, int b, long nbatch,
                            int adjoint, void* st) {
  if (!U || !x || !z || b < 1 || nbatch < 1 || nbatch > 0x7fffffffL / (2 * b))
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_rotate_spectrum: bad argument");
  RotateParams p;
  p.U = (const float2*)U; p.x = (const float2*)x; p.z = (float2*)z;
  p.nl = b; p.adjoint = adjoint != 0; p.nbatch = nbatch;
  return S2C_LAUNCH(so3_rotate_rows, rot_blocks(b, nbatch), kRotThreads, rot_smem_bytes(b), as_stream(st), p);
}


}  // extern "C"

// ================================================================================================
// s2c_so3_rifft_static: the SO(3) synthesis without any device allocation.
//
// Some callers of this library cannot obtain device memory at call time: a serving process whose
// whole GPU is pre-reserved by another allocator at start-up (a later cudaMalloc simply fails), or
// a control loop that must not take the device-wide synchronisation a cudaMalloc/cudaFree implies.
// For them the scratch arrays of the synthesis and the constant tables it reads live in the two
// file-scope device arrays below, which every GPU that loads this library holds until the process
// exits (kStaticScratchBytes + kStaticTableBytes = 36 MiB per GPU).
//
// In host code the array names are host-side stand-ins, not device addresses; the device address
// is fetched once per device with cudaGetSymbolAddress (with that device current) and handed to
// the kernels.  That set-up, and the (synchronous) upload of the tables for the requested
// bandwidths, happen on the first call on a device and again whenever a call asks for different
// bandwidths / weighting than the tables currently held - make such a call before any stream
// capture.  All calls on a device share the arrays: the scratch keeps the previous call's
// contents (every element a pass reads has been written by the pass before it in the same call,
// so nothing needs clearing), and two calls that overlap on the GPU - different streams or host
// threads - race on it.
// ================================================================================================
namespace s2c {

constexpr size_t kStaticScratchBytes = (size_t)32 << 20;
constexpr size_t kStaticTableBytes = (size_t)4 << 20;

#ifndef S2C_EMUL
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
static __device__ __align__(256) unsigned char g_static_tables[kStaticTableBytes];
#else
alignas(256) static unsigned char g_static_scratch[kStaticScratchBytes];
alignas(256) static unsigned char g_static_tables[kStaticTableBytes];
#endif

struct StaticDeviceState {
  bool ready = false;
  unsigned char* scratch = nullptr;  // device addresses of the two arrays on this device
  unsigned char* tables = nullptr;
  int b_beta = -1, K = -1, weighted = -1;  // configuration the table array currently holds
  FftDev fft;
  PanelsDev pan;
};

static std::mutex g_static_mu;
static std::map<int, StaticDeviceState> g_static_state;

static int static_setup(StaticDeviceState& st) {
  if (st.ready) return S2C_OK;
#ifndef S2C_EMUL
  void* p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
  if (e != cudaSuccess) return cuda_check(e, "cudaGetSymbolAddress(scratch)");
  st.scratch = (unsigned char*)p;
  e = cudaGetSymbolAddress(&p, g_static_tables);
  if (e != cudaSuccess) return cuda_check(e, "cudaGetSymbolAddress(tables)");
  st.tables = (unsigned char*)p;
#else
  st.scratch = g_static_scratch;
  st.tables = g_static_tables;
#endif
  st.ready = true;
  return S2C_OK;
}

// Builds the FFT and Wigner tables for (b_beta, K, weighted) on the host and copies them into the
// static table array (no allocation; cudaMemcpy waits for the copy).
static int static_load_tables(StaticDeviceState& st, int b_beta, int K, bool weighted,
                              stream_t stream) {
  if (st.b_beta == b_beta && st.K == K && st.weighted == (int)weighted) return S2C_OK;
  const int N = 2 * b_beta;
  FftDev f;
  if (!fft_plan(N, f.desc))
    return fail(S2C_ERR_UNSUPPORTED, "s2c_so3_rifft_static: unsupported FFT length");
  std::vector<float> tw;
  std::vector<unsigned short> pos;
  fft_twiddles(N, tw);
  fft_positions(f.desc, pos);
  std::vector<float> pdata;
  std::vector<long long> poff;
  TableCache::build_panels(b_beta, K, K, weighted, false, pdata, poff);
  const size_t o_tw = 0;
  const size_t o_pos = align_up(o_tw + tw.size() * sizeof(float), 256);
  const size_t o_off = align_up(o_pos + pos.size() * sizeof(unsigned short), 256);
  const size_t o_dat = align_up(o_off + poff.size() * sizeof(long long), 256);
  const size_t total = o_dat + pdata.size() * sizeof(float);
  if (total > kStaticTableBytes)
    return fail(S2C_ERR_UNSUPPORTED,
                "s2c_so3_rifft_static: tables for these bandwidths need " + std::to_string(total) +
                    " bytes, the static table array holds " + std::to_string(kStaticTableBytes));
#ifndef S2C_EMUL
  // Kernels of an earlier call on this stream may still be reading the old tables.  Only the
  // caller's stream is waited for: calls on other streams must not overlap this one anyway (they
  // would race on the shared arrays, as the header says).
  S2C_TRY(cuda_check(cudaStreamSynchronize(stream), "stream sync before table reload"));
#endif
  (void)stream;
  // From here on the array no longer holds a complete table set: forget the old key first, so that
  // a failed upload cannot leave a later call with the old bandwidths reading a half-written array.
  st.b_beta = st.K = st.weighted = -1;
  S2C_TRY(dev_upload(st.tables + o_tw, tw.data(), tw.size() * sizeof(float)));
  S2C_TRY(dev_upload(st.tables + o_pos, pos.data(), pos.size() * sizeof(unsigned short)));
  S2C_TRY(dev_upload(st.tables + o_off, poff.data(), poff.size() * sizeof(long long)));
  S2C_TRY(dev_upload(st.tables + o_dat, pdata.data(), pdata.size() * sizeof(float)));
  f.tw = (const float2*)(st.tables + o_tw);
  f.pos = (const unsigned short*)(st.tables + o_pos);
  st.fft = f;
  st.pan.nbeta = N;
  st.pan.nl = K;
  st.pan.K = K;
  st.pan.npairs = (int)poff.size() - 1;
  st.pan.s2 = 0;
  st.pan.nrows = (int)(poff.back() / N);
  st.pan.rowmap = nullptr;
  st.pan.data_g = nullptr;
  st.pan.g_bg = 0;
  st.pan.g_stride = 0;
  st.pan.order = nullptr;
  st.pan.off = (const long long*)(st.tables + o_off);
  st.pan.data = (const float*)(st.tables + o_dat);
  st.b_beta = b_beta;
  st.K = K;
  st.weighted = (int)weighted;
  return S2C_OK;
}

}  // namespace s2c

extern "C" {

size_t s2c_so3_rifft_static_max_bytes(void) { return kStaticScratchBytes; }

int s2c_so3_rifft_static(const float* x, float* out, long nbatch, int b_in, int b_out,
                         int for_grad, const float* bias, int nfeature, void* stream) {
  S2C_TRY(check_b(b_in, b_out));
  if (!x || !out || nbatch < 1) return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft_static: bad argument");
  if (bias && nfeature < 1)
    return fail(S2C_ERR_BAD_ARG, "s2c_so3_rifft_static: nfeature must be >= 1 with a bias");
  const int N = 2 * b_out, K = std::min(b_in, b_out);
  // scratch of the synthesis: both arrays are laid out on the OUTPUT grid (2 b_out samples per axis)
  const size_t need = so3_ws_per_z(N, K) * (size_t)nbatch;
  if (need > kStaticScratchBytes)
    return fail(S2C_ERR_WORKSPACE,
                "s2c_so3_rifft_static: this call needs " + std::to_string(need) +
                    " bytes of scratch, the static array holds " +
                    std::to_string(kStaticScratchBytes) + " (use s2c_so3_rifft with a workspace)");
  stream_t st = as_stream(stream);
  std::lock_guard<std::mutex> lock(g_static_mu);
  StaticDeviceState& dev = g_static_state[dev_current()];
  S2C_TRY(static_setup(dev));
  S2C_TRY(static_load_tables(dev, b_out, K, for_grad != 0, st));

  const int G = fft_group(N, N), Gg = fft_group(N, N / 2);  // alpha passes, gamma passes
  const size_t fft_smem = fft_smem_bytes(N, G);
  float2* t = (float2*)dev.scratch;                   // [z][K][N][N]
  float2* s = t + (size_t)nbatch * K * N * N;         // [K][2K-1][z][N]
  InvWignerParams w;
  w.x = (const float2*)x;
  w.x_zstride = nbatch;
  w.s = s;
  w.pan = dev.pan;
  w.nbatch = (int)nbatch; w.N = N; w.K = K;
  w.ZT = (int)std::min<long>(32, nbatch);
  w.nzt = (int)((nbatch + w.ZT - 1) / w.ZT);
  w.mode = kSo3Real;
  const size_t wsm = align_up((size_t)K * N * sizeof(float), 16) + (size_t)K * w.ZT * sizeof(float2);
  S2C_TRY(S2C_LAUNCH(so3_inv_wigner, (long)dev.pan.npairs * w.nzt, kThreads, wsm, st, w));
  InvAlphaParams a;
  a.s = s;
  a.out = (float*)t;
  a.out_real = 0;
  a.herm_n0 = 1;
  a.nbatch = (int)nbatch; a.N = N; a.K = K; a.Kn = K; a.G = G;
  a.nrows = nbatch * K * N;
  a.fft = dev.fft;
  S2C_TRY(S2C_LAUNCH(so3_inv_alpha, (a.nrows + G - 1) / G, kThreads, fft_smem, st, a));
  InvGammaParams g;
  g.t = t;
  g.out = out;
  g.out_stride = 1;
  g.out_off = 0;
  g.bias = bias;
  g.nfeat = nfeature > 0 ? nfeature : 1;
  g.z0 = 0;
  g.N = N; g.b = b_out; g.K = K; g.G = Gg;
  g.npairs = nbatch * N * b_out;
  g.fft = dev.fft;
  return S2C_LAUNCH(so3_inv_gamma, (g.npairs + Gg - 1) / Gg, kThreads, fft_smem_bytes(N, Gg), st, g);
}

}  // extern "C"
