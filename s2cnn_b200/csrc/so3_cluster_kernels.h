// SO(3) transforms for small bandwidths (N = 2b <= 32) and few batch elements: one kernel per direction, and
// one for a synthesis followed by the next layer's analysis, like so3_fused_kernels.h and
// so3_relay_kernels.h, whose blocks walk beta sequentially and so leave most SMs idle (or one block of 16
// warps alone on its SM) while the batch is small.
//
// A thread-block CLUSTER owns ZG = 4 consecutive batch elements (whole 32-byte sectors of the
// [spectrum][batch] layout).  Its C blocks split the work two ways:
//
//   * the FFTs by beta: block r holds the planes of betas r BC .. r BC + BC - 1 (all four batch elements)
//     in shared memory; every 1-D FFT runs in the registers of one thread (fft_reg.h);
//   * the Wigner contractions by frequency pair (m, n): the pairs, sorted by their number of degrees, are
//     dealt round-robin to the blocks.  A synthesis thread contracts one pair over l for the BC betas of one
//     block and stores the sums into that block's planes; an analysis thread reads one pair's values of ALL
//     betas out of the blocks' planes and accumulates in registers.  Both go through distributed shared
//     memory, with one cluster barrier between the two splits.
//
//   so3_inv_cl     symmetrised half spectrum (or the s2_mm product computed on the fly) -> Wigner over l ->
//                  column FFTs (m -> alpha) -> Hermitian row FFTs (n -> gamma, two real rows per complex
//                  transform) -> (+ bias) -> store, or integrate max(., 0)
//   so3_fwd_cl     row FFTs of two real rows (optional ReLU on load) -> column FFTs -> Wigner over beta ->
//                  spectrum and Hermitian mirror
//   so3_relay_cl   the synthesis, + bias, ReLU and forward row transform in the registers of the thread that
//                  finished two rows, then the rest of the analysis
//
// Sums keep the order of the sequential walk (l ascending, beta ascending, one fused multiply-add per
// term), so the results are the same bit for bit.
//
// Measured against the walking kernels: analysis b = 16, 20 signals 61 -> 19 us, 100 signals 61 -> 35 us; synthesis
// 61 -> 15 and 22 us; b = 10, 20 signals 22 -> 10 us; relay b = 16, 20 - 3200 signals 461 - 2624 -> 27 - 1036 us,
// b = 10 -> 6, 20 signals 33 -> 13 us.  With many batch elements the remote accesses bound them (analysis b = 16,
// 3200 signals 378 -> 736 us): see so3_prefers_cluster (lib.cu) for where the line lies.
#pragma once

#include <string>
#include <type_traits>

#include "backend.h"
#include "fft_reg.h"
#include "so3_fused_kernels.h"
#include "so3_kernels.h"
#include "tables.h"

namespace s2c {

// Planes hold the four batch elements innermost, [beta][N rows][KP][z]: what the contractions move between
// blocks is then 32 contiguous bytes per (beta, m, n) - with one plane per batch element the 8-byte remote
// accesses bound the kernels (analysis of 3200 signals at b = 16: 0.86 ms against 0.29 ms) -, and with an odd KP
// both the column phase (lanes over z, n) and the row phase (lanes over z, alpha) are free of bank conflicts.
S2C_HD constexpr int cl_kp(int K) { return K | 1; }
constexpr int kClSlots = 8 * kFusedZG;   // floats: partial integrals of the cluster's blocks
// complex numbers of the planes (at least one float per thread: the integral sums over the threads there)
S2C_HD int cl_plane_count(int N, int kmax) {
  const int planes = cl_betas(N) * N * cl_kp(kmax) * kFusedZG, least = cl_threads(N) / 2;
  return planes > least ? planes : least;
}
inline size_t cl_smem_bytes(int N, int kmax, int spec_rows) {
  return ((size_t)spec_rows * kFusedZG + cl_plane_count(N, kmax)) * sizeof(float2) + kClSlots * sizeof(float);
}

// ---------------------------------------------------------------------------------------------
struct ClSpectrumIn {
  const float2* x;     // spectrum rows of x_zstride complex
  long x_zstride;
  int mode;            // kSo3Real, kSo3RotI, or
  // kS2Product: the spectrum is never materialised; row (l,m,n), batch z = (i, j) is
  //   sum_k xs[l,m,i,k] conj(ys[l,n,k,j])        (s2_mm evaluated while the spectrum is staged)
  const float2* xs;    // [K*K, s2_nb, s2_fin]
  const float2* ys;    // [K*K, s2_fin, s2_fout]
  int s2_nb, s2_fin, s2_fout;
  int s2_real;         // (s2_mirror)
};
struct ClInvParams {
  ClSpectrumIn in;
  ClTables tab;        // beta grid of b_out, nl = K
  float* out;          // element e of the real signal at out[e * out_stride + out_off]
  long out_stride, out_off;
  const float* bias;
  int nfeat;
  int nbatch, K;
  // optional tail of a network: instead of writing the signal, integrate max(signal, 0) over SO(3)
  // (so3_integrate(relu(.)), s2cnn/soft/so3_integrate.py:7-29) and write one number per batch element
  const float* iw;     // quadrature weights [N] (null: write the signal)
  float* isum;         // [nbatch]
  // optional: a signal of the output's shape (unit stride); output samples where it is <= 0 are
  // written as 0 - the gradient of a ReLU that was applied while this signal was read
  const float* mask;
  int wide;            // out (and mask) are 32-byte aligned and N % 4 == 0: 32-byte stores
};
struct ClFwdParams {
  const float* x;      // element e of the real signal at x[e * in_stride + in_off]
  long in_stride, in_off;
  float2* out;         // spectrum rows of out_zstride complex
  long out_zstride;
  ClTables tab;        // beta grid of b_in, nl = b_out, K
  int nbatch, K, mode, relu;
  int wide;            // x is 32-byte aligned, unit stride and N % 4 == 0: 32-byte loads
  // optional by-product [nbatch]: the plain sum of every signal over its (2b)^3 samples (the
  // (m, n) = (0, 0) bin of each beta plane, summed over beta) - what the gradient of a bias that
  // was added to the signal needs, without another pass over the signal
  float* sums;
};
struct ClRelayParams {
  ClSpectrumIn in;
  ClTables tin;        // beta grid of b, nl = Kin (unweighted)
  const float* bias;   // optional [nfeat]
  int nfeat;
  ClTables tout;       // beta grid of b, nl = b_next, K = Kout (weighted)
  float2* out;         // spectrum rows of out_zstride complex
  long out_zstride;
  int nbatch, Kin, Kout;
};

// ---------------------------------------------------------------------------------------------
// The phases.  `planes` = [beta of this block][N rows][KP][z] complex.
template <int N>
struct Cl {
  static constexpr int C = cl_size(N), BC = cl_betas(N), ZG = kFusedZG, H = N / 2;
  static constexpr bool FULL = C * BC == N;      // every block has BC betas
  static_assert(ZG == 4, "two 16-byte accesses per (beta, m, n)");

  struct Block {
    float2* planes;
    int RS, BS;              // row and beta strides of the planes (complex)
    int rank, beta0, bc;     // this block's betas: beta0 .. beta0 + bc - 1
    long z0;
    int zc;
  };
  static S2C_D Block block(const ClCtx& ctx, float2* planes, int kmax, int nbatch) {
    Block b;
    b.planes = planes;
    b.RS = cl_kp(kmax) * ZG;
    b.BS = N * b.RS;
    b.rank = ctx.rank;
    b.beta0 = ctx.rank * BC;
    b.bc = N - b.beta0 < BC ? (N - b.beta0 > 0 ? N - b.beta0 : 0) : BC;
    b.z0 = (long)ctx.bid * ZG;
    b.zc = (int)(nbatch - b.z0 < ZG ? nbatch - b.z0 : ZG);
    return b;
  }

  // ---- symmetrised half spectrum of this block's pairs, Xs = (X[l,m,n] + (-1)^(m-n) conj X[l,-m,-n]) / 2,
  //      rows of four batch elements; one row per work item when the block's batch elements are whole
  //      sectors (or, with the product, share the batch index of xs), else one (row, element) -----------
  static S2C_D float2 symmetrise(float2 a, float2 b, int mn, int mode) {
    if (mode == kSo3RotI) {   // multiply the spectrum by -i
      a = make_float2(a.y, -a.x);
      b = make_float2(b.y, -b.x);
    }
    const float fudge = (mn & 1) ? -1.f : 1.f;
    return make_float2(0.5f * (a.x + fudge * b.x), 0.5f * (a.y - fudge * b.y));
  }
  static S2C_D void load_spectrum(const ClCtx& ctx, const ClSpectrumIn& p, const ClTables& t, const Block& b, float2* Xs) {
    const int nr = t.nrows[b.rank];
    const int2* rows = t.rows + (long)b.rank * t.max_rows;
    const bool prod = p.mode == kS2Product;
    const bool fast = b.zc == ZG && (prod ? p.s2_fout % ZG == 0 : p.x_zstride % 2 == 0);
    if (fast && prod) {
      const int pi = (int)(b.z0 / p.s2_fout), pj = (int)(b.z0 - (long)pi * p.s2_fout);
      for (int i = ctx.tid; i < nr; i += ctx.nthr) {
        const int2 row = rows[i];
        int l, m, n;
        rowmap_unpack(row.x, l, m, n);
        const float2* xa = p.xs + ((long)(l * l + l + m) * p.s2_nb + pi) * p.s2_fin;
        const float2* xb = p.xs + ((long)(l * l + l - m) * p.s2_nb + pi) * p.s2_fin;
        const float2* ya = p.ys + (long)(l * l + l + n) * p.s2_fin * p.s2_fout + pj;
        const float2* yb = p.ys + (long)(l * l + l - n) * p.s2_fin * p.s2_fout + pj;
        float2 av[ZG], bv[ZG];
#pragma unroll
        for (int z = 0; z < ZG; ++z) { av[z] = make_float2(0.f, 0.f); bv[z] = make_float2(0.f, 0.f); }
        for (int k = 0; k < p.s2_fin; ++k) {
          s2_multiply_add(xa[k], ya + (long)k * p.s2_fout, av);
          if (!p.s2_real) s2_multiply_add(xb[k], yb + (long)k * p.s2_fout, bv);
        }
        if (p.s2_real) {
#pragma unroll
          for (int z = 0; z < ZG; ++z) bv[z] = s2_mirror(av[z], m - n);
        }
#pragma unroll
        for (int z = 0; z < ZG; ++z) Xs[row.y * ZG + z] = symmetrise(av[z], bv[z], m - n, p.mode);
      }
    } else if (fast) {
      for (int i = ctx.tid; i < nr; i += ctx.nthr) {
        const int2 row = rows[i];
        int l, m, n;
        rowmap_unpack(row.x, l, m, n);
        const float4* pa = reinterpret_cast<const float4*>(p.x + so3_row(l, m, n) * p.x_zstride + b.z0);
        const float4* pb = reinterpret_cast<const float4*>(p.x + so3_row(l, -m, -n) * p.x_zstride + b.z0);
        const float4 a01 = pa[0], a23 = pa[1], b01 = pb[0], b23 = pb[1];
        const float2 v0 = symmetrise(make_float2(a01.x, a01.y), make_float2(b01.x, b01.y), m - n, p.mode);
        const float2 v1 = symmetrise(make_float2(a01.z, a01.w), make_float2(b01.z, b01.w), m - n, p.mode);
        const float2 v2 = symmetrise(make_float2(a23.x, a23.y), make_float2(b23.x, b23.y), m - n, p.mode);
        const float2 v3 = symmetrise(make_float2(a23.z, a23.w), make_float2(b23.z, b23.w), m - n, p.mode);
        float4* d = reinterpret_cast<float4*>(Xs + row.y * ZG);
        d[0] = make_float4(v0.x, v0.y, v1.x, v1.y);
        d[1] = make_float4(v2.x, v2.y, v3.x, v3.y);
      }
    } else {
      for (int it = ctx.tid; it < nr * ZG; it += ctx.nthr) {
        const int i = it / ZG, zz = it - i * ZG;
        const int2 row = rows[i];
        int l, m, n;
        rowmap_unpack(row.x, l, m, n);
        float2 a = make_float2(0.f, 0.f), c = make_float2(0.f, 0.f);
        if (zz < b.zc) {
          if (prod) {
            const int z = (int)(b.z0 + zz), zi = z / p.s2_fout, zj = z - zi * p.s2_fout;
            a = s2_product_entry(p, l, m, n, zi, zj);
            c = p.s2_real ? s2_mirror(a, m - n) : s2_product_entry(p, l, -m, -n, zi, zj);
          } else {
            a = p.x[so3_row(l, m, n) * p.x_zstride + b.z0 + zz];
            c = p.x[so3_row(l, -m, -n) * p.x_zstride + b.z0 + zz];
          }
        }
        Xs[row.y * ZG + zz] = symmetrise(a, c, m - n, p.mode);
      }
    }
  }
  static S2C_D float2 s2_product_entry(const ClSpectrumIn& p, int l, int m, int n, int i, int j) {
    const float2* xr = p.xs + ((long)(l * l + l + m) * p.s2_nb + i) * p.s2_fin;
    const float2* yr = p.ys + (long)(l * l + l + n) * p.s2_fin * p.s2_fout + j;
    float re = 0.f, im = 0.f;
    for (int k = 0; k < p.s2_fin; ++k) {
      const float2 a = xr[k], b = yr[(long)k * p.s2_fout];
      re = fmaf(a.x, b.x, re);
      re = fmaf(a.y, b.y, re);
      im = fmaf(a.y, b.x, im);
      im = fmaf(-a.x, b.y, im);
    }
    return make_float2(re, im);
  }

  // ---- Wigner contraction over l of this block's pairs, for every block's betas: work item = (pair,
  //      destination block), BC x 4 sums in registers, stored into that block's planes ---------------------
  static S2C_D void wigner_in(const ClCtx& ctx, const ClTables& t, const Block& b, const float2* Xs) {
    const int npl = (t.npairs - b.rank + C - 1) / C;
    for (int it = ctx.tid; it < npl * C; it += ctx.nthr) {
      const int k = it / C, c = it - k * C;
      const int4 pr = t.pairs[k * C + b.rank];      // {first panel row, L, FFT row of m, n}
      const float* w = t.w + (long)pr.x * N + c * BC;
      const float4* x4 = reinterpret_cast<const float4*>(Xs) + 2 * t.lrow[k * C + b.rank];
      float2 s[BC][ZG];
#pragma unroll
      for (int bi = 0; bi < BC; ++bi)
#pragma unroll
        for (int z = 0; z < ZG; ++z) s[bi][z] = make_float2(0.f, 0.f);
      for (int li = 0; li < pr.y; ++li) {
        float wv[BC];
        if constexpr (BC == 4 && FULL) {
          const float4 w4 = *reinterpret_cast<const float4*>(w + (long)li * N);
          wv[0] = w4.x; wv[1] = w4.y; wv[2] = w4.z; wv[3] = w4.w;
        } else {
#pragma unroll
          for (int bi = 0; bi < BC; ++bi) wv[bi] = (FULL || c * BC + bi < N) ? w[(long)li * N + bi] : 0.f;
        }
        const float4 xa = x4[2 * li], xb = x4[2 * li + 1];
        const float2 xv[ZG] = {make_float2(xa.x, xa.y), make_float2(xa.z, xa.w),
                               make_float2(xb.x, xb.y), make_float2(xb.z, xb.w)};
#pragma unroll
        for (int bi = 0; bi < BC; ++bi)
#pragma unroll
          for (int z = 0; z < ZG; ++z) {
            s[bi][z] = fma2(make_float2(wv[bi], wv[bi]), xv[z], s[bi][z]);
          }
      }
      const cl_addr dst = cl_map(ctx, b.planes + pr.z * b.RS + pr.w * ZG, c);
      const bool mirror = pr.w == 0 && pr.z > 0;    // n = 0, m > 0: row N - m holds the conjugate
#pragma unroll
      for (int bi = 0; bi < BC; ++bi)
        if (FULL || c * BC + bi < N) {
          const int off = bi * b.BS;
          cl_store4(dst, off, make_float4(s[bi][0].x, s[bi][0].y, s[bi][1].x, s[bi][1].y));
          cl_store4(dst, off + 2, make_float4(s[bi][2].x, s[bi][2].y, s[bi][3].x, s[bi][3].y));
          if (mirror) {
            const int om = off + (N - 2 * pr.z) * b.RS;
            cl_store4(dst, om, make_float4(s[bi][0].x, -s[bi][0].y, s[bi][1].x, -s[bi][1].y));
            cl_store4(dst, om + 2, make_float4(s[bi][2].x, -s[bi][2].y, s[bi][3].x, -s[bi][3].y));
          }
        }
    }
  }

  // ---- column FFTs m -> alpha: one thread per (z, beta, n < K) ------------------------------------------
  static S2C_D void columns_inv(const ClCtx& ctx, const Block& b, int K) {
    for (int it = ctx.tid; it < ZG * b.bc * K; it += ctx.nthr) {
      const int z = it % ZG, nb = it / ZG;
      const int bi = nb / K, n = nb - bi * K;
      float2* col = b.planes + bi * b.BS + n * ZG + z;
      float2 v[N];
#pragma unroll
      for (int i = 0; i < N; ++i)
        v[i] = (i < K || i > N - K) ? col[i * b.RS] : make_float2(0.f, 0.f);
      fft_reg<N, +1>(v, nullptr);
      static_for<0, N>([&](auto ic) {
        constexpr int a = decltype(ic)::value;
        col[a * b.RS] = v[fft_reg_pos<N>(a)];
      });
    }
  }
  // ---- column FFTs alpha -> m -----------------------------------------------------------------------------
  static S2C_D void columns_fwd(const ClCtx& ctx, const Block& b, int K) {
    for (int it = ctx.tid; it < ZG * b.bc * K; it += ctx.nthr) {
      const int z = it % ZG, nb = it / ZG;
      const int bi = nb / K, n = nb - bi * K;
      float2* col = b.planes + bi * b.BS + n * ZG + z;
      float2 v[N];
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = col[i * b.RS];
      fft_reg<N, -1>(v, nullptr);
      static_for<0, N>([&](auto ic) {
        constexpr int f = decltype(ic)::value;
        if (f < K || f > N - K) col[f * b.RS] = v[fft_reg_pos<N>(f)];
      });
    }
  }

  // the thread's pair of rows (alpha, alpha + N/2) of a row phase
  struct Rows {
    int ap, bi, z;
    float2 *r1, *r2;
  };
  static S2C_D Rows rows_of(const Block& b, int it) {
    Rows r;
    r.z = it % ZG;
    const int ab = it / ZG;
    r.bi = ab / H;
    r.ap = ab - r.bi * H;
    r.r1 = b.planes + r.bi * b.BS + r.ap * b.RS + r.z;
    r.r2 = r.r1 + H * b.RS;
    return r;
  }
  // packed Hermitian rows: v[n] = T1 + i T2, v[N - n] = conj(T1) + i conj(T2)
  static S2C_D void pack_rows(const Rows& r, int K, float2 (&v)[N]) {
    {
      const float2 t1 = r.r1[0], t2 = r.r2[0];
      v[0] = make_float2(t1.x, t2.x);  // T[alpha][0] is real for a Hermitian spectrum
    }
    if constexpr (N > 1) v[H] = make_float2(0.f, 0.f);
#pragma unroll
    for (int n = 1; n < H; ++n) {
      if (n < K) {
        const float2 t1 = r.r1[n * ZG], t2 = r.r2[n * ZG];
        v[n] = make_float2(t1.x - t2.y, t1.y + t2.x);
        v[N - n] = make_float2(t1.x + t2.y, t2.x - t1.y);
      } else {
        v[n] = make_float2(0.f, 0.f);
        v[N - n] = make_float2(0.f, 0.f);
      }
    }
  }
  // half spectra (n < K) of the two real rows whose packed transform is in v
  static S2C_D void split_rows(const Rows& r, int K, const float2 (&v)[N]) {
    static_for<0, H>([&](auto ic) {
      constexpr int n = decltype(ic)::value;
      constexpr int pn = fft_reg_pos<N>(n), pq = fft_reg_pos<N>(n == 0 ? 0 : N - n);
      if (n < K) {
        const float2 zk = v[pn], zq = v[pq];
        r.r1[n * ZG] = make_float2(0.5f * (zk.x + zq.x), 0.5f * (zk.y - zq.y));
        r.r2[n * ZG] = make_float2(0.5f * (zk.y + zq.y), -0.5f * (zk.x - zq.x));
      }
    });
  }

  // ---- Wigner contraction over all betas of this block's pairs -> spectrum rows.  Work item = up to two
  //      degrees of one pair, ZT of the four batch elements (all, or one when there are few items) ----------
  template <int ZT>
  static S2C_D void wigner_out(const ClCtx& ctx, const ClTables& t, const Block& b, float2* out, long zstride, int mode) {
    const int nt = t.ntasks[b.rank];
    const int4* tasks = t.tasks + (long)b.rank * t.max_tasks;
    for (int it = ctx.tid; it < nt * (ZG / ZT); it += ctx.nthr) {
      const int4 tk = tasks[it / (ZG / ZT)];    // {panel row, degrees (1 or 2), FFT row of m, n | l << 8}
      const int zf = ZT == ZG ? 0 : it % ZG;
      const float* w0 = t.w + (long)tk.x * N;
      const float* w1 = w0 + (tk.y > 1 ? N : 0);
      const int n = tk.w & 0xff, l = tk.w >> 8, m = tk.z < H ? tk.z : tk.z - N;
      const float2* local = b.planes + tk.z * b.RS + n * ZG + zf;
      float2 a0[ZT], a1[ZT];
#pragma unroll
      for (int z = 0; z < ZT; ++z) a0[z] = a1[z] = make_float2(0.f, 0.f);
#pragma unroll 1
      for (int c = 0; c < C; ++c) {
        const cl_addr src = cl_map(ctx, local, c);
        float u0[BC], u1[BC];
        float2 xv[BC][ZT];
        if constexpr (BC == 4 && FULL) {
          const float4 p0 = *reinterpret_cast<const float4*>(w0 + c * BC), p1 = *reinterpret_cast<const float4*>(w1 + c * BC);
          u0[0] = p0.x; u0[1] = p0.y; u0[2] = p0.z; u0[3] = p0.w;
          u1[0] = p1.x; u1[1] = p1.y; u1[2] = p1.z; u1[3] = p1.w;
        } else {
#pragma unroll
          for (int bi = 0; bi < BC; ++bi) {
            const bool in = FULL || c * BC + bi < N;
            u0[bi] = in ? w0[c * BC + bi] : 0.f;
            u1[bi] = in ? w1[c * BC + bi] : 0.f;
          }
        }
#pragma unroll
        for (int bi = 0; bi < BC; ++bi) {
          if (FULL || c * BC + bi < N) {
            if constexpr (ZT == ZG) {
              const float4 q0 = cl_load4(src, bi * b.BS), q1 = cl_load4(src, bi * b.BS + 2);
              xv[bi][0] = make_float2(q0.x, q0.y); xv[bi][1] = make_float2(q0.z, q0.w);
              xv[bi][2] = make_float2(q1.x, q1.y); xv[bi][3] = make_float2(q1.z, q1.w);
            } else {
              xv[bi][0] = cl_load(src, bi * b.BS);
            }
          } else {
#pragma unroll
            for (int z = 0; z < ZT; ++z) xv[bi][z] = make_float2(0.f, 0.f);
          }
        }
#pragma unroll
        for (int bi = 0; bi < BC; ++bi)
#pragma unroll
          for (int z = 0; z < ZT; ++z) {
            a0[z] = fma2(make_float2(u0[bi], u0[bi]), xv[bi][z], a0[z]);
            a1[z] = fma2(make_float2(u1[bi], u1[bi]), xv[bi][z], a1[z]);
          }
      }
      emit<ZT>(out, zstride, b, zf, l, m, n, a0, mode);
      if (tk.y > 1) emit<ZT>(out, zstride, b, zf, l + 1, m, n, a1, mode);
    }
  }
  // one spectrum row and its Hermitian mirror
  template <int ZT>
  static S2C_D void emit(float2* out, long zstride, const Block& b, int zf, int l, int m, int n, const float2 (&a)[ZT], int mode) {
    const float fudge = ((m - n) & 1) ? -1.f : 1.f;
    float2* o1 = out + so3_row(l, m, n) * zstride + b.z0 + zf;
    float2* o2 = out + so3_row(l, -m, -n) * zstride + b.z0 + zf;
    const bool self = (m == 0 && n == 0);
    if (ZT == ZG && mode == kSo3Real && b.zc == ZG && zstride % 2 == 0) {
      float4* q1 = reinterpret_cast<float4*>(o1);
      q1[0] = make_float4(a[0].x, a[0].y, a[ZT > 1 ? 1 : 0].x, a[ZT > 1 ? 1 : 0].y);
      q1[1] = make_float4(a[ZT > 2 ? 2 : 0].x, a[ZT > 2 ? 2 : 0].y, a[ZT > 3 ? 3 : 0].x, a[ZT > 3 ? 3 : 0].y);
      if (!self) {
        float4* q2 = reinterpret_cast<float4*>(o2);
        q2[0] = make_float4(fudge * a[0].x, -fudge * a[0].y, fudge * a[ZT > 1 ? 1 : 0].x, -fudge * a[ZT > 1 ? 1 : 0].y);
        q2[1] = make_float4(fudge * a[ZT > 2 ? 2 : 0].x, -fudge * a[ZT > 2 ? 2 : 0].y, fudge * a[ZT > 3 ? 3 : 0].x,
                            -fudge * a[ZT > 3 ? 3 : 0].y);
      }
      return;
    }
#pragma unroll
    for (int z = 0; z < ZT; ++z) {
      if (zf + z >= b.zc) continue;
      if (mode == kSo3Real) {
        o1[z] = a[z];
        if (!self) o2[z] = make_float2(fudge * a[z].x, -fudge * a[z].y);
      } else {  // += i * a ; mirror += i * fudge * conj(a)
        float2 c = o1[z];
        o1[z] = make_float2(c.x - a[z].y, c.y + a[z].x);
        if (!self) {
          c = o2[z];
          o2[z] = make_float2(c.x + fudge * a[z].y, c.y + fudge * a[z].x);
        }
      }
    }
  }
  static S2C_D void wigner_out_any(const ClCtx& ctx, const ClTables& t, const Block& b, float2* out, long zstride, int mode) {
    if (t.max_tasks * ZG <= 2 * ctx.nthr) wigner_out<1>(ctx, t, b, out, zstride, mode);
    else wigner_out<ZG>(ctx, t, b, out, zstride, mode);
  }
};

// ---------------------------------------------------------------------------------------------
template <int N>
struct so3_inv_cl_impl {
  static S2C_D void run(const ClCtx& ctx, const ClInvParams& p, unsigned char* smem) {
    using K_ = Cl<N>;
    constexpr int H = N / 2, ZG = kFusedZG;
    const int K = p.K;
    float2* Xs = reinterpret_cast<float2*>(smem);
    float2* planes = Xs + (long)p.tab.max_rows * ZG;
    const typename K_::Block b = K_::block(ctx, planes, K, p.nbatch);
    float* slots = reinterpret_cast<float*>(planes + cl_plane_count(N, K));   // [rank][z]
    K_::load_spectrum(ctx, p.in, p.tab, b, Xs);
    ctx.sync_cluster();          // (also: every block of the cluster has started, its memory may be written)
    K_::wigner_in(ctx, p.tab, b, Xs);
    ctx.sync_cluster();
    K_::columns_inv(ctx, b, K);
    ctx.sync();
    // ---- Hermitian row FFTs n -> gamma: one thread per (z, beta, alpha pair) -----------------------------
    float ipart = 0.f;
    for (int it = ctx.tid; it < ZG * b.bc * H; it += ctx.nthr) {
      const typename K_::Rows r = K_::rows_of(b, it);
      float2 v[N];
      K_::pack_rows(r, K, v);
      fft_reg<N, +1>(v, nullptr);
      float add = 0.f;
      if (p.bias) add = p.bias[(b.z0 + r.z) % p.nfeat];
      if (p.iw) {
        // the signal is not written: max(x, 0) of both rows, summed over gamma, times w_beta
        float rs = 0.f;
#pragma unroll
        for (int g = 0; g < N; ++g) {
          const float a1 = v[g].x + add, a2 = v[g].y + add;
          rs += relu(a1) + relu(a2);
        }
        ipart = fmaf(p.iw[b.beta0 + r.bi], rs, ipart);
        continue;
      }
      if (r.z >= b.zc) continue;
      // store the two finished rows straight from registers (the plane is contiguous in memory)
      const long row1 = (((b.z0 + r.z) * N + b.beta0 + r.bi) * (long)N + r.ap) * N;   // first float of row ap
      const long row2 = row1 + (long)H * N;
      auto keep = [](float4 val, float4 k) {
        return make_float4(relu_grad(k.x, val.x), relu_grad(k.y, val.y), relu_grad(k.z, val.z),
                           relu_grad(k.w, val.w));
      };
      auto quad = [&](auto gc, float4& o1, float4& o2) {
        constexpr int g = decltype(gc)::value;
        constexpr int p0 = fft_reg_pos<N>(g), p1 = fft_reg_pos<N>(g + 1);
        constexpr int p2 = fft_reg_pos<N>(g + 2), p3 = fft_reg_pos<N>(g + 3);
        o1 = make_float4(v[p0].x + add, v[p1].x + add, v[p2].x + add, v[p3].x + add);
        o2 = make_float4(v[p0].y + add, v[p1].y + add, v[p2].y + add, v[p3].y + add);
      };
      auto st4 = [&](auto gc) {
        constexpr int g = decltype(gc)::value;
        float4 o1, o2;
        quad(gc, o1, o2);
        if (p.mask) {
          o1 = keep(o1, *reinterpret_cast<const float4*>(p.mask + row1 + g));
          o2 = keep(o2, *reinterpret_cast<const float4*>(p.mask + row2 + g));
        }
        *reinterpret_cast<float4*>(p.out + row1 + g) = o1;
        *reinterpret_cast<float4*>(p.out + row2 + g) = o2;
      };
      if constexpr (N % 4 == 0) {
        if (p.wide) {
          // 32-byte stores, one whole sector per lane and instruction (with 16-byte stores every
          // sector would reach L2 in two halves).  Rows of N % 8 == 4 floats start on a sector
          // boundary only every other row (the planes themselves do, 4 N^2 bytes apart): even
          // rows end, odd rows begin with a 16-byte piece.
          auto st8 = [&](auto gc) {
            constexpr int g = decltype(gc)::value;
            float8 o1, o2;
            quad(gc, o1.lo, o2.lo);
            quad(std::integral_constant<int, g + 4>{}, o1.hi, o2.hi);
            if (p.mask) {
              const float8 k1 = ld_global_256(p.mask + row1 + g), k2 = ld_global_256(p.mask + row2 + g);
              o1.lo = keep(o1.lo, k1.lo); o1.hi = keep(o1.hi, k1.hi);
              o2.lo = keep(o2.lo, k2.lo); o2.hi = keep(o2.hi, k2.hi);
            }
            st_global_256(p.out + row1 + g, o1);
            st_global_256(p.out + row2 + g, o2);
          };
          if constexpr (N % 8 == 0) {
            static_for<0, N / 8>([&](auto ic) { st8(std::integral_constant<int, 8 * decltype(ic)::value>{}); });
          } else if (r.ap & 1) {
            st4(std::integral_constant<int, 0>{});
            static_for<0, N / 8>([&](auto ic) { st8(std::integral_constant<int, 4 + 8 * decltype(ic)::value>{}); });
          } else {
            static_for<0, N / 8>([&](auto ic) { st8(std::integral_constant<int, 8 * decltype(ic)::value>{}); });
            st4(std::integral_constant<int, N - 4>{});
          }
          continue;
        }
      }
      if (p.out_stride == 1) {
        if constexpr (N % 4 == 0) {
          static_for<0, N / 4>([&](auto ic) { st4(std::integral_constant<int, 4 * decltype(ic)::value>{}); });
        } else {
          static_for<0, N / 2>([&](auto ic) {
            constexpr int g = 2 * decltype(ic)::value;
            constexpr int p0 = fft_reg_pos<N>(g), p1 = fft_reg_pos<N>(g + 1);
            float2 o1 = make_float2(v[p0].x + add, v[p1].x + add);
            float2 o2 = make_float2(v[p0].y + add, v[p1].y + add);
            if (p.mask) {
              const float2 k1 = *reinterpret_cast<const float2*>(p.mask + row1 + g);
              const float2 k2 = *reinterpret_cast<const float2*>(p.mask + row2 + g);
              o1 = make_float2(relu_grad(k1.x, o1.x), relu_grad(k1.y, o1.y));
              o2 = make_float2(relu_grad(k2.x, o2.x), relu_grad(k2.y, o2.y));
            }
            *reinterpret_cast<float2*>(p.out + row1 + g) = o1;
            *reinterpret_cast<float2*>(p.out + row2 + g) = o2;
          });
        }
      } else {
        static_for<0, N>([&](auto ic) {
          constexpr int g = decltype(ic)::value;
          constexpr int pg = fft_reg_pos<N>(g);
          p.out[(row1 + g) * p.out_stride + p.out_off] = v[pg].x + add;
          p.out[(row2 + g) * p.out_stride + p.out_off] = v[pg].y + add;
        });
      }
    }
    if (p.iw) {
      // thread t served batch element t mod 4: sum the threads of each element in a fixed order, then the
      // blocks of the cluster
      ctx.sync();
      float* red = reinterpret_cast<float*>(planes);
      red[ctx.tid] = ipart;
      ctx.sync();
      if (ctx.tid < ZG) {
        float sum = 0.f;
        for (int t = ctx.tid; t < ctx.nthr; t += ZG) sum += red[t];
        cl_store_float(cl_map(ctx, reinterpret_cast<float2*>(slots), 0), b.rank * ZG + ctx.tid, sum);
      }
      ctx.sync_cluster();
      if (b.rank == 0 && ctx.tid < b.zc) {
        float sum = 0.f;
        for (int r = 0; r < K_::C; ++r) sum += slots[r * ZG + ctx.tid];
        p.isum[b.z0 + ctx.tid] = sum;
      }
    }
  }
};

// ---------------------------------------------------------------------------------------------
template <int N>
struct so3_fwd_cl_impl {
  static S2C_D void run(const ClCtx& ctx, const ClFwdParams& p, unsigned char* smem) {
    using K_ = Cl<N>;
    constexpr int H = N / 2, ZG = kFusedZG;
    const int K = p.K;
    float2* planes = reinterpret_cast<float2*>(smem);
    const typename K_::Block b = K_::block(ctx, planes, K, p.nbatch);
    // ---- row FFTs gamma -> n: each thread reads two real rows (alpha, alpha + N/2) straight from global
    //      memory into registers (optional ReLU), transforms them as one complex sequence and leaves the
    //      n < K half spectra of both rows in shared memory -------------------------------------------------
    for (int it = ctx.tid; it < ZG * b.bc * H; it += ctx.nthr) {
      const typename K_::Rows r = K_::rows_of(b, it);
      float2 v[N];
      if (r.z < b.zc) {
        const long row1 = (((b.z0 + r.z) * N + b.beta0 + r.bi) * (long)N + r.ap) * N;
        const long row2 = row1 + (long)H * N;
        if (N % 4 == 0 && p.wide) {
          // 32-byte loads, one whole sector per lane and instruction; rows of N % 8 == 4 floats
          // start on a sector boundary only every other row (see the synthesis kernel)
          auto ld4 = [&](auto gc) {
            constexpr int g = decltype(gc)::value;
            const float4 a = *reinterpret_cast<const float4*>(p.x + row1 + g);
            const float4 c = *reinterpret_cast<const float4*>(p.x + row2 + g);
            v[g] = make_float2(a.x, c.x);
            v[g + 1] = make_float2(a.y, c.y);
            v[g + 2] = make_float2(a.z, c.z);
            v[g + 3] = make_float2(a.w, c.w);
          };
          auto ld8 = [&](auto gc) {
            constexpr int g = decltype(gc)::value;
            const float8 a = ld_global_256(p.x + row1 + g), c = ld_global_256(p.x + row2 + g);
            v[g] = make_float2(a.lo.x, c.lo.x);
            v[g + 1] = make_float2(a.lo.y, c.lo.y);
            v[g + 2] = make_float2(a.lo.z, c.lo.z);
            v[g + 3] = make_float2(a.lo.w, c.lo.w);
            v[g + 4] = make_float2(a.hi.x, c.hi.x);
            v[g + 5] = make_float2(a.hi.y, c.hi.y);
            v[g + 6] = make_float2(a.hi.z, c.hi.z);
            v[g + 7] = make_float2(a.hi.w, c.hi.w);
          };
          if constexpr (N % 8 == 0) {
            static_for<0, N / 8>([&](auto ic) { ld8(std::integral_constant<int, 8 * decltype(ic)::value>{}); });
          } else if (r.ap & 1) {
            ld4(std::integral_constant<int, 0>{});
            static_for<0, N / 8>([&](auto ic) { ld8(std::integral_constant<int, 4 + 8 * decltype(ic)::value>{}); });
          } else {
            static_for<0, N / 8>([&](auto ic) { ld8(std::integral_constant<int, 8 * decltype(ic)::value>{}); });
            ld4(std::integral_constant<int, N - 4>{});
          }
        } else if (p.in_stride == 1) {
          constexpr int V = (N % 4 == 0) ? 4 : 2;
          static_for<0, N / V>([&](auto ic) {
            constexpr int g = V * decltype(ic)::value;
            if constexpr (V == 4) {
              const float4 a = *reinterpret_cast<const float4*>(p.x + row1 + g);
              const float4 c = *reinterpret_cast<const float4*>(p.x + row2 + g);
              v[g] = make_float2(a.x, c.x);
              v[g + 1] = make_float2(a.y, c.y);
              v[g + 2] = make_float2(a.z, c.z);
              v[g + 3] = make_float2(a.w, c.w);
            } else {
              const float2 a = *reinterpret_cast<const float2*>(p.x + row1 + g);
              const float2 c = *reinterpret_cast<const float2*>(p.x + row2 + g);
              v[g] = make_float2(a.x, c.x);
              v[g + 1] = make_float2(a.y, c.y);
            }
          });
        } else {
#pragma unroll
          for (int g = 0; g < N; ++g)
            v[g] = make_float2(p.x[(row1 + g) * p.in_stride + p.in_off], p.x[(row2 + g) * p.in_stride + p.in_off]);
        }
        if (p.relu) {
#pragma unroll
          for (int g = 0; g < N; ++g) {
            v[g].x = relu(v[g].x);
            v[g].y = relu(v[g].y);
          }
        }
      } else {
#pragma unroll
        for (int g = 0; g < N; ++g) v[g] = make_float2(0.f, 0.f);
      }
      fft_reg<N, -1>(v, nullptr);
      K_::split_rows(r, K, v);
    }
    ctx.sync();
    K_::columns_fwd(ctx, b, K);
    ctx.sync_cluster();
    if (p.sums && b.rank == 0 && ctx.tid < b.zc) {
      float s = 0.f;
      for (int c = 0; c < K_::C; ++c) {
        const cl_addr src = cl_map(ctx, planes + ctx.tid, c);
        for (int bi = 0; bi < K_::BC && c * K_::BC + bi < N; ++bi) s += cl_load(src, bi * b.BS).x;
      }
      p.sums[b.z0 + ctx.tid] = s;
    }
    K_::wigner_out_any(ctx, p.tab, b, p.out, p.out_zstride, p.mode);
    ctx.sync_cluster();          // no block leaves while another still reads its planes
  }
};

// ---------------------------------------------------------------------------------------------
template <int N>
struct so3_relay_cl_impl {
  static S2C_D void run(const ClCtx& ctx, const ClRelayParams& p, unsigned char* smem) {
    using K_ = Cl<N>;
    constexpr int H = N / 2, ZG = kFusedZG;
    const int Kin = p.Kin, Kout = p.Kout;
    float2* Xs = reinterpret_cast<float2*>(smem);
    float2* planes = Xs + (long)p.tin.max_rows * ZG;
    const typename K_::Block b = K_::block(ctx, planes, Kin > Kout ? Kin : Kout, p.nbatch);
    K_::load_spectrum(ctx, p.in, p.tin, b, Xs);
    ctx.sync_cluster();
    K_::wigner_in(ctx, p.tin, b, Xs);
    ctx.sync_cluster();
    K_::columns_inv(ctx, b, Kin);
    ctx.sync();
    // ---- rows: Hermitian inverse transform n -> gamma of rows (alpha, alpha + N/2), + bias, ReLU, forward
    //      transform gamma -> n of the same two rows, in place (a thread owns its two rows) ------------------
    for (int it = ctx.tid; it < ZG * b.bc * H; it += ctx.nthr) {
      const typename K_::Rows r = K_::rows_of(b, it);
      float2 v[N];
      K_::pack_rows(r, Kin, v);
      fft_reg<N, +1>(v, nullptr);
      float add = 0.f;
      if (p.bias) add = p.bias[(b.z0 + r.z) % p.nfeat];
      float2 u[N];
      static_for<0, N>([&](auto gc) {
        constexpr int g = decltype(gc)::value;
        constexpr int pg = fft_reg_pos<N>(g);
        const float a1 = v[pg].x + add, a2 = v[pg].y + add;   // samples gamma = g of both rows
        u[g] = make_float2(relu(a1), relu(a2));
      });
      fft_reg<N, -1>(u, nullptr);
      K_::split_rows(r, Kout, u);
    }
    ctx.sync();
    K_::columns_fwd(ctx, b, Kout);
    ctx.sync_cluster();
    K_::wigner_out_any(ctx, p.tout, b, p.out, p.out_zstride, kSo3Real);
    ctx.sync_cluster();
  }
};

#ifndef S2C_EMUL
#define S2C_CLUSTER_KERNEL(name, P)                                                                      \
  template <int N>                                                                                       \
  __global__ void __cluster_dims__(cl_size(N), 1, 1) __launch_bounds__(cl_threads(N), cl_min_blocks(N))  \
  name(const P p) {                                                                                      \
    extern __shared__ float4 s2c_dyn_smem[];                                                             \
    constexpr int C = cl_size(N);                                                                        \
    ClCtx ctx{(int)threadIdx.x, (int)blockDim.x, (int)(blockIdx.x / C), (int)(blockIdx.x % C)};          \
    stream_order_wait();                                                                                 \
    name##_impl<N>::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));                         \
    stream_order_next();  \
  }
S2C_CLUSTER_KERNEL(so3_inv_cl, ClInvParams)
S2C_CLUSTER_KERNEL(so3_fwd_cl, ClFwdParams)
S2C_CLUSTER_KERNEL(so3_relay_cl, ClRelayParams)
S2C_LAUNCHER_N(so3_inv_cl, ClInvParams)
S2C_LAUNCHER_N(so3_fwd_cl, ClFwdParams)
S2C_LAUNCHER_N(so3_relay_cl, ClRelayParams)
// one cluster per kFusedZG batch elements
#define S2C_LAUNCH_CL(name, N, nclusters, smem, stream, params) \
  s2c::launch_##name<N>((long)(nclusters) * cl_size(N), cl_threads(N), (size_t)(smem), stream, params)
#else
#define S2C_LAUNCH_CL(name, N, nclusters, smem, stream, params) \
  s2c::emu_launch_cluster<name##_impl<N>>(#name, (long)(nclusters), cl_size(N), cl_threads(N), (size_t)(smem), params)
#endif

}  // namespace s2c
