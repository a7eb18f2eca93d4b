// Wigner-d contractions for 2b <= 32 and large batches: one batch element per thread.
//
// Same inputs, outputs and sums (same order) as wigner_tiled.h, between spectrum rows and V[n][m][beta][z] - the
// batch innermost on both sides, so that every access of a warp is one run of 256 bytes and nothing but the table
// goes through shared memory.  At b = 16 a frequency pair has 5 degrees on average: the tiles of 4 x 2 outputs
// there share too little (512 signals: 44 us analysis, of which the copies into shared memory and the padded
// tiles are most), while a thread that owns all degrees of one batch element reads each sample of V once and
// each table entry as a broadcast of 16 bytes.  512 signals at b = 16: 23 us, bound by the
// latency of V's loads (24 warps per SM), not by their rate.
#pragma once

#include "backend.h"
#include "so3_kernels.h"

namespace s2c {

constexpr int kColZT = 128;          // batch elements (threads) per block
constexpr int kColMaxDegrees = 16;   // degrees a thread keeps in registers

S2C_HD constexpr int col_nb(int N) { return (N + 7) / 8 * 8; }
inline size_t wigner_col_smem(int N, int nl) { return (size_t)col_nb(N) * ((nl + 3) / 4 * 4) * sizeof(float); }

// spectrum rows of successive degrees, in 32-bit arithmetic: row (l, m, n) is (l, 0, 0) + m (2l + 1) + n
struct ColRows {
  int l, centre;
  S2C_D explicit ColRows(int l0) : l(l0), centre((int)so3_row(l0, 0, 0)) {}
  S2C_D long at(int m, int n) const { return centre + m * (2 * l + 1) + n; }
  S2C_D void next() { centre += 4 * l * (l + 2) + 5; ++l; }
};

// X[l][z] = sum_beta W[l][beta] V[beta][z]   (+ Hermitian mirror row); table as [beta][l], zero-padded
S2C_KERNEL_BOUNDS(so3_fwd_wigner_col, FwdWignerParams, kColZT, 6) {
  const int N = p.N;
  const int pair = ctx.bid / p.nzt, zt = ctx.bid - pair * p.nzt;
  int m, n;
  so3_pair_decode(pair, p.K, m, n);
  const int am = m < 0 ? -m : m;
  const int lmin = am > n ? am : n;
  const int L = p.nl - lmin;
  if (L <= 0) return;
  const int LT = (L + 3) / 4;
  // eight samples of V at a time, in flight while the table is staged or the eight before them are used
  const int nm = 2 * p.K - 1, mi = m + p.K - 1;
  const int z = zt * p.ZT + ctx.tid;
  const float2* vb = p.v + ((long)n * nm + mi) * N * p.nbatch + z;
  float2 next[8];
  auto fetch = [&](int b0) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (b0 + u < N && z < p.nbatch) next[u] = *vb;
      vb += p.nbatch;
    }
  };
  fetch(0);
  float* Ws = reinterpret_cast<float*>(smem);   // [beta][4 LT]
  const float* panel = p.pan.data + p.pan.off[pair];
  for (int i = ctx.tid; i < 4 * LT * N; i += ctx.nthr) {
    const int l = i / N, bt = i - l * N;
    Ws[bt * 4 * LT + l] = l < L ? panel[i] : 0.f;
  }
  ctx.sync();
  if (z >= p.nbatch) return;
  const float fudge = ((m - n) & 1) ? -1.f : 1.f;
  const bool self = (m == 0 && n == 0);
  auto degrees = [&](auto tiles) {
    constexpr int T = decltype(tiles)::value;
    float2 re[2 * T], im[2 * T];                // two degrees each
#pragma unroll
    for (int i = 0; i < 2 * T; ++i) re[i] = im[i] = make_float2(0.f, 0.f);
    for (int b0 = 0; b0 < N; b0 += 8) {
      float2 c[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) c[u] = next[u];
      fetch(b0 + 8);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (b0 + u < N) {
          const float2 cr = make_float2(c[u].x, c[u].x), ci = make_float2(c[u].y, c[u].y);
          const float4* w = reinterpret_cast<const float4*>(Ws + (b0 + u) * 4 * T);
#pragma unroll
          for (int t = 0; t < T; ++t) {
            const float4 w4 = w[t];
            const float2 lo = make_float2(w4.x, w4.y), hi = make_float2(w4.z, w4.w);
            re[2 * t] = fma2(lo, cr, re[2 * t]);
            im[2 * t] = fma2(lo, ci, im[2 * t]);
            re[2 * t + 1] = fma2(hi, cr, re[2 * t + 1]);
            im[2 * t + 1] = fma2(hi, ci, im[2 * t + 1]);
          }
        }
      }
    }
    ColRows row(lmin);
#pragma unroll
    for (int li = 0; li < 4 * T; ++li) {
      if (li >= L) continue;
      const float x = li & 1 ? re[li / 2].y : re[li / 2].x, y = li & 1 ? im[li / 2].y : im[li / 2].x;
      float2* o1 = p.out + row.at(m, n) * p.out_zstride + z;
      float2* o2 = p.out + row.at(-m, -n) * p.out_zstride + z;
      row.next();
      if (p.mode == kSo3Real) {
        *o1 = make_float2(x, y);
        if (!self) *o2 = make_float2(fudge * x, -fudge * y);
      } else {  // += i * (x + i y); mirror += i * fudge * conj
        float2 q = *o1;
        *o1 = make_float2(q.x - y, q.y + x);
        if (!self) {
          q = *o2;
          *o2 = make_float2(q.x + fudge * y, q.y + fudge * x);
        }
      }
    }
  };
  if (LT == 1) degrees(std::integral_constant<int, 1>{});
  else if (LT == 2) degrees(std::integral_constant<int, 2>{});
  else if (LT == 3) degrees(std::integral_constant<int, 3>{});
  else degrees(std::integral_constant<int, 4>{});
}

// S[beta][z] = sum_l W[l][beta] Xs[l][z],  Xs = symmetrised spectrum (or S2 product); table as [l][beta]
enum ColProduct { kColPlain, kColProduct, kColRealProduct };     // (kColRealProduct: s2_mirror)
template <ColProduct kProduct>
S2C_D void inv_wigner_col(const Ctx& ctx, const InvWignerParams& p, unsigned char* smem) {
  const int N = p.N, NP = col_nb(N);
  const int pair = ctx.bid / p.nzt, zt = ctx.bid - pair * p.nzt;
  int m, n;
  so3_pair_decode(pair, p.K, m, n);
  const int am = m < 0 ? -m : m;
  const int lmin = am > n ? am : n;
  const int L = p.pan.nl - lmin;
  if (L <= 0) return;
  const int LT = (L + 3) / 4;
  float* Ws = reinterpret_cast<float*>(smem);   // [4 LT][NP]
  const float* panel = p.pan.data + p.pan.off[pair];
  const int z = zt * p.ZT + ctx.tid;
  const float fudge = ((m - n) & 1) ? -1.f : 1.f;
  const int nm = 2 * p.K - 1, mi = m + p.K - 1;
  float2* s = p.s + ((long)n * nm + mi) * N * p.nbatch + z;
  auto degrees = [&](auto tiles) {
    constexpr int T = decltype(tiles)::value;
    float2 x[4 * T];
    if constexpr (kProduct != kColPlain) {
      // the loads of four degrees are in flight together (one product after the other: 101 us at b = 10, 5120
      // signals; all degrees at once do not fit the registers); multiply-adds in the order of the single-kernel transforms
      const unsigned zz = (unsigned)(p.z0 + z), i = zz / (unsigned)p.s2_fout, j = zz - i * (unsigned)p.s2_fout;
      const long xs = (long)p.s2_nb * p.s2_fin, ys = (long)p.s2_fin * p.s2_fout;
      const float2* x0 = p.xs + (long)(lmin * lmin + lmin) * xs + (long)i * p.s2_fin;   // row (l, 0), l = lmin
      const float2* y0 = p.ys + (long)(lmin * lmin + lmin) * ys + j;
      int l = lmin;
      static_for<0, T>([&](auto tc) {
        constexpr int t = decltype(tc)::value;
        float2 a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) a[q] = b[q] = make_float2(0.f, 0.f);
        if (z < p.nbatch) {
          for (int k = 0; k < p.s2_fin; ++k) {
            const float2 *xr = x0 + k, *yr = y0 + (long)k * p.s2_fout;
            float2 u[4], v[4], u2[4], v2[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (4 * t + q < L) {
                u[q] = xr[m * xs];
                v[q] = yr[n * ys];
                if constexpr (kProduct == kColProduct) { u2[q] = xr[-m * xs]; v2[q] = yr[-n * ys]; }
              }
              xr += 2L * (l + q + 1) * xs;
              yr += 2L * (l + q + 1) * ys;
            }
            auto mul = [](float2 c, float2 d, float2& acc) {
              acc.x = fmaf(c.x, d.x, acc.x);
              acc.x = fmaf(c.y, d.y, acc.x);
              acc.y = fmaf(c.y, d.x, acc.y);
              acc.y = fmaf(-c.x, d.y, acc.y);
            };
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (4 * t + q >= L) continue;
              mul(u[q], v[q], a[q]);
              if constexpr (kProduct == kColProduct) mul(u2[q], v2[q], b[q]);
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if constexpr (kProduct == kColRealProduct) x[4 * t + q] = a[q];
          else x[4 * t + q] = make_float2(0.5f * (a[q].x + fudge * b[q].x), 0.5f * (a[q].y - fudge * b[q].y));
        }
        // rows (l, 0) -> (l + 4, 0): l (l + 1) grows by 8 l + 20
        x0 += (8L * l + 20) * xs;
        y0 += (8L * l + 20) * ys;
        l += 4;
      });
    } else {
      ColRows row(lmin);
#pragma unroll
      for (int li = 0; li < 4 * T; ++li) {
        x[li] = make_float2(0.f, 0.f);
        if (li >= L || z >= p.nbatch) continue;
        float2 a = p.x[row.at(m, n) * p.x_zstride + z];
        float2 b = p.x[row.at(-m, -n) * p.x_zstride + z];
        row.next();
        if (p.mode == kSo3RotI) {  // multiply the spectrum by -i
          a = make_float2(a.y, -a.x);
          b = make_float2(b.y, -b.x);
        }
        x[li] = make_float2(0.5f * (a.x + fudge * b.x), 0.5f * (a.y - fudge * b.y));
      }
    }
    for (int i = ctx.tid; i < 4 * T * NP; i += ctx.nthr) {
      const int l = i / NP, bt = i - l * NP;
      Ws[i] = l < L && bt < N ? panel[l * N + bt] : 0.f;
    }
    ctx.sync();
    if (z >= p.nbatch) return;
    float2* o = s;
    for (int b0 = 0; b0 < N; b0 += 4, o += 4L * p.nbatch) {
      float2 r0 = make_float2(0.f, 0.f), r1 = r0, i0 = r0, i1 = r0;   // two betas each
#pragma unroll
      for (int li = 0; li < 4 * T; ++li) {
        const float4 w4 = *reinterpret_cast<const float4*>(Ws + li * NP + b0);
        const float2 lo = make_float2(w4.x, w4.y), hi = make_float2(w4.z, w4.w);
        const float2 xr = make_float2(x[li].x, x[li].x), xi = make_float2(x[li].y, x[li].y);
        r0 = fma2(lo, xr, r0);
        i0 = fma2(lo, xi, i0);
        r1 = fma2(hi, xr, r1);
        i1 = fma2(hi, xi, i1);
      }
      o[0] = make_float2(r0.x, i0.x);
      o[p.nbatch] = make_float2(r0.y, i0.y);
      if (b0 + 2 < N) {
        o[2L * p.nbatch] = make_float2(r1.x, i1.x);
        o[3L * p.nbatch] = make_float2(r1.y, i1.y);
      }
    }
  };
  if (LT == 1) degrees(std::integral_constant<int, 1>{});
  else if (LT == 2) degrees(std::integral_constant<int, 2>{});
  else if (LT == 3) degrees(std::integral_constant<int, 3>{});
  else degrees(std::integral_constant<int, 4>{});
}
S2C_KERNEL_BOUNDS(so3_inv_wigner_col, InvWignerParams, kColZT, 6) { inv_wigner_col<kColPlain>(ctx, p, smem); }
S2C_KERNEL_BOUNDS(so3_inv_wigner_col_s2, InvWignerParams, kColZT, 6) { inv_wigner_col<kColProduct>(ctx, p, smem); }
S2C_KERNEL_BOUNDS(so3_inv_wigner_col_s2real, InvWignerParams, kColZT, 6) { inv_wigner_col<kColRealProduct>(ctx, p, smem); }

}  // namespace s2c
