// Register-tiled Wigner-d contractions for the general (large bandwidth) SO(3) path.
//
// Same inputs, outputs and arithmetic as so3_fwd_wigner / so3_inv_wigner (so3_kernels.h), i.e. the
// beta / l contraction of the reference's so3fft.cu / so3ifft.cu tile loops
// (s2cnn/soft/so3_fft.py:296-336 and :391-431), but organised as a small GEMM per frequency pair:
// a block stages the whole Wigner panel and a tile of up to 64 batch elements in shared memory and
// every thread owns 4 x 2 complex outputs, so that one pair of 16-byte shared-memory loads feeds
// 16 fused multiply-adds.
#pragma once

#include "backend.h"
#include "fft_device.h"
#include "so3_kernels.h"

namespace s2c {

constexpr int kWigZT = 64;  // batch elements per block tile (even): SO(3), and the most for S2
// kHalf, S2 transforms of real signals: the frequencies m >= 0 alone.  The two signs are then one sum, no longer two with
// independent roundings, of which whatever reads them takes the mean: terms are summed in chains of this many, which join
// the sum.  Relative errors at b = 64 with all frequencies / half in one chain / half in these, in 1e-7: symmetric part of a
// spectrum of 64 degrees 1.94 / 2.08 / 1.39, there and back 2.45 / 2.68 / 1.87, the signal of such a spectrum 1.28 / 1.45 /
// 1.10.  (Not quite for few degrees of a long grid, where the row transforms are most of the error: 20 degrees 0.92 / 1.05 /
// 1.00.)  192 signals at b = 64 with 64 degrees, one chain -> these: analysis 24.1 -> 25.0 us, synthesis 23.5 -> 24.2.
constexpr int kWigChain = 8, kWigChainBeta = 32;     // degrees (synthesis), betas (analysis)

// Rows of N mod 4 = 2 betas are staged with two columns of zeros.
S2C_HD constexpr int wig_np(int N) { return (N + 3) / 4 * 4; }
inline size_t fwd_wigner_t_smem(int N, int nl, int zt = kWigZT) {
  return (size_t)((nl + 3) / 4 * 4) * (wig_np(N) + 4) * sizeof(float) +
         (size_t)zt * (wig_np(N) + 2) * sizeof(float2);
}
// the kernels take 4 x 2 (or 4 x 1) outputs per thread and tile, two tiles per thread
inline bool fwd_wigner_t_fits(int N, int nl, int zt, int smem_limit) {
  return (nl + 3) / 4 * ((zt + 1) / 2) <= 2 * kThreads && fwd_wigner_t_smem(N, nl, zt) <= (size_t)smem_limit - 1024;
}
// Batch elements per block for the S2 transforms: only 2K - 1 table panels exist, so small batches take
// smaller tiles until about two blocks per SM are there.
inline int wig_s2_zt(int npairs, long nbatch) {
  int zt = kWigZT;
  while (zt > 8 && npairs * ((nbatch + zt - 1) / zt) < 2 * 148) zt /= 2;
  return zt;
}

// X[l][z] = sum_beta W[l][beta] V[z][beta]   (+ Hermitian mirror row)
//
// Panel rows and batch rows are staged exactly as they lie in memory (no transposition): the beta loop
// runs four samples at a time, a thread reads W[l][beta..beta+3] for its four degrees (the whole warp
// shares the address: broadcast) and V[z][beta..beta+3] for its two batch elements z = tz and
// tz + ceil(zc/2) (row stride N + 2 complex numbers, so the 8 lanes of a 16-byte access phase hit 8
// different bank groups).  S2 transforms (kS2) are the n = 0 column without mirror rows.
template <bool kHalf>
S2C_D void fwd_wigner_tiled(const Ctx& ctx, const FwdWignerParams& p, unsigned char* smem) {
  const int N = p.N, NH = wig_np(N);
  const int bt0 = ctx.bid / p.nzt, zt = ctx.bid - bt0 * p.nzt, pair = bt0 + (kHalf ? p.K - 1 : 0);
  int m, n;
  if (p.mode == kS2) { m = pair - (p.K - 1); n = 0; } else so3_pair_decode(pair, p.K, m, n);
  const int am = m < 0 ? -m : m;
  const int lmin = am > n ? am : n;
  const int L = p.nl - lmin;
  if (L <= 0) return;
  const int z0 = zt * p.ZT;
  const int zc = (p.nbatch - z0) < p.ZT ? (p.nbatch - z0) : p.ZT;
  const int LDW = NH + 4, LDV = NH + 2, ZH = (zc + 1) / 2;   // a thread's batch elements: tz, tz + ZH
  float* Ws = reinterpret_cast<float*>(smem);                                        // [nl up to 4][LDW]
  float2* Vs = reinterpret_cast<float2*>(Ws + (size_t)((p.nl + 3) / 4 * 4) * LDW);    // [ZT][LDV]
  const int LT = (L + 3) / 4;
  const float* panel = p.pan.data + p.pan.off[pair];
  const int nm = 2 * p.K - 1, mi = m + p.K - 1;
  const float2* vsrc = p.v + (((long)n * nm + mi) * p.nbatch + z0) * N;
  // 4 x 2 tiles (degrees x batch elements), or 4 x 1 when the pair has few degrees so that more
  // threads share the beta loop; at most two tiles per thread either way (LT <= 16, 256 threads)
  const bool narrow = LT * ZH < ctx.nthr;
  const int ntiles = narrow ? LT * zc : LT * ZH;
  float ar[2][4][2], ai[2][4][2];
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) { ar[t][i][0] = ar[t][i][1] = ai[t][i][0] = ai[t][i][1] = 0.f; }

  // kHalf: what is in the accumulators joins the sums of the chains before
  float sr[4][2], si[4][2];
  const int chain = kHalf ? kWigChainBeta : NH;
  auto next_chain = [&](int t) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        sr[i][j] += ar[t][i][j];
        si[i][j] += ai[t][i][j];
        ar[t][i][j] = ai[t][i][j] = 0.f;
      }
  };

  {
    if (N % 4 == 0) {
      const int n4 = NH / 4, total = LT * 4 * n4;                    // rows past L are zero
      for (int base = ctx.tid; base < total; base += 4 * ctx.nthr) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int idx = base + u * ctx.nthr;
          v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (idx < total && idx / n4 < L) {
            const int l = idx / n4, c4 = idx - l * n4;
            v[u] = *reinterpret_cast<const float4*>(panel + (long)l * N + 4 * c4);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int idx = base + u * ctx.nthr;
          if (idx < total) {
            const int l = idx / n4, c4 = idx - l * n4;
            *reinterpret_cast<float4*>(Ws + l * LDW + 4 * c4) = v[u];
          }
        }
      }
    } else {   // panel rows start on 8-byte boundaries only
      const int n2 = NH / 2, total = LT * 4 * n2;
      for (int idx = ctx.tid; idx < total; idx += ctx.nthr) {
        const int l = idx / n2, c2 = idx - l * n2;
        float2 v = make_float2(0.f, 0.f);
        if (l < L && 2 * c2 < N) v = *reinterpret_cast<const float2*>(panel + (long)l * N + 2 * c2);
        *reinterpret_cast<float2*>(Ws + l * LDW + 2 * c2) = v;
      }
    }
    {
      const int n2 = NH / 2, total = 2 * ZH * n2;                     // a row past zc is zero
      for (int base = ctx.tid; base < total; base += 4 * ctx.nthr) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int idx = base + u * ctx.nthr;
          v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (idx < total && idx / n2 < zc) {
            const int zz = idx / n2, c2 = idx - zz * n2;
            if (2 * c2 < N) v[u] = *reinterpret_cast<const float4*>(vsrc + (long)zz * N + 2 * c2);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int idx = base + u * ctx.nthr;
          if (idx < total) {
            const int zz = idx / n2, c2 = idx - zz * n2;
            *reinterpret_cast<float4*>(Vs + zz * LDV + 2 * c2) = v[u];
          }
        }
      }
    }
    ctx.sync();
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int tile = ctx.tid + t * ctx.nthr;
      if (tile >= ntiles) continue;
      if constexpr (kHalf) {
#pragma unroll
        for (int i = 0; i < 4; ++i) sr[i][0] = sr[i][1] = si[i][0] = si[i][1] = 0.f;
      }
      if (narrow) {
        const int tl = tile / zc, zz = tile - tl * zc;
        const float* wp = Ws + 4 * tl * LDW;
        const float2* vp = Vs + zz * LDV;
        for (int first = 0; first < NH; first += chain) {
          const int end = NH - first < chain ? NH : first + chain;
          for (int bt = first; bt < end; bt += 4) {
            const float4 va = *reinterpret_cast<const float4*>(vp + bt);
            const float4 vb = *reinterpret_cast<const float4*>(vp + bt + 2);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 w4 = *reinterpret_cast<const float4*>(wp + i * LDW + bt);
              ar[t][i][0] = fmaf(w4.x, va.x, ar[t][i][0]); ai[t][i][0] = fmaf(w4.x, va.y, ai[t][i][0]);
              ar[t][i][0] = fmaf(w4.y, va.z, ar[t][i][0]); ai[t][i][0] = fmaf(w4.y, va.w, ai[t][i][0]);
              ar[t][i][0] = fmaf(w4.z, vb.x, ar[t][i][0]); ai[t][i][0] = fmaf(w4.z, vb.y, ai[t][i][0]);
              ar[t][i][0] = fmaf(w4.w, vb.z, ar[t][i][0]); ai[t][i][0] = fmaf(w4.w, vb.w, ai[t][i][0]);
            }
          }
          if (kHalf) next_chain(t);
        }
      } else {
        const int tl = tile / ZH, tz = tile - tl * ZH;
        const float* wp = Ws + 4 * tl * LDW;
        const float2* v0 = Vs + tz * LDV;
        const float2* v1 = Vs + (tz + ZH) * LDV;
        for (int first = 0; first < NH; first += chain) {
          const int end = NH - first < chain ? NH : first + chain;
          for (int bt = first; bt < end; bt += 4) {
            float4 w4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w4[i] = *reinterpret_cast<const float4*>(wp + i * LDW + bt);
            const float4 a0 = *reinterpret_cast<const float4*>(v0 + bt);       // beta, beta+1 of z = tz
            const float4 b0 = *reinterpret_cast<const float4*>(v0 + bt + 2);   // beta+2, beta+3
            const float4 a1 = *reinterpret_cast<const float4*>(v1 + bt);       // z = tz + ZH
            const float4 b1 = *reinterpret_cast<const float4*>(v1 + bt + 2);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              ar[t][i][0] = fmaf(w4[i].x, a0.x, ar[t][i][0]); ai[t][i][0] = fmaf(w4[i].x, a0.y, ai[t][i][0]);
              ar[t][i][0] = fmaf(w4[i].y, a0.z, ar[t][i][0]); ai[t][i][0] = fmaf(w4[i].y, a0.w, ai[t][i][0]);
              ar[t][i][0] = fmaf(w4[i].z, b0.x, ar[t][i][0]); ai[t][i][0] = fmaf(w4[i].z, b0.y, ai[t][i][0]);
              ar[t][i][0] = fmaf(w4[i].w, b0.z, ar[t][i][0]); ai[t][i][0] = fmaf(w4[i].w, b0.w, ai[t][i][0]);
              ar[t][i][1] = fmaf(w4[i].x, a1.x, ar[t][i][1]); ai[t][i][1] = fmaf(w4[i].x, a1.y, ai[t][i][1]);
              ar[t][i][1] = fmaf(w4[i].y, a1.z, ar[t][i][1]); ai[t][i][1] = fmaf(w4[i].y, a1.w, ai[t][i][1]);
              ar[t][i][1] = fmaf(w4[i].z, b1.x, ar[t][i][1]); ai[t][i][1] = fmaf(w4[i].z, b1.y, ai[t][i][1]);
              ar[t][i][1] = fmaf(w4[i].w, b1.z, ar[t][i][1]); ai[t][i][1] = fmaf(w4[i].w, b1.w, ai[t][i][1]);
            }
          }
          if (kHalf) next_chain(t);
        }
      }
      if constexpr (kHalf) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) { ar[t][i][j] = sr[i][j]; ai[t][i][j] = si[i][j]; }
      }
    }
  }

  const float fudge = ((m - n) & 1) ? -1.f : 1.f;
  const bool self = (m == 0 && n == 0);
  auto emit = [&](int li, int zz, float re, float im) {
    if (li >= L || zz >= zc) return;
    const int l = lmin + li;
    if (p.mode == kS2) {
      float2* o = p.out + ((long)l * l + l) * p.out_zstride + z0 + zz;
      o[m * p.out_zstride] = make_float2(re, im);
      if (kHalf && m > 0) o[-m * p.out_zstride] = make_float2(fudge * re, -fudge * im);
      return;
    }
    float2* o1 = p.out + so3_row(l, m, n) * p.out_zstride + z0 + zz;
    float2* o2 = p.out + so3_row(l, -m, -n) * p.out_zstride + z0 + zz;
    if (p.mode == kSo3Real) {
      *o1 = make_float2(re, im);
      if (!self) *o2 = make_float2(fudge * re, -fudge * im);
    } else {  // += i * (re + i im); mirror += i * fudge * conj
      float2 c = *o1;
      *o1 = make_float2(c.x - im, c.y + re);
      if (!self) {
        c = *o2;
        *o2 = make_float2(c.x + fudge * im, c.y + fudge * re);
      }
    }
  };
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int tile = ctx.tid + t * ctx.nthr;
    if (tile >= ntiles) continue;
    if (narrow) {
      const int tl = tile / zc, zz = tile - tl * zc;
#pragma unroll
      for (int i = 0; i < 4; ++i) emit(4 * tl + i, zz, ar[t][i][0], ai[t][i][0]);
    } else {
      const int tl = tile / ZH, tz = tile - tl * ZH;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        emit(4 * tl + i, tz, ar[t][i][0], ai[t][i][0]);
        emit(4 * tl + i, tz + ZH, ar[t][i][1], ai[t][i][1]);
      }
    }
  }
}

S2C_KERNEL(so3_fwd_wigner_t, FwdWignerParams) { fwd_wigner_tiled<false>(ctx, p, smem); }
S2C_KERNEL_BOUNDS(s2_fwd_wigner_t_half, FwdWignerParams, kThreads, 3) { fwd_wigner_tiled<true>(ctx, p, smem); }

inline size_t inv_wigner_t_smem(int N, int K, int zt = kWigZT) {
  return (size_t)K * wig_np(N) * sizeof(float) + (size_t)K * (zt + 2) * sizeof(float2);
}

// one entry of s2_mm(xs, ys), multiply-adds in the order of cgemm_grouped
S2C_D float2 wig_s2_product(const InvWignerParams& p, int l, int m, int n, int i, int j) {
  const float2* xr = p.xs + ((long)(l * l + l + m) * p.s2_nb + i) * p.s2_fin;
  const float2* yr = p.ys + (long)(l * l + l + n) * p.s2_fin * p.s2_fout + j;
  float re = 0.f, im = 0.f;
  for (int k = 0; k < p.s2_fin; ++k) {
    const float2 a = xr[k], b = yr[(long)k * p.s2_fout];
    re = fmaf(a.x, b.x, re);
    re = fmaf(a.y, b.y, re);
    im = fmaf(a.x, -b.y, im);
    im = fmaf(a.y, b.x, im);
  }
  return make_float2(re, im);
}

// S[z][beta] = sum_l W[l][beta] Xs[l][z],  Xs = symmetrised spectrum
template <bool kHalf>
S2C_D void inv_wigner_tiled(const Ctx& ctx, const InvWignerParams& p, unsigned char* smem) {
  const int N = p.N, NP = wig_np(N);
  const int bt0 = ctx.bid / p.nzt, zt = ctx.bid - bt0 * p.nzt, pair = bt0 + (kHalf ? p.K - 1 : 0);
  int m, n;
  if (p.mode == kS2) { m = pair - (p.K - 1); n = 0; } else so3_pair_decode(pair, p.K, m, n);
  const int am = m < 0 ? -m : m;
  const int lmin = am > n ? am : n;
  const int L = p.pan.nl - lmin;
  if (L <= 0) return;
  const int z0 = zt * p.ZT;
  const int zc = (p.nbatch - z0) < p.ZT ? (p.nbatch - z0) : p.ZT;
  const int ZP = p.ZT + 2;
  float* Ws = reinterpret_cast<float*>(smem);                            // [L][NP]
  float2* Xs = reinterpret_cast<float2*>(Ws + (size_t)p.pan.nl * NP);     // [L][ZP]
  const int Z2 = (zc + 1) / 2;
  const float* panel = p.pan.data + p.pan.off[pair];
  if (N % 4 == 0) {
    const float4* src = reinterpret_cast<const float4*>(panel);
    float4* dst4 = reinterpret_cast<float4*>(Ws);
    const int total = L * N / 4;
    for (int base = ctx.tid; base < total; base += 4 * ctx.nthr) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (base + u * ctx.nthr < total) v[u] = src[base + u * ctx.nthr];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (base + u * ctx.nthr < total) dst4[base + u * ctx.nthr] = v[u];
    }
  } else {   // panel rows start on 8-byte boundaries only; two columns of padding
    const int n2 = NP / 2;
    for (int idx = ctx.tid; idx < L * n2; idx += ctx.nthr) {
      const int li = idx / n2, c2 = idx - li * n2;
      float2 v = make_float2(0.f, 0.f);
      if (2 * c2 < N) v = *reinterpret_cast<const float2*>(panel + (long)li * N + 2 * c2);
      *reinterpret_cast<float2*>(Ws + li * NP + 2 * c2) = v;
    }
  }
  const float fudge = ((m - n) & 1) ? -1.f : 1.f;
  for (int it = ctx.tid; it < L * Z2 * 2; it += ctx.nthr) {
    const int li = it / (Z2 * 2), zz = it - li * (Z2 * 2);
    float2 v = make_float2(0.f, 0.f);
    if (zz < zc && p.mode == kS2) {
      const long l = lmin + li;
      v = p.x[(l * l + l + m) * p.x_zstride + z0 + zz];
      if (kHalf) {
        const float2 w = p.x[(l * l + l - m) * p.x_zstride + z0 + zz];
        v = make_float2(0.5f * (v.x + fudge * w.x), 0.5f * (v.y - fudge * w.y));
      }
    } else if (zz < zc && p.xs) {
      const int l = lmin + li;
      const int z = (int)(p.z0 + z0 + zz), i = z / p.s2_fout, j = z - i * p.s2_fout;
      const float2 a = wig_s2_product(p, l, m, n, i, j);
      const float2 b = p.s2_real ? s2_mirror(a, m - n) : wig_s2_product(p, l, -m, -n, i, j);
      v = make_float2(0.5f * (a.x + fudge * b.x), 0.5f * (a.y - fudge * b.y));
    } else if (zz < zc) {
      const int l = lmin + li;
      float2 a = p.x[so3_row(l, m, n) * p.x_zstride + z0 + zz];
      float2 b = p.x[so3_row(l, -m, -n) * p.x_zstride + z0 + zz];
      if (p.mode == kSo3RotI) {  // multiply the spectrum by -i
        a = make_float2(a.y, -a.x);
        b = make_float2(b.y, -b.x);
      }
      v = make_float2(0.5f * (a.x + fudge * b.x), 0.5f * (a.y - fudge * b.y));
    }
    Xs[li * ZP + zz] = v;
  }
  ctx.sync();
  const int nm = 2 * p.K - 1, mi = m + p.K - 1;
  float2* dst = p.s + (((long)n * nm + mi) * p.nbatch + z0) * N;
  const int B4 = NP / 4;
  for (int tile = ctx.tid; tile < B4 * Z2; tile += ctx.nthr) {
    const int tz = tile / B4, tb = tile - tz * B4;  // consecutive threads -> consecutive beta
    float2 acc[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[j][i] = make_float2(0.f, 0.f);
    const float* wp = Ws + 4 * tb;
    const float2* xp = Xs + 2 * tz;
    float2 sum[2][4];
    const int chain = kHalf ? kWigChain : L;
    auto next_chain = [&]() {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sum[j][i] = fma2(acc[j][i], make_float2(1.f, 1.f), sum[j][i]);
          acc[j][i] = make_float2(0.f, 0.f);
        }
    };
    if constexpr (kHalf) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[j][i] = make_float2(0.f, 0.f);
    }
    for (int first = 0; first < L; first += chain) {
      const int end = L - first < chain ? L : first + chain;
      for (int li = first; li < end; ++li) {
        const float4 w4 = *reinterpret_cast<const float4*>(wp + li * NP);
        const float4 x4 = *reinterpret_cast<const float4*>(xp + li * ZP);  // (re0, im0, re1, im1)
        const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[0][i] = fma2(make_float2(w[i], w[i]), make_float2(x4.x, x4.y), acc[0][i]);
          acc[1][i] = fma2(make_float2(w[i], w[i]), make_float2(x4.z, x4.w), acc[1][i]);
        }
      }
      if (kHalf) next_chain();
    }
    if constexpr (kHalf) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = sum[j][i];
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int zz = 2 * tz + j;
      if (zz >= zc) continue;
      float4* o = reinterpret_cast<float4*>(dst + (long)zz * N + 4 * tb);
      o[0] = make_float4(acc[j][0].x, acc[j][0].y, acc[j][1].x, acc[j][1].y);
      if (4 * tb + 2 < N) o[1] = make_float4(acc[j][2].x, acc[j][2].y, acc[j][3].x, acc[j][3].y);
    }
  }
}

S2C_KERNEL(so3_inv_wigner_t, InvWignerParams) { inv_wigner_tiled<false>(ctx, p, smem); }
S2C_KERNEL_BOUNDS(s2_inv_wigner_t_half, InvWignerParams, kThreads, 4) { inv_wigner_tiled<true>(ctx, p, smem); }

}  // namespace s2c
