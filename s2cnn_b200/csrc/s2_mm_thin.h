// Gradients of s2_mm for layers with few input features (f_in <= kThinFi = 8; the first layer of
// the reference's models has 1 to 6):
//   gx[l,m,i,k] = sum_{n,j} gz[l,m,n,i,j] y[l,n,k,j]            (s2cnn/s2_mm.py:38-46, kernel :222-262)
//   gy[l,n,k,j] = sum_{m,i} conj(gz[l,m,n,i,j]) x[l,m,i,k]      (s2cnn/s2_mm.py:48-58, kernel :265-312)
// With f_in that small both are reductions over the large tensor gz with a handful of outputs per
// row or column - matrix-vector shaped, so the 64 x 64 tiles of cgemm_grouped would sit almost
// empty.  Here gz is streamed exactly once; the small operand is broadcast from shared memory
// (grad x) or read at a warp-uniform address (grad y).
#pragma once

#include "backend.h"
#include "fft_device.h"
#include "host_math.h"

namespace s2c {

constexpr int kThinFi = 8;           // largest f_in these kernels take
constexpr int kThinRows = 64;        // batch rows per block of the grad-x kernel
constexpr int kThinSlices = 4;       // slices of the n range per block of the grad-x kernel
// Terms that are summed in one chain before they join the rest.  With `real` a coefficient and its
// mirror are one sum, no longer two whose mean the transforms behind take: without the short chains the error of
// what they read grew by 1.25 - 1.45.
constexpr int kThinChain = 4;

struct S2ThinParams {
  const float2* gz;     // [nspec3(nl)][nb][fo]
  const float2* other;  // grad x: y [nl^2][fi][fo];  grad y: x [nl^2][nb][fi]
  float2* out;          // grad x: gx [nl^2][nb][fi]; grad y: gy [nl^2][fi][fo]
  int nl, nb, fi, fo;
  int real;             // gz and other are spectra of real signals: rows (l, m >= 0) of out, the others are their mirrors
};

// row (l, m) of block t of a tile: all rows l^2 + m, or those of m >= 0 (index l .. 2l) in order of l
struct ThinRow {
  int l, m;
};
S2C_D ThinRow thin_row(int t, int real);
S2C_HD int thin_rows(int nl, int real) { return real ? nl * (nl + 1) / 2 : nl * nl; }
// the mirror of a row's value: out[l, -m] = (-1)^m conj out[l, m]
S2C_D float2 thin_mirror(float2 v, int l, int m) { return ((m - l) & 1) ? make_float2(-v.x, v.y) : make_float2(v.x, -v.y); }

S2C_D int thin_isqrt(int v) {   // floor(sqrt(v)) for the small row indices used here
  int r = (int)sqrtf((float)v);
  while (r * r > v) --r;
  while ((r + 1) * (r + 1) <= v) ++r;
  return r;
}
S2C_D ThinRow thin_row(int t, int real) {
  ThinRow r;
  if (real) {
    r.l = (thin_isqrt(8 * t + 1) - 1) / 2;
    r.m = r.l + t - r.l * (r.l + 1) / 2;
  } else {
    r.l = thin_isqrt(t);
    r.m = t - r.l * r.l;
  }
  return r;
}

inline size_t s2_gradx_thin_smem(int nl, int fi, int fo) {
  const size_t ys = (size_t)(2 * nl - 1) * fi * fo * sizeof(float2);
  const size_t red = (size_t)kThinSlices * kThinRows * kThinFi * sizeof(float2);
  return ys + red;
}

// block = (l, m, tile of kThinRows batch rows); thread = (row, slice of n)
S2C_KERNEL(s2_mm_gradx_thin, S2ThinParams) {
  const int tiles_i = (p.nb + kThinRows - 1) / kThinRows;
  // largest degrees first: a block's work grows with 2l + 1, and the blocks that start last should
  // be the short ones
  const int rbid = ctx.nblk - 1 - ctx.bid;
  const int lm = rbid / tiles_i, itile = rbid - lm * tiles_i;
  const ThinRow tr = thin_row(lm, p.real);
  const int l = tr.l, m = tr.m;
  const int L = 2 * l + 1;
  float2* ys = reinterpret_cast<float2*>(smem);                     // [L][fi][fo]
  float2* red = ys + (size_t)(2 * p.nl - 1) * p.fi * p.fo;          // [slices][rows][kThinFi]
  {
    const float2* ysrc = p.other + (size_t)l * l * p.fi * p.fo;     // rows l^2 .. l^2 + L - 1
    for (int e = ctx.tid; e < L * p.fi * p.fo; e += ctx.nthr) ys[e] = ysrc[e];
  }
  ctx.sync();
  const int r = ctx.tid % kThinRows, slice = ctx.tid / kThinRows;
  const int i = itile * kThinRows + r;
  float2 acc[kThinFi];
#pragma unroll
  for (int k = 0; k < kThinFi; ++k) acc[k] = make_float2(0.f, 0.f);
  if (i < p.nb) {
    const long row0 = (long)so3_offset(l) + (long)m * L;
    for (int n = slice; n < L; n += kThinSlices) {
      const float2* g = p.gz + ((row0 + n) * p.nb + i) * p.fo;
      const float2* yn = ys + (size_t)n * p.fi * p.fo;
      for (int j0 = 0; j0 < p.fo; j0 += kThinChain) {
        float2 gv[kThinChain];
#pragma unroll
        for (int u = 0; u < kThinChain; ++u) gv[u] = j0 + u < p.fo ? g[j0 + u] : make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < kThinFi; ++k) {
          if (k < p.fi) {
            float2 part = make_float2(0.f, 0.f);
#pragma unroll
            for (int u = 0; u < kThinChain; ++u) {
              if (j0 + u < p.fo) {
                const float2 yv = yn[k * p.fo + j0 + u];
                part.x = fmaf(gv[u].x, yv.x, part.x);
                part.x = fmaf(-gv[u].y, yv.y, part.x);
                part.y = fmaf(gv[u].x, yv.y, part.y);
                part.y = fmaf(gv[u].y, yv.x, part.y);
              }
            }
            acc[k] = cadd(acc[k], part);
          }
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kThinFi; ++k) red[(slice * kThinRows + r) * kThinFi + k] = acc[k];
  ctx.sync();
  if (slice == 0 && i < p.nb) {
    float2* dst = p.out + ((long)(l * l + m) * p.nb + i) * p.fi;
#pragma unroll
    for (int k = 0; k < kThinFi; ++k) {
      if (k < p.fi) {
        float2 s = red[r * kThinFi + k];
        for (int sl = 1; sl < kThinSlices; ++sl) {
          const float2 t = red[(sl * kThinRows + r) * kThinFi + k];
          s.x += t.x;
          s.y += t.y;
        }
        dst[k] = s;
        if (p.real && m > l) p.out[((long)(l * l + 2 * l - m) * p.nb + i) * p.fi + k] = thin_mirror(s, l, m);
      }
    }
  }
}

inline int s2_grady_thin_threads(int fo) {
  int t = (1024 / fo) * fo;          // whole slices of fo threads
  return t < fo ? fo : t;
}
S2C_HD int s2_grady_sharers(int nthr, int outputs) {
  const int s = nthr / outputs;
  return s < 1 ? 1 : s > 16 ? 16 : s;
}
inline size_t s2_grady_thin_smem(int fo) {
  return (size_t)s2_grady_thin_threads(fo) * kThinFi * sizeof(float2);
}

// block = (l, n); thread = (slice of the batch rows, j); all of (m, i) is summed inside the block
S2C_KERNEL_BOUNDS(s2_mm_grady_thin, S2ThinParams, 1024, 1) {
  const int rbid = ctx.nblk - 1 - ctx.bid;     // largest degrees (the long blocks) first
  const ThinRow tr = thin_row(rbid, p.real);
  const int l = tr.l, n = tr.m;
  const int L = 2 * l + 1;
  const int nsl = ctx.nthr / p.fo;
  const int j = ctx.tid % p.fo, sl = ctx.tid / p.fo;
  float2* red = reinterpret_cast<float2*>(smem);   // [nthr][kThinFi]
  float2 acc[kThinFi];
#pragma unroll
  for (int k = 0; k < kThinFi; ++k) acc[k] = make_float2(0.f, 0.f);
  // the rows (m, i) in one run over the slices, eight in flight: with a loop over m around one over i a batch
  // smaller than the slices left most threads idle and every m waited for its own loads (f_out = 8, batch 32,
  // b = 30: 168 us)
  if (sl < nsl) {
    const float2* g0 = p.gz + ((long)so3_offset(l) + n) * p.nb * p.fo + j;
    const float2* x0 = p.other + (long)l * l * p.nb * p.fi;
    const long gm = (long)L * p.nb * p.fo;                  // from m to m + 1
    const int rows = L * p.nb, dm = nsl / p.nb, di = nsl - dm * p.nb;
    int m = sl / p.nb, i = sl - m * p.nb;
    for (int q = sl; q < rows; q += 8 * nsl) {
      float2 gv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        gv[u] = make_float2(0.f, 0.f);
        if (q + u * nsl < rows) gv[u] = g0[m * gm + (long)i * p.fo];
        m += dm;
        i += di;
        if (i >= p.nb) { i -= p.nb; ++m; }
      }
#pragma unroll
      for (int u0 = 0; u0 < 8; u0 += kThinChain) {
        // (one feature's chain at a time: the chains of all would not fit the 64 registers)
#pragma unroll
        for (int k = 0; k < kThinFi; ++k) {
          if (k < p.fi) {
            float2 part = make_float2(0.f, 0.f);
#pragma unroll
            for (int u = u0; u < u0 + kThinChain; ++u) {
              const int r = q + u * nsl;
              if (r < rows) {
                const float2 xv = x0[(long)r * p.fi + k];   // rows of x are contiguous in (m, i);  conj(gv) * xv
                part.x = fmaf(gv[u].x, xv.x, part.x);
                part.x = fmaf(gv[u].y, xv.y, part.x);
                part.y = fmaf(gv[u].x, xv.y, part.y);
                part.y = fmaf(-gv[u].y, xv.x, part.y);
              }
            }
            acc[k] = cadd(acc[k], part);
          }
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kThinFi; ++k) red[ctx.tid * kThinFi + k] = acc[k];
  ctx.sync();
  // The sum over the slices, in a fixed order and rounded once: it is the longest chain of all (128 slices at f_out = 8).  With
  // few outputs up to 16 threads share one (1 -> 8 channels, nl = 30, batch 7: 26.6 -> 19.6 us).
  const int outputs = p.fo * p.fi, sharers = s2_grady_sharers(ctx.nthr, outputs);
  struct Sum {
    double re = 0, im = 0;
  };
  auto write = [&](int e, const Sum& t) {
    const int k = e / p.fo, jj = e - k * p.fo;
    const float2 s = make_float2((float)t.re, (float)t.im);
    p.out[((long)(l * l + n) * p.fi + k) * p.fo + jj] = s;
    if (p.real && n > l) p.out[((long)(l * l + 2 * l - n) * p.fi + k) * p.fo + jj] = thin_mirror(s, l, n);
  };
  auto slices = [&](int e, int first) {
    const int k = e / p.fo, jj = e - k * p.fo;
    Sum t;
    for (int s2 = first; s2 < nsl; s2 += sharers) {
      const float2 v = red[(s2 * p.fo + jj) * kThinFi + k];
      t.re += v.x;
      t.im += v.y;
    }
    return t;
  };
  if (sharers == 1) {
    for (int e = ctx.tid; e < outputs; e += ctx.nthr) write(e, slices(e, 0));
  } else {
    Sum t;
    if (ctx.tid < outputs * sharers) t = slices(ctx.tid % outputs, ctx.tid / outputs);
    ctx.sync();                  // (the parts take the place of what they were made from)
    Sum* parts = reinterpret_cast<Sum*>(smem);
    if (ctx.tid < outputs * sharers) parts[ctx.tid] = t;
    ctx.sync();
    if (ctx.tid < outputs) {
      for (int g = 1; g < sharers; ++g) {
        t.re += parts[g * outputs + ctx.tid].re;
        t.im += parts[g * outputs + ctx.tid].im;
      }
      write(ctx.tid, t);
    }
  }
}

inline bool s2_mm_thin_supported(int nl, int fi, int fo) {
  return fi <= kThinFi && fo <= 1024 && s2_gradx_thin_smem(nl, fi, fo) <= 200 * 1024;
}

}  // namespace s2c
