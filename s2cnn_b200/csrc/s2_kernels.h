// S2 transforms for the lengths N = 2b <= 128 (compile-time, fft_twopart.h / fft_reg.h).
//
//   s2_fwd_fused   analysis of a real signal with at most 32 degrees, one block per signal: the first
//                  layer of every network on this path.  The 2b rows are transformed over alpha two at a
//                  time (rows beta and beta + b packed into one complex FFT), separated, and one thread
//                  per coefficient (l, m) runs the Wigner contraction over beta from shared memory.
//   s2_fwd_rows    the row transforms of larger analyses (the contraction follows in so3_fwd_wigner_t,
//                  which reuses a table panel over many signals) ...
//   s2_inv_rows    ... and of every synthesis.
//
// Same values as the reference's s2_fft / s2_ifft (s2cnn/soft/s2_fft.py:13-107, kernels :151-223).
//
// The generic shared-memory FFT these replace ran every radix stage through shared memory with run-time
// index divisions; the contraction of the single-kernel analysis read one table row per lane (32 sectors
// per load) and now reads the table transposed, [beta][l, m] (whole lines per warp).
#pragma once

#include "backend.h"
#include "fft_twopart.h"
#include "so3_kernels.h"
#include "tables.h"

namespace s2c {

// ---- one row transform in two register steps, for any supported length ------------------------------
// head: x[j + R2 k], k < R1 -> values stored at [j + R2 k]; tail: block b of R2 contiguous values -> emit(q,
// value) for the frequency block_freq(b) + R1 q, to be stored at [b R2 + slot(q)] if it stays in place.
template <int N>
struct RowFft {
  static constexpr bool kTwoStep = N == 64 || N == 128;     // as fft_twostep.h: 8 x 8, 8 x 16
  static constexpr int R1 = kTwoStep ? 8 : two_r1(N), R2 = N / R1;
  template <int DIR>
  static S2C_D void head(float2 (&v)[R1], int j, const float2* tw) {
    if constexpr (kTwoStep) {
      fft_reg<R1, DIR>(v, tw);
      float2 u[R1];
      static_for<0, R1>([&](auto pc) {
        constexpr int p = decltype(pc)::value;
        u[p] = p == 0 ? v[fft_reg_pos<R1>(p)] : two_ctw<DIR>(v[fft_reg_pos<R1>(p)], tw[j * p]);
      });
      static_for<0, R1>([&](auto pc) { v[decltype(pc)::value] = u[decltype(pc)::value]; });
    } else {
      two_head<N, DIR>(v, j, tw);
    }
  }
  template <int DIR, class F>
  static S2C_D void tail(float2 (&v)[R2], const float2* tw, F&& emit) {
    if constexpr (kTwoStep) {
      fft_reg<R2, DIR>(v, tw);
      static_for<0, R2>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        emit(q, v[fft_reg_pos<R2>(q)]);
      });
    } else {
      two_tail<N, DIR>(v, tw, emit);
    }
  }
  static S2C_D int block_freq(int b) { return kTwoStep ? b : two_block_freq(N, R1, b); }
  static S2C_D int freq_block(int f) { return kTwoStep ? f : two_freq_block(N, R1, f); }   // its inverse, f < R1
};

S2C_HD constexpr bool s2_length(int N) {      // even, up to 128, prime factors up to 31
  if (N < 2 || N > 128 || N % 2) return false;
  int r = N;
  for (int p = 2; p <= 31; ++p)
    while (r % p == 0) r /= p;
  return r == 1;
}
constexpr int kS2FusedK = 32;                  // degrees of the single-kernel analysis
constexpr int kS2Rows = 32;                    // rows (betas) per block of the row kernels

// ---------------------------------------------------------------------------------------------
struct S2FwdFusedParams {
  const float* x;      // [nbatch][N][N] real
  float2* out;         // rows l*l + l + m of out_zstride complex
  long out_zstride;
  const float* wt;     // Wigner table [beta][K * K]
  const float2* tw;
  int K;               // b_out = number of degrees <= kS2FusedK
};
inline size_t s2_fwd_fused_smem(int N, int K) {
  return ((size_t)N + (size_t)(N / 2) * (N + 1) + 1) * sizeof(float2) + (size_t)(N / 2) * K * sizeof(float4);
}

template <int N>
struct s2_fwd_fused_impl {
  static S2C_D void run(const Ctx& ctx, const S2FwdFusedParams& p, unsigned char* smem) {
    using F = RowFft<N>;
    constexpr int R1 = F::R1, R2 = F::R2, H = N / 2, LD = N + 1;
    const int K = p.K, KK = K * K;
    float4* Vs = reinterpret_cast<float4*>(smem);                 // [t < H][m < K]: rows t and t + H
    float2* tw = reinterpret_cast<float2*>(Vs + H * K);
    float2* A = tw + N;                                            // packed rows [t < H][LD]
    const long z = ctx.bid;
    const float* src = p.x + z * (long)N * N;
    for (int i = ctx.tid; i < N; i += ctx.nthr) tw[i] = p.tw[i];
    ctx.sync();
    for (int it = ctx.tid; it < H * R2; it += ctx.nthr) {
      const int t = it / R2, j = it - t * R2;
      const float* e = src + t * N + j;
      float2 v[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) v[k] = make_float2(e[k * R2], e[H * N + k * R2]);
      F::template head<-1>(v, j, tw);
      float2* a = A + t * LD + j;
#pragma unroll
      for (int k = 0; k < R1; ++k) a[k * R2] = v[k];
    }
    ctx.sync();
    // every block stays in place, frequency block_freq(b) + R1 q at [b R2 + q]
    for (int it = ctx.tid; it < H * R1; it += ctx.nthr) {
      const int b = it / H, t = it - b * H;
      float2* a = A + t * LD + b * R2;
      float2 v[R2];
#pragma unroll
      for (int i = 0; i < R2; ++i) v[i] = a[i];
      F::template tail<-1>(v, tw, [&](int q, float2 val) { a[q] = val; });
    }
    ctx.sync();
    // row t: (zk + conj zc) / 2,  row t + H: (zk - conj zc) / (2 i), frequencies 0 <= m < K
    for (int it = ctx.tid; it < H * R1; it += ctx.nthr) {
      const int b = it / H, t = it - b * H, f0 = F::block_freq(b);
      const int bc = F::freq_block(f0 == 0 ? 0 : R1 - f0);
      const float2* ak = A + t * LD + b * R2;
      const float2* ac = A + t * LD + bc * R2;
      for (int q = 0, m = f0; m < K; ++q, m += R1) {
        // N - m = (R1 - f0) + R1 (R2 - 1 - q) for f0 > 0, R1 (R2 - q) for f0 = 0
        const float2 zk = ak[q], zc = ac[f0 == 0 ? (q == 0 ? 0 : R2 - q) : R2 - 1 - q];
        Vs[t * K + m] = make_float4(0.5f * (zk.x + zc.x), 0.5f * (zk.y - zc.y), 0.5f * (zk.y + zc.y),
                                    -0.5f * (zk.x - zc.x));
      }
    }
    ctx.sync();
    for (int o = ctx.tid; o < KK; o += ctx.nthr) {
      int l = (int)sqrtf((float)o);
      while (l * l > o) --l;
      while ((l + 1) * (l + 1) <= o) ++l;
      const int m = o - l * l - l;
      const float4* v = Vs + (m < 0 ? -m : m);
      const float sg = m < 0 ? -1.f : 1.f;      // a real signal: the coefficients of -m are conjugates
      const float* w = p.wt + o;
      float ar = 0.f, ai = 0.f;
#pragma unroll 4
      for (int t = 0; t < H; ++t) {
        const float w1 = w[t * KK], w2 = w[(t + H) * KK];
        const float4 u = v[t * K];
        ar = fmaf(w1, u.x, ar);
        ai = fmaf(w1, sg * u.y, ai);
        ar = fmaf(w2, u.z, ar);
        ai = fmaf(w2, sg * u.w, ai);
      }
      p.out[(long)o * p.out_zstride + z] = make_float2(ar, ai);
    }
  }
};

// ---------------------------------------------------------------------------------------------
struct S2RowsParams {
  const float* x;      // analysis: rows of N real, or of N complex when `complex`
  float* out;          // synthesis: the same
  int complex;
  float2* v;           // [m + K - 1][z][beta]
  const float2* tw;
  int nbatch, K;
  int half;            // only m >= 0 is written / read: real signals, V[-m] = conj V[m]
};
S2C_HD constexpr int s2_rows_groups(int N) { return (N + kS2Rows - 1) / kS2Rows; }
inline size_t s2_fwd_rows_smem(int N) { return ((size_t)N + (size_t)kS2Rows * (N + 1)) * sizeof(float2); }
inline size_t s2_inv_rows_smem(int N) { return ((size_t)N + 2 * (size_t)kS2Rows * (N + 1)) * sizeof(float2); }

template <int N>
struct s2_fwd_rows_impl {
  static S2C_D void run(const Ctx& ctx, const S2RowsParams& p, unsigned char* smem) {
    using F = RowFft<N>;
    constexpr int R1 = F::R1, R2 = F::R2, H = N / 2, LD = N + 1, G = s2_rows_groups(N);
    float2* tw = reinterpret_cast<float2*>(smem);
    float2* A = tw + N;
    const int K = p.K;
    const long z = ctx.bid / G;
    const int beta0 = (int)(ctx.bid - z * G) * kS2Rows;
    const int rows = N - beta0 < kS2Rows ? N - beta0 : kS2Rows;
    for (int i = ctx.tid; i < N; i += ctx.nthr) tw[i] = p.tw[i];
    ctx.sync();
    for (int it = ctx.tid; it < rows * R2; it += ctx.nthr) {
      const int row = it / R2, j = it - row * R2;
      const long e = (z * N + beta0 + row) * N + j;
      float2 v[R1];
      if (p.complex) {
#pragma unroll
        for (int k = 0; k < R1; ++k) v[k] = reinterpret_cast<const float2*>(p.x)[e + k * R2];
      } else {
#pragma unroll
        for (int k = 0; k < R1; ++k) v[k] = make_float2(p.x[e + k * R2], 0.f);
      }
      F::template head<-1>(v, j, tw);
      float2* a = A + row * LD + j;
#pragma unroll
      for (int k = 0; k < R1; ++k) a[k * R2] = v[k];
    }
    ctx.sync();
    // lanes over the rows: for every frequency a run of `rows` numbers in beta
    for (int it = ctx.tid; it < kS2Rows * R1; it += ctx.nthr) {
      const int b = it / kS2Rows, row = it - b * kS2Rows;
      if (row >= rows) continue;
      const float2* a = A + row * LD + b * R2;
      float2 v[R2];
#pragma unroll
      for (int i = 0; i < R2; ++i) v[i] = a[i];
      const int f0 = F::block_freq(b);
      float2* o = p.v + z * N + beta0 + row;
      F::template tail<-1>(v, tw, [&](int q, float2 val) {
        const int f = f0 + R1 * q, m = f < H ? f : f - N;
        if (m < K && m > (p.half ? -1 : -K)) o[(long)(m + K - 1) * p.nbatch * N] = val;
      });
    }
  }
};

template <int N>
struct s2_inv_rows_impl {
  static S2C_D void run(const Ctx& ctx, const S2RowsParams& p, unsigned char* smem) {
    using F = RowFft<N>;
    constexpr int R1 = F::R1, R2 = F::R2, H = N / 2, LD = N + 1, G = s2_rows_groups(N);
    float2* tw = reinterpret_cast<float2*>(smem);
    float2* A = tw + N;
    float2* B = A + kS2Rows * LD;
    const int K = p.K;
    const long z = ctx.bid / G;
    const int beta0 = (int)(ctx.bid - z * G) * kS2Rows;
    const int rows = N - beta0 < kS2Rows ? N - beta0 : kS2Rows;
    for (int i = ctx.tid; i < N; i += ctx.nthr) tw[i] = p.tw[i];
    ctx.sync();
    for (int it = ctx.tid; it < kS2Rows * R2; it += ctx.nthr) {
      const int j = it / kS2Rows, row = it - j * kS2Rows;
      if (row >= rows) continue;
      const float2* s = p.v + z * N + beta0 + row;
      float2 v[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        const int f = j + k * R2, m = f < H ? f : f - N;
        const bool other = p.half && m < 0;
        v[k] = (m < K && m > -K) ? s[(long)((other ? -m : m) + K - 1) * p.nbatch * N] : make_float2(0.f, 0.f);
        if (other) v[k].y = -v[k].y;
      }
      F::template head<+1>(v, j, tw);
      float2* a = A + row * LD + j;
#pragma unroll
      for (int k = 0; k < R1; ++k) a[k * R2] = v[k];
    }
    ctx.sync();
    for (int it = ctx.tid; it < kS2Rows * R1; it += ctx.nthr) {
      const int b = it / kS2Rows, row = it - b * kS2Rows;
      if (row >= rows) continue;
      const float2* a = A + row * LD + b * R2;
      float2 v[R2];
#pragma unroll
      for (int i = 0; i < R2; ++i) v[i] = a[i];
      float2* o = B + row * LD + F::block_freq(b);
      F::template tail<+1>(v, tw, [&](int q, float2 val) { o[R1 * q] = val; });
    }
    ctx.sync();
    const long e0 = (z * N + beta0) * (long)N;
    for (int it = ctx.tid; it < rows * N; it += ctx.nthr) {
      const int row = it / N, a = it - row * N;
      const float2 val = B[row * LD + a];
      if (p.complex) reinterpret_cast<float2*>(p.out)[e0 + it] = val;
      else p.out[e0 + it] = val.x;
    }
  }
};

#ifndef S2C_EMUL
template <int N>
__global__ void __launch_bounds__(256) s2_fwd_fused(const S2FwdFusedParams p) {
  extern __shared__ float4 s2c_dyn_smem[];
  Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};
  stream_order_wait();
  s2_fwd_fused_impl<N>::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));
  stream_order_next();
}
template <int N>
__global__ void __launch_bounds__(256) s2_fwd_rows(const S2RowsParams p) {
  extern __shared__ float4 s2c_dyn_smem[];
  Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};
  stream_order_wait();
  s2_fwd_rows_impl<N>::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));
  stream_order_next();
}
template <int N>
__global__ void __launch_bounds__(256) s2_inv_rows(const S2RowsParams p) {
  extern __shared__ float4 s2c_dyn_smem[];
  Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};
  stream_order_wait();
  s2_inv_rows_impl<N>::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));
  stream_order_next();
}
S2C_LAUNCHER_N(s2_fwd_fused, S2FwdFusedParams)
S2C_LAUNCHER_N(s2_fwd_rows, S2RowsParams)
S2C_LAUNCHER_N(s2_inv_rows, S2RowsParams)
#endif

// run-time N -> compile-time N, by bisection over 2, 4, ..., 128; lengths that s2_length refuses do not exist
template <int LO, int HI, class F>
inline int s2_dispatch(int N, F&& f) {
  if constexpr (LO == HI) {
    if constexpr (s2_length(2 * LO)) return f(std::integral_constant<int, 2 * LO>{});
    else return fail(S2C_ERR_UNSUPPORTED, "no S2 kernel for this length");
  } else {
    constexpr int MID = (LO + HI) / 2;
    return N <= 2 * MID ? s2_dispatch<LO, MID>(N, f) : s2_dispatch<MID + 1, HI>(N, f);
  }
}

}  // namespace s2c
