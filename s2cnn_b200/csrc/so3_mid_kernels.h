// Plane kernels of the SO(3) transform for 32 < N = 2b < 64: both row transforms of NB neighbouring
// (z, beta) planes in one kernel, between the signal and the [n][m][z][beta] array of the Wigner kernels
// (wigner_tiled.h).  Same arithmetic as so3_fwd_gamma + so3_fwd_alpha and so3_inv_alpha + so3_inv_gamma
// (so3_kernels.h; s2cnn/soft/so3_fft.py:40-42, 89-92, 181-199), bit for bit.
//
// What this replaces: two kernels per direction with a [z][n][beta][alpha] scratch array of 8 K N^2
// bytes per signal written and read between them (3.5 times the signal), each FFT stage a pass through
// shared memory with run-time index divisions and a block barrier.  At N = 60, 256 signals, the pair took
// 308 us (analysis) and 319 us (synthesis) - issue bound at 1.3 TB/s.
//
// Here a plane crosses shared memory four times (two two-step FFTs, fft_twopart.h), alternating between
// two buffers so that every step is separated by one block barrier and can write in the order the next one
// reads.  NB planes (2, or 4 where they fit) share a block because the Wigner side keeps beta innermost: a
// block then writes / reads runs of 16 - 32 bytes instead of 8.  Lanes run over the planes first, then
// over n, in every step that touches V or a column, with row strides = 2 mod 4 and plane strides that
// spread the planes over the remaining banks.
#pragma once

#include "backend.h"
#include "fft_twopart.h"
#include "so3_kernels.h"

namespace s2c {

S2C_HD constexpr bool mid_supported(int N) { return N > 32 && N < 64 && N % 2 == 0; }
S2C_HD constexpr int mid_nb(int N) { return N <= 44 ? 4 : 2; }
// Row strides (complex).  Odd, so that lanes that run down a column hit all banks (16 numbers of 8 bytes); where the
// leading step of a row transform writes R2 neighbours per row, the stride is R2 modulo 16 if that costs at most four
// numbers: lanes that go on to the next row then go on through the banks.  The synthesis reads two numbers at a time from
// buffer B, whose stride is 2 modulo 4.
S2C_HD constexpr int mid_lda(int N) {
  for (int ld = N + 1; ld <= N + 4; ++ld)
    if (ld % 2 == 1 && (ld - two_r2(N)) % 16 == 0) return ld;
  return N + 1;
}
S2C_HD constexpr int mid_ldb(int N, bool synthesis) { return !synthesis ? N + 1 : N % 4 == 2 ? N : N + 2; }
// plane strides: the planes of a block, which are the fastest index of the lanes where columns are touched, share the banks
S2C_HD constexpr int mid_plane(int N, int ld) {
  int ps = (N / 2) * ld;
  while (ps % 16 != 16 / mid_nb(N)) ++ps;
  return ps;
}
constexpr int kMidThreads = 256;
inline size_t mid_smem_bytes(int N) {
  const int b = std::max(mid_plane(N, mid_ldb(N, false)), mid_plane(N, mid_ldb(N, true)));
  return ((size_t)(N + 1) / 2 * 2 + (size_t)mid_nb(N) * (mid_plane(N, mid_lda(N)) + b) + 2) * sizeof(float2);
}

struct MidParams {
  const float* x;      // analysis: real signal, element e at x[e * stride + off]
  float* out;          // synthesis: the same
  long stride, off;
  float2* v;           // [n < K][m + K - 1][z < nbatch][beta]
  const float2* tw;
  const float* bias;   // synthesis, optional [nfeat]; feature of signal z is (z0 + z) % nfeat
  int nfeat;
  long z0;
  int nbatch, K;
  int relu;            // analysis: transform max(x, 0)
  const float* mask;   // synthesis, optional (unit stride): samples where this signal is <= 0 are written as 0
  float inv_k;         // 1 / K (index split without an integer division)
};

// it -> it / K, exact for the few thousand items of a block
S2C_D int mid_div(int it, float inv_k) { return (int)(((float)it + 0.5f) * inv_k); }

S2C_D void mid_ld(const float* p, float (&v)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
S2C_D void mid_ld(const float* p, float (&v)[2]) {
  const float2 a = *reinterpret_cast<const float2*>(p);
  v[0] = a.x; v[1] = a.y;
}

template <int N>
struct so3_fwd_mid_impl {
  static S2C_D void run(const Ctx& ctx, const MidParams& p, unsigned char* smem) {
    constexpr int R1 = two_r1(N), R2 = two_r2(N), H = N / 2, NB = mid_nb(N), LD = mid_lda(N), LDB = mid_ldb(N, false);
    constexpr int PSA = mid_plane(N, LD), PSB = mid_plane(N, LDB), G = (N + NB - 1) / NB;
    float2* tw = reinterpret_cast<float2*>(smem);
    float2* B = tw + (N + 1) / 2 * 2;
    float2* A = B + NB * PSB;
    const long z = ctx.bid / G;
    const int beta0 = (int)(ctx.bid - z * G) * NB;
    const int bc = N - beta0 < NB ? N - beta0 : NB;
    const int K = p.K;
    for (int i = ctx.tid; i < N; i += ctx.nthr) tw[i] = p.tw[i];
    ctx.sync();
    // ---- FFT over gamma of the packed row pairs (2 t, 2 t + 1), first step from global memory ------
    const long e00 = ((z * N + beta0) * N) * (long)N;
    for (int it = ctx.tid; it < bc * H * R2; it += ctx.nthr) {
      const int j = it % R2, row = it / R2, pl = row / H, t = row - pl * H;
      const long e0 = e00 + (long)row * 2 * N + j;       // planes of one z are adjacent: row = pl * H + t
      float2 v[R1];
      if (p.stride == 1) {
#pragma unroll
        for (int k = 0; k < R1; ++k) v[k] = make_float2(p.x[e0 + k * R2], p.x[e0 + N + k * R2]);
      } else {
#pragma unroll
        for (int k = 0; k < R1; ++k)
          v[k] = make_float2(p.x[(e0 + k * R2) * p.stride + p.off], p.x[(e0 + N + k * R2) * p.stride + p.off]);
      }
      if (p.relu) {
#pragma unroll
        for (int k = 0; k < R1; ++k) v[k] = make_float2(relu(v[k].x), relu(v[k].y));
      }
      two_head<N, -1>(v, j, tw);
      float2* a = A + pl * PSA + t * LD + j;
#pragma unroll
      for (int k = 0; k < R1; ++k) a[k * R2] = v[k];
    }
    ctx.sync();
    for (int it = ctx.tid; it < NB * H * R1; it += ctx.nthr) {
      const int b = it / (NB * H), row = it % (NB * H), pl = row / H, t = row - pl * H;
      if (pl >= bc) continue;
      const float2* a = A + pl * PSA + t * LD + b * R2;
      float2 v[R2];
#pragma unroll
      for (int i = 0; i < R2; ++i) v[i] = a[i];
      float2* o = B + pl * PSB + t * LDB + two_block_freq(N, R1, b);
      two_tail<N, -1>(v, tw, [&](int q, float2 val) { o[R1 * q] = val; });
    }
    ctx.sync();
    // ---- FFT over alpha of the kept columns, the Hermitian split of the packed pairs on load --------
    for (int it = ctx.tid; it < NB * K * R2; it += ctx.nthr) {
      const int pl = it % NB, jn = it / NB, j = mid_div(jn, p.inv_k), n = jn - j * K;
      if (pl >= bc) continue;
      const float2* bk = B + pl * PSB + n;
      const float2* bq = B + pl * PSB + (n == 0 ? 0 : N - n);
      float2 v[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        const int al = j + k * R2;                          // alpha: row 2 t (even) or 2 t + 1 (odd)
        const float2 zk = bk[(al >> 1) * LDB], zc = bq[(al >> 1) * LDB];
        v[k] = (al & 1) ? make_float2(0.5f * (zk.y + zc.y), -0.5f * (zk.x - zc.x))
                        : make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y - zc.y));
      }
      two_head<N, -1>(v, j, tw);
      float2* a = A + pl * PSA + n * LD + j;
#pragma unroll
      for (int k = 0; k < R1; ++k) a[k * R2] = v[k];
    }
    ctx.sync();
    const long mstride = (long)p.nbatch * N;
    for (int it = ctx.tid; it < NB * K * R1; it += ctx.nthr) {
      const int pl = it % NB, bn = it / NB, b = mid_div(bn, p.inv_k), n = bn - b * K;
      if (pl >= bc) continue;
      const float2* a = A + pl * PSA + n * LD + b * R2;
      float2 v[R2];
#pragma unroll
      for (int i = 0; i < R2; ++i) v[i] = a[i];
      const int f0 = two_block_freq(N, R1, b);
      float2* o = p.v + ((long)n * (2 * K - 1) * p.nbatch + z) * N + beta0 + pl;
      two_tail<N, -1>(v, tw, [&](int q, float2 val) {
        const int f = f0 + R1 * q, m = f < H ? f : f - N;
        if (m < K && m > (n == 0 ? -1 : -K)) o[(m + K - 1) * mstride] = val;   // n = 0: only m >= 0 is read
      });
    }
  }
};

template <int N>
struct so3_inv_mid_impl {
  static S2C_D void run(const Ctx& ctx, const MidParams& p, unsigned char* smem) {
    constexpr int R1 = two_r1(N), R2 = two_r2(N), H = N / 2, NB = mid_nb(N), LD = mid_lda(N), LDB = mid_ldb(N, true);
    constexpr int PSA = mid_plane(N, LD), PSB = mid_plane(N, LDB), G = (N + NB - 1) / NB;
    float2* tw = reinterpret_cast<float2*>(smem);
    float2* B = tw + (N + 1) / 2 * 2;                        // 16-byte aligned: read two numbers at a time
    float2* A = B + NB * PSB;
    const long z = ctx.bid / G;
    const int beta0 = (int)(ctx.bid - z * G) * NB;
    const int bc = N - beta0 < NB ? N - beta0 : NB;
    const int K = p.K;
    for (int i = ctx.tid; i < N; i += ctx.nthr) tw[i] = p.tw[i];
    ctx.sync();
    // ---- inverse FFT over m -> alpha of the kept columns ----------------------------------------------
    const long mstride = (long)p.nbatch * N;
    for (int it = ctx.tid; it < NB * K * R2; it += ctx.nthr) {
      const int pl = it % NB, jn = it / NB, j = mid_div(jn, p.inv_k), n = jn - j * K;
      if (pl >= bc) continue;
      const float2* s = p.v + ((long)n * (2 * K - 1) * p.nbatch + z) * N + beta0 + pl;
      float2 v[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        const int f = j + k * R2, m = f < H ? f : f - N;
        v[k] = make_float2(0.f, 0.f);
        if (m < K && m > -K) {
          if (n == 0 && m < 0) {                             // only m >= 0 is stored: Hermitian
            const float2 c = s[(K - 1 - m) * mstride];
            v[k] = make_float2(c.x, -c.y);
          } else {
            v[k] = s[(m + K - 1) * mstride];
          }
        }
      }
      two_head<N, +1>(v, j, tw);
      float2* a = A + pl * PSA + n * LD + j;
#pragma unroll
      for (int k = 0; k < R1; ++k) a[k * R2] = v[k];
    }
    ctx.sync();
    for (int it = ctx.tid; it < NB * K * R1; it += ctx.nthr) {
      const int pl = it % NB, bn = it / NB, b = mid_div(bn, p.inv_k), n = bn - b * K;
      const float2* a = A + pl * PSA + n * LD + b * R2;
      float2 v[R2];
#pragma unroll
      for (int i = 0; i < R2; ++i) v[i] = a[i];
      float2* o = B + pl * PSB + n * LDB + two_block_freq(N, R1, b);
      if (pl < bc) two_tail<N, +1>(v, tw, [&](int q, float2 val) { o[R1 * q] = val; });
    }
    ctx.sync();
    // ---- Hermitian inverse FFT over n -> gamma of the row pairs (2 t, 2 t + 1), packed on load ----------
    for (int it = ctx.tid; it < bc * H * R2; it += ctx.nthr) {
      const int t = it % H, pj = it / H, pl = pj / R2, j = pj - pl * R2;
      const float2* src = B + pl * PSB + 2 * t;
      float2 v[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        const int n = j + k * R2;
        if (n < K) {
          const float4 u = *reinterpret_cast<const float4*>(src + n * LDB);        // alpha = 2 t, 2 t + 1
          // T[alpha][0] is real for a Hermitian spectrum; its rounding-level imaginary part is dropped
          v[k] = n == 0 ? make_float2(u.x, u.z) : make_float2(u.x - u.w, u.y + u.z);   // T1 + i T2
        } else if (N - n < K) {
          const float4 u = *reinterpret_cast<const float4*>(src + (N - n) * LDB);
          v[k] = make_float2(u.x + u.w, u.z - u.y);                                    // conj(T1) + i conj(T2)
        } else {
          v[k] = make_float2(0.f, 0.f);
        }
      }
      two_head<N, +1>(v, j, tw);
      float2* a = A + pl * PSA + t * LD + j;
#pragma unroll
      for (int k = 0; k < R1; ++k) a[k * R2] = v[k];
    }
    ctx.sync();
    for (int it = ctx.tid; it < NB * H * R1; it += ctx.nthr) {
      const int b = it / (NB * H), row = it % (NB * H), pl = row / H, t = row - pl * H;
      if (pl >= bc) continue;
      const float2* a = A + pl * PSA + t * LD + b * R2;
      float2 v[R2];
#pragma unroll
      for (int i = 0; i < R2; ++i) v[i] = a[i];
      float2* o = B + pl * PSB + t * LDB + two_block_freq(N, R1, b);
      two_tail<N, +1>(v, tw, [&](int q, float2 val) { o[R1 * q] = val; });
    }
    ctx.sync();
    // ---- + bias, whole rows out ---------------------------------------------------------------------------
    float add = 0.f;
    if (p.bias) add = p.bias[(p.z0 + z) % p.nfeat];
    const long e00 = ((z * N + beta0) * N) * (long)N;
    constexpr int W = N % 4 == 0 ? 4 : 2, PR = N / W;        // samples per store, stores per row
    // the mask's loads of four steps are in flight together, ahead of the stores the compiler keeps them
    // behind (256 signals at b = 30: 409 us, 390 without a mask)
    constexpr int U = 4;
    const int total = bc * H * PR;
    for (int base = ctx.tid; base < total; base += U * ctx.nthr) {
      float k0[U][W], k1[U][W];
      if (p.mask) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int it = base + u * ctx.nthr;
          if (it >= total) break;
          const float* k = p.mask + e00 + (long)(it / PR) * 2 * N + it % PR * W;
          mid_ld(k, k0[u]);
          mid_ld(k + N, k1[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int it = base + u * ctx.nthr;
        if (it >= total) break;
        const int c = it % PR, row = it / PR, pl = row / H, t = row - pl * H;
        const float4* src = reinterpret_cast<const float4*>(B + pl * PSB + t * LDB + c * W);
        const long e0 = e00 + (long)row * 2 * N + c * W;
        float r0[W], r1[W];
#pragma unroll
        for (int i = 0; i < W / 2; ++i) {
          const float4 v = src[i];
          r0[2 * i] = v.x + add; r1[2 * i] = v.y + add;
          r0[2 * i + 1] = v.z + add; r1[2 * i + 1] = v.w + add;
        }
        if (p.mask) {
#pragma unroll
          for (int i = 0; i < W; ++i) {
            r0[i] = relu_grad(k0[u][i], r0[i]);
            r1[i] = relu_grad(k1[u][i], r1[i]);
          }
        }
        if (p.stride == 1) {
          if constexpr (W == 4) {
            *reinterpret_cast<float4*>(p.out + e0) = make_float4(r0[0], r0[1], r0[2], r0[3]);
            *reinterpret_cast<float4*>(p.out + e0 + N) = make_float4(r1[0], r1[1], r1[2], r1[3]);
          } else {
            *reinterpret_cast<float2*>(p.out + e0) = make_float2(r0[0], r0[1]);
            *reinterpret_cast<float2*>(p.out + e0 + N) = make_float2(r1[0], r1[1]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < W; ++i) {
            p.out[(e0 + i) * p.stride + p.off] = r0[i];
            p.out[(e0 + N + i) * p.stride + p.off] = r1[i];
          }
        }
      }
    }
  }
};

// by-product of the analysis: the plain sum of every signal, i.e. its (0, 0) bins summed over beta
struct MidSumsParams {
  const float2* v;     // V[n = 0][m = 0], element (z, beta) at v[z * zs + beta * bs]
  float* sums;
  int nbatch, N, zs, bs;
};
S2C_KERNEL(so3_mid_sums, MidSumsParams) {
  const int z = ctx.bid * ctx.nthr + ctx.tid;
  if (z >= p.nbatch) return;
  float s = 0.f;
  for (int b = 0; b < p.N; ++b) s += p.v[(long)z * p.zs + (long)b * p.bs].x;
  p.sums[z] = s;
}

#ifndef S2C_EMUL
template <int N>
__global__ void __launch_bounds__(kMidThreads, 3) so3_fwd_mid(const MidParams p) {
  extern __shared__ float4 s2c_dyn_smem[];
  Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};
  stream_order_wait();
  so3_fwd_mid_impl<N>::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));
  stream_order_next();
}
template <int N>
__global__ void __launch_bounds__(kMidThreads, 3) so3_inv_mid(const MidParams p) {
  extern __shared__ float4 s2c_dyn_smem[];
  Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};
  stream_order_wait();
  so3_inv_mid_impl<N>::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));
  stream_order_next();
}
S2C_LAUNCHER_N(so3_fwd_mid, MidParams)
S2C_LAUNCHER_N(so3_inv_mid, MidParams)
#endif

#define S2C_DISPATCH_MID(N, CALL)                                                            \
  switch (N) {                                                                               \
    case 34: { constexpr int kN = 34; CALL; } break;                                         \
    case 36: { constexpr int kN = 36; CALL; } break;                                         \
    case 38: { constexpr int kN = 38; CALL; } break;                                         \
    case 40: { constexpr int kN = 40; CALL; } break;                                         \
    case 42: { constexpr int kN = 42; CALL; } break;                                         \
    case 44: { constexpr int kN = 44; CALL; } break;                                         \
    case 46: { constexpr int kN = 46; CALL; } break;                                         \
    case 48: { constexpr int kN = 48; CALL; } break;                                         \
    case 50: { constexpr int kN = 50; CALL; } break;                                         \
    case 52: { constexpr int kN = 52; CALL; } break;                                         \
    case 54: { constexpr int kN = 54; CALL; } break;                                         \
    case 56: { constexpr int kN = 56; CALL; } break;                                         \
    case 58: { constexpr int kN = 58; CALL; } break;                                         \
    case 60: { constexpr int kN = 60; CALL; } break;                                         \
    case 62: { constexpr int kN = 62; CALL; } break;                                         \
    default: rc = s2c::fail(s2c::S2C_ERR_UNSUPPORTED, "no plane kernel for this length");    \
  }

}  // namespace s2c
