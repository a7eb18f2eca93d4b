// Plane kernels of the SO(3) transform for small bandwidths (18 <= N = 2b <= 32) and LARGE batches: both row
// transforms of P neighbouring (z, beta) planes in one block, every 1-D FFT in the registers of one thread
// (fft_reg.h), between the signal and the V[n][m][beta][z] array of wigner_columns.h.
//
// The single-kernel transforms (so3_fused_kernels.h) keep the spectrum of four batch elements, the Wigner slice and
// the planes of a beta group in one block: at b = 16 that is 210 KB, one block of 16 warps per SM whose eight beta
// groups pass four block barriers each (0.34 instructions per clock and scheduler, 4 of 12 stall cycles at
// barriers).  For a large batch the Wigner contraction is better off on its own - a block shares each table row
// among 128 signals - and what is left needs one barrier and 35 KB: several blocks per SM overlap their loads,
// transforms and stores.  2560 signals at b = 15: analysis 398 -> 198 us, synthesis 437 -> 218 (floor, the signal
// once: 44 us); half of it is this file's kernels (latency: 20 warps per SM, L1 at 65 %), half the Wigner step.
//
//   so3_fwd_small    two real rows per thread (optional ReLU on load) -> n -> columns alpha -> m -> V
//   so3_inv_small    V -> columns m -> alpha -> two rows per thread n -> gamma (+ bias, mask) -> store
//   so3_relay_small  the synthesis, + bias, ReLU, forward row transform in the same registers, then the rest of
//                    the analysis: the signal between two layers never exists in memory
//
// The planes of a block are consecutive in (beta, z), so that V is moved in runs of 8 P bytes.  Same FFTs, same
// sums in the same order as the single-kernel transforms: the results are the same bit for bit.
#pragma once

#include "backend.h"
#include "fft_reg.h"
#include "so3_fused_kernels.h"
#include "so3_kernels.h"

namespace s2c {

S2C_HD constexpr bool small_supported(int N) { return N >= 18 && N <= 32 && N % 2 == 0; }
S2C_HD constexpr int small_planes(int N) { return 256 / N / 4 * 4 < 8 ? 8 : 256 / N / 4 * 4; }
S2C_HD constexpr int small_threads(int N) { return (small_planes(N) * (N / 2) + 31) / 32 * 32; }
S2C_HD constexpr int small_kp(int N) { return N / 2 | 1; }                 // odd row stride (complex)
// plane stride: the lanes of a column phase run over the planes, then over n
S2C_HD constexpr int small_ps(int N) {
  int ps = N * small_kp(N);
  while (ps % 16 != (small_planes(N) < 12 ? 2 : 1)) ++ps;
  return ps;
}
inline size_t small_smem_bytes(int N) { return (size_t)small_planes(N) * small_ps(N) * sizeof(float2); }

struct SmallParams {
  const float* x;      // analysis: real signal, element e at x[e * stride + off]
  float* out;          // synthesis: the same
  long stride, off;
  float2* v;           // [n < K][m + K - 1][beta][z]: analysis output, synthesis / relay input
  float2* v2;          // relay output, bandwidth K2
  const float* bias;   // optional [nfeat]; feature of signal z is (z0 + z) % nfeat
  int nfeat;
  long z0;
  const float* mask;   // synthesis, optional (unit stride): samples where this signal is <= 0 are written as 0
  int relu;
  long nplanes;        // signals * N, plane q is (beta = q / nz, z = q % nz)
  int nz;              // signals
  int K, K2;
};

// 8 bytes from global to shared memory, not through registers
#ifndef S2C_EMUL
S2C_D void small_copy(float2* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
S2C_D void small_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
#else
S2C_D void small_copy(float2* dst, const float* src) { *dst = *reinterpret_cast<const float2*>(src); }
S2C_D void small_copy_wait() {}
#endif

template <int N>
struct Small {
  static constexpr int P = small_planes(N), H = N / 2, KP = small_kp(N), PS = small_ps(N);

  // columns of the K kept frequencies n: thread = (plane, n)
  static S2C_D void columns_inv(const Ctx& ctx, const SmallParams& p, long q0, float2* planes) {
    const int pl = ctx.tid % P, n = ctx.tid / P, K = p.K;
    if (n >= K || q0 + pl >= p.nplanes) return;
    const float2* s = p.v + ((long)n * (2 * K - 1) + K - 1) * p.nplanes + q0 + pl;      // frequency m = 0
    float2 v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int m = i < H ? i : i - N;
      v[i] = make_float2(0.f, 0.f);
      if (m < K && m > -K) v[i] = s[(m < 0 && n == 0 ? -m : m) * p.nplanes];
    }
    if (n == 0) {                                            // only m >= 0 is stored: Hermitian
#pragma unroll
      for (int i = H; i < N; ++i) v[i].y = -v[i].y;
    }
    fft_reg<N, +1>(v, nullptr);
    float2* col = planes + pl * PS + n;
    static_for<0, N>([&](auto ic) {
      constexpr int a = decltype(ic)::value;
      col[a * KP] = v[fft_reg_pos<N>(a)];
    });
  }
  static S2C_D void columns_fwd(const Ctx& ctx, const SmallParams& p, long q0, const float2* planes, float2* out, int K) {
    const int pl = ctx.tid % P, n = ctx.tid / P;
    if (n >= K || q0 + pl >= p.nplanes) return;
    const float2* col = planes + pl * PS + n;
    float2 v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = col[i * KP];
    fft_reg<N, -1>(v, nullptr);
    float2* o = out + ((long)n * (2 * K - 1) + K - 1) * p.nplanes + q0 + pl;
    static_for<0, N>([&](auto ic) {
      constexpr int f = decltype(ic)::value;
      constexpr int m = f < H ? f : f - N;
      if (m < K && m > (n == 0 ? -1 : -K)) o[m * p.nplanes] = v[fft_reg_pos<N>(f)];
    });
  }

  // rows alpha = ap, ap + N/2 of a plane: one complex transform for two real rows
  static S2C_D void pack_rows(const float2* r1, int K, float2 (&v)[N]) {
    const float2* r2 = r1 + H * KP;
    {
      const float2 t1 = r1[0], t2 = r2[0];
      v[0] = make_float2(t1.x, t2.x);  // T[alpha][0] is real for a Hermitian spectrum
    }
    v[H] = make_float2(0.f, 0.f);
#pragma unroll
    for (int n = 1; n < H; ++n) {
      if (n < K) {
        const float2 t1 = r1[n], t2 = r2[n];
        v[n] = make_float2(t1.x - t2.y, t1.y + t2.x);      // T1 + i T2
        v[N - n] = make_float2(t1.x + t2.y, t2.x - t1.y);  // conj(T1) + i conj(T2)
      } else {
        v[n] = make_float2(0.f, 0.f);
        v[N - n] = make_float2(0.f, 0.f);
      }
    }
  }
  static S2C_D void split_rows(float2* r1, int K, const float2 (&v)[N]) {
    float2* r2 = r1 + H * KP;
    static_for<0, H>([&](auto ic) {
      constexpr int n = decltype(ic)::value;
      constexpr int pn = fft_reg_pos<N>(n), pq = fft_reg_pos<N>(n == 0 ? 0 : N - n);
      if (n < K) {
        const float2 zk = v[pn], zq = v[pq];
        r1[n] = make_float2(0.5f * (zk.x + zq.x), 0.5f * (zk.y - zq.y));
        r2[n] = make_float2(0.5f * (zk.y + zq.y), -0.5f * (zk.x - zq.x));
      }
    });
  }

  // Planes of a real signal go through the rows' own places in shared memory (row stride KP complex >= N floats), so
  // that the lanes of a warp touch neighbouring samples in memory: a row per thread would take 32 cache lines per
  // access (b = 15: 81 % of the L1 rate).  f(alpha, place in shared memory, offset in the signal) for every two samples; a
  // thread keeps its plane and gamma and steps over alpha, so that all addresses are constants apart.
  template <int A0 = 0, int A1 = N, class F>
  static S2C_D void samples(const Ctx& ctx, const SmallParams& p, long q0, float2* planes, F&& f) {
    const int c = ctx.tid % H, pl = ctx.tid / H;
    if (pl >= P || q0 + pl >= p.nplanes) return;
    const int beta = (int)((q0 + pl) / p.nz), z = (int)(q0 + pl - (long)beta * p.nz);
    const long base = ((long)z * N + beta) * (N * N) + 2 * c;
    float2* place = planes + pl * PS + c;
#pragma unroll
    for (int a = A0; a < A1; ++a) f(a, place + a * KP, base + a * N);
  }
};

template <int N>
struct so3_fwd_small_impl {
  static S2C_D void run(const Ctx& ctx, const SmallParams& p, unsigned char* smem) {
    using S = Small<N>;
    constexpr int H = N / 2;
    float2* planes = reinterpret_cast<float2*>(smem);
    const long q0 = (long)ctx.bid * S::P;
    if (p.stride == 1) {
      S::samples(ctx, p, q0, planes, [&](int, float2* place, long at) { small_copy(place, p.x + at); });
      small_copy_wait();
      ctx.sync();
    }
    const int ap = ctx.tid % H, pl = ctx.tid / H;
    if (pl < S::P && q0 + pl < p.nplanes) {
      float2* r1 = planes + pl * S::PS + ap * S::KP;
      float2 v[N];
      if (p.stride == 1) {
#pragma unroll
        for (int c = 0; c < H; ++c) {
          const float2 a = r1[c], b = r1[H * S::KP + c];
          v[2 * c] = make_float2(a.x, b.x);
          v[2 * c + 1] = make_float2(a.y, b.y);
        }
      } else {
        const int beta = (int)((q0 + pl) / p.nz), z = (int)(q0 + pl - (long)beta * p.nz);
        const long row1 = (((long)z * N + beta) * N + ap) * (long)N, row2 = row1 + (long)H * N;
#pragma unroll
        for (int g = 0; g < N; ++g)
          v[g] = make_float2(p.x[(row1 + g) * p.stride + p.off], p.x[(row2 + g) * p.stride + p.off]);
      }
      if (p.relu) {
#pragma unroll
        for (int g = 0; g < N; ++g) v[g] = make_float2(relu(v[g].x), relu(v[g].y));
      }
      fft_reg<N, -1>(v, nullptr);
      S::split_rows(r1, p.K, v);        // in place: a thread owns its two rows
    }
    ctx.sync();
    S::columns_fwd(ctx, p, q0, planes, p.v, p.K);
  }
};

template <int N>
struct so3_inv_small_impl {
  static S2C_D void run(const Ctx& ctx, const SmallParams& p, unsigned char* smem) {
    using S = Small<N>;
    constexpr int H = N / 2;
    float2* planes = reinterpret_cast<float2*>(smem);
    const long q0 = (long)ctx.bid * S::P;
    S::columns_inv(ctx, p, q0, planes);
    ctx.sync();
    const int ap = ctx.tid % H, pl = ctx.tid / H;
    if (pl < S::P && q0 + pl < p.nplanes) {
      float2* r1 = planes + pl * S::PS + ap * S::KP;
      float2 v[N];
      S::pack_rows(r1, p.K, v);
      fft_reg<N, +1>(v, nullptr);
      const int beta = (int)((q0 + pl) / p.nz), z = (int)(q0 + pl - (long)beta * p.nz);
      float add = 0.f;
      if (p.bias) add = p.bias[(p.z0 + z) % p.nfeat];
      if (p.stride == 1) {
        static_for<0, H>([&](auto ic) {
          constexpr int c = decltype(ic)::value, pa = fft_reg_pos<N>(2 * c), pb = fft_reg_pos<N>(2 * c + 1);
          r1[c] = make_float2(v[pa].x + add, v[pb].x + add);
          r1[H * S::KP + c] = make_float2(v[pa].y + add, v[pb].y + add);
        });
      } else {
        const long row1 = (((long)z * N + beta) * N + ap) * (long)N, row2 = row1 + (long)H * N;
        static_for<0, N>([&](auto ic) {
          constexpr int g = decltype(ic)::value;
          constexpr int pg = fft_reg_pos<N>(g);
          p.out[(row1 + g) * p.stride + p.off] = v[pg].x + add;
          p.out[(row2 + g) * p.stride + p.off] = v[pg].y + add;
        });
      }
    }
    if (p.stride != 1) return;
    ctx.sync();
    if (!p.mask) {
      S::samples(ctx, p, q0, planes, [&](int, float2* place, long at) { *reinterpret_cast<float2*>(p.out + at) = *place; });
      return;
    }
    // the mask's loads of a quarter of the rows are in flight together: the compiler keeps a load behind the stores
    // before it (one by one: 434 us for 3200 signals at b = 16, 839 MB; so: 190)
    constexpr int G = (N + 3) / 4;
    static_for<0, 4>([&](auto gc) {
      constexpr int A0 = decltype(gc)::value * G, A1 = A0 + G < N ? A0 + G : N;
      float2 keep[G];
      S::template samples<A0, A1>(ctx, p, q0, planes, [&](int a, float2*, long at) {
        keep[a - A0] = *reinterpret_cast<const float2*>(p.mask + at);
      });
      S::template samples<A0, A1>(ctx, p, q0, planes, [&](int a, float2* place, long at) {
        const float2 k = keep[a - A0], v = *place;
        *reinterpret_cast<float2*>(p.out + at) = make_float2(relu_grad(k.x, v.x), relu_grad(k.y, v.y));
      });
    });
  }
};

template <int N>
struct so3_relay_small_impl {
  static S2C_D void run(const Ctx& ctx, const SmallParams& p, unsigned char* smem) {
    using S = Small<N>;
    constexpr int H = N / 2;
    float2* planes = reinterpret_cast<float2*>(smem);
    const long q0 = (long)ctx.bid * S::P;
    S::columns_inv(ctx, p, q0, planes);
    ctx.sync();
    const int ap = ctx.tid % H, pl = ctx.tid / H;
    if (pl < S::P && q0 + pl < p.nplanes) {
      float2* r1 = planes + pl * S::PS + ap * S::KP;
      float2 v[N];
      S::pack_rows(r1, p.K, v);
      fft_reg<N, +1>(v, nullptr);
      float add = 0.f;
      if (p.bias) add = p.bias[(p.z0 + (q0 + pl) % p.nz) % p.nfeat];
      float2 u[N];
      static_for<0, N>([&](auto gc) {
        constexpr int g = decltype(gc)::value;
        constexpr int pg = fft_reg_pos<N>(g);
        const float a1 = v[pg].x + add, a2 = v[pg].y + add;   // samples gamma = g of both rows
        u[g] = make_float2(relu(a1), relu(a2));
      });
      fft_reg<N, -1>(u, nullptr);
      S::split_rows(r1, p.K2, u);      // in place: a thread owns its two rows
    }
    ctx.sync();
    S::columns_fwd(ctx, p, q0, planes, p.v2, p.K2);
  }
};

// Six blocks of 128 threads per SM (85 registers); N = 32 needs a few more and is faster with five (2560 signals:
// 259 against 294 us) - the spills of 80 registers cost more than the sixth block gives.
#ifndef S2C_EMUL
#define S2C_SMALL_KERNEL(name)                                                                   \
  template <int N>                                                                               \
  __global__ void __launch_bounds__(small_threads(N), N == 32 ? 5 : 768 / small_threads(N)) name(const SmallParams p) {                \
    extern __shared__ float4 s2c_dyn_smem[];                                                     \
    Ctx ctx{(int)threadIdx.x, (int)blockDim.x, (int)blockIdx.x, (int)gridDim.x};                 \
    stream_order_wait();                                                                           \
    name##_impl<N>::run(ctx, p, reinterpret_cast<unsigned char*>(s2c_dyn_smem));                 \
    stream_order_next();  \
  }                                                                                              \
  S2C_LAUNCHER_N(name, SmallParams)
S2C_SMALL_KERNEL(so3_fwd_small)
S2C_SMALL_KERNEL(so3_inv_small)
S2C_SMALL_KERNEL(so3_relay_small)
#endif
#define S2C_LAUNCH_SMALL(name, N, stream, params)                                                \
  S2C_LAUNCH_N(name, N, ((params).nplanes + small_planes(N) - 1) / small_planes(N), small_threads(N), small_smem_bytes(N), stream, params)
#define S2C_DISPATCH_SMALL(N, CALL)                                                              \
  switch (N) {                                                                                   \
    case 18: { constexpr int kN = 18; CALL; } break;                                             \
    case 20: { constexpr int kN = 20; CALL; } break;                                             \
    S2C_CASES_32(CALL)                                                                           \
    default: rc = s2c::fail(s2c::S2C_ERR_UNSUPPORTED, "no plane kernel for this length");        \
  }

}  // namespace s2c
