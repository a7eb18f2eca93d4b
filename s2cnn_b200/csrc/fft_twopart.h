// Mixed-radix FFT of compile-time length N = R1 * R2 in two register steps: the in-place decimation in
// frequency of fft_device.h (radices 4, 2, then odd primes ascending, digit-reversed output), its first
// stages - product R1 - run by one thread on the R1 elements j, j + R2, ..., its remaining stages - product
// R2 - by one thread on a block of R2 contiguous elements.  Every butterfly and twiddle is the one that
// fft_dif_inplace evaluates, in the same order and with the same table values, so the results are the
// same bit for bit; an element crosses shared memory once between the steps instead of once per stage,
// indices are compile-time, and the twiddles of the second step are immediates.
#pragma once

#include "fft_device.h"
#include "fft_reg.h"

namespace s2c {

// first radix of the plan for a length (host_math.h: fft_plan)
S2C_HD constexpr int two_radix(int len) { return fft_pick_radix(len); }
// R1: the shortest run of leading stages that leaves at most 16 elements, or one prime, for the second step
S2C_HD constexpr int two_r1(int n) {
  int r1 = 1, rest = n;
  while (rest > 16 && two_radix(rest) != rest) {
    const int r = two_radix(rest);
    r1 *= r;
    rest /= r;
  }
  return r1;
}
S2C_HD constexpr int two_r2(int n) { return n / two_r1(n); }
// frequency offset of block b after the leading stages of plan n (product r1): digits reversed
S2C_HD constexpr int two_block_freq(int n, int r1, int b) {
  int len = n, span = r1, f = 0, mul = 1;
  while (span > 1) {
    const int r = two_radix(len);
    len /= r;
    span /= r;
    f += (b / span) * mul;
    b %= span;
    mul *= r;
  }
  return f;
}

// ... and the block whose frequencies are f + r1 q (f < r1)
S2C_HD constexpr int two_freq_block(int n, int r1, int f) {
  int len = n, span = r1, b = 0;
  while (span > 1) {
    const int r = two_radix(len);
    len /= r;
    span /= r;
    b += (f % r) * span;
    f /= r;
  }
  return b;
}

// a * w^DIR with the roundings spelled out: which of the two products of a component is fused into the
// addition is the compiler's choice in ctw() (and changes with constant operands), but it decides the last
// bit, and a training step of a deep network amplifies last bits through its ReLUs and batch
// normalisation.  With this choice - in the general prime radices (PRIME: 7 and above) the imaginary part of
// the inverse direction fused the other way round - the outputs equal those of the three-pass kernels, whose
// stages call fft_dif_inplace, bit for bit on the GPU (tests/test_mid_bandwidths.py).
#ifndef S2C_EMUL
__device__ __forceinline__ float two_mul(float a, float b) { return __fmul_rn(a, b); }
#else
inline float two_mul(float a, float b) { return a * b; }
#endif
template <int DIR, bool PRIME = false>
S2C_D float2 two_ctw(float2 a, float2 w) {
  if constexpr (DIR > 0)
    return make_float2(fmaf(a.x, w.x, -two_mul(a.y, w.y)),
                       PRIME ? fmaf(a.y, w.x, two_mul(a.x, w.y)) : fmaf(a.x, w.y, two_mul(a.y, w.x)));
  else
    return make_float2(fmaf(a.x, w.x, two_mul(a.y, w.y)), fmaf(a.y, w.x, -two_mul(a.x, w.y)));
}
// ... with w a compile-time table entry; a multiplication by 1 is left out (it is exact)
template <int DIR, int K, int N, bool PRIME = false>
S2C_D float2 two_ctw_const(float2 a) {
  if constexpr (K % N == 0) return a;
  else return two_ctw<DIR, PRIME>(a, make_float2(Twiddle<K, N>::re, Twiddle<K, N>::im));
}

// butterfly of radix R within a transform of length N (table step N / R), as fft_butterfly
template <int DIR, int R, int N>
S2C_D void two_butterfly(float2 (&t)[R]) {
  if constexpr (R == 2 || R == 4) {
    reg_butterfly<DIR, R>(t);
  } else {
    float2 u[R];
    static_for<0, R>([&](auto pc) {
      constexpr int p = decltype(pc)::value;
      float2 acc = t[0];
      static_for<1, R>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        const float2 w = two_ctw_const<DIR, ((p * k) % R) * (N / R), N, (R > 5)>(t[k]);
        acc.x += w.x;
        acc.y += w.y;
      });
      u[p] = acc;
    });
    static_for<0, R>([&](auto pc) { t[decltype(pc)::value] = u[decltype(pc)::value]; });
  }
}

// First step: v[k] = x[j + R2 k]; S = elements (in k) per block at this stage.
template <int N, int R1, int S, int DIR>
S2C_D void two_head_stages(float2 (&v)[R1], int j, const float2* tw) {
  if constexpr (S > 1) {
    constexpr int R2 = N / R1, LEN = S * R2, R = two_radix(LEN), M = S / R, STEP = N / LEN;
    static_for<0, R1 / S>([&](auto bc) {
      constexpr int blk = decltype(bc)::value;
      static_for<0, M>([&](auto kc) {
        constexpr int k0 = decltype(kc)::value;
        float2 t[R];
        static_for<0, R>([&](auto qc) { t[decltype(qc)::value] = v[blk * S + k0 + decltype(qc)::value * M]; });
        two_butterfly<DIR, R, N>(t);
        v[blk * S + k0] = t[0];
        static_for<1, R>([&](auto pc) {
          constexpr int p = decltype(pc)::value;
          v[blk * S + k0 + p * M] = two_ctw<DIR>(t[p], tw[(j + k0 * R2) * p * STEP]);
        });
      });
    });
    two_head_stages<N, R1, M, DIR>(v, j, tw);
  }
}
template <int N, int DIR>
S2C_D void two_head(float2 (&v)[two_r1(N)], int j, const float2* tw) {
  two_head_stages<N, two_r1(N), two_r1(N), DIR>(v, j, tw);
}

// Second step on a block of R2 elements; output digit-reversed within the block.
template <int N, int R2, int LEN, int DIR>
S2C_D void two_tail_stages(float2 (&v)[R2]) {
  if constexpr (LEN > 1) {
    constexpr int R = two_radix(LEN), M = LEN / R, STEP = N / LEN;
    static_for<0, R2 / LEN>([&](auto bc) {
      constexpr int blk = decltype(bc)::value;
      static_for<0, M>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        float2 t[R];
        static_for<0, R>([&](auto qc) { t[decltype(qc)::value] = v[blk * LEN + j + decltype(qc)::value * M]; });
        two_butterfly<DIR, R, N>(t);
        static_for<0, R>([&](auto pc) {
          constexpr int p = decltype(pc)::value;
          v[blk * LEN + j + p * M] = two_ctw_const<DIR, j * p * STEP, N>(t[p]);
        });
      });
    });
    two_tail_stages<N, R2, M, DIR>(v);
  }
}

// Runs the second step and hands every result to emit(q, value): the value belongs to frequency
// two_block_freq(block) + R1 q.  A prime block above 13 is one direct transform whose rows run in a
// rolled loop with table twiddles (unrolled, 29 x 29 complex products would not fit the instruction cache).
template <int N, int DIR, class F>
S2C_D void two_tail(float2 (&v)[two_r2(N)], const float2* tw, F&& emit) {
  constexpr int R2 = two_r2(N);
  if constexpr (R2 > 13 && two_radix(R2) == R2) {
    constexpr int STEP = N / R2;
#pragma unroll 1
    for (int p = 0; p < R2; ++p) {
      float2 acc = v[0];
      int idx = 0;
#pragma unroll
      for (int k = 1; k < R2; ++k) {
        idx += p;
        idx = idx >= R2 ? idx - R2 : idx;
        const float2 w = two_ctw<DIR, true>(v[k], tw[idx * STEP]);
        acc.x += w.x;
        acc.y += w.y;
      }
      emit(p, acc);
    }
  } else {
    two_tail_stages<N, R2, R2, DIR>(v);
    static_for<0, R2>([&](auto qc) {
      constexpr int q = decltype(qc)::value;
      emit(q, v[fft_reg_pos<R2>(q)]);
    });
  }
}

}  // namespace s2c
