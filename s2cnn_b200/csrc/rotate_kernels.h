// Rotation of an SO(3) spectrum by block-diagonal Wigner-D matrices (s2cnn/soft/so3_rotation.py:22-41):
//   adjoint = 0:  z[l,m,n,b]  = sum_k conj(U^l[m,k]) x[l,k,n,b]
//   adjoint = 1:  gx[l,k,n,b] = sum_m      U^l[m,k]  gz[l,m,n,b]      (transpose of the above)
// U is the concatenation over l of the L x L matrices, L = 2l+1; x / z are [nspec3, nbatch], so for a degree
// this is an L x L matrix times an L x (L nbatch) one.  L is at most a few dozen: the 64 x 64 x 16 tiles of
// cgemm_grouped were mostly padding, their K loop two barriers per 16 (256 signals, b = 12: 29 us).  Here a block
// keeps kRotRows rows of the matrix in shared memory, a thread owns two columns and those rows, and x streams
// through registers; the tiles of one column range run side by side, so x comes from HBM once and from L2 after
// that.
#pragma once

#include "backend.h"
#include "host_math.h"

namespace s2c {

constexpr int kRotRows = 8, kRotThreads = 128;

struct RotateParams {
  const float2* U;
  const float2* x;
  float2* z;
  int nl, adjoint;
  long nbatch;
};

S2C_HD long rot_col_tiles(int l, long nbatch) { return ((2 * l + 1) * nbatch + 2 * kRotThreads - 1) / (2 * kRotThreads); }
S2C_HD long rot_row_tiles(int l) { return (2 * l + 1 + kRotRows - 1) / kRotRows; }
inline long rot_blocks(int nl, long nbatch) {
  long t = 0;
  for (int l = 0; l < nl; ++l) t += rot_col_tiles(l, nbatch) * rot_row_tiles(l);
  return t;
}
inline size_t rot_smem_bytes(int nl) { return (size_t)(2 * nl - 1) * kRotRows * sizeof(float2); }

S2C_KERNEL(so3_rotate_rows, RotateParams) {
  int l = p.nl - 1;            // largest degrees first
  long t = ctx.bid;
  for (;; --l) {
    const long c = rot_col_tiles(l, p.nbatch) * rot_row_tiles(l);
    if (t < c) break;
    t -= c;
  }
  const int L = 2 * l + 1, rt = (int)rot_row_tiles(l);
  const int row0 = (int)(t % rt) * kRotRows;
  const long col0 = t / rt * (2 * kRotThreads), C = L * p.nbatch;
  const long spec0 = (long)l * (4L * l * l - 1) / 3;
  float2* Us = reinterpret_cast<float2*>(smem);               // [k][kRotRows], zeros past the last row
  const float2* U = p.U + spec0;
  for (int e = ctx.tid; e < L * kRotRows; e += ctx.nthr) {
    const int k = e / kRotRows, r = row0 + (e - k * kRotRows);
    float2 u = make_float2(0.f, 0.f);
    if (r < L) u = p.adjoint ? U[(long)k * L + r] : U[(long)r * L + k];
    if (!p.adjoint) u.y = -u.y;
    Us[e] = u;
  }
  ctx.sync();
  const long c = col0 + 2 * ctx.tid;
  if (c >= C) return;
  const bool pair = c + 1 < C;
  const float2* x = p.x + spec0 * p.nbatch + c;
  // both columns in one 16-byte access
  const bool vec = pair && C % 2 == 0 && reinterpret_cast<unsigned long long>(x) % 16 == 0 &&
                   reinterpret_cast<unsigned long long>(p.z + spec0 * p.nbatch + c) % 16 == 0;
  float2 s[kRotRows][2];
#pragma unroll
  for (int r = 0; r < kRotRows; ++r) s[r][0] = s[r][1] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < L; ++k) {
    float2 x0, x1 = make_float2(0.f, 0.f);
    if (vec) {
      const float4 v = *reinterpret_cast<const float4*>(x + k * C);
      x0 = make_float2(v.x, v.y);
      x1 = make_float2(v.z, v.w);
    } else {
      x0 = x[k * C];
      if (pair) x1 = x[k * C + 1];
    }
    const float2 i0 = make_float2(-x0.y, x0.x), i1 = make_float2(-x1.y, x1.x);     // i x
    const float4* u4 = reinterpret_cast<const float4*>(Us + k * kRotRows);
#pragma unroll
    for (int r = 0; r < kRotRows; r += 2) {
      const float4 u = u4[r / 2];
      s[r][0] = fma2(make_float2(u.x, u.x), x0, s[r][0]);
      s[r][1] = fma2(make_float2(u.x, u.x), x1, s[r][1]);
      s[r][0] = fma2(make_float2(u.y, u.y), i0, s[r][0]);
      s[r][1] = fma2(make_float2(u.y, u.y), i1, s[r][1]);
      s[r + 1][0] = fma2(make_float2(u.z, u.z), x0, s[r + 1][0]);
      s[r + 1][1] = fma2(make_float2(u.z, u.z), x1, s[r + 1][1]);
      s[r + 1][0] = fma2(make_float2(u.w, u.w), i0, s[r + 1][0]);
      s[r + 1][1] = fma2(make_float2(u.w, u.w), i1, s[r + 1][1]);
    }
  }
  float2* z = p.z + spec0 * p.nbatch + c;
#pragma unroll
  for (int r = 0; r < kRotRows; ++r) {
    if (row0 + r >= L) break;
    float2* o = z + (row0 + r) * C;
    if (vec) {
      *reinterpret_cast<float4*>(o) = make_float4(s[r][0].x, s[r][0].y, s[r][1].x, s[r][1].y);
    } else {
      o[0] = s[r][0];
      if (pair) o[1] = s[r][1];
    }
  }
}

}  // namespace s2c
