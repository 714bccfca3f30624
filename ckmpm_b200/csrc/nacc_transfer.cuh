// Particle-grid transfers of Cam-clay particles, included by kernels.cuh.
//
// The law leaves F = U diag(S) V with V not transposed (mpm_math.cuh, stress_nacc), which
// jumps when two nearly equal stretches change order: a last-bit difference in what F is
// made from shows in F itself (12 % of F's norm for a sphere of 60 thousand particles after
// 24 substeps), although F F^T, the only part of F that the motion depends on, agrees. So
// that a saved state continues to the same F, these transfers keep one order of operations,
// the one node by node, with the fused products written out, so that no instantiation of a
// kernel contracts them otherwise (but for D^-1 tau, whose diagonal shares products in an order
// that is the compiler's, the same in every instantiation); the other materials, whose F is
// continuous, take the cheaper forms of kernels.cuh. For this law, whose SVD takes most of the time, the cheaper forms gained
// nothing: 1.88 ms for the 24 substeps of that sphere with them, 1.78 to 1.88 with these.
#pragma once

namespace ckmpm {
namespace clay {

// a b + c d, the first product fused into the rounded second, and a b + c d + e f.
__device__ __forceinline__ float sum2(float a, float b, float c, float d) { return fmaf(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ float sum3(float a, float b, float c, float d, float e, float f) {
  return fmaf(e, f, sum2(a, b, c, d));
}

__device__ __forceinline__ float ck_w0(float o) {
  const float kTwoPi = 6.283185307179586f;
  const float kInvTwoPi = 0.15915494309189535f;
  return fmaf(kInvTwoPi, __sinf(kTwoPi * o), 1.0f - o);
}

__device__ __forceinline__ void inv_sym3(float d00, float d11, float d22, float d01, float d02, float d12, float* r) {
  const float c00 = sum2(d11, d22, -d12, d12);
  const float c01 = sum2(d02, d12, -d01, d22);
  const float c02 = sum2(d01, d12, -d02, d11);
  const float det = sum3(d00, c00, d01, c01, d02, c02);
  const float id = 1.0f / det;
  r[0] = id * c00;
  r[1] = id * sum2(d00, d22, -d02, d02);
  r[2] = id * sum2(d00, d11, -d01, d01);
  r[3] = id * c01;
  r[4] = id * c02;
  r[5] = id * sum2(d01, d02, -d00, d12);
}

// Stencil of one grid (G = -1 or +1) along one axis at position x.  The base cell on grid
// -dx/4 is the binning's, so a particle's stencil lies in the window of its block.
struct AxisStencil {
  int base;
  float o, w0;
};

template <int G>
__device__ __forceinline__ AxisStencil axis_stencil(float x, float inv_dx) {
  AxisStencil s;
  s.base = G < 0 ? cell_of(x, inv_dx) : static_cast<int>(fmaf(x, inv_dx, -0.25f));
  s.o = fmaf(x, inv_dx, -static_cast<float>(s.base)) - 0.25f * G;
  s.w0 = ck_w0(s.o);
  return s;
}

// m1 = sum_d w_d (d - o) dx and m2 = sum_d w_d (d - o)^2 dx of one grid along one axis.
__device__ __forceinline__ void axis_moments(const AxisStencil& s, float dx, float& m1, float& m2) {
  const float w1 = 1.0f - s.w0;
  m1 = (w1 - s.o) * dx;
  const float a = s.o, b = 1.0f - s.o;
  m2 = sum2(w1 * b, b, s.w0 * a, a) * dx;
}

// D, summed over both grids (00, 11, 22, 01, 02, 12).
__device__ __forceinline__ void d_matrix(const AxisStencil (&st)[2][3], float dx, float* D6) {
  float m1[2][3], m2[2][3];
#pragma unroll
  for (int g = 0; g < 2; ++g)
#pragma unroll
    for (int a = 0; a < 3; ++a) axis_moments(st[g][a], dx, m1[g][a], m2[g][a]);
#pragma unroll
  for (int a = 0; a < 3; ++a) D6[a] = sum2(m2[0][a], dx, m2[1][a], dx);
  D6[3] = sum2(m1[0][0], m1[0][1], m1[1][0], m1[1][1]);
  D6[4] = sum2(m1[0][0], m1[0][2], m1[1][0], m1[1][2]);
  D6[5] = sum2(m1[0][1], m1[0][2], m1[1][1], m1[1][2]);
}

// Halved velocity v, C = B D^-1 and D of the G2P at x.
__device__ __forceinline__ void g2p(const float4* __restrict__ vtile, const float (&x)[3], int4 key, float dx,
                                    float inv_dx, float* v, float* C, bool& inside, float* D6) {
  AxisStencil st[2][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    st[0][a] = axis_stencil<-1>(x[a], inv_dx);
    st[1][a] = axis_stencil<1>(x[a], inv_dx);
  }
  float B[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) B[k] = 0.f;
  float vs[3] = {0.f, 0.f, 0.f};
  const int kb[3] = {key.x * 4, key.y * 4, key.z * 4};
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    int l[3];
    const int lo = g == 0 ? 2 : 1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      l[a] = st[g][a].base - kb[a];
      if (l[a] < lo || l[a] > 5) {
        inside = false;
        l[a] = min(max(l[a], lo), 5);
      }
    }
    const float wx[2] = {st[g][0].w0, 1.f - st[g][0].w0};
    const float wy[2] = {st[g][1].w0, 1.f - st[g][1].w0};
    const float wz[2] = {st[g][2].w0, 1.f - st[g][2].w0};
    float S[3] = {0.f, 0.f, 0.f}, T[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) T[r][0] = T[r][1] = T[r][2] = 0.f;
    const int sx = g == 0 ? 25 : 36, sy = g == 0 ? 5 : 6;
    const float4* base = vtile + vtile_index(g, l[0], l[1], l[2]);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int dxn = (n >> 2) & 1, dyn = (n >> 1) & 1, dzn = n & 1;
      const float w = wx[dxn] * wy[dyn] * wz[dzn];
      const float4 vi = base[dxn * sx + dyn * sy + dzn];
      const float vn[3] = {vi.x, vi.y, vi.z};
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        S[r] = fmaf(w, vn[r], S[r]);
        if (dxn) T[r][0] = fmaf(w, vn[r], T[r][0]);
        if (dyn) T[r][1] = fmaf(w, vn[r], T[r][1]);
        if (dzn) T[r][2] = fmaf(w, vn[r], T[r][2]);
      }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      vs[r] += S[r];
#pragma unroll
      for (int a = 0; a < 3; ++a) B[r * 3 + a] = fmaf(dx, fmaf(-st[g][a].o, S[r], T[r][a]), B[r * 3 + a]);
    }
  }
  float Di6[6], Di[9];
  d_matrix(st, dx, D6);
  inv_sym3(D6[0], D6[1], D6[2], D6[3], D6[4], D6[5], Di6);
  sym_to_full(Di6, Di);
  matmul3_nacc(B, Di, C);
#pragma unroll
  for (int r = 0; r < 3; ++r) v[r] = 0.5f * vs[r];
}

// kernels.cuh, p2g_scatter.
__device__ __forceinline__ void p2g_scatter(unsigned* __restrict__ ptile, const AxisStencil (&st)[2][3],
                                            const int (&lbase)[2][3], const float* v, const float* Ah) {
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    float Q[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
      Q[r] = v[r] - sum3(Ah[r * 3], st[g][0].o, Ah[r * 3 + 1], st[g][1].o, Ah[r * 3 + 2], st[g][2].o);
    const float wx[2] = {st[g][0].w0 * kFixScale, (1.f - st[g][0].w0) * kFixScale};
    const float wy[2] = {st[g][1].w0, 1.f - st[g][1].w0};
    const float wz[2] = {st[g][2].w0, 1.f - st[g][2].w0};
    unsigned* base = ptile + ((g * 8 + lbase[g][0]) * kTileRow + lbase[g][1] * 8 + lbase[g][2]);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int dxn = (n >> 2) & 1, dyn = (n >> 1) & 1, dzn = n & 1;
      const float w = wx[dxn] * wy[dyn] * wz[dzn];
      float val[3];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        val[r] = Q[r];
        if (dxn) val[r] += Ah[r * 3];
        if (dyn) val[r] += Ah[r * 3 + 1];
        if (dzn) val[r] += Ah[r * 3 + 2];
      }
      unsigned* node = base + (dxn * kTileRow + dyn * 8 + dzn);
      const long long fx[4] = {__float2ll_rn(w), __float2ll_rn(w * val[0]), __float2ll_rn(w * val[1]),
                               __float2ll_rn(w * val[2])};
#pragma unroll
      for (int c = 0; c < 4; ++c) fixed_add(node + c * kTileNodes, fx[c]);
    }
  }
}

}  // namespace clay
}  // namespace ckmpm
