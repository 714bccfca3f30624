// Device math for the CK-MPM substep: 3x3 helpers, the FP32 SVD, and
// the constitutive models of the hot path.
//
// Matrices are row-major float[9] like the reference's Matrix<float,3,3>
// (AppledoreM/CKMPM include/data_type.cuh:32-425).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ckmpm {

#define CKMPM_DEV __device__ __forceinline__

// Sums of products are written as explicit fused multiply-adds: the compiler may
// contract a b + c d either way, and not the same way in every instantiation of a
// kernel, while results must not depend on the launch shape.
CKMPM_DEV float dot2(float a, float b, float c, float d) { return fmaf(c, d, a * b); }
CKMPM_DEV float dot3(float a, float b, float c, float d, float e, float f) { return fmaf(e, f, fmaf(c, d, a * b)); }

CKMPM_DEV float det3(const float* a) {
  return dot3(a[0], dot2(a[4], a[8], -a[5], a[7]), -a[1], dot2(a[3], a[8], -a[5], a[6]), a[2],
              dot2(a[3], a[7], -a[4], a[6]));
}

// Adjugate inverse (include/data_type.cuh:369-386).
CKMPM_DEV void inv3(const float* a, float* r) {
  const float id = 1.0f / det3(a);
  r[0] = id * (a[4] * a[8] - a[5] * a[7]);
  r[1] = id * (a[2] * a[7] - a[1] * a[8]);
  r[2] = id * (a[1] * a[5] - a[2] * a[4]);
  r[3] = id * (a[5] * a[6] - a[3] * a[8]);
  r[4] = id * (a[0] * a[8] - a[2] * a[6]);
  r[5] = id * (a[2] * a[3] - a[0] * a[5]);
  r[6] = id * (a[3] * a[7] - a[4] * a[6]);
  r[7] = id * (a[1] * a[6] - a[0] * a[7]);
  r[8] = id * (a[0] * a[4] - a[1] * a[3]);
}

// Inverse of a symmetric matrix given by its 6 unique entries
// (d00, d11, d22, d01, d02, d12); writes the 6 unique entries of the inverse.
CKMPM_DEV void inv_sym3(float d00, float d11, float d22, float d01, float d02, float d12, float* r) {
  const float c00 = dot2(d11, d22, -d12, d12);
  const float c01 = dot2(d02, d12, -d01, d22);
  const float c02 = dot2(d01, d12, -d02, d11);
  const float det = dot3(d00, c00, d01, c01, d02, c02);
  const float id = 1.0f / det;
  r[0] = id * c00;
  r[1] = id * dot2(d00, d22, -d02, d02);
  r[2] = id * dot2(d00, d11, -d01, d01);
  r[3] = id * c01;
  r[4] = id * c02;
  r[5] = id * dot2(d01, d02, -d00, d12);
}

CKMPM_DEV void matmul3(const float* a, const float* b, float* r) {
  float t[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) t[i * 3 + j] = dot3(a[i * 3], b[j], a[i * 3 + 1], b[3 + j], a[i * 3 + 2], b[6 + j]);
#pragma unroll
  for (int k = 0; k < 9; ++k) r[k] = t[k];
}

// For the Cam-clay path (nacc_transfer.cuh): the first product fused into the rounded second, then the third.
CKMPM_DEV void matmul3_nacc(const float* a, const float* b, float* r) {
  float t[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      t[i * 3 + j] = fmaf(a[i * 3 + 2], b[6 + j], fmaf(a[i * 3], b[j], __fmul_rn(a[i * 3 + 1], b[3 + j])));
#pragma unroll
  for (int k = 0; k < 9; ++k) r[k] = t[k];
}

// The same with the compiler's own contraction (Cam-clay's D^-1 tau).
CKMPM_DEV void matmul3_plain(const float* a, const float* b, float* r) {
  float t[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) t[i * 3 + j] = a[i * 3] * b[j] + a[i * 3 + 1] * b[3 + j] + a[i * 3 + 2] * b[6 + j];
#pragma unroll
  for (int k = 0; k < 9; ++k) r[k] = t[k];
}

// ------------------------------------------------------------------ SVD
//
// A = U diag(S) V^T with U, V proper rotations, |S0| >= |S1| >= |S2|, S0, S1 >= 0
// and the sign of det(A) on S2 -- the convention of the method of
// McAdams, Selle, Tamstorf, Teran, Sifakis, "Computing the Singular Value
// Decomposition of 3x3 matrices with minimal branching and elementary floating
// point operations", UW-Madison TR1690 (2011), which the reference vendors
// (include/mpm_math.cuh:1-18).  Implemented here from the published outline:
//   1. symmetric eigenproblem of A^T A by cyclic Jacobi (fixed sweep count,
//      exact rotation angles from the 2x2 Schur form).  Three sweeps reach
//      FP32 rounding: in an FP32 emulation of these steps over 4000 random
//      F = R1 diag(s) R2 per family, with s in [0.1, 3] and
//      e^[-2, 2], and I + N(0, 0.5) shears, the singular values agree with an
//      FP64 SVD to 4e-7 relative (max) with three sweeps and with four; the
//      off-diagonal residual of (A V)^T (A V) is ~1.6e-7 at the 99th percentile
//      either way, and up to 6e-6 for about 1 matrix in 1000 with three
//      (2.7e-7 at worst with four); the fourth sweep costs ~2 % of the substep
//      (tests/test_svd_sweeps.py restates these steps and checks the bounds);
//   2. B = A V, columns sorted by decreasing norm (sign flips keep det V = 1);
//   3. Givens QR of B gives U and the diagonal S.

// 1/sqrt(x) from the hardware estimate (up to 2 ulp) with one Newton step: ~1 ulp,
// and exactly 1 for x = 1, so that a pair left unrotated keeps c = 1, s = 0.
CKMPM_DEV float rsqrt_refined(float x) {
  const float r = rsqrtf(x);
  return r * fmaf(-0.5f * x * r, r, 1.5f);
}

// Off-diagonal entries of A^T A below this magnitude are left in place, as the
// reference's SVD leaves a pair unrotated when (a_pq / 2)^2 < 1e-20
// (include/mpm_math.cuh:117-123).  Without it a deformation gradient within
// rounding of the identity (every particle of a rigidly moving or free-falling
// body) has equal diagonal entries and a 1e-11 off-diagonal, which an exact
// Jacobi step rotates by 45 degrees; the re-projected F = U V^T of the
// Drucker-Prager tension branch then carries ~1e-7 of rounding back into F
// every substep.
constexpr float kJacobiNegligible = 2e-10f;

CKMPM_DEV void jacobi_rotate(float& app, float& aqq, float& apq, float& arp, float& arq, float* V, int p, int q) {
  if (!(fabsf(apq) >= kJacobiNegligible)) return;
  // Zero apq.  t = tan(theta) of the smaller rotation solving
  // t^2 + 2 tau t - 1 = 0 with tau = (aqq - app) / (2 apq).
  const float d = aqq - app;
  const float e = 2.0f * apq;
  const float h = sqrtf(d * d + e * e);
  const float den = d + copysignf(h, d);
  float t = den != 0.0f ? e / den : 0.0f;
  const float c = rsqrt_refined(1.0f + t * t);
  const float s = t * c;
  app = app - t * apq;
  aqq = aqq + t * apq;
  apq = 0.0f;
  const float rp = arp, rq = arq;
  arp = c * rp - s * rq;
  arq = s * rp + c * rq;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float vp = V[k * 3 + p], vq = V[k * 3 + q];
    V[k * 3 + p] = c * vp - s * vq;
    V[k * 3 + q] = s * vp + c * vq;
  }
}

// Entries below this are already zero for the QR (the reference's threshold
// for its QR Givens steps, include/mpm_math.cuh:735-741).
constexpr float kQrNegligible = 1e-12f;

CKMPM_DEV void givens_qr_step(float* B, float* U, int p, int q, int col) {
  const float a = B[p * 3 + col], b = B[q * 3 + col];
  float c = a < 0.0f ? -1.0f : 1.0f, s = 0.0f;
  if (fabsf(b) >= kQrNegligible) {
    const float ir = rsqrt_refined(a * a + b * b);
    c = a * ir;
    s = b * ir;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float bp = B[p * 3 + k], bq = B[q * 3 + k];
    B[p * 3 + k] = c * bp + s * bq;
    B[q * 3 + k] = -s * bp + c * bq;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float up = U[k * 3 + p], uq = U[k * 3 + q];
    U[k * 3 + p] = c * up + s * uq;
    U[k * 3 + q] = -s * up + c * uq;
  }
}

CKMPM_DEV void swap_cols(float* V, float& la, float& lb, int a, int b) {
  const float t = la;
  la = lb;
  lb = t;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float va = V[k * 3 + a];
    V[k * 3 + a] = V[k * 3 + b];
    V[k * 3 + b] = -va;
  }
}

template <int kSweeps = 3, bool NACC = false>
CKMPM_DEV void svd3(const float* A, float* U, float* S, float* V) {
  // M = A^T A (symmetric; 6 unique entries)
  float m00 = A[0] * A[0] + A[3] * A[3] + A[6] * A[6];
  float m11 = A[1] * A[1] + A[4] * A[4] + A[7] * A[7];
  float m22 = A[2] * A[2] + A[5] * A[5] + A[8] * A[8];
  float m01 = A[0] * A[1] + A[3] * A[4] + A[6] * A[7];
  float m02 = A[0] * A[2] + A[3] * A[5] + A[6] * A[8];
  float m12 = A[1] * A[2] + A[4] * A[5] + A[7] * A[8];
#pragma unroll
  for (int k = 0; k < 9; ++k) V[k] = (k & 3) ? 0.0f : 1.0f;
#pragma unroll
  for (int sweep = 0; sweep < kSweeps; ++sweep) {
    jacobi_rotate(m00, m11, m01, m02, m12, V, 0, 1);  // r = 2: (m20, m21)
    jacobi_rotate(m00, m22, m02, m01, m12, V, 0, 2);  // r = 1: (m10, m12)
    jacobi_rotate(m11, m22, m12, m01, m02, V, 1, 2);  // r = 0: (m01, m02)
  }
  float l0 = m00, l1 = m11, l2 = m22;
  if (l0 < l1) swap_cols(V, l0, l1, 0, 1);
  if (l0 < l2) swap_cols(V, l0, l2, 0, 2);
  if (l1 < l2) swap_cols(V, l1, l2, 1, 2);
  float B[9];
  if (NACC) matmul3_nacc(A, V, B);
  else matmul3(A, V, B);
#pragma unroll
  for (int k = 0; k < 9; ++k) U[k] = (k & 3) ? 0.0f : 1.0f;
  givens_qr_step(B, U, 0, 1, 0);
  givens_qr_step(B, U, 0, 2, 0);
  givens_qr_step(B, U, 1, 2, 1);
  S[0] = B[0];
  S[1] = B[4];
  S[2] = B[8];
}

// ------------------------------------------------------------------ left eigenvectors
//
// The isotropic stresses need F = U diag(S) V^T only through U, S and
// F itself: tau = U diag(f(S)) U^T, and a return map that scales the
// principal stretches by r_i gives F <- U diag(r) U^T F.  So the substep takes the
// eigenvectors U of b = F F^T by the same cyclic Jacobi as svd3 and the stretches
// as the column norms of W = F^T U (W_i = S_i V_i), and needs neither V, nor the
// sorting, nor the QR of svd3.  Norms of F^T u_i keep S_i to rounding of |F|
// where square roots of the eigenvalues would not.
//
// A pair is left unrotated when its off-diagonal is below kLeftNegligible times
// the trace: leaving it changes U diag(f(S)) U^T by at most that fraction of f,
// below the rounding of forming b.
constexpr float kLeftNegligible = 1e-9f;

// c = cos, s = sin and t = tan of the rotation that zeroes apq; (1, 0, 0) when
// |apq| < tiny.
CKMPM_DEV void jacobi_angle(float app, float aqq, float apq, float tiny, float& t, float& c, float& s) {
  const float d = aqq - app, e = 2.0f * apq;
  const float h2 = fmaf(d, d, e * e);
  const float den = d + copysignf(h2 * rsqrtf(h2), d);
  t = fabsf(apq) >= tiny ? __fdividef(e, den) : 0.0f;
  c = rsqrt_refined(fmaf(t, t, 1.0f));
  s = t * c;
}

CKMPM_DEV void left_rotate(float& app, float& aqq, float& apq, float& arp, float& arq, float tiny, float* U, int p,
                           int q) {
  if (!(fabsf(apq) >= tiny)) return;
  float t, c, s;
  jacobi_angle(app, aqq, apq, tiny, t, c, s);
  app = fmaf(-t, apq, app);
  aqq = fmaf(t, apq, aqq);
  apq = 0.0f;
  const float rp = arp, rq = arq;
  arp = dot2(c, rp, -s, rq);
  arq = dot2(s, rp, c, rq);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float up = U[k * 3 + p], uq = U[k * 3 + q];
    U[k * 3 + p] = dot2(c, up, -s, uq);
    U[k * 3 + q] = dot2(s, up, c, uq);
  }
}

// U (columns: eigenvectors of F F^T, a proper rotation), W = F^T U and the
// stretches S = |W_i| >= 0, in no order.
CKMPM_DEV void left_stretch(const float* F, float* U, float* W, float* S) {
  float m00 = dot3(F[0], F[0], F[1], F[1], F[2], F[2]);
  float m11 = dot3(F[3], F[3], F[4], F[4], F[5], F[5]);
  float m22 = dot3(F[6], F[6], F[7], F[7], F[8], F[8]);
  float m01 = dot3(F[0], F[3], F[1], F[4], F[2], F[5]);
  float m02 = dot3(F[0], F[6], F[1], F[7], F[2], F[8]);
  float m12 = dot3(F[3], F[6], F[4], F[7], F[5], F[8]);
  const float tiny = fmaxf(kLeftNegligible * (m00 + m11 + m22), 1e-18f);  // 1e-18 squared stays normal
#pragma unroll
  for (int k = 0; k < 9; ++k) U[k] = (k & 3) ? 0.0f : 1.0f;
  if (!(fmaxf(fmaxf(fabsf(m01), fabsf(m02)), fabsf(m12)) < tiny)) {
    // First sweep written out on U = I.
    float t, c, s;
    jacobi_angle(m00, m11, m01, tiny, t, c, s);
    m00 = fmaf(-t, m01, m00);
    m11 = fmaf(t, m01, m11);
    const float q02 = dot2(c, m02, -s, m12), q12 = dot2(s, m02, c, m12);
    float t2, c2, s2;
    jacobi_angle(m00, m22, q02, tiny, t2, c2, s2);
    m00 = fmaf(-t2, q02, m00);
    m22 = fmaf(t2, q02, m22);
    m01 = -s2 * q12;
    m12 = c2 * q12;
    U[0] = c2 * c;
    U[3] = -c2 * s;
    U[6] = -s2;
    const float u02 = s2 * c, u12 = -s2 * s;
    float t3, c3, s3;
    jacobi_angle(m11, m22, m12, tiny, t3, c3, s3);
    m11 = fmaf(-t3, m12, m11);
    m22 = fmaf(t3, m12, m22);
    m02 = s3 * m01;
    m01 = c3 * m01;
    m12 = 0.0f;
    U[1] = dot2(c3, s, -s3, u02);
    U[4] = dot2(c3, c, -s3, u12);
    U[7] = -s3 * c2;
    U[2] = dot2(s3, s, c3, u02);
    U[5] = dot2(s3, c, c3, u12);
    U[8] = c3 * c2;
#pragma unroll
    for (int sweep = 1; sweep < 3; ++sweep) {
      left_rotate(m00, m11, m01, m02, m12, tiny, U, 0, 1);
      left_rotate(m00, m22, m02, m01, m12, tiny, U, 0, 2);
      left_rotate(m11, m22, m12, m01, m02, tiny, U, 1, 2);
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int k = 0; k < 3; ++k) W[k * 3 + i] = dot3(F[k], U[i], F[3 + k], U[3 + i], F[6 + k], U[6 + i]);
    const float n2 = dot3(W[i], W[i], W[3 + i], W[3 + i], W[6 + i], W[6 + i]);
    S[i] = n2 > 0.0f ? n2 * rsqrt_refined(n2) : n2;
  }
}

// U diag(d) U^T (symmetric).
CKMPM_DEV void left_diag(const float* U, const float* d, float* r9) {
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const float a = U[r * 3] * d[0], b = U[r * 3 + 1] * d[1], e = U[r * 3 + 2] * d[2];
#pragma unroll
    for (int c = r; c < 3; ++c) {
      const float v = dot3(a, U[c * 3], b, U[c * 3 + 1], e, U[c * 3 + 2]);
      r9[r * 3 + c] = v;
      r9[c * 3 + r] = v;
    }
  }
}

// F += U diag(r) W^T.  A return map that scales the stretches by q_i adds
// U diag(q - 1) U^T F: the error of U then enters times q - 1, not times q (the product
// form's F was 1.2x as far from 64 bits after a frame of von Mises flow, this one's is not).
CKMPM_DEV void left_rescale(const float* U, const float* r, const float* W, float* F) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float a = U[i * 3] * r[0], b = U[i * 3 + 1] * r[1], e = U[i * 3 + 2] * r[2];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      F[i * 3 + k] = fmaf(e, W[k * 3 + 2], fmaf(b, W[k * 3 + 1], fmaf(a, W[k * 3], F[i * 3 + k])));
  }
}

// Whether the smallest stretch is large enough against the largest for W_i / S_i
// to stand for V_i: the error of W_i is that of |F|, so V_i's is S_max / S_min
// times rounding.  Beyond 4 (and for a NaN) the return maps take svd3's V.
CKMPM_DEV bool left_well_conditioned(const float* S) {
  return fminf(fminf(S[0], S[1]), S[2]) > 0.25f * fmaxf(fmaxf(S[0], S[1]), S[2]);
}

// ------------------------------------------------------------------ materials
// Numbering of MPMConstitutiveModel (include/mpm_material.cuh:10-18).
enum MaterialKind : int32_t {
  kFixedCorotated = 0,
  kLinear = 1,
  kDruckerPrager = 2,
  kFluid = 3,
  kVonMises = 4,
  kNacc = 5,
};

constexpr int kMaterialParams = 8;

struct MaterialParams {
  int32_t kind;
  // FC / DP / Linear: lambda, mu.  Fluid: bulk, gamma, viscosity, J0.  Von Mises: mu, lambda, yield
  // stress.  NACC: mu, lambda, alpha0, beta, hardening factor, M, hardening on (0 / 1).
  float p[kMaterialParams];
};

// Fixed-corotated Kirchhoff stress, tau = U diag(2 mu s (s - 1) + lambda J (J - 1)) U^T
// (include/mpm_material.cuh:320-357), where the smallest stretch takes the sign of det F.
CKMPM_DEV void stress_fixed_corotated(float lambda, float mu, const float* F, float* tau) {
  float U[9], W[9], S[3];
  left_stretch(F, U, W, S);
  const float J = det3(F);
  if (J < 0.0f) {
    const float least = fminf(fminf(S[0], S[1]), S[2]);
    if (S[2] == least) S[2] = -S[2];
    else if (S[1] == least) S[1] = -S[1];
    else S[0] = -S[0];
  }
  const float lj = lambda * J * (J - 1.0f);
  float sc[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) sc[i] = fmaf(2.0f * mu * S[i], S[i] - 1.0f, lj);
  left_diag(U, sc, tau);
}

// Drucker-Prager StVK-Hencky return map with the reference's constants:
// zero cohesion, beta = 1, volume correction on, sin(phi) = 0.5
// (include/mpm_material.cuh:362-464).  Updates F and logJp in place.
//
// The reference computes tau = U diag(p) V^T F^T with p = (2 mu log s + lambda tr log s) / s
// after F <- U diag(s) V^T; V^T F^T = diag(s) U^T, so tau = U diag(2 mu log s + lambda tr log s) U^T,
// and log s is known: 0 on the tension branch (s = 1), H elsewhere.
// An elastic step (dg <= 0, stretches within the clamp) leaves F as it is.
// An inverted F takes svd3's rotations U and V: F <- U diag(s) V^T with s > 0 undoes the
// reflection, which the additive map and the untouched elastic step would keep.
CKMPM_DEV void stress_drucker_prager(float lambda, float mu, float* F, float& logJp, float* tau) {
  const float kYs = 0.816496580927726f * 2.0f * 0.5f / (3.0f - 0.5f);
  const float smu = 2.0f * mu;
  float U[9], W[9], S[3];
  left_stretch(F, U, W, S);
  const bool good = left_well_conditioned(S) && S[0] > 4e-4f && det3(F) > 0.0f;
  if (!good) {
    float V[9];
    svd3(F, U, S, V);
#pragma unroll
    for (int i = 0; i < 9; ++i) W[i] = V[i];
  }
  float eps[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) eps[i] = logf(fmaxf(fabsf(S[i]), 1e-4f));
  const float esum = eps[0] + eps[1] + eps[2];
  const float etr = esum + logJp;
  float eh[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) eh[i] = fmaf(etr, -1.0f / 3.0f, eps[i]);
  const float ehn = sqrtf(dot3(eh[0], eh[0], eh[1], eh[1], eh[2], eh[2]));
  const bool tension = etr >= 0.0f;
  logJp = tension ? etr : 0.0f;
  const float dg = fmaf(fmaf(3.0f, lambda, smu) / smu * kYs, etr, ehn);
  const float k = !tension && dg > 0.0f ? dg / ehn : 0.0f;
  float h[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) h[i] = tension ? 0.0f : fmaf(-k, eh[i], eps[i]);
  if (tension || k > 0.0f || !good) {
    // Change of the stretch over |W_i| (S_i); where W holds V, the stretch itself onto F = 0.
    float r[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) r[i] = good ? expf(h[i] - eps[i]) - 1.0f : expf(h[i]);
    if (!good) {
#pragma unroll
      for (int i = 0; i < 9; ++i) F[i] = 0.0f;
    }
    left_rescale(U, r, W, F);
  }
  const float trh = h[0] + h[1] + h[2];
  float sc[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) sc[i] = dot2(smu, h[i], lambda, trh);
  left_diag(U, sc, tau);
}

// Von Mises plasticity on the Hencky strain of the trial elastic F, then the
// StVK-Hencky stress of the projected F (include/mpm_algorithm.cuh:404-520,
// include/mpm_material.cuh:480-518):
//   eps = log S, eps_hat = eps - tr(eps) / 3, f = |eps_hat| - yield / (2 mu);
//   f > 0: S <- exp(eps - f eps_hat / |eps_hat|), Fe <- U diag(S) V^T;
//   tau = U diag((2 mu log S + lambda tr log S) / S) V^T Fe^T = U diag(2 mu log S + lambda tr log S) U^T.
// The reference takes a second SVD for the projected Fe; its U and log S are
// the ones at hand.  Fe holds the trial elastic F on entry and the projected one on exit.
// An inverted Fe (S_2 < 0) has no Hencky strain: NaN, as log S gives.
CKMPM_DEV void stress_von_mises(float mu, float lambda, float yield, float* Fe, float* tau) {
  float U[9], W[9], S[3];
  left_stretch(Fe, U, W, S);
  const bool good = left_well_conditioned(S) && det3(Fe) > 0.0f;
  if (!good) {
    float V[9];
    svd3(Fe, U, S, V);
#pragma unroll
    for (int i = 0; i < 9; ++i) W[i] = V[i];
  }
  float eps[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) eps[i] = logf(S[i]);
  const float etr = eps[0] + eps[1] + eps[2];
  float eh[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) eh[i] = fmaf(etr, -1.0f / 3.0f, eps[i]);
  const float ehn = sqrtf(dot3(eh[0], eh[0], eh[1], eh[1], eh[2], eh[2]));
  const float yf = ehn - yield / (2.0f * mu);
  float h[3] = {eps[0], eps[1], eps[2]};
  if (yf > 0.0f) {
    const float k = yf / ehn;
    float r[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      h[i] = fmaf(-k, eh[i], eps[i]);
      r[i] = good ? expf(-k * eh[i]) - 1.0f : expf(h[i]);
    }
    if (!good) {
#pragma unroll
      for (int i = 0; i < 9; ++i) Fe[i] = 0.0f;
    }
    left_rescale(U, r, W, Fe);
  }
  const float trh = h[0] + h[1] + h[2];
  float sc[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) sc[i] = dot2(2.0f * mu, h[i], lambda, trh);
  left_diag(U, sc, tau);
}

// Non-associated Cam-clay (include/mpm_material.cuh:520-669, driven from
// include/mpm_algorithm.cuh:330-402), restated step for step, including what
// it does beyond the textbook model, so that results match the reference:
//  * the projected F is U diag(S) V (V itself, not its transpose); the stress
//    only sees F F^T = U S^2 U^T, so V never affects the motion, but the stored
//    F is fixed only up to a rotation on the right;
//  * the hardening update of the yield-surface branch sits in a loop of 9
//    identical iterations, so logJp takes the same increment 9 times;
//  * thresholds written as double literals (1e-4) compare in double.
// Both branches (pressure clamped to [pMin, p0], or the return to the yield
// surface) end in the same stress: mu Je_trial^(-2/3) dev(F F^T) + K/2 (J^2 - 1) I.
// F holds dW F_old on entry and the projected F on exit.
CKMPM_DEV void stress_nacc(const float* prm, float* F, float& logJp, float* tau) {
  const float mu = prm[0], lambda = prm[1], beta = prm[3], xi = prm[4], msq = prm[5] * prm[5];
  const bool hardening = prm[6] != 0.0f;
  const float K = 2.0f * mu / 3.0f + lambda;
  float U[9], S[3], V[9];
  svd3<3, true>(F, U, S, V);
  const float p0 = K * (1e-5f + sinhf(xi * (-logJp > 0.0f ? -logJp : 0.0f)));
  const float pmin = -beta * p0;
  const float je = S[0] * S[1] * S[2];
  const float bh[3] = {S[0] * S[0], S[1] * S[1], S[2] * S[2]};
  const float btr3 = (bh[0] + bh[1] + bh[2]) / 3.0f;
  const float devf = mu * powf(je, -2.0f / 3.0f);
  const float sh[3] = {devf * (bh[0] - btr3), devf * (bh[1] - btr3), devf * (bh[2] - btr3)};
  const float hydro = K * 0.5f * (je - 1.0f / je);
  const float ptrial = -hydro * je;
  const float ysh = 3.0f / 2.0f * (1.0f + 2.0f * beta);
  const float yph = msq * (ptrial - pmin) * (ptrial - p0);
  const float sn2 = sh[0] * sh[0] + sh[1] * sh[1] + sh[2] * sh[2];
  const float y = ysh * sn2 + yph;
  float Sn[3] = {S[0], S[1], S[2]};
  if (ptrial > p0 || ptrial < pmin) {
    const float pp = ptrial > p0 ? p0 : pmin;
    const float jn = sqrtf(-2.0f * pp / K + 1.0f);
    const float sc = powf(jn, 1.0f / 3.0f);
    Sn[0] = Sn[1] = Sn[2] = sc;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        F[r * 3 + c] = sc * (U[r * 3] * V[c] + U[r * 3 + 1] * V[3 + c] + U[r * 3 + 2] * V[6 + c]);
    if (hardening) logJp += logf(je / jn);
  } else if (static_cast<double>(y) >= 1e-4) {
    const float coef = powf(je, 2.0f / 3.0f) / mu * sqrtf(-yph / ysh) / sqrtf(sn2);
#pragma unroll
    for (int i = 0; i < 3; ++i) Sn[i] = sqrtf(sh[i] * coef + btr3);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        F[r * 3 + c] = U[r * 3] * Sn[0] * V[c] + U[r * 3 + 1] * Sn[1] * V[3 + c] + U[r * 3 + 2] * Sn[2] * V[6 + c];
    if (hardening && static_cast<double>(p0) > 1e-4 && static_cast<double>(ptrial) < static_cast<double>(p0) - 1e-4 &&
        static_cast<double>(ptrial) > 1e-4 + static_cast<double>(pmin)) {
      const float pc = (1.0f - beta) * p0 / 2.0f;
      const float qt = sqrtf(3.0f / 2.0f * sn2);
      float d0 = pc - ptrial, d1 = -qt;
      const float dn = sqrtf(d0 * d0 + d1 * d1);
      d0 /= dn;
      d1 /= dn;
      const float A = msq * d0 * d0 + (1.0f + 2.0f * beta) * d1 * d1;
      const float B = msq * d0 * (2.0f * pc - p0 - pmin);
      const float C = msq * (pc - pmin) * (pc - p0);
      const float disc = B * B - 4.0f * A * C;
      const float l1 = (-B + sqrtf(disc)) / (2.0f * A);
      const float l2 = (-B - sqrtf(disc)) / (2.0f * A);
      const float p1 = pc + l1 * d0, p2 = pc + l2 * d0;
      const float pf = (ptrial - pc) * (p1 - pc) > 0.0f ? p1 : p2;
      const float jsq = -2.0f * pf / K + 1.0f;
      const float jn = sqrtf(jsq > 0.0f ? jsq : -jsq);
      if (static_cast<double>(jn) > 1e-4) {
        const float inc = logf(je / jn);
        for (int it = 0; it < 9; ++it) logJp += inc;
      }
    }
  }
  const float J = Sn[0] * Sn[1] * Sn[2];
  float b[9];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) b[r * 3 + c] = F[r * 3] * F[c * 3] + F[r * 3 + 1] * F[c * 3 + 1] + F[r * 3 + 2] * F[c * 3 + 2];
  const float btr = (b[0] + b[4] + b[8]) / 3.0f;
  const float hc = K * 0.5f * (J * J - 1.0f);
#pragma unroll
  for (int k = 0; k < 9; ++k) tau[k] = devf * (b[k] - ((k & 3) ? 0.0f : btr));
  tau[0] += hc;
  tau[4] += hc;
  tau[8] += hc;
}

// Linear model as the reference updates it (include/mpm_algorithm.cuh:107-191):
// F <- dW F (done by the caller); the stored stress Q <- (Q + 50 (C + C^T - I) dt)
// det(F), with its rows 1 and 2 zeroed; tau = Q.  lambda and mu are not read.
CKMPM_DEV void stress_linear(const float* C, float dt, const float* F, float* Q, float* tau) {
  const float detF = det3(F);
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int k = r * 3 + c;
      const float t = 50.0f * (C[k] + C[c * 3 + r] - ((k & 3) ? 0.0f : 1.0f)) * dt;
      Q[k] = r == 0 ? (Q[k] + t) * detF : 0.0f;
    }
#pragma unroll
  for (int k = 0; k < 9; ++k) tau[k] = Q[k];
}

// J-fluid: J += tr(C) dt J; p = bulk (J^-gamma - 1); tau = J (visc (C + C^T) - p I)
// (include/mpm_algorithm.cuh:528-569, include/mpm_material.cuh:468-477).
CKMPM_DEV void stress_fluid(float bulk, float gamma, float visc, const float* C, float dt, float& J, float* tau) {
  J = fmaf((C[0] + C[4] + C[8]) * dt, J, J);
  const float p = __fmul_rn(bulk, powf(J, -gamma) - 1.0f);
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      tau[r * 3 + c] = r == c ? fmaf(2.0f * C[r * 3 + c], visc, -p) : (C[r * 3 + c] + C[c * 3 + r]) * visc;
#pragma unroll
  for (int k = 0; k < 9; ++k) tau[k] *= J;
}

}  // namespace ckmpm
