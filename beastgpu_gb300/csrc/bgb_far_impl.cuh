// Far-pair tile kernels (plain FP64 and mixed FP32) with the deterministic gather write.
//
// A CTA owns one output tile: a block of test functions (rows) x a block of trial
// functions (columns), each a compact patch of a recursive coordinate bisection of the functions.
// It stages the triangles supporting those functions ("halo" included) in shared memory,
// sweeps the trial triangles in chunks, computes the 3x3 local matrix of every (test
// triangle, trial triangle) pair of the chunk into shared memory, and then lets each thread
// add the chunk's contributions to the output entries it owns.  Every entry Z[m, n]
// therefore accumulates its contributions in one fixed order -- trial triangle ascending,
// then test triangle ascending -- no matter how the tiles are shaped: results are
// bit-identical across tile configurations and runs, with no atomics.  Each output entry is
// written exactly once.  Non-far pairs (singular or near, found by the classifier) are
// taken from the FP64 singular-pair buffer instead of the far rule.
//
// The tile kernel serves the mixed path and FP64 batches; single FP64 assemblies compute the local matrices of
// panels of pairs (k_pair64, below) and gather them in a second kernel: at 1/62 of the FP32 rate the halo's
// FP64 work costs more than writing the matrices once (level-4 EFIE: 84.3 -> 46 ms when it was split, 33 ms now).
//
// Roofline: compute-bound on FP32 issue (mixed) or FP64 issue (plain), plus MUFU (rsqrt, rcp, sin, cos: 4 per
// point pair).  The default rule pair (3 x 4 points) has its own pair code (bgb_far_pair34.cuh); the other rules
// take 21 packed FP32 operations per two point pairs (EFIE).
//
// Mixed precision (FP32) keeps the phase k R accurate without FP64: per pair, the centroid
// distance D = c_tau - c_sigma is formed in double-float, R0 is any FP32 number close to |D|,
// and phi0 = k R0 mod 2 pi is reduced exactly (Dekker product + Cody-Waite); per point pair
// only delta = R - R0 = q / (R + R0) with q = |D_hi + s|^2 - R0^2 computed cancellation-free
// in FP32 enters the phase (psi = phi0 + k delta), so the absolute phase error stays ~1e-7
// rad regardless of k R.  Shape functions use coordinates relative to each triangle's
// centroid, so the EFIE/MFIE bilinear forms carry no cancellation either.
// Far-pair kernel templates; instantiated per precision and operator in bgb_far_*_op*.cu.
#pragma once
#include "bgb_df.cuh"
#include "bgb_kernels.cuh"

#include <algorithm>

namespace bgb {
namespace farimpl {

constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr float kPiA = 6.28125f;
constexpr float kPiB = (float)(kTwoPi - 6.28125);
constexpr float kPiC = (float)(kTwoPi - 6.28125 - (double)(float)(kTwoPi - 6.28125));
constexpr float kInv2Pi = (float)(1.0 / kTwoPi);
// Hardware approximations (PTX .approx with flush-to-zero).  Their arguments in the FP32 pair loop
// are normal numbers (squared distances, sums of distances, phases within a few pi), so the
// denormal handling that the non-flushing forms add to each call is dead weight there.
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_ftz(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void sincos_ftz(float x, float* s, float* c) {
  asm("sin.approx.ftz.f32 %0, %1;" : "=f"(*s) : "f"(x));
  asm("cos.approx.ftz.f32 %0, %1;" : "=f"(*c) : "f"(x));
}
// e^x = 2^(x log2 e)
__device__ __forceinline__ float exp_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}

// Operators on Lagrange hats: Helmholtz single layer, double layer, transposed double layer,
// hypersingular.  They share the hat accumulation of the single layer.
__host__ __device__ constexpr bool is_lagrange_op(int op) {
  return op == BGB_OP_HELMHOLTZ3D_SL || op == BGB_OP_HELMHOLTZ3D_DL || op == BGB_OP_HELMHOLTZ3D_DLT ||
         op == BGB_OP_HELMHOLTZ3D_HS;
}
// Unit normal (v0 - v2) x (v1 - v2) / (2A) from the centroid-relative vertices vo[3][3].
template <class T>
__device__ __forceinline__ void tri_normal(const T* vo, T inv2a, T n[3]) {
  const T a0 = vo[0] - vo[6], a1 = vo[1] - vo[7], a2 = vo[2] - vo[8];
  const T b0 = vo[3] - vo[6], b1 = vo[4] - vo[7], b2 = vo[5] - vo[8];
  n[0] = (a1 * b2 - a2 * b1) * inv2a;
  n[1] = (a2 * b0 - a0 * b2) * inv2a;
  n[2] = (a0 * b1 - a1 * b0) * inv2a;
}
// Surface curls of the hats, n x grad(lambda_i) = (v_{i+1} - v_{i+2}) / (2A).
template <class T>
__device__ __forceinline__ void tri_curls(const T* vo, T inv2a, T c[3][3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) c[i][k] = (vo[3 * ((i + 1) % 3) + k] - vo[3 * ((i + 2) % 3) + k]) * inv2a;
}

}  // namespace farimpl
}  // namespace bgb
#include "bgb_far_pair34.cuh"
namespace bgb {
namespace farimpl {

// Records of the generic rules (the 3 x 4 rule pair has its own, bgb_far_pair34.cuh).
// FP32 record of a triangle, in 16-byte groups read with 128-bit shared-memory loads:
// [CH.xyz CL.x] [CL.yz - -] [VO (9) INV2A - -], two groups [x0 x1 y0 y1] [z0 z1 w0 w1] per two quadrature points
// (the operands of packed operations; a last odd point is paired with itself at weight zero).  The stride follows
// the rule's points (6 or 7: 52 floats) and is an odd number of groups, so the records of different triangles
// start in different bank groups.
__host__ __device__ constexpr int off32_size(int q) { return 4 * ((5 + q + (q & 1)) | 1); }
struct Off32 {
  static constexpr int CH = 0, CL = 3, VO = 8, INV2A = VO + 9, X = 20;
  static __host__ __device__ constexpr int px(int I) { return X + 8 * (I >> 1) + (I & 1); }  // x; y, z: 2, 4 on
  static __host__ __device__ constexpr int pw(int I) { return px(I) + 6; }                  // weight
};
template <int Q>
struct Off64 {
  static constexpr int C = 0, X = 3, W = 3 + 3 * Q, VO = 3 + 4 * Q, INV2A = 12 + 4 * Q, SIZE = 13 + 4 * Q;
};

struct PMixed {
  using R = float;
  using C = float2;
  static constexpr int kThreads = 256, kMinBlocks = 3;  // 24 warps per SM (<= 85 registers)
  template <int Q>  // stride of the records of a rule of q points (q <= Q)
  static __host__ __device__ constexpr int rec(int q) { return Q <= 4 ? kRec34F : off32_size(q); }
  static __device__ __forceinline__ C mk(double a, double b) { return make_float2((float)a, (float)b); }
};
struct PFp64 {
  using R = double;
  using C = double2;
  static constexpr int kThreads = 256, kMinBlocks = 1;
  template <int Q>
  static __host__ __device__ constexpr int rec(int = 0) { return Q <= 4 ? kRec34D : Off64<Q>::SIZE; }
  static __device__ __forceinline__ C mk(double a, double b) { return make_double2(a, b); }
};

// ----------------------------------------------------------------------------------------
// Mixed FP32 far pair
// ----------------------------------------------------------------------------------------
// the 9 vertex offsets of an FP32 record (three 16-byte groups)
__device__ __forceinline__ void load_vo(const float4* __restrict__ g, float V[3][3]) {
  const float4 v0 = g[0], v1 = g[1], v2 = g[2];
  V[0][0] = v0.x; V[0][1] = v0.y; V[0][2] = v0.z;
  V[1][0] = v0.w; V[1][1] = v1.x; V[1][2] = v1.y;
  V[2][0] = v1.z; V[2][1] = v1.w; V[2][2] = v2.x;
}

using f2x = unsigned long long;  // two FP32 numbers, the operand of packed operations
__device__ __forceinline__ f2x both(float x) { return pk2(x, x); }
__device__ __forceinline__ float half_sum(f2x a) {
  float x, y;
  upk2(a, x, y);
  return x + y;
}

// Bound by FP32 issue and MUFU (4 per point pair).  Trial points two at a time in packed operations, loops rolled: the
// scalar form, unrolled over 13 x 13 points with an exit per point, ran ~120 KB of code per pair.  The MFIE's
// sums come from sum H and sum H y like the EFIE's from sum G and sum G y.  Level-4 EFIE, 6 x 7 points: far stage
// 6.9 -> 3.9 ms with the per-chunk trial records and strides by the rule's points (60 x 80 tiles instead of
// 60 x 64 cut to fit, 1.56 instead of 1.86 times the pairs); unrolled by two 4.7 ms, two CTAs per SM 4.4 - 4.8 ms.
template <int OP, int QT, int QB>
__device__ __forceinline__ void far_pair_mixed(const FarScalars& K, const float (*__restrict__ shpT)[3],
                                               const float (*__restrict__ shpB)[BGB_MAXQ + 1], const float* __restrict__ a,
                                               const float* __restrict__ b, float2 L[9]) {
  using OA = Off32;
  using OB = Off32;
  const float4* __restrict__ a4 = reinterpret_cast<const float4*>(a);
  const float4* __restrict__ b4 = reinterpret_cast<const float4*>(b);
  float Dh[3], Dl[3];
  {
    const float4 a0 = a4[0], a1 = a4[1], b0 = b4[0], b1 = b4[1];
    const float ach[3] = {a0.x, a0.y, a0.z}, acl[3] = {a0.w, a1.x, a1.y};
    const float bch[3] = {b0.x, b0.y, b0.z}, bcl[3] = {b0.w, b1.x, b1.y};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float s, e;
      two_sum(ach[c], -bch[c], s, e);
      e = __fadd_rn(e, __fsub_rn(acl[c], bcl[c]));
      fast_two_sum(s, e, Dh[c], Dl[c]);
    }
  }
  const float n2 = fmaf(Dh[0], Dh[0], fmaf(Dh[1], Dh[1], Dh[2] * Dh[2]));
  const float R0 = near_root(n2);
  // c0 = |D_hi|^2 - R0^2, exact to double-float accuracy
  float p0, e0, p1, e1, p2, e2, s1, f1, s2, f2, r2h, r2l;
  two_prod(Dh[0], Dh[0], p0, e0);
  two_prod(Dh[1], Dh[1], p1, e1);
  two_prod(Dh[2], Dh[2], p2, e2);
  two_sum(p0, p1, s1, f1);
  two_sum(s1, p2, s2, f2);
  const float lo = __fadd_rn(__fadd_rn(__fadd_rn(f1, f2), __fadd_rn(e0, e1)), e2);
  two_prod(R0, R0, r2h, r2l);
  const float c0 = __fadd_rn(__fsub_rn(s2, r2h), __fsub_rn(lo, r2l));
  // phi0 = k R0 mod 2 pi
  float ph, pl;
  two_prod(K.k_hi, R0, ph, pl);
  pl = fmaf(K.k_lo, R0, pl);
  const float nq = rintf(ph * kInv2Pi);
  float phi0 = fmaf(-nq, kPiA, ph);
  phi0 = fmaf(-nq, kPiB, phi0);
  phi0 = fmaf(-nq, kPiC, phi0);
  phi0 = __fadd_rn(phi0, pl);
  const float D2x = 2.f * Dh[0], D2y = 2.f * Dh[1], D2z = 2.f * Dh[2];
  const float kh = K.k_hi;
  const float amp0 = K.lossy ? exp_ftz(-K.gre * R0) : 1.f;
  constexpr bool kHH = is_lagrange_op(OP);
  constexpr bool kGrad = OP == BGB_OP_HELMHOLTZ3D_DL || OP == BGB_OP_HELMHOLTZ3D_DLT || OP == BGB_OP_MAXWELL3D_DL;
  float nA[3] = {0.f, 0.f, 0.f}, nB[3] = {0.f, 0.f, 0.f};
  if (OP == BGB_OP_HELMHOLTZ3D_DLT || OP == BGB_OP_HELMHOLTZ3D_HS) tri_normal(a + OA::VO, a[OA::INV2A], nA);
  if (OP == BGB_OP_HELMHOLTZ3D_DL || OP == BGB_OP_HELMHOLTZ3D_HS) tri_normal(b + OB::VO, b[OB::INV2A], nB);
  const int qt = QT < BGB_MAXQ ? QT : K.qt;
  const int qb2 = (QB < BGB_MAXQ ? QB + 1 : K.qb + 1) / 2;

  // accumulators
  float2 S = make_float2(0.f, 0.f), P0 = make_float2(0.f, 0.f);
  float2 Px[3], Py[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) Px[c] = Py[c] = make_float2(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 9; ++k) L[k] = make_float2(0.f, 0.f);

  const f2x R0sq2 = both(R0 * R0), R02 = both(R0), kh2 = both(kh), phi2 = both(phi0);
#pragma unroll 1
  for (int I = 0; I < qt; ++I) {
    const float* __restrict__ pi = a + OA::px(I);
    const float Xx = pi[0], Xy = pi[2], Xz = pi[4], wI = pi[6];
    const float ax = Dl[0] + Xx, ay = Dl[1] + Xy, az = Dl[2] + Xz;
    // q = |D + X_I - y|^2 - R0^2 = KI + y . (y - 2 (D + X_I))
    const f2x KI = both(fmaf(ax, ax + D2x, fmaf(ay, ay + D2y, fmaf(az, az + D2z, c0))));
    const f2x ex = both(-fmaf(2.f, ax, D2x)), ey = both(-fmaf(2.f, ay, D2y)), ez = both(-fmaf(2.f, az, D2z));
    // sums of G (or of its radial derivative over R) times the weights, points y and hats; halves: even and odd points
    f2x Tr = 0, Ti = 0, Ur[3] = {0, 0, 0}, Ui[3] = {0, 0, 0};
#pragma unroll 1
    for (int J = 0; J < qb2; ++J) {
      const ulonglong2 g0 = *reinterpret_cast<const ulonglong2*>(b + OB::X + 8 * J);
      const ulonglong2 g1 = *reinterpret_cast<const ulonglong2*>(b + OB::X + 8 * J + 4);
      const f2x yx = g0.x, yy = g0.y, yz = g1.x, w = g1.y;
      const f2x q = fma2(add2(yx, ex), yx, fma2(add2(yy, ey), yy, fma2(add2(yz, ez), yz, KI)));
      const f2x R2 = add2(R0sq2, q);
      float u0, u1, s0, s1, k0, k1;
      upk2(R2, u0, u1);
      const f2x rs = pk2(rsqrt_ftz(u0), rsqrt_ftz(u1));
      upk2(fma2(R2, rs, R02), u0, u1);
      const f2x delta = mul2(q, pk2(rcp_ftz(u0), rcp_ftz(u1)));
      f2x psi = fma2(kh2, delta, phi2);
      if (!K.phase_direct) {  // |psi| may exceed 2 pi: reduce again (rounding by the 1.5 2^23 addend)
        const f2x magic = both(12582912.f);
        const f2x n = sub2(magic, fma2(psi, both(kInv2Pi), magic));
        psi = fma2(n, both(kPiB), fma2(n, both(kPiA), psi));
      }
      upk2(psi, u0, u1);
      sincos_ftz(u0, &s0, &k0);
      sincos_ftz(u1, &s1, &k1);
      f2x amp = mul2(w, rs);
      if (K.lossy) {
        upk2(mul2(both(-K.gre), delta), u0, u1);
        amp = mul2(amp, mul2(both(amp0), pk2(exp_ftz(u0), exp_ftz(u1))));
      }
      f2x hr = mul2(amp, pk2(k0, k1)), hi = mul2(amp, pk2(-s0, -s1));  // G
      if (kGrad) {  // (gamma + 1 / R) G / R
        const f2x t = mul2(add2(both(K.gre), rs), rs), u = mul2(kh2, rs);
        const f2x gr = hr, gi = hi;
        hr = fma2(t, gr, neg2(mul2(u, gi)));
        hi = fma2(t, gi, mul2(u, gr));
      }
      if (kHH) {
        if (OP == BGB_OP_HELMHOLTZ3D_DLT) {  // times -(x - y) . n_x = -(D - y) . n_x
          const f2x e = fma2(sub2(yx, both(Dl[0] + Dh[0])), both(nA[0]),
                             fma2(sub2(yy, both(Dl[1] + Dh[1])), both(nA[1]), mul2(sub2(yz, both(Dl[2] + Dh[2])), both(nA[2]))));
          hr = mul2(hr, e);
          hi = mul2(hi, e);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const f2x g = *reinterpret_cast<const f2x*>(&shpB[j][2 * J]);
          Ur[j] = fma2(hr, g, Ur[j]);
          Ui[j] = fma2(hi, g, Ui[j]);
        }
      } else {
        Tr = add2(Tr, hr);
        Ti = add2(Ti, hi);
        Ur[0] = fma2(hr, yx, Ur[0]); Ui[0] = fma2(hi, yx, Ui[0]);
        Ur[1] = fma2(hr, yy, Ur[1]); Ui[1] = fma2(hi, yy, Ui[1]);
        Ur[2] = fma2(hr, yz, Ur[2]); Ui[2] = fma2(hi, yz, Ui[2]);
      }
    }
    const float2 T = make_float2(half_sum(Tr), half_sum(Ti));
    float2 U[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) U[c] = make_float2(half_sum(Ur[c]), half_sum(Ui[c]));
    if (kHH) {
      // double layer: (x - y) . n_y = (D + X_I) . n_y, constant over the trial points
      const float cI = OP == BGB_OP_HELMHOLTZ3D_DL
                           ? wI * fmaf(Dh[0] + ax, nB[0], fmaf(Dh[1] + ay, nB[1], (Dh[2] + az) * nB[2]))
                           : wI;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const float f = shpT[I][i] * cI;
#pragma unroll
        for (int j = 0; j < 3; ++j) L[i * 3 + j] = cfm(U[j], f, L[i * 3 + j]);
      }
    } else if (OP == BGB_OP_MAXWELL3D_SL) {
      const float x = wI * Xx, y = wI * Xy, z = wI * Xz;
      S = cfm(U[0], x, cfm(U[1], y, cfm(U[2], z, S)));
      Px[0] = cfm(T, x, Px[0]);
      Px[1] = cfm(T, y, Px[1]);
      Px[2] = cfm(T, z, Px[2]);
#pragma unroll
      for (int c = 0; c < 3; ++c) Py[c] = cfm(U[c], wI, Py[c]);
      P0 = cfm(T, wI, P0);
    } else {
      // H = -(gamma + 1 / R) G / R, d = x - y = e + (X_I - y), e = D: with T = -sum H, U = -sum H y,
      // E = sum H d = U - (D + X_I) T and B = sum H d x y = U x (D + X_I)
      const float dx = -wI * (Dh[0] + ax), dy = -wI * (Dh[1] + ay), dz = -wI * (Dh[2] + az);
      const float2 E0 = cfm(T, dx, csc(U[0], wI)), E1 = cfm(T, dy, csc(U[1], wI)), E2 = cfm(T, dz, csc(U[2], wI));
      const float2 B0 = cfm(U[2], dy, csc(U[1], -dz)), B1 = cfm(U[0], dz, csc(U[2], -dx)),
                   B2 = cfm(U[1], dx, csc(U[0], -dy));
      // C += X x E (Px), A1 += X . B (S), B (Py), E (L[0..2])
      Px[0] = cfm(E2, Xy, cfm(E1, -Xz, Px[0]));
      Px[1] = cfm(E0, Xz, cfm(E2, -Xx, Px[1]));
      Px[2] = cfm(E1, Xx, cfm(E0, -Xy, Px[2]));
      S = cfm(B0, Xx, cfm(B1, Xy, cfm(B2, Xz, S)));
      Py[0] = cad(Py[0], B0);
      Py[1] = cad(Py[1], B1);
      Py[2] = cad(Py[2], B2);
      L[0] = cad(L[0], E0);
      L[1] = cad(L[1], E1);
      L[2] = cad(L[2], E2);
    }
  }
  const float2 alpha = make_float2(K.alpha32[0], K.alpha32[1]);
  if (OP == BGB_OP_HELMHOLTZ3D_HS) {
    // alpha (n_x . n_y) int int f g G + beta (curl f . curl g) int int G, int int G = sum of L
    float2 P = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 9; ++k) { P.x += L[k].x; P.y += L[k].y; }
    const float nn = fmaf(nA[0], nB[0], fmaf(nA[1], nB[1], nA[2] * nB[2]));
    const float2 an = make_float2(alpha.x * nn, alpha.y * nn);
    const float2 bP = cmulf(make_float2(K.beta32[0], K.beta32[1]), P);
    float cA[3][3], cB[3][3];
    tri_curls(a + OA::VO, a[OA::INV2A], cA);
    tri_curls(b + OB::VO, b[OB::INV2A], cB);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const float cc = fmaf(cA[i][0], cB[j][0], fmaf(cA[i][1], cB[j][1], cA[i][2] * cB[j][2]));
        const float2 t = cmulf(an, L[i * 3 + j]);
        L[i * 3 + j] = make_float2(fmaf(cc, bP.x, t.x), fmaf(cc, bP.y, t.y));
      }
    return;
  }
  if (kHH) {
#pragma unroll
    for (int k = 0; k < 9; ++k) L[k] = cmulf(alpha, L[k]);
    return;
  }
  const float inv4AA = a[OA::INV2A] * b[OB::INV2A];
  const float2 ca = make_float2(alpha.x * inv4AA, alpha.y * inv4AA);
  if (OP == BGB_OP_MAXWELL3D_SL) {
    // L_ij = alpha/(4 A A) (S - V_i.Py - W_j.Px + (V_i.W_j) P0) + beta/(A A) P0
    const float invAA = 4.f * inv4AA;
    const float2 cb = make_float2(K.beta32[0] * invAA, K.beta32[1] * invAA);
    const float2 tb = cmulf(cb, P0);
    float V[3][3], W[3][3];
    load_vo(a4 + OA::VO / 4, V);
    load_vo(b4 + OB::VO / 4, W);
    float2 Ai[3], Bj[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      Ai[i].x = S.x - fmaf(V[i][0], Py[0].x, fmaf(V[i][1], Py[1].x, V[i][2] * Py[2].x));
      Ai[i].y = S.y - fmaf(V[i][0], Py[0].y, fmaf(V[i][1], Py[1].y, V[i][2] * Py[2].y));
      Bj[i].x = fmaf(W[i][0], Px[0].x, fmaf(W[i][1], Px[1].x, W[i][2] * Px[2].x));
      Bj[i].y = fmaf(W[i][0], Px[0].y, fmaf(W[i][1], Px[1].y, W[i][2] * Px[2].y));
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const float vw = fmaf(V[i][0], W[j][0], fmaf(V[i][1], W[j][1], V[i][2] * W[j][2]));
        const float tx = fmaf(vw, P0.x, Ai[i].x - Bj[j].x);
        const float ty = fmaf(vw, P0.y, Ai[i].y - Bj[j].y);
        L[i * 3 + j] = make_float2(fmaf(ca.x, tx, fmaf(-ca.y, ty, tb.x)), fmaf(ca.x, ty, fmaf(ca.y, tx, tb.y)));
      }
    return;
  }
  // MFIE: L = alpha/(4AA) (A1 - W_j . C - V_i . B + V_i . (E x W_j))
  const float2 E0 = L[0], E1 = L[1], E2 = L[2];
  float2 vb[3], wc[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float vx = a[OA::VO + 3 * i], vy = a[OA::VO + 3 * i + 1], vz = a[OA::VO + 3 * i + 2];
    vb[i].x = vx * Py[0].x + vy * Py[1].x + vz * Py[2].x;
    vb[i].y = vx * Py[0].y + vy * Py[1].y + vz * Py[2].y;
    const float wx = b[OB::VO + 3 * i], wy = b[OB::VO + 3 * i + 1], wz = b[OB::VO + 3 * i + 2];
    wc[i].x = wx * Px[0].x + wy * Px[1].x + wz * Px[2].x;
    wc[i].y = wx * Px[0].y + wy * Px[1].y + wz * Px[2].y;
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const float wx = b[OB::VO + 3 * j], wy = b[OB::VO + 3 * j + 1], wz = b[OB::VO + 3 * j + 2];
    // E x W_j
    const float2 x0 = make_float2(E1.x * wz - E2.x * wy, E1.y * wz - E2.y * wy);
    const float2 x1 = make_float2(E2.x * wx - E0.x * wz, E2.y * wx - E0.y * wz);
    const float2 x2 = make_float2(E0.x * wy - E1.x * wx, E0.y * wy - E1.y * wx);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const float vx = a[OA::VO + 3 * i], vy = a[OA::VO + 3 * i + 1], vz = a[OA::VO + 3 * i + 2];
      float2 t;
      t.x = S.x - wc[j].x - vb[i].x + (vx * x0.x + vy * x1.x + vz * x2.x);
      t.y = S.y - wc[j].y - vb[i].y + (vx * x0.y + vy * x1.y + vz * x2.y);
      L[i * 3 + j] = cmulf(ca, t);
    }
  }
}

// ----------------------------------------------------------------------------------------
// Plain FP64 far pair (same accumulation structure, FP64 throughout, CUDA sincos / exp)
// ----------------------------------------------------------------------------------------
template <int OP, int QT, int QB>
__device__ __forceinline__ void far_pair_fp64(const FarScalars& K, const double (*__restrict__ shpT)[3],
                                              const double (*__restrict__ shpB)[3], const double* __restrict__ tay_s,
                                              const double* __restrict__ tay_c, const double* __restrict__ a,
                                              const double* __restrict__ b, double2 L[9]) {
  using OA = Off64<QT>;
  using OB = Off64<QB>;
  constexpr bool kHH = is_lagrange_op(OP);
  const double Dx = a[OA::C] - b[OB::C], Dy = a[OA::C + 1] - b[OB::C + 1], Dz = a[OA::C + 2] - b[OB::C + 2];
  const double gre = K.gamma[0], gim = K.gamma[1];
  // Phase k R = k R0 + k (R - R0) with R0 the centroid distance: sin / cos of k R0 once per pair, and
  // of the small k (R - R0) (|.| <= 2) from K.tay_n series terms per point pair (sincos otherwise).
  const int tn = gim != 0.0 ? K.tay_n : 0;
  double R0 = 0.0, s0 = 0.0, c0 = 1.0;
  if (tn > 0) {
    R0 = sqrt(Dx * Dx + Dy * Dy + Dz * Dz);
    sincos(gim * R0, &s0, &c0);
  }
  double nA[3] = {0, 0, 0}, nB[3] = {0, 0, 0};
  if (OP == BGB_OP_HELMHOLTZ3D_DLT || OP == BGB_OP_HELMHOLTZ3D_HS) tri_normal(a + OA::VO, a[OA::INV2A], nA);
  if (OP == BGB_OP_HELMHOLTZ3D_DL || OP == BGB_OP_HELMHOLTZ3D_HS) tri_normal(b + OB::VO, b[OB::INV2A], nB);
  const int qt = QT < BGB_MAXQ ? QT : K.qt;
  const int qb = QB < BGB_MAXQ ? QB : K.qb;
  double2 S = make_double2(0, 0), P0 = make_double2(0, 0);
  double2 Px[3], Py[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) Px[c] = Py[c] = make_double2(0, 0);
#pragma unroll
  for (int k = 0; k < 9; ++k) L[k] = make_double2(0, 0);
#pragma unroll
  for (int I = 0; I < QT; ++I) {
    if (I >= qt) break;
    const double Xx = a[OA::X + 3 * I], Xy = a[OA::X + 3 * I + 1], Xz = a[OA::X + 3 * I + 2];
    const double ax = Dx + Xx, ay = Dy + Xy, az = Dz + Xz;
    const double wI = a[OA::W + I];
    // double layer: (x - y) . n_y = (D + X_I) . n_y, constant over the trial points
    const double cI = OP == BGB_OP_HELMHOLTZ3D_DL ? ax * nB[0] + ay * nB[1] + az * nB[2] : 1.0;
    double2 TI = make_double2(0, 0);
    double2 UI[3], EI[3], BI[3], M[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) UI[c] = EI[c] = BI[c] = M[c] = make_double2(0, 0);
#pragma unroll
    for (int J = 0; J < QB; ++J) {
      if (J >= qb) break;
      const double Yx = b[OB::X + 3 * J], Yy = b[OB::X + 3 * J + 1], Yz = b[OB::X + 3 * J + 2];
      const double dx = ax - Yx, dy = ay - Yy, dz = az - Yz;
      const double R2 = dx * dx + dy * dy + dz * dz;
      const double rinv = rsqrt(R2);
      const double R = R2 * rinv;
      double sn = 0.0, cs = 1.0;
      if (tn > 0) {
        const double x = gim * (R - R0), x2 = x * x;
        double ps = tay_s[tn - 1], pc = tay_c[tn - 1];
        for (int j = tn - 2; j >= 0; --j) {
          ps = fma(ps, x2, tay_s[j]);
          pc = fma(pc, x2, tay_c[j]);
        }
        const double s1 = x * ps;
        sn = fma(s0, pc, c0 * s1);  // sin(k R0 + x)
        cs = fma(c0, pc, -s0 * s1); // cos(k R0 + x)
      } else if (gim != 0.0) {
        sincos(gim * R, &sn, &cs);
      }
      double amp = wI * b[OB::W + J] * rinv;
      if (gre != 0.0) amp *= exp(-gre * R);
      const double gr = amp * cs, gi = -amp * sn;
      if (kHH) {
        double hr = gr, hi = gi;
        if (OP == BGB_OP_HELMHOLTZ3D_DL || OP == BGB_OP_HELMHOLTZ3D_DLT) {
          // (gamma + 1/R) G / R, times -(x - y) . n_x for the transposed double layer
          const double t = (gre + rinv) * rinv, u = gim * rinv;
          hr = t * gr - u * gi;
          hi = t * gi + u * gr;
          if (OP == BGB_OP_HELMHOLTZ3D_DLT) {
            const double e = -(dx * nA[0] + dy * nA[1] + dz * nA[2]);
            hr *= e;
            hi *= e;
          }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const double g = shpB[J][j];
          M[j].x = fma(hr, g, M[j].x);
          M[j].y = fma(hi, g, M[j].y);
        }
      } else if (OP == BGB_OP_MAXWELL3D_SL) {
        TI.x += gr;
        TI.y += gi;
        UI[0].x = fma(gr, Yx, UI[0].x); UI[0].y = fma(gi, Yx, UI[0].y);
        UI[1].x = fma(gr, Yy, UI[1].x); UI[1].y = fma(gi, Yy, UI[1].y);
        UI[2].x = fma(gr, Yz, UI[2].x); UI[2].y = fma(gi, Yz, UI[2].y);
      } else {
        const double g2r = gr * rinv, g2i = gi * rinv;
        const double re = gre + rinv;
        const double Hx = -(re * g2r - gim * g2i), Hy = -(re * g2i + gim * g2r);
        EI[0].x = fma(Hx, dx, EI[0].x); EI[0].y = fma(Hy, dx, EI[0].y);
        EI[1].x = fma(Hx, dy, EI[1].x); EI[1].y = fma(Hy, dy, EI[1].y);
        EI[2].x = fma(Hx, dz, EI[2].x); EI[2].y = fma(Hy, dz, EI[2].y);
        const double c0x = dy * Yz - dz * Yy, c0y = dz * Yx - dx * Yz, c0z = dx * Yy - dy * Yx;
        BI[0].x = fma(Hx, c0x, BI[0].x); BI[0].y = fma(Hy, c0x, BI[0].y);
        BI[1].x = fma(Hx, c0y, BI[1].x); BI[1].y = fma(Hy, c0y, BI[1].y);
        BI[2].x = fma(Hx, c0z, BI[2].x); BI[2].y = fma(Hy, c0z, BI[2].y);
      }
    }
    if (kHH) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double f = shpT[I][i] * cI;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          L[i * 3 + j].x = fma(f, M[j].x, L[i * 3 + j].x);
          L[i * 3 + j].y = fma(f, M[j].y, L[i * 3 + j].y);
        }
      }
    } else if (OP == BGB_OP_MAXWELL3D_SL) {
      S.x = fma(Xx, UI[0].x, fma(Xy, UI[1].x, fma(Xz, UI[2].x, S.x)));
      S.y = fma(Xx, UI[0].y, fma(Xy, UI[1].y, fma(Xz, UI[2].y, S.y)));
      Px[0].x = fma(Xx, TI.x, Px[0].x); Px[0].y = fma(Xx, TI.y, Px[0].y);
      Px[1].x = fma(Xy, TI.x, Px[1].x); Px[1].y = fma(Xy, TI.y, Px[1].y);
      Px[2].x = fma(Xz, TI.x, Px[2].x); Px[2].y = fma(Xz, TI.y, Px[2].y);
#pragma unroll
      for (int c = 0; c < 3; ++c) { Py[c].x += UI[c].x; Py[c].y += UI[c].y; }
      P0.x += TI.x;
      P0.y += TI.y;
    } else {
      Px[0].x += Xy * EI[2].x - Xz * EI[1].x; Px[0].y += Xy * EI[2].y - Xz * EI[1].y;
      Px[1].x += Xz * EI[0].x - Xx * EI[2].x; Px[1].y += Xz * EI[0].y - Xx * EI[2].y;
      Px[2].x += Xx * EI[1].x - Xy * EI[0].x; Px[2].y += Xx * EI[1].y - Xy * EI[0].y;
      S.x = fma(Xx, BI[0].x, fma(Xy, BI[1].x, fma(Xz, BI[2].x, S.x)));
      S.y = fma(Xx, BI[0].y, fma(Xy, BI[1].y, fma(Xz, BI[2].y, S.y)));
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        Py[c].x += BI[c].x; Py[c].y += BI[c].y;
        L[c].x += EI[c].x; L[c].y += EI[c].y;
      }
    }
  }
  const double2 alpha = make_double2(K.alpha[0], K.alpha[1]);
  if (OP == BGB_OP_HELMHOLTZ3D_HS) {
    // alpha (n_x . n_y) int int f g G + beta (curl f . curl g) int int G, int int G = sum of L
    double2 P = make_double2(0, 0);
#pragma unroll
    for (int k = 0; k < 9; ++k) { P.x += L[k].x; P.y += L[k].y; }
    const double nn = nA[0] * nB[0] + nA[1] * nB[1] + nA[2] * nB[2];
    const double2 an = make_double2(alpha.x * nn, alpha.y * nn);
    const double2 bP = cmul(make_double2(K.beta[0], K.beta[1]), P);
    double cA[3][3], cB[3][3];
    tri_curls(a + OA::VO, a[OA::INV2A], cA);
    tri_curls(b + OB::VO, b[OB::INV2A], cB);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double cc = cA[i][0] * cB[j][0] + cA[i][1] * cB[j][1] + cA[i][2] * cB[j][2];
        const double2 t = cmul(an, L[i * 3 + j]);
        L[i * 3 + j] = make_double2(fma(cc, bP.x, t.x), fma(cc, bP.y, t.y));
      }
    return;
  }
  if (kHH) {
#pragma unroll
    for (int k = 0; k < 9; ++k) L[k] = cmul(alpha, L[k]);
    return;
  }
  const double inv4AA = a[OA::INV2A] * b[OB::INV2A];
  const double2 ca = make_double2(alpha.x * inv4AA, alpha.y * inv4AA);
  if (OP == BGB_OP_MAXWELL3D_SL) {
    const double invAA = 4.0 * inv4AA;
    const double2 cb = make_double2(K.beta[0] * invAA, K.beta[1] * invAA);
    const double2 tb = cmul(cb, P0);
    double2 av[3], bv[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double vx = a[OA::VO + 3 * i], vy = a[OA::VO + 3 * i + 1], vz = a[OA::VO + 3 * i + 2];
      av[i].x = vx * Py[0].x + vy * Py[1].x + vz * Py[2].x;
      av[i].y = vx * Py[0].y + vy * Py[1].y + vz * Py[2].y;
      const double wx = b[OB::VO + 3 * i], wy = b[OB::VO + 3 * i + 1], wz = b[OB::VO + 3 * i + 2];
      bv[i].x = wx * Px[0].x + wy * Px[1].x + wz * Px[2].x;
      bv[i].y = wx * Px[0].y + wy * Px[1].y + wz * Px[2].y;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double vw = a[OA::VO + 3 * i] * b[OB::VO + 3 * j] + a[OA::VO + 3 * i + 1] * b[OB::VO + 3 * j + 1] +
                          a[OA::VO + 3 * i + 2] * b[OB::VO + 3 * j + 2];
        double2 t;
        t.x = S.x - av[i].x - bv[j].x + vw * P0.x;
        t.y = S.y - av[i].y - bv[j].y + vw * P0.y;
        const double2 r = cmul(ca, t);
        L[i * 3 + j] = make_double2(r.x + tb.x, r.y + tb.y);
      }
    return;
  }
  const double2 E0 = L[0], E1 = L[1], E2 = L[2];
  double2 vb[3], wc[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double vx = a[OA::VO + 3 * i], vy = a[OA::VO + 3 * i + 1], vz = a[OA::VO + 3 * i + 2];
    vb[i].x = vx * Py[0].x + vy * Py[1].x + vz * Py[2].x;
    vb[i].y = vx * Py[0].y + vy * Py[1].y + vz * Py[2].y;
    const double wx = b[OB::VO + 3 * i], wy = b[OB::VO + 3 * i + 1], wz = b[OB::VO + 3 * i + 2];
    wc[i].x = wx * Px[0].x + wy * Px[1].x + wz * Px[2].x;
    wc[i].y = wx * Px[0].y + wy * Px[1].y + wz * Px[2].y;
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double wx = b[OB::VO + 3 * j], wy = b[OB::VO + 3 * j + 1], wz = b[OB::VO + 3 * j + 2];
    const double2 x0 = make_double2(E1.x * wz - E2.x * wy, E1.y * wz - E2.y * wy);
    const double2 x1 = make_double2(E2.x * wx - E0.x * wz, E2.y * wx - E0.y * wz);
    const double2 x2 = make_double2(E0.x * wy - E1.x * wx, E0.y * wy - E1.y * wx);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double vx = a[OA::VO + 3 * i], vy = a[OA::VO + 3 * i + 1], vz = a[OA::VO + 3 * i + 2];
      double2 t;
      t.x = S.x - wc[j].x - vb[i].x + (vx * x0.x + vy * x1.x + vz * x2.x);
      t.y = S.y - wc[j].y - vb[i].y + (vx * x0.y + vy * x1.y + vz * x2.y);
      L[i * 3 + j] = cmul(ca, t);
    }
  }
}

__device__ __forceinline__ FarScalars far_scalars(const FarConst& K) {
  FarScalars S;
  S.qt = K.qt;
  S.qb = K.qb;
  S.lossy = K.lossy;
  S.phase_direct = K.phase_direct;
  S.tay_n = K.tay_n;
  S.k_hi = K.k_hi;
  S.k_lo = K.k_lo;
  S.gre = K.gre;
  for (int c = 0; c < 2; ++c) {
    S.alpha32[c] = K.alpha32[c];
    S.beta32[c] = K.beta32[c];
    S.alpha[c] = K.alpha[c];
    S.beta[c] = K.beta[c];
    S.gamma[c] = K.gamma[c];
    S.far_a[c] = K.far_a[c];
    S.far_b[c] = K.far_b[c];
    S.far_a32[c] = (float)K.far_a[c];
    S.far_b32[c] = (float)K.far_b[c];
  }
  return S;
}

// Points that lie close to each other against the centroid distance (a small triangle over the inside of a large one):
// E + H + d, a sum of terms of size |D|^2, carries eps (R0 / R)^2 into R^2, the points' difference eps R0 / R, as far as
// the points themselves are known.  A function of its own: as a branch inside the pair code it cost the level-4 EFIE 6%
// (33.2 -> 35.4 ms), by the registers that stay live and the code that no longer overlaps.
template <int OP>
__device__ __noinline__ void far_pair34_fp64_close(const FarConst& K, const double* __restrict__ a,
                                                   const double* __restrict__ b, double2* __restrict__ L) {
  double2 t[9];
  far_pair34_fp64<OP, true>(far_scalars(K), K.tay_s, K.tay_c, a, b, t);
#pragma unroll
  for (int k = 0; k < 9; ++k) L[k] = t[k];
}
// True below R0 = 2.3 - 2.45 times the larger of the point radii, by exponents (n < 5.3 - 6 times the radius squared),
// beside the FP64 pipe.  Beyond, points may still be as close as R0 / 6 where triangles of about one size overlap;
// overlapping plates (8 x 8 on 8 x 8, 12 x 12) are within 1e-15 of a pair's matrix there, as below 3.4 radii before.
// Triangles that do not overlap come this near on stretched meshes only; 3.4 radii took in pairs of every plate and box,
// 25 of 700 us of a small call.
__device__ __forceinline__ bool far_pair34_is_close(const double* __restrict__ a, const double* __restrict__ b) {
  double n = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) n = fm(sb(a[k], b[k]), sb(a[k], b[k]), n);
  int top = max(__double2hiint(a[12]), __double2hiint(b[12]));
#pragma unroll
  for (int i = 1; i < 3; ++i) top = max(top, max(__double2hiint(a[12 + i]), __double2hiint(b[12 + i])));
  return __double2hiint(n) < top + 0x00280000;
}

template <class P, int OP, int QT, int QB>
__device__ __forceinline__ void far_pair(const FarScalars& S, const FarConst& K, const typename P::R* a,
                                         const typename P::R* b, typename P::C L[9]) {
  if constexpr (QT == 3 && QB == 4 && sizeof(typename P::R) == 4)
    far_pair34_mixed<OP>(S, a, b, L);
  else if constexpr (QT == 3 && QB == 4) {
    if (far_pair34_is_close(a, b)) {
      double2 t[9];
      far_pair34_fp64_close<OP>(K, a, b, t);
#pragma unroll
      for (int k = 0; k < 9; ++k) L[k] = t[k];
    } else {
      far_pair34_fp64<OP, false>(S, K.tay_s, K.tay_c, a, b, L);
    }
  } else if constexpr (sizeof(typename P::R) == 4)
    far_pair_mixed<OP, QT, QB>(S, K.shpT, K.shpB, a, b, L);
  else
    far_pair_fp64<OP, QT, QB>(S, K.shpT64, K.shpB64, K.tay_s, K.tay_c, a, b, L);
}

__device__ __forceinline__ int64_t find_sigma(const int64_t* __restrict__ off, const int* __restrict__ sig, int tau,
                                              int sigma) {
  int64_t lo = off[tau], hi = off[tau + 1];
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    int v = sig[mid];
    if (v == sigma) return mid;
    if (v < sigma) lo = mid + 1;
    else hi = mid;
  }
  return -1;
}

// ----------------------------------------------------------------------------------------
// Tile kernel
// ----------------------------------------------------------------------------------------
// A support of a trial function in a chunk: its offset in a pair's local matrices, its coefficient.
template <class R>
struct Support {
  int col;
  R w;
};

template <class P>
struct Smem {
  float4* bndT;
  float4* bndB;
  int* triT;
  int* triB;
  int* row;        // output row of each test function
  typename P::R* recT;
  typename P::R* recB;
  int* fcnt;
  int* fcode;
  typename P::R* fcoef;
  typename P::C* Lbuf;
  typename P::C* Zs;
  int2* grp;       // per group of the trial block: offset of its function in Zs, first support << 5 | count
  int* chGrp;      // per chunk: first group (block-relative)
  Support<typename P::R>* gs;
};

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

// Trial records staged per chunk (two chunk buffers, the next copied in while the current one is
// computed) instead of per tile: for the large records of the generic FP32 rules, which would
// otherwise bound the tile's width.
template <class P, int OP, int QB>
__host__ __device__ constexpr bool chunk_trial_records() {
  return sizeof(typename P::R) == 4 && QB > 4;
}

template <class P>
__host__ __device__ inline size_t carve(unsigned char* base, int tmax, int nmax, int rt, int rb, int FM, int FN,
                                        int MAXS, int SC, int gmax, int gsmax, bool chunk_recb, Smem<P>* s) {
  using R = typename P::R;
  using C = typename P::C;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off = align16(off + bytes);
    return base ? base + o : nullptr;
  };
  unsigned char* p;
  p = take(sizeof(float4) * tmax); if (s) s->bndT = (float4*)p;
  p = take(sizeof(float4) * nmax); if (s) s->bndB = (float4*)p;
  p = take(sizeof(int) * tmax); if (s) s->triT = (int*)p;
  p = take(sizeof(int) * nmax); if (s) s->triB = (int*)p;
  p = take(sizeof(int) * FM); if (s) s->row = (int*)p;
  p = take(sizeof(R) * (size_t)tmax * rt); if (s) s->recT = (R*)p;
  p = take(sizeof(R) * (size_t)(chunk_recb ? 2 * SC : nmax) * rb); if (s) s->recB = (R*)p;
  p = take(sizeof(int) * FM); if (s) s->fcnt = (int*)p;
  p = take(sizeof(int) * (size_t)FM * MAXS); if (s) s->fcode = (int*)p;
  p = take(sizeof(R) * (size_t)FM * MAXS); if (s) s->fcoef = (R*)p;
  p = take(sizeof(C) * 9 * (size_t)tmax * SC); if (s) s->Lbuf = (C*)p;
  p = take(sizeof(C) * (size_t)FM * FN); if (s) s->Zs = (C*)p;
  const int nch = (nmax + SC - 1) / SC;
  p = take(sizeof(int2) * (size_t)gmax); if (s) s->grp = (int2*)p;
  p = take(sizeof(int) * (size_t)(nch + 1)); if (s) s->chGrp = (int*)p;
  p = take(sizeof(Support<R>) * (size_t)gsmax); if (s) s->gs = (Support<R>*)p;
  return off;
}

// 16-byte asynchronous global -> shared copies (completion awaited by the issuing thread).
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// One output tile (test-function block bm x trial-function block bn).
template <class P, int OP, int QT, int QB>
__device__ __forceinline__ void tile_body(const FarConst& K, const TilePlan& p, int bm, int bn, unsigned char* smem,
                                          int* s_nonfar) {
  using R = typename P::R;
  using C = typename P::C;
  constexpr int kThreads = P::kThreads;
  const int tid = threadIdx.x;
  const FarScalars S = far_scalars(K);  // registers, not shared-memory loads in the pair loop
  const int RT = P::template rec<QT>(S.qt), RB = P::template rec<QB>(S.qb);
  const int SC = p.SC, MAXS = p.MAXS;
  Smem<P> s;
  constexpr bool kChunkB = chunk_trial_records<P, OP, QB>();
  carve<P>(smem, p.tmax, p.nmax, RT, RB, p.FM, p.FN, MAXS, SC, p.gmax, p.gsmax, kChunkB, &s);

  const int t0 = p.tb_off[bm], tm = p.tb_off[bm + 1] - t0;
  const int b0 = p.bb_off[bn], nbk = p.bb_off[bn + 1] - b0;
  const int f0 = p.tb_fn_off[bm], fm = p.tb_fn_off[bm + 1] - f0;
  const int g0 = p.bb_fn_off[bn], fn = p.bb_fn_off[bn + 1] - g0;
  const R* __restrict__ gRT = (const R*)p.rec_t;
  const R* __restrict__ gRB = (const R*)p.rec_b;

  for (int i = tid; i < tm; i += kThreads) {
    const int t = p.tb_tris[t0 + i];
    s.triT[i] = t;
    s.bndT[i] = p.bnd_t[t];
  }
  for (int i = tid; i < nbk; i += kThreads) {
    const int t = p.bb_tris[b0 + i];
    s.triB[i] = t;
    s.bndB[i] = p.bnd_b[t];
  }
  if constexpr (sizeof(R) == 4) {  // FP32 records: whole 16-byte groups
    const int RT4 = RT / 4, RB4 = RB / 4;
    const float4* __restrict__ gT4 = reinterpret_cast<const float4*>(gRT);
    const float4* __restrict__ gB4 = reinterpret_cast<const float4*>(gRB);
    for (int i = tid; i < tm * RT4; i += kThreads) {
      const int r = i / RT4, c = i - r * RT4;
      reinterpret_cast<float4*>(s.recT)[i] = gT4[(int64_t)p.tb_tris[t0 + r] * RT4 + c];
    }
    for (int i = tid; i < (kChunkB ? min(SC, nbk) : nbk) * RB4; i += kThreads) {  // kChunkB: the first chunk's
      const int r = i / RB4, c = i - r * RB4;
      reinterpret_cast<float4*>(s.recB)[i] = gB4[(int64_t)p.bb_tris[b0 + r] * RB4 + c];
    }
  } else {
    for (int i = tid; i < tm * RT; i += kThreads) {
      const int r = i / RT, c = i - r * RT;
      s.recT[i] = gRT[(int64_t)p.tb_tris[t0 + r] * RT + c];
    }
    for (int i = tid; i < nbk * RB; i += kThreads) {
      const int r = i / RB, c = i - r * RB;
      s.recB[i] = gRB[(int64_t)p.bb_tris[b0 + r] * RB + c];
    }
  }
  const bool f32 = sizeof(R) == 4;
  // local matrices of a chunk: entry (i, j) of pair (ti, si) at Lbuf[(i * 3 + j) * LS + ti * SC + si];
  // supports are staged as their offsets in it (test: (i * 3) * LS + ti * SC, trial: j * LS + si)
  const int LS = p.tmax * SC;
  for (int m = tid; m < fm; m += kThreads) {
    const int a0 = p.fs_off[f0 + m], a1 = p.fs_off[f0 + m + 1];
    const int cnt = min(a1 - a0, MAXS);
    s.fcnt[m] = cnt;
    s.row[m] = (int)p.rows[f0 + m];
    for (int k = 0; k < cnt; ++k) {
      const int fc = p.fs_code[a0 + k];  // test triangle << 2 | local
      s.fcode[m * MAXS + k] = (fc & 3) * 3 * LS + (fc >> 2) * SC;
      s.fcoef[m * MAXS + k] = f32 ? (R)p.fs_coef32[a0 + k] : (R)p.fs_coef[a0 + k];
    }
  }
  // the trial block's gather groups (all chunks), block-relative
  const int c0 = p.bb_chunk_off[bn], nch = p.bb_chunk_off[bn + 1] - c0;
  const int gb0 = p.ch_grp_off[c0], gb1 = p.ch_grp_off[c0 + nch];
  const int sb0 = p.grp_sup_off[gb0], sb1 = p.grp_sup_off[gb1];
  for (int i = tid; i < gb1 - gb0; i += kThreads) {
    const int q0 = p.grp_sup_off[gb0 + i], q1 = p.grp_sup_off[gb0 + i + 1];  // at most SC <= 16 supports
    s.grp[i] = make_int2(p.grp_fn[gb0 + i] * fm, (q0 - sb0) << 5 | (q1 - q0));
  }
  for (int i = tid; i <= nch; i += kThreads) s.chGrp[i] = p.ch_grp_off[c0 + i] - gb0;
  for (int i = tid; i < sb1 - sb0; i += kThreads) {
    const int code = p.gs_code[sb0 + i];  // trial slot << 2 | local
    s.gs[i].col = (code & 3) * LS + (code >> 2) % SC;
    s.gs[i].w = f32 ? (R)p.gs_coef32[sb0 + i] : (R)p.gs_coef[sb0 + i];
  }
  for (int i = tid; i < fm * fn; i += kThreads) s.Zs[i] = P::mk(0.0, 0.0);
  if (tid == 0) *s_nonfar = 0;
  __syncthreads();
  // Does the tile hold any non-far pair?  Most tiles do not, and skip the per-pair test.  First a
  // sphere around each block's triangle spheres (warp 0: test block, warp 1: trial block): blocks
  // whose spheres are clearly apart hold no pair that passes the per-pair sphere test, so no
  // non-far pair; only the other tiles scan their test triangles' lists of non-far pairs.
  __shared__ float4 s_blk[2];
  if (tid < 64) {
    const int w = tid >> 5, lane = tid & 31;
    const float4* __restrict__ bl = w ? s.bndB : s.bndT;
    const int nb = w ? nbk : tm;
    float cx = 0.f, cy = 0.f, cz = 0.f;
    for (int i = lane; i < nb; i += 32) {
      cx += bl[i].x;
      cy += bl[i].y;
      cz += bl[i].z;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      cx += __shfl_xor_sync(0xffffffffu, cx, o);
      cy += __shfl_xor_sync(0xffffffffu, cy, o);
      cz += __shfl_xor_sync(0xffffffffu, cz, o);
    }
    const float inv = 1.f / (float)max(nb, 1);
    cx *= inv;
    cy *= inv;
    cz *= inv;
    float r = 0.f;
    for (int i = lane; i < nb; i += 32) {
      const float dx = bl[i].x - cx, dy = bl[i].y - cy, dz = bl[i].z - cz;
      r = fmaxf(r, sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) + bl[i].w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
    if (lane == 0) s_blk[w] = make_float4(cx, cy, cz, r);
  }
  __syncthreads();
  bool blocks_apart;
  {
    const float4 A = s_blk[0], B = s_blk[1];
    const float dx = A.x - B.x, dy = A.y - B.y, dz = A.z - B.z;
    // margin over the FP32 rounding of the block spheres (sums of ~64 centres: relative to the
    // coordinates' size) and of the per-pair test
    const float mag = fmaxf(fmaxf(fabsf(A.x), fabsf(A.y)), fmaxf(fabsf(A.z), fmaxf(fmaxf(fabsf(B.x), fabsf(B.y)), fabsf(B.z))));
    const float lim = 1.001f * (A.w + B.w) + 1e-5f * mag + 1e-30f;
    blocks_apart = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > lim * lim;  // false for NaN: scan
  }
  bool check = false;
  if (!blocks_apart) {  // the same in every thread
    for (int i = tid; i < tm; i += kThreads) {
      const int T = s.triT[i];
      for (int64_t e = p.sing_off[T], e1 = p.sing_off[T + 1]; e < e1; ++e) {
        const int sg = p.sing_sigma[e];
        int lo = 0, hi = nbk;  // triB is sorted ascending
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (s.triB[mid] < sg) lo = mid + 1;
          else hi = mid;
        }
        if (lo < nbk && s.triB[lo] == sg) {
          *s_nonfar = 1;
          break;
        }
      }
    }
    __syncthreads();
    check = *s_nonfar != 0;
  }
  // fixed roles of this thread: pairs (ti0 + k * tstep, si) of a chunk; gather row m, groups gq + k * gstep
  const int tstep = kThreads / SC, ti0 = tid / SC, si = tid - ti0 * SC;
  // gather rows in whole warps (one group stream per warp) when that keeps the groups in flight
  const int FM32 = (p.FM + 31) & ~31;
  const int FMb = kThreads / FM32 == kThreads / p.FM ? FM32 : p.FM;
  const int gstep = kThreads / FMb, gq = tid / FMb, m = tid - gq * FMb;
  const bool gather_on = m < fm && gq < gstep;
  // this row's test supports: two (RWG) in registers
  int cnt = 0, fcA = 0, fcB = 0;
  R fwA = 0, fwB = 0;
  if (gather_on) {
    cnt = s.fcnt[m];
    if (MAXS <= 2) {
      if (cnt > 0) {
        fcA = s.fcode[m * MAXS];
        fwA = s.fcoef[m * MAXS];
      }
      if (cnt > 1) {
        fcB = s.fcode[m * MAXS + 1];
        fwB = s.fcoef[m * MAXS + 1];
      }
    }
  }

  for (int c = 0; c < nch; ++c) {
    {
      const int sbase = c * SC;
      const int scn = min(SC, nbk - sbase);
      C* __restrict__ Lb = s.Lbuf;
      const R* __restrict__ recb = s.recB + (kChunkB ? (c & 1) * SC * RB : sbase * RB);  // this chunk's trial records
      if constexpr (kChunkB) {
        const int RB4 = RB / 4;
        const int nn = c + 1 < nch ? min(SC, nbk - sbase - SC) : 0;  // the next chunk's records
        for (int i = tid; i < nn * RB4; i += kThreads) {
          const int r = i / RB4, k = i - r * RB4;
          cp_async16(s.recB + ((((c + 1) & 1) * SC + r) * RB + 4 * k),
                     (const float4*)gRB + (int64_t)s.triB[sbase + SC + r] * RB4 + k);
        }
        cp_async_commit();
      }
      if (si < scn) {
        const int sb = sbase + si;
        for (int ti = ti0; ti < tm; ti += tstep) {
          C L[9];
          bool done = false;
          if (check && sphere_candidate(s.bndT[ti], s.bndB[sb])) {
            const int64_t e = find_sigma(p.sing_off, p.sing_sigma, s.triT[ti], s.triB[sb]);
            if (e >= 0) {
#pragma unroll
              for (int k = 0; k < 9; ++k) {
                const double2 v = p.sing_L[e * 9 + k];
                L[k] = P::mk(v.x, v.y);
              }
              done = true;
            }
          }
          if (!done) far_pair<P, OP, QT, QB>(S, K, s.recT + ti * RT, recb + si * RB, L);
          const int li = ti * SC + si;
#pragma unroll
          for (int k = 0; k < 9; ++k) Lb[k * LS + li] = L[k];
        }
      }
    }
    if constexpr (kChunkB) cp_async_wait_all();  // the next chunk's records, before the barrier
    __syncthreads();
    if (gather_on) {
      const C* __restrict__ Lb = s.Lbuf;
      const int gg1 = s.chGrp[c + 1];
      for (int g = s.chGrp[c] + gq; g < gg1; g += gstep) {
        const int2 G = s.grp[g];
        C* z = s.Zs + G.x + m;
        C acc = *z;
        const Support<R>* __restrict__ q = s.gs + (G.y >> 5);
        const Support<R>* __restrict__ q1 = q + (G.y & 31);
        for (; q != q1; ++q) {
          const Support<R> u = *q;
          if (MAXS <= 2) {
            if (cnt > 0) {
              const R w = fwA * u.w;
              const C l = Lb[fcA + u.col];
              acc.x = fma(w, l.x, acc.x);
              acc.y = fma(w, l.y, acc.y);
            }
            if (cnt > 1) {
              const R w = fwB * u.w;
              const C l = Lb[fcB + u.col];
              acc.x = fma(w, l.x, acc.x);
              acc.y = fma(w, l.y, acc.y);
            }
          } else {
            for (int a = 0; a < cnt; ++a) {
              const R w = s.fcoef[m * MAXS + a] * u.w;
              const C l = Lb[s.fcode[m * MAXS + a] + u.col];
              acc.x = fma(w, l.x, acc.x);
              acc.y = fma(w, l.y, acc.y);
            }
          }
        }
        *z = acc;
      }
    }
    __syncthreads();
  }
  // output columns by warps, rows by lanes
  for (int n = tid >> 5; n < fn; n += kThreads / 32) {
    const int64_t col = p.cols[g0 + n] * p.ld;
    for (int mm = tid & 31; mm < fm; mm += 32) {
      const C v = s.Zs[n * fm + mm];
      const int64_t idx = col + s.row[mm];
      if (p.out_c64) ((double2*)p.out)[idx] = make_double2(v.x, v.y);
      else ((float2*)p.out)[idx] = make_float2((float)v.x, (float)v.y);
    }
  }
}

// The far kernel: persistent CTAs pull tiles (problem, bm, bn) from a work queue (an atomic
// counter; no CTA ever waits on another): items[t], or without a list the tiles of plans[0] with
// the row block fastest.  A single assembly is a one-problem queue.  Each
// problem has its own constants (wave number, alpha, beta) and plan; the tile shape and rules
// are common to the launch.  The problem's constants and plan are copied to shared memory
// when a CTA's tile belongs to another problem than its previous one; each CTA claims its next
// tile when it starts a tile.
template <class P, int OP, int QT, int QB>
__global__ void __launch_bounds__(P::kThreads, P::kMinBlocks) k_far_persistent(const FarConst* __restrict__ Ks,
                                                             const TilePlan* __restrict__ plans,
                                                             const int4* __restrict__ items, int nitems,
                                                             int* __restrict__ counter,
                                                             const volatile int* abort_flag) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int next, nonfar;
  __shared__ FarConst sK;
  __shared__ TilePlan sP;
  if (threadIdx.x == 0) next = (abort_flag && *abort_flag) ? nitems : atomicAdd(counter, 1);
  __syncthreads();
  int cur = -1;  // the problem whose constants and plan are in shared memory (the same in all threads)
  for (;;) {
    const int t = next;
    if (t >= nitems) return;
    // an item list (batches), or tile t = bn * n_tblocks + bm of the single plan
    int4 it;
    if (items) {
      it = items[t];
    } else {
      const int ntb = plans[0].n_tblocks;
      it = make_int4(0, t % ntb, t / ntb, 0);
    }
    if (it.x != cur) {
      for (int i = threadIdx.x; i < (int)(sizeof(FarConst) / 4); i += P::kThreads)
        ((int*)&sK)[i] = ((const int*)&Ks[it.x])[i];
      for (int i = threadIdx.x; i < (int)(sizeof(TilePlan) / 4); i += P::kThreads)
        ((int*)&sP)[i] = ((const int*)&plans[it.x])[i];
      cur = it.x;
    }
    __syncthreads();
    // claim the next tile now: the atomic completes while this one is computed
    int claimed = 0;
    if (threadIdx.x == 0) claimed = (abort_flag && *abort_flag) ? nitems : atomicAdd(counter, 1);
    tile_body<P, OP, QT, QB>(sK, sP, it.y, it.z, smem, &nonfar);
    if (threadIdx.x == 0) next = claimed;
    __syncthreads();
  }
}

// ----------------------------------------------------------------------------------------
// Plain FP64: the local matrices of a panel, every pair once (the gather is in bgb_gather64.cu).
//
// One pair per thread, 16 test x 16 trial triangles per CTA, records in shared memory; the matrix of
// (row, column) goes to ws[(row * ncols + column) * 9].  Bound by the FP64 pipe: two CTAs per SM
// (at most 128 registers) keep it fed through the latencies of its 2-lanes-per-clock instructions.
// ----------------------------------------------------------------------------------------
constexpr int kPairSide = 16;
template <int OP, int QT, int QB>
__global__ void __launch_bounds__(kPairSide * kPairSide, 2) k_pair64(const FarConst* __restrict__ Kp,
                                                                     const double* __restrict__ rec_t,
                                                                     const double* __restrict__ rec_b,
                                                                     const int* __restrict__ rows, int nrows,
                                                                     const int* __restrict__ cols, int ncols,
                                                                     const int64_t* __restrict__ sing_off,
                                                                     const int* __restrict__ sing_sigma,
                                                                     double2* __restrict__ ws,
                                                                     const volatile int* abort_flag) {
  constexpr int RT = PFp64::rec<QT>(), RB = PFp64::rec<QB>();
  __shared__ FarConst K;
  __shared__ double sT[kPairSide * RT], sB[kPairSide * RB];
  __shared__ int stop, nclose;
  __shared__ unsigned char close[kPairSide * kPairSide];
  const int tid = threadIdx.x;
  const int r0 = blockIdx.y * kPairSide, c0 = blockIdx.x * kPairSide;
  const int nr = min(kPairSide, nrows - r0), nc = min(kPairSide, ncols - c0);
  for (int i = tid; i < (int)(sizeof(FarConst) / 4); i += kPairSide * kPairSide) ((int*)&K)[i] = ((const int*)Kp)[i];
  for (int i = tid; i < nr * RT; i += kPairSide * kPairSide) {
    const int r = i / RT;
    sT[i] = rec_t[(int64_t)rows[r0 + r] * RT + (i - r * RT)];
  }
  for (int i = tid; i < nc * RB; i += kPairSide * kPairSide) {
    const int r = i / RB;
    sB[i] = rec_b[(int64_t)cols[c0 + r] * RB + (i - r * RB)];
  }
  if (tid == 0) {
    stop = abort_flag && *abort_flag;
    nclose = 0;
  }
  __syncthreads();
  if (stop) return;
  const int ti = tid / kPairSide, si = tid - ti * kPairSide;
  auto out = [&](int t, int s) { return ws + ((int64_t)(r0 + t) * ncols + c0 + s) * 9; };
  bool on = ti < nr && si < nc;
  const double *a = sT + ti * RT, *b = sB + si * RB;
  if constexpr (QT == 3 && QB == 4) {
    // singular and near pairs, whose matrices are placed afterwards, and a few others: those are listed and computed
    // by full warps at the end (a second pass of every warp that holds one: ellipsoid of 320 long triangles, far
    // stage 156 -> 238 us)
    if (on && far_pair34_is_close(a, b)) {
      on = false;
      if (find_sigma(sing_off, sing_sigma, rows[r0 + ti], cols[c0 + si]) < 0) close[atomicAdd(&nclose, 1)] = (unsigned char)tid;
    }
  }
  if (on) {
    double2 L[9];
    if constexpr (QT == 3 && QB == 4) far_pair34_fp64<OP, false>(far_scalars(K), K.tay_s, K.tay_c, a, b, L);
    else far_pair<PFp64, OP, QT, QB>(far_scalars(K), K, a, b, L);
    double2* o = out(ti, si);
#pragma unroll
    for (int k = 0; k < 9; ++k) o[k] = L[k];
  }
  if constexpr (QT == 3 && QB == 4) {
    __syncthreads();
    if (tid < nclose) {  // at most one per thread
      const int t = close[tid] / kPairSide, s = close[tid] % kPairSide;
      far_pair34_fp64_close<OP>(K, sT + t * RT, sB + s * RB, out(t, s));
    }
  }
}

template <int OP, int QT, int QB>
int launch_pair64_t(const FarConst* K, const void* rt, const void* rb, const int* rows, int nrows, const int* cols,
                    int ncols, const int64_t* sing_off, const int* sing_sigma, double2* ws, const volatile int* abort_flag,
                    cudaStream_t st) {
  if (nrows <= 0 || ncols <= 0) return 0;
  // rows along y in runs of at most 65535 blocks (a grid's limit)
  const int step = 65535 * kPairSide;
  for (int r = 0; r < nrows; r += step) {
    const int n = std::min(step, nrows - r);
    const dim3 grid((ncols + kPairSide - 1) / kPairSide, (n + kPairSide - 1) / kPairSide);
    k_pair64<OP, QT, QB><<<grid, kPairSide * kPairSide, 0, st>>>(K, (const double*)rt, (const double*)rb, rows + r, n,
                                                                 cols, ncols, sing_off, sing_sigma,
                                                                 ws + (int64_t)r * ncols * 9, abort_flag);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "k_pair64 launch");
}

// ----------------------------------------------------------------------------------------
// Records
// ----------------------------------------------------------------------------------------
template <int Q>  // rules of at most Q points
__global__ void k_prepare_rec32(const Geo64* __restrict__ g, int nt, const __grid_constant__ RuleTable rules, int rule,
                                double wscale, float* __restrict__ out) {
  using O = Off32;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const Geo64& T = g[t];
  const int q = rules.npoints[rule], stride = off32_size(q);
  float* r = out + (int64_t)t * stride;
  double c[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) c[k] = (T.v[0][k] + T.v[1][k] + T.v[2][k]) / 3.0;
  for (int k = 0; k < stride; ++k) r[k] = 0.f;  // spare slots
  for (int k = 0; k < 3; ++k) {
    const float hi = (float)c[k];
    r[O::CH + k] = hi;
    r[O::CL + k] = (float)(c[k] - (double)hi);
  }
  r[O::INV2A] = (float)(1.0 / (2.0 * T.area));
  for (int I = 0; I < q + (q & 1); ++I) {
    // the pad of an odd rule is its last point with weight zero: another place (a vertex) may be a test point
    const double* p = rules.uvw[rules.offset[rule] + min(I, q - 1)];
    const double u = p[0], v = p[1], w = I < q ? p[2] : 0.0;
    for (int k = 0; k < 3; ++k) {
      const double x = (T.v[2][k] + T.t[0][k] * u) + T.t[1][k] * v;
      r[O::px(I) + 2 * k] = (float)(x - c[k]);
    }
    r[O::pw(I)] = (float)((w / 2.0) * (2.0 * T.area) * wscale);
  }
  for (int i = 0; i < 3; ++i)
    for (int k = 0; k < 3; ++k) r[O::VO + 3 * i + k] = (float)(T.v[i][k] - c[k]);
}

template <int Q>
__global__ void k_prepare_rec64(const Geo64* __restrict__ g, int nt, const __grid_constant__ RuleTable rules, int rule,
                                double wscale, double* __restrict__ out) {
  using O = Off64<Q>;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const Geo64& T = g[t];
  double* r = out + (int64_t)t * O::SIZE;
  double c[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) c[k] = (T.v[0][k] + T.v[1][k] + T.v[2][k]) / 3.0;
  for (int k = 0; k < 3; ++k) r[O::C + k] = c[k];
  const int q = rules.npoints[rule];
  for (int I = 0; I < Q; ++I) {
    double u = 0, v = 0, w = 0;
    if (I < q) {
      u = rules.uvw[rules.offset[rule] + I][0];
      v = rules.uvw[rules.offset[rule] + I][1];
      w = rules.uvw[rules.offset[rule] + I][2];
    }
    for (int k = 0; k < 3; ++k) {
      const double x = (T.v[2][k] + T.t[0][k] * u) + T.t[1][k] * v;
      r[O::X + 3 * I + k] = x - c[k];
    }
    r[O::W + I] = (w / 2.0) * (2.0 * T.area) * wscale;
  }
  for (int i = 0; i < 3; ++i)
    for (int k = 0; k < 3; ++k) r[O::VO + 3 * i + k] = T.v[i][k] - c[k];
  r[O::INV2A] = 1.0 / (2.0 * T.area);
}

// Diagnostic kernel: far rule of explicit pairs, one thread per pair, records from HBM.
template <class P, int OP, int QT, int QB>
__global__ void k_far_pairs_diag(const __grid_constant__ FarConst K, const typename P::R* __restrict__ rt,
                                 const typename P::R* __restrict__ rb, const int* __restrict__ tau,
                                 const int* __restrict__ sigma, int64_t n, double2* __restrict__ out) {
  const int RT = P::template rec<QT>(K.qt), RB = P::template rec<QB>(K.qb);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    typename P::C L[9];
    far_pair<P, OP, QT, QB>(far_scalars(K), K, rt + (int64_t)tau[e] * RT, rb + (int64_t)sigma[e] * RB, L);
#pragma unroll
    for (int k = 0; k < 9; ++k) out[e * 9 + k] = make_double2(L[k].x, L[k].y);
  }
}

// The dynamic shared-memory limit of a kernel is set to the device maximum less its static
// shared memory (not to one launch's size), so that concurrent callers never lower it under
// each other's launches.
template <class K>
inline int max_dynamic_smem(K kern) {
  int dev = 0, v = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return v;
  return v - (int)fa.sharedSizeBytes;
}

template <class P, int OP, int QT, int QB>
int launch_persistent_t(const FarConst* Ks, const TilePlan* plans, const int4* items, int nitems, int* counter,
                        size_t smem_bytes, int ctas, const volatile int* abort_flag, cudaStream_t st) {
  auto kern = k_far_persistent<P, OP, QT, QB>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dynamic_smem(kern));
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(far persistent)");
  if (nitems <= 0) return 0;
  kern<<<ctas, P::kThreads, smem_bytes, st>>>(Ks, plans, items, nitems, counter, abort_flag);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "k_far_persistent launch");
}

template <class P, int OP, int QT, int QB>
int occupancy_t(size_t smem_bytes, int* per_sm) {
  cudaError_t e = cudaFuncSetAttribute(k_far_persistent<P, OP, QT, QB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       max_dynamic_smem(k_far_persistent<P, OP, QT, QB>));
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(far persistent)");
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_far_persistent<P, OP, QT, QB>, P::kThreads,
                                                    smem_bytes);
  return e == cudaSuccess ? 0 : cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
}

template <class P, int OP, int QT, int QB>
size_t smem_t(const TilePlan& p, int qt, int qb) {
  return carve<P>(nullptr, p.tmax, p.nmax, P::template rec<QT>(qt), P::template rec<QB>(qb), p.FM, p.FN, p.MAXS, p.SC,
                  p.gmax, p.gsmax, chunk_trial_records<P, OP, QB>(), nullptr);
}

template <class P, int OP, int QT, int QB>
int launch_diag_t(const FarConst& K, const void* rt, const void* rb, const int* tau, const int* sigma, int64_t n,
                  double2* out, cudaStream_t st) {
  if (n <= 0) return 0;
  const int blocks = (int)std::min<int64_t>((n + 127) / 128, 65535);
  using R = typename P::R;
  k_far_pairs_diag<P, OP, QT, QB><<<blocks, 128, 0, st>>>(K, (const R*)rt, (const R*)rb, tau, sigma, n, out);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "k_far_pairs_diag launch");
}

// Instances live in bgb_far_{mixed,fp64}_op{0,1,2,3,4,5}.cu.
#define BGB_FAR_EXTERN(P, OP)                                                                                   \
  extern template int launch_diag_t<P, OP, 3, 4>(const FarConst&, const void*, const void*, const int*,        \
                                                 const int*, int64_t, double2*, cudaStream_t);                \
  extern template int launch_diag_t<P, OP, BGB_MAXQ, BGB_MAXQ>(const FarConst&, const void*, const void*,      \
                                                               const int*, const int*, int64_t, double2*,     \
                                                               cudaStream_t);                                 \
  extern template int launch_persistent_t<P, OP, 3, 4>(const FarConst*, const TilePlan*, const int4*, int, int*, \
                                                       size_t, int, const volatile int*, cudaStream_t);        \
  extern template int launch_persistent_t<P, OP, BGB_MAXQ, BGB_MAXQ>(const FarConst*, const TilePlan*,       \
                                                                     const int4*, int, int*, size_t, int,      \
                                                                     const volatile int*, cudaStream_t);       \
  extern template int occupancy_t<P, OP, 3, 4>(size_t, int*);                                                 \
  extern template int occupancy_t<P, OP, BGB_MAXQ, BGB_MAXQ>(size_t, int*);

#define BGB_PAIR64_EXTERN(OP)                                                                                       \
  extern template int launch_pair64_t<OP, 3, 4>(const FarConst*, const void*, const void*, const int*, int,        \
                                                const int*, int, const int64_t*, const int*, double2*,             \
                                                const volatile int*, cudaStream_t);                                \
  extern template int launch_pair64_t<OP, BGB_MAXQ, BGB_MAXQ>(const FarConst*, const void*, const void*, const int*, \
                                                              int, const int*, int, const int64_t*, const int*,      \
                                                              double2*, const volatile int*, cudaStream_t);

}  // namespace farimpl
}  // namespace bgb
