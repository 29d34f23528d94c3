// Far-pair local matrices of the default rule pair (3 test points x 4 trial points), both precisions.
//
// The points of these two symmetric rules are multiples of the vertex offsets from the centroid, so no
// point coordinate is stored or multiplied per point pair.  With V_i, W_j the vertex offsets (sum 0):
//   test points  x_I = c_t + V_I / 2            (weights A_t / 3)
//   trial points y_0 = c_s, y_q = c_s + 0.4 W_q (weights -0.5625 A_s, then 25/48 A_s)
// and with w_q = -0.4 W_q, D = c_t - c_s and the table d_Iq = V_I . w_q,
//   |x_I - y_q|^2 = E_I + H_q + d_Iq,  E_I = |D|^2 + V_I.D + |V_I|^2/4,  H_q = 2 w_q.D + |w_q|^2,
//   |x_I - y_0|^2 = E_I:
// two additions per point pair (none for the centroid point) instead of five or six operations.  The
// kernel values are used without weights: the ratio -27/25 of the two trial weights is a constant of
// the sums T_I = G_I1 + G_I2 + G_I3 - 1.08 G_I0, and all other factors (rule weights, areas against the
// 1/(2A) of the RWG shapes, 1/(4 pi)) go into one constant per launch.
//
// Local matrices from the 12 kernel values (C_q = sum_I G_Iq, TT = sum_I T_I):
//   hats   M_Ij = G_Ij + (G_I1 + G_I2 + G_I3)/2 - 0.9 G_I0,  L_ij ~ M_ij + (M_0j + M_1j + M_2j)/3
//   EFIE   sum G (x - V_i).(y - W_j) = -A/2 + F_i + 1.25 B_j - 2.5 TT d_ij
//          with A = sum G_Iq d_Iq, F_i = sum C_q d_iq, B_j = sum T_I d_Ij
//   MFIE   f.(d x g) = P.(g x f) with P = D + V_i - W_j for every point pair (d differs from P by
//          multiples of f and g), so the triple products reduce to t_Iq = w_q.(V_I x D), a_q = w_q.(V_0 x V_1)
//          and b_I = V_I.(w_0 x w_1) (V_0 x V_1 = V_1 x V_2 = V_2 x V_0).
// The EFIE takes 171 operations after the kernel values instead of 291 (8 moment updates per point
// pair and their expansion), the MFIE about 200 instead of 460.
#pragma once
#include "bgb_kernels.cuh"

namespace bgb {
namespace farimpl {

// FP32 record: five 16-byte groups [CH.xyz area] [CL.xyz 1/(2A)] [V_i.xyz |x_i|^2] x 3, V_i scaled by -0.4
// on the trial side (an odd number of groups: the records of different triangles start in different banks).
// FP64 record: centroid, the three offsets, |x_i|^2, area, 1/(2A), unit normal; an odd stride (the 8-byte reads of
// different triangles start in different banks).
constexpr int kRec34F = 20, kRec34D = 21;
// Factor of the trial records' areas: the hats' constants (rule weights, 1/(4 pi), 1/5), in FP64 before
// the FP32 records are rounded.
constexpr double kHatScale34 = 0.2 * 25.0 / 144.0 * BGB_INV_4PI_D;

__device__ __forceinline__ float fm(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float ml(float a, float b) { return a * b; }
__device__ __forceinline__ float ad(float a, float b) { return a + b; }
__device__ __forceinline__ float sb(float a, float b) { return a - b; }
// FP64: round-to-nearest intrinsics, never contracted or reassociated, so that every kernel that inlines
// this code gives the same bits.
__device__ __forceinline__ double fm(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double ml(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ad(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sb(double a, double b) { return __dsub_rn(a, b); }

__device__ __forceinline__ float2 mk2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 mk2(double a, double b) { return make_double2(a, b); }
// Complex FP32 sums in packed f32x2 instructions: one issue slot for the real and the imaginary part.
__device__ __forceinline__ unsigned long long pk(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 upk(unsigned long long a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ float2 cfm(float2 g, float s, float2 acc) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pk(g)), "l"(pk(make_float2(s, s))), "l"(pk(acc)));
  return upk(r);
}
__device__ __forceinline__ float2 csc(float2 g, float s) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(g)), "l"(pk(make_float2(s, s))));
  return upk(r);
}
__device__ __forceinline__ float2 cad(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
  return upk(r);
}
template <class T, class C>
__device__ __forceinline__ C cfm(C g, T s, C acc) { return mk2(fm(g.x, s, acc.x), fm(g.y, s, acc.y)); }
template <class T, class C>
__device__ __forceinline__ C csc(C g, T s) { return mk2(ml(g.x, s), ml(g.y, s)); }
template <class C>
__device__ __forceinline__ C cad(C a, C b) { return mk2(ad(a.x, b.x), ad(a.y, b.y)); }
template <class C>
__device__ __forceinline__ C csb(C a, C b) { return mk2(sb(a.x, b.x), sb(a.y, b.y)); }
// a * b
template <class C>
__device__ __forceinline__ C cml(C a, C b) {
  return mk2(fm(a.x, b.x, -ml(a.y, b.y)), fm(a.x, b.y, ml(a.y, b.x)));
}
// a * b + c
template <class C>
__device__ __forceinline__ C cma(C a, C b, C c) {
  return mk2(fm(a.x, b.x, fm(-a.y, b.y, c.x)), fm(a.x, b.y, fm(a.y, b.x, c.y)));
}
template <class T>
__device__ __forceinline__ T dot(const T a[3], const T b[3]) { return fm(a[0], b[0], fm(a[1], b[1], ml(a[2], b[2]))); }
// d_Iq = V_I . w_q from the first two of each: the offsets of a triangle sum to zero
__device__ __forceinline__ void dot_table(const float V[3][3], const float W[3][3], float d[3][3]) {
#pragma unroll
  for (int I = 0; I < 2; ++I) {
    d[I][0] = dot(V[I], W[0]);
    d[I][1] = dot(V[I], W[1]);
    d[I][2] = -ad(d[I][0], d[I][1]);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) d[2][q] = -ad(d[0][q], d[1][q]);
}
template <class T>
__device__ __forceinline__ void cross(const T a[3], const T b[3], T c[3]) {
  c[0] = fm(a[1], b[2], -ml(a[2], b[1]));
  c[1] = fm(a[2], b[0], -ml(a[0], b[2]));
  c[2] = fm(a[0], b[1], -ml(a[1], b[0]));
}

// Sums over the kernel values, one test point at a time.
template <int OP, class T, class C>
struct Sums34 {
  static constexpr bool kHat = OP != BGB_OP_MAXWELL3D_SL && OP != BGB_OP_MAXWELL3D_DL;
  static constexpr bool kMfie = OP == BGB_OP_MAXWELL3D_DL;
  C M[kHat ? 9 : 1];
  C T_[3], Cq[3], A, U[kMfie ? 3 : 1], Vq[kMfie ? 3 : 1];
  // g: values of test point I (centroid point first).  t: d_Iq (EFIE) or t_Iq (MFIE); e: the double
  // layer's factor (x_I - y).n; a, b: the MFIE's a_q and b_I.
  __device__ __forceinline__ void point(int I, const C g[4], const T t[3], T e, const T a[3], T b) {
    if (kHat) {
      const C s = cad(cad(g[1], g[2]), g[3]);
      const C base = cfm(g[0], (T)-0.9, csc(s, (T)0.5));
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        M[3 * I + j] = cad(g[j + 1], base);
        if (OP == BGB_OP_HELMHOLTZ3D_DL) M[3 * I + j] = csc(M[3 * I + j], e);
      }
    } else {
      T_[I] = cfm(g[0], (T)-1.08, cad(cad(g[1], g[2]), g[3]));
      if (I == 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) Cq[q] = g[q + 1];
        A = csc(g[1], t[0]);
      } else {
#pragma unroll
        for (int q = 0; q < 3; ++q) Cq[q] = cad(Cq[q], g[q + 1]);
        A = cfm(g[1], t[0], A);
      }
      A = cfm(g[3], t[2], cfm(g[2], t[1], A));
      if (kMfie) {
        U[I] = cfm(g[3], a[2], cfm(g[2], a[1], csc(g[1], a[0])));
#pragma unroll
        for (int q = 0; q < 3; ++q) Vq[q] = I == 0 ? csc(g[q + 1], b) : cfm(g[q + 1], b, Vq[q]);
      }
    }
  }
};

template <class T>
struct PairGeo34 {
  T V[3][3], W[3][3];  // vertex offsets (test), -0.4 x vertex offsets (trial)
  T t[3][3];           // d_Iq, or t_Iq (MFIE)
  T a[3], b[3];        // MFIE
};

// L_ij from the sums; sa: the factor of the alpha part, sbeta: of the beta part (EFIE: of TT; hypersingular:
// of int int G (curl . curl)), nn: n_t . n_s and inv2a the 1/(2A) of both sides (hypersingular).
template <int OP, class T, class C>
__device__ __forceinline__ void finish34(const Sums34<OP, T, C>& S, const PairGeo34<T>& G, C sa, C sbeta, T nn, T inv2at,
                                         T inv2as, C L[9]) {
  if (S.kHat) {
    C s3[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) s3[j] = cad(cad(S.M[j], S.M[3 + j]), S.M[6 + j]);
    if (OP == BGB_OP_HELMHOLTZ3D_HS) {
      const C an = csc(sa, nn);
      // curl_i = (V_{i+1} - V_{i+2}) / (2A), the trial side's offsets carry -0.4
      const C bP = csc(cml(sbeta, cad(cad(s3[0], s3[1]), s3[2])), ml(ml(inv2at, inv2as), (T)-2.5));
      T cA[3][3], cB[3][3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          cA[i][k] = sb(G.V[(i + 1) % 3][k], G.V[(i + 2) % 3][k]);
          cB[i][k] = sb(G.W[(i + 1) % 3][k], G.W[(i + 2) % 3][k]);
        }
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          L[3 * i + j] = cfm(bP, dot(cA[i], cB[j]), cml(an, cfm(s3[j], (T)(1.0 / 3.0), S.M[3 * i + j])));
      return;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) L[3 * i + j] = cml(sa, cfm(s3[j], (T)(1.0 / 3.0), S.M[3 * i + j]));
    return;
  }
  const C TT = cad(cad(S.T_[0], S.T_[1]), S.T_[2]);
  const C TT25 = csc(TT, (T)-2.5);
  C F[3], B[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    F[i] = cfm(S.Cq[2], G.t[i][2], cfm(S.Cq[1], G.t[i][1], cfm(S.Cq[0], G.t[i][0], csc(S.A, (T)-0.5))));
    B[i] = csc(cfm(S.T_[2], G.t[2][i], cfm(S.T_[1], G.t[1][i], csc(S.T_[0], G.t[0][i]))), (T)1.25);
  }
  if (OP == BGB_OP_MAXWELL3D_SL) {
    const C tb = cml(sbeta, TT);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) L[3 * i + j] = cma(sa, cfm(TT25, G.t[i][j], cad(F[i], B[j])), tb);
    return;
  }
  // MFIE
  C h[3], c[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int p = (i + 2) % 3, n = (i + 1) % 3;
    F[i] = cfm(csb(S.U[p], S.U[n]), (T)-0.5, F[i]);
    B[i] = cfm(csb(S.Vq[n], S.Vq[p]), (T)-1.25, B[i]);
    h[i] = csc(csb(S.T_[p], S.T_[n]), (T)1.25);
    c[i] = csc(csb(S.Cq[n], S.Cq[p]), (T)2.5);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      L[3 * i + j] = cml(sa, cfm(TT25, G.t[i][j], cfm(h[i], G.a[j], cfm(c[j], G.b[i], cad(F[i], B[j])))));
}

// The MFIE's tables: t_Iq = w_q.(V_I x D), a_q, b_I (all nine and three: from their zero sums, as in dot_table,
// the error against 64 bits grew from 2.4e-7 to 2.9e-7 on folded plates).
template <class T>
__device__ __forceinline__ void mfie_tables(PairGeo34<T>& G, const T D[3]) {
  T m[3], x[3];
  cross(G.V[0], G.V[1], m);
#pragma unroll
  for (int q = 0; q < 3; ++q) G.a[q] = dot(G.W[q], m);
  cross(G.W[0], G.W[1], m);
#pragma unroll
  for (int I = 0; I < 3; ++I) {
    G.b[I] = dot(G.V[I], m);
    cross(G.V[I], D, x);
#pragma unroll
    for (int q = 0; q < 3; ++q) G.t[I][q] = dot(G.W[q], x);
  }
}

// FP32: unit normal V_0 x V_1 * 3 / (2A) (the trial side's offsets carry -0.4: scale 18.75).  It takes the offsets' sum
// for zero, which holds to eps64 times the centroid's coordinates: below FP32, so the FP64 path has the normal in its
// record instead, from edges (10 to 15 times the error at 1000 edges from the origin otherwise).
__device__ __forceinline__ void normal34(const float V[3][3], float inv2a, float scale, float n[3]) {
  cross(V[0], V[1], n);
  const float s = ml(inv2a, scale);
#pragma unroll
  for (int k = 0; k < 3; ++k) n[k] = ml(n[k], s);
}

// An FP32 number near sqrt(x): 0 below the normal numbers (equal centroids: a triangle and the middle one of its
// refinement), where the flushed reciprocal root is infinite.
__device__ __forceinline__ float near_root(float x) { return x >= 1.17549435e-38f ? x * rsqrt_ftz(x) : 0.f; }

// ---- mixed: FP32 with the double-float phase base of far_pair_mixed -------------------------------
template <int OP>
__device__ __forceinline__ void far_pair34_mixed(const FarScalars& K, const float* __restrict__ a,
                                                 const float* __restrict__ b, float2 L[9]) {
  constexpr bool kDL = OP == BGB_OP_HELMHOLTZ3D_DL, kDLT = OP == BGB_OP_HELMHOLTZ3D_DLT, kHS = OP == BGB_OP_HELMHOLTZ3D_HS,
                 kMfie = OP == BGB_OP_MAXWELL3D_DL;
  const float4* __restrict__ a4 = reinterpret_cast<const float4*>(a);
  const float4* __restrict__ b4 = reinterpret_cast<const float4*>(b);
  PairGeo34<float> G;
  float D[3], E[3], H[3], c0, R0, phi0, area_t, area_s, i2t, i2s;
  {
    // D = Dh + Dl in double-float, R0 an FP32 number near |D|, c0 = |D|^2 - R0^2, phi0 = k R0 mod 2 pi
    const float4 a0 = a4[0], a1 = a4[1], b0 = b4[0], b1 = b4[1];
    area_t = a0.w;
    area_s = b0.w;
    i2t = a1.w;
    i2s = b1.w;
    float Dh[3], Dl[3];
    two_sum(a0.x, -b0.x, Dh[0], Dl[0]);
    two_sum(a0.y, -b0.y, Dh[1], Dl[1]);
    two_sum(a0.z, -b0.z, Dh[2], Dl[2]);
    Dl[0] = __fadd_rn(Dl[0], __fsub_rn(a1.x, b1.x));
    Dl[1] = __fadd_rn(Dl[1], __fsub_rn(a1.y, b1.y));
    Dl[2] = __fadd_rn(Dl[2], __fsub_rn(a1.z, b1.z));
    const float n2 = fmaf(Dh[0], Dh[0], fmaf(Dh[1], Dh[1], Dh[2] * Dh[2]));
    R0 = near_root(n2);
    float p0, e0, p1, e1, p2, e2, s1, f1, s2, f2, r2h, r2l;
    two_prod(Dh[0], Dh[0], p0, e0);
    two_prod(Dh[1], Dh[1], p1, e1);
    two_prod(Dh[2], Dh[2], p2, e2);
    two_sum(p0, p1, s1, f1);
    two_sum(s1, p2, s2, f2);
    const float lo = __fadd_rn(__fadd_rn(__fadd_rn(f1, f2), __fadd_rn(e0, e1)), e2);
    two_prod(R0, R0, r2h, r2l);
    c0 = __fadd_rn(__fsub_rn(s2, r2h), __fsub_rn(lo, r2l));
    // the low parts: 2 Dh.Dl + |Dl|^2
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      c0 = fmaf(Dl[k], fmaf(2.f, Dh[k], Dl[k]), c0);
      D[k] = __fadd_rn(Dh[k], Dl[k]);
    }
    float ph, pl;
    two_prod(K.k_hi, R0, ph, pl);
    pl = fmaf(K.k_lo, R0, pl);
    const float nq = rintf(ph * kInv2Pi);
    phi0 = fmaf(-nq, kPiA, ph);
    phi0 = fmaf(-nq, kPiB, phi0);
    phi0 = fmaf(-nq, kPiC, phi0);
    phi0 = __fadd_rn(phi0, pl);
  }
  const float D2[3] = {2.f * D[0], 2.f * D[1], 2.f * D[2]};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float4 v = a4[2 + i], w = b4[2 + i];
    G.V[i][0] = v.x; G.V[i][1] = v.y; G.V[i][2] = v.z;
    G.W[i][0] = w.x; G.W[i][1] = w.y; G.W[i][2] = w.z;
    E[i] = fmaf(v.x, D[0], fmaf(v.y, D[1], fmaf(v.z, D[2], v.w + c0)));
    H[i] = fmaf(w.x, D2[0], fmaf(w.y, D2[1], fmaf(w.z, D2[2], w.w)));
  }
  float d[3][3];
  dot_table(G.V, G.W, d);
  float eI[3] = {0.f, 0.f, 0.f}, eq[4] = {0.f, 0.f, 0.f, 0.f}, nn = 0.f;
  if (kDL || kDLT || kHS) {
    float nt[3] = {0.f, 0.f, 0.f}, ns[3] = {0.f, 0.f, 0.f};
    if (kDLT || kHS) normal34(G.V, i2t, 3.f, nt);
    if (kDL || kHS) normal34(G.W, i2s, 18.75f, ns);
    if (kDL) {  // (x_I - y).n_s, constant over the trial points
      const float e = dot(D, ns);
#pragma unroll
      for (int I = 0; I < 3; ++I) eI[I] = fmaf(0.5f, dot(G.V[I], ns), e);
    }
    if (kDLT) {  // -(x - y_q).n_t, constant over the test points
      eq[0] = -dot(D, nt);
#pragma unroll
      for (int q = 0; q < 3; ++q) eq[q + 1] = eq[0] - dot(G.W[q], nt);
    }
    if (kHS) nn = dot(nt, ns);
  }
  if (kMfie) {
    mfie_tables(G, D);
  } else {
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
      for (int q = 0; q < 3; ++q) G.t[I][q] = d[I][q];
  }
  const float R0sq = R0 * R0, kh = K.k_hi;
  const float amp0 = K.lossy ? exp_ftz(-K.gre * R0) : 1.f;
  Sums34<OP, float, float2> S;
#pragma unroll
  for (int I = 0; I < 3; ++I) {
    float2 g[4];
#pragma unroll
    for (int J = 0; J < 4; ++J) {
      const float q = J == 0 ? E[I] : (E[I] + H[J - 1]) + d[I][J - 1];  // R^2 - R0^2
      const float R2 = R0sq + q;
      const float rs = rsqrt_ftz(R2);
      const float delta = q * rcp_ftz(fmaf(R2, rs, R0));  // R - R0
      float psi = fmaf(kh, delta, phi0);
      if (!K.phase_direct) {  // |psi| may exceed 2 pi: reduce again
        const float m = rintf(psi * kInv2Pi);
        psi = fmaf(-m, kPiA, psi);
        psi = fmaf(-m, kPiB, psi);
      }
      float sn, cs;
      sincos_ftz(psi, &sn, &cs);
      float amp = rs;
      if (K.lossy) amp *= amp0 * exp_ftz(-K.gre * delta);
      if (kMfie || kDL || kDLT) {  // (gamma + 1/R) G / R (the MFIE's sign is in its constant)
        const float t = (K.gre + rs) * rs, u = kh * rs;
        g[J] = make_float2(amp * fmaf(t, cs, u * sn), amp * fmaf(u, cs, -t * sn));
        if (kDLT) g[J] = csc(g[J], eq[J]);
      } else {
        g[J] = make_float2(amp * cs, -amp * sn);
      }
    }
    S.point(I, g, G.t[I], eI[I], G.a, G.b[I]);
  }
  float2 sa = make_float2(K.far_a32[0], K.far_a32[1]), sbeta = make_float2(K.far_b32[0], K.far_b32[1]);
  if (S.kHat) {
    const float aa = area_t * area_s;
    sa = csc(sa, aa);
    sbeta = csc(sbeta, aa);
  }
  finish34<OP>(S, G, sa, sbeta, nn, i2t, i2s, L);
}

// ---- plain FP64 -----------------------------------------------------------------------------------
// The phase is k R = k R0 + k (R - R0) with R0 the centroid distance: exp(-i k R0) is a factor of the whole
// local matrix, and cos / sin of the small k (R - R0) come from tay_n terms of their series for all
// four trial points together (sincos of k R where the series would be long).
// CLOSE: the points' differences are squared; otherwise R^2 = E + H + d.
template <int OP, bool CLOSE>
__device__ __forceinline__ void far_pair34_fp64(const FarScalars& K, const double* __restrict__ tay_s,
                                                const double* __restrict__ tay_c, const double* __restrict__ a,
                                                const double* __restrict__ b, double2 L[9]) {
  constexpr bool kDL = OP == BGB_OP_HELMHOLTZ3D_DL, kDLT = OP == BGB_OP_HELMHOLTZ3D_DLT, kHS = OP == BGB_OP_HELMHOLTZ3D_HS,
                 kMfie = OP == BGB_OP_MAXWELL3D_DL;
  const double gre = K.gamma[0], gim = K.gamma[1];
  PairGeo34<double> G;
  double D[3], E[3], H[3], nD = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    D[k] = sb(a[k], b[k]);
    nD = fm(D[k], D[k], nD);
  }
  const double D2[3] = {ad(D[0], D[0]), ad(D[1], D[1]), ad(D[2], D[2])};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      G.V[i][k] = a[3 + 3 * i + k];
      G.W[i][k] = b[3 + 3 * i + k];
    }
    E[i] = fm(G.V[i][0], D[0], fm(G.V[i][1], D[1], fm(G.V[i][2], D[2], ad(a[12 + i], nD))));
    H[i] = fm(G.W[i][0], D2[0], fm(G.W[i][1], D2[1], fm(G.W[i][2], D2[2], b[12 + i])));
  }
  double d[3][3];  // nine independent dots: the shorter dot_table was no faster here (its chains)
#pragma unroll
  for (int I = 0; I < 3; ++I)
#pragma unroll
    for (int q = 0; q < 3; ++q) d[I][q] = dot(G.V[I], G.W[q]);
  double eI[3] = {0, 0, 0}, eq[4] = {0, 0, 0, 0}, nn = 0.0;
  if (kDL || kDLT || kHS) {
    const double nt[3] = {a[17], a[18], a[19]}, ns[3] = {b[17], b[18], b[19]};
    if (kDL) {
      const double e = dot(D, ns);
#pragma unroll
      for (int I = 0; I < 3; ++I) eI[I] = fm(0.5, dot(G.V[I], ns), e);
    }
    if (kDLT) {
      eq[0] = -dot(D, nt);
#pragma unroll
      for (int q = 0; q < 3; ++q) eq[q + 1] = sb(eq[0], dot(G.W[q], nt));
    }
    if (kHS) nn = dot(nt, ns);
  }
  if (kMfie) {
    mfie_tables(G, D);
  } else {
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
      for (int q = 0; q < 3; ++q) G.t[I][q] = d[I][q];
  }
  const int tn = gim != 0.0 ? K.tay_n : 0;
  double th0 = 0.0;
  double2 rot = make_double2(1.0, 0.0);
  if (tn > 0) {
    // 0 for equal centroids (a triangle and the middle one of its refinement); an integer compare
    if (__double2hiint(nD) >= 0x00100000) th0 = ml(gim, ml(nD, rsqrt_newton(nD)));
    double s0, c0;
    sincos(th0, &s0, &c0);
    rot = make_double2(c0, -s0);
  }
  Sums34<OP, double, double2> S;
#pragma unroll
  for (int I = 0; I < 3; ++I) {
    double rinv[4], R[4], sn[4], cs[4];
    double2 g[4];
#pragma unroll
    for (int J = 0; J < 4; ++J) {
      double R2;
      if (CLOSE) {
        double x[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          x[k] = fm(0.5, G.V[I][k], D[k]);
          if (J > 0) x[k] = ad(x[k], G.W[J - 1][k]);
        }
        R2 = dot(x, x);
      } else {
        R2 = J == 0 ? E[I] : ad(ad(E[I], H[J - 1]), d[I][J - 1]);
      }
      rinv[J] = rsqrt_newton(R2);
      R[J] = ml(R2, rinv[J]);
    }
    if (tn > 0) {
      double x[4], x2[4];
#pragma unroll
      for (int J = 0; J < 4; ++J) {
        x[J] = fm(gim, R[J], -th0);
        x2[J] = ml(x[J], x[J]);
        sn[J] = tay_s[tn - 1];
        cs[J] = tay_c[tn - 1];
      }
      for (int j = tn - 2; j >= 0; --j) {
        const double ts = tay_s[j], tc = tay_c[j];
#pragma unroll
        for (int J = 0; J < 4; ++J) {
          sn[J] = fm(sn[J], x2[J], ts);
          cs[J] = fm(cs[J], x2[J], tc);
        }
      }
#pragma unroll
      for (int J = 0; J < 4; ++J) sn[J] = ml(sn[J], x[J]);
    } else {
#pragma unroll
      for (int J = 0; J < 4; ++J) {
        sn[J] = 0.0;
        cs[J] = 1.0;
        if (gim != 0.0) sincos(ml(gim, R[J]), &sn[J], &cs[J]);
      }
    }
#pragma unroll
    for (int J = 0; J < 4; ++J) {
      double amp = rinv[J];
      if (gre != 0.0) amp = ml(amp, exp(-ml(gre, R[J])));
      g[J] = make_double2(ml(amp, cs[J]), -ml(amp, sn[J]));
      if (kMfie || kDL || kDLT) {  // (gamma + 1/R) G / R
        const double t = ml(ad(gre, rinv[J]), rinv[J]), u = ml(gim, rinv[J]);
        g[J] = make_double2(fm(t, g[J].x, -ml(u, g[J].y)), fm(t, g[J].y, ml(u, g[J].x)));
        if (kDLT) g[J] = csc(g[J], eq[J]);
      }
    }
    S.point(I, g, G.t[I], eI[I], G.a, G.b[I]);
  }
  double2 sa = cml(make_double2(K.far_a[0], K.far_a[1]), rot), sbeta = cml(make_double2(K.far_b[0], K.far_b[1]), rot);
  if (S.kHat) {
    const double aa = ml(a[15], b[15]);
    sa = csc(sa, aa);
    sbeta = csc(sbeta, aa);
  }
  finish34<OP>(S, G, sa, sbeta, nn, a[16], b[16], L);
}

// ---- records --------------------------------------------------------------------------------------
// scale: factor of the vertex offsets (1 test, -0.4 trial); x2: |x_i|^2 = x2 |V_i|^2 (1/4, 0.16); warea: factor
// of the area.
template <class T>
__global__ void k_prepare_rec34(const Geo64* __restrict__ g, int nt, double scale, double x2, double warea,
                                T* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const Geo64& S = g[t];
  double c[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) c[k] = (S.v[0][k] + S.v[1][k] + S.v[2][k]) / 3.0;
  const double inv2a = 1.0 / (2.0 * S.area);
  constexpr bool f32 = sizeof(T) == 4;
  T* r = out + (int64_t)t * (f32 ? kRec34F : kRec34D);
  for (int k = 0; k < 3; ++k) {
    r[k] = (T)c[k];
    if (f32) r[4 + k] = (T)(c[k] - (double)(T)c[k]);
  }
  r[f32 ? 3 : 15] = (T)(warea * S.area);
  r[f32 ? 7 : 16] = (T)inv2a;
  for (int i = 0; i < 3; ++i) {
    double s = 0.0;
    for (int k = 0; k < 3; ++k) {
      const double v = S.v[i][k] - c[k];
      s += v * v;
      r[(f32 ? 8 + 4 * i : 3 + 3 * i) + k] = (T)(scale * v);
    }
    r[f32 ? 11 + 4 * i : 12 + i] = (T)(x2 * s);
  }
  if (!f32) {
    double n[3];
    cross(S.t[0], S.t[1], n);
    for (int k = 0; k < 3; ++k) r[17 + k] = (T)(n[k] * inv2a);
    r[20] = (T)0;
  }
}

}  // namespace farimpl
}  // namespace bgb
