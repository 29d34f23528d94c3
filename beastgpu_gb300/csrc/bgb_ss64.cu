// Sauter-Schwab integrals of singular pairs in FP64 (plain path, and the operators the double-float kernel
// does not cover).
//
// In every region of the rules (SauterSchwab.jl:265-297) both chart points move on rays from the
// shared vertex P0: x = P0 + xi X, y = P0 + xi Y with X, Y depending on (eta1, eta2, eta3) only, so
// R = xi |X - Y|.  The sum over xi is therefore done in closed form per (eta, region) point: with
// theta = k |X - Y|,
//   T_m = sum_l w_l xi_l^(2+m) exp(-i theta xi_l) = sum_n (-i theta)^n / n! S_(m+n),
//   S_p = sum_l w_l xi_l^(2+p),
// and a moment of degree m in (x - P0, y - P0) takes one T_m.  One reciprocal square root and three
// short series serve the n_xi points of a ray: ~27 FP64 operations per Sauter-Schwab point at n = 4
// instead of ~95 (a sincos at each).  The points (X, Y in terms of the triangles' edges, weights) are
// tables built on the host, and about the common origin P0 the Maxwell double layer's moments reduce to
// X x Y and X - Y.
//
// Bound by the FP64 pipe.  One warp per pair; the per-lane sums are reduced through shared memory
// (16 additions per lane instead of five butterfly steps per moment) and nine lanes each form one
// entry.  theta up to 3 takes the series (its terms stay below 5); beyond, and for lossy wave numbers,
// the sum over xi is taken point by point.  Pairs whose coincident vertices are not bit-equal (flagged by
// the classifier) have no common origin and stay with k_singular.
#include "bgb_kernels.cuh"
#include "bgb_ss.cuh"

#include <cmath>
#include <vector>

namespace bgb {
namespace {

constexpr int kWarps = 8;

__host__ __device__ constexpr bool ss_hat_op(int op) {
  return op == BGB_OP_HELMHOLTZ3D_SL || op == BGB_OP_HELMHOLTZ3D_DL || op == BGB_OP_HELMHOLTZ3D_DLT ||
         op == BGB_OP_HELMHOLTZ3D_HS;
}
__host__ __device__ constexpr bool ss_double_layer(int op) {
  return op == BGB_OP_MAXWELL3D_DL || op == BGB_OP_HELMHOLTZ3D_DL || op == BGB_OP_HELMHOLTZ3D_DLT;
}
// Moments (complex): hats 9 (p_a q_b, p = (1, alpha xi, beta xi)); EFIE S, Px, Py, P0; MFIE sum H X x Y, sum H (X - Y).
template <int OP>
struct SsMoments {
  static constexpr int N = OP == BGB_OP_MAXWELL3D_SL ? 8 : (OP == BGB_OP_MAXWELL3D_DL ? 6 : 9);
  static constexpr int M0 = ss_double_layer(OP) ? -1 : 0;               // lowest T_m used
  static constexpr int NT = OP == BGB_OP_HELMHOLTZ3D_DL || OP == BGB_OP_HELMHOLTZ3D_DLT ? 4 : 3;
};

__device__ __forceinline__ void sub3(const double* a, const double* b, double c[3]) {
  c[0] = a[0] - b[0];
  c[1] = a[1] - b[1];
  c[2] = a[2] - b[2];
}
__device__ __forceinline__ double dot3(const double a[3], const double b[3]) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
__device__ __forceinline__ void tri_unit_normal(const Geo64& T, double n[3]) {
  const double inv = 1.0 / (2.0 * T.area);
  n[0] = (T.t[0][1] * T.t[1][2] - T.t[0][2] * T.t[1][1]) * inv;
  n[1] = (T.t[0][2] * T.t[1][0] - T.t[0][0] * T.t[1][2]) * inv;
  n[2] = (T.t[0][0] * T.t[1][1] - T.t[0][1] * T.t[1][0]) * inv;
}

// Entry (i, j) of the local matrix from the reduced moments v[2 q], v[2 q + 1].
template <int OP>
__device__ double2 ss_entry(const OpParams& op, const Geo64& A, const Geo64& B, const int I[3], const int J[3],
                            const double* v, int i, int j) {
  const double2 alpha = make_double2(op.alpha[0], op.alpha[1]);
  auto m = [&](int q) { return make_double2(v[2 * q], v[2 * q + 1]); };
  const double i4p = BGB_INV_4PI_D;
  if (ss_hat_op(OP)) {
    // hats of the reordered vertices: 1 - p1, p2, p1 - p2
    const double H[3][3] = {{1, -1, 0}, {0, 0, 1}, {0, 1, -1}};
    const int r = I[0] == i + 1 ? 0 : (I[1] == i + 1 ? 1 : 2), c = J[0] == j + 1 ? 0 : (J[1] == j + 1 ? 1 : 2);
    double2 s = make_double2(0, 0);
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b) {
        const double t = H[r][a] * H[c][b];
        if (t != 0.0) s = cadd(s, cscale(m(a * 3 + b), t));
      }
    const double w = 4.0 * A.area * B.area * i4p;
    if (OP != BGB_OP_HELMHOLTZ3D_HS) return cmul(cscale(alpha, w), s);
    double nA[3], nB[3];
    tri_unit_normal(A, nA);
    tri_unit_normal(B, nB);
    double cA[3], cB[3];  // (v_{i+1} - v_{i+2}); the 1/(2A) of both sides cancel the 4 A A' of w
    sub3(A.v[(i + 1) % 3], A.v[(i + 2) % 3], cA);
    sub3(B.v[(j + 1) % 3], B.v[(j + 2) % 3], cB);
    return cadd(cmul(cscale(alpha, w * dot3(nA, nB)), s), cmul(make_double2(op.beta[0], op.beta[1]), cscale(m(0), i4p * dot3(cA, cB))));
  }
  double V[3], W[3];
  sub3(A.v[i], A.v[I[0] - 1], V);
  sub3(B.v[j], B.v[J[0] - 1], W);
  if (OP == BGB_OP_MAXWELL3D_SL) {
    // (1/(4 A A') of the shapes cancels the Jacobians; the divergences leave 4)
    double2 t = m(0);
    for (int c = 0; c < 3; ++c) {
      t.x -= V[c] * v[2 * (4 + c)] + W[c] * v[2 * (1 + c)];
      t.y -= V[c] * v[2 * (4 + c) + 1] + W[c] * v[2 * (1 + c) + 1];
    }
    t = cadd(t, cscale(m(7), dot3(V, W)));
    return cadd(cmul(cscale(alpha, i4p), t), cmul(make_double2(op.beta[0] * (4.0 * i4p), op.beta[1] * (4.0 * i4p)), m(7)));
  }
  // MFIE: A1 - W.C - V.B + V.(E x W) with A1 = 0, B = sum H X x Y, C = -B, E = sum H (X - Y)
  double2 t = make_double2(0, 0);
  for (int c = 0; c < 3; ++c) t = cadd(t, cscale(m(c), W[c] - V[c]));
  const double x[3] = {W[1] * V[2] - W[2] * V[1], W[2] * V[0] - W[0] * V[2], W[0] * V[1] - W[1] * V[0]};  // W x V
  for (int c = 0; c < 3; ++c) t = cadd(t, cscale(m(3 + c), x[c]));  // V.(E x W) = E.(W x V)
  return cmul(cscale(alpha, -i4p), t);
}

template <int OP>
__global__ void __launch_bounds__(32 * kWarps, 2) k_ss64(OpParams op1, const OpParams* __restrict__ ops,
                                                         const int* __restrict__ tri_problem,
                                                         const __grid_constant__ SsTab64 M, const double* __restrict__ pts,
                                                         const Geo64* __restrict__ tg, const Geo64* __restrict__ bg,
                                                         const int* __restrict__ ent_tau, const int* __restrict__ ent_sigma,
                                                         const int8_t* __restrict__ ent_cls,
                                                         const int16_t* __restrict__ ent_mask, int64_t n,
                                                         double2* __restrict__ out, const volatile int* abort_flag,
                                                         const int* __restrict__ perm, const int64_t* __restrict__ range) {
  constexpr int NA = SsMoments<OP>::N, NV = 2 * NA, M0 = SsMoments<OP>::M0, NT = SsMoments<OP>::NT;
  __shared__ double part[kWarps][NV][33];
  __shared__ double red[kWarps][NV];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  // perm: the entries perm[range[0] .. range[1]) (one output block's group); otherwise 0 .. n
  const int64_t i0 = perm ? range[0] : 0, i1 = perm ? range[1] : n;
  for (int64_t it = i0 + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); it < i1; it += warps) {
    if (abort_flag && *abort_flag) return;
    const int64_t e = perm ? (int64_t)perm[it] : it;
    const int cls = ent_cls[e], mask = ent_mask[e];
    if (cls == BGB_CLASS_NEAR || (mask & BGB_MASK_INEXACT)) continue;  // k_singular
    if (ss_double_layer(OP) && cls == BGB_CLASS_CF) {  // vanishes on a flat face
      if (lane < 9) out[e * 9 + lane] = make_double2(0.0, 0.0);
      continue;
    }
    const int tau = ent_tau[e];
    const Geo64 &A = tg[tau], &B = bg[ent_sigma[e]];
    const OpParams& op = ops ? ops[tri_problem[tau]] : op1;  // one instance for both: the same bits
    const double gre = op.gamma[0], gim = op.gamma[1];
    int I[3], J[3];
    ss_permutation_mask(cls, mask, I, J);
    for (int k = 0; k < 3; ++k) {  // guard against an inconsistent mask
      I[k] = I[k] < 1 ? 1 : (I[k] > 3 ? 3 : I[k]);
      J[k] = J[k] < 1 ? 1 : (J[k] > 3 ? 3 : J[k]);
    }
    double a1[3], a2[3], b1[3], b2[3], nrm[3] = {0, 0, 0};
    sub3(A.v[I[2] - 1], A.v[I[0] - 1], a1);
    sub3(A.v[I[1] - 1], A.v[I[2] - 1], a2);
    sub3(B.v[J[2] - 1], B.v[J[0] - 1], b1);
    sub3(B.v[J[1] - 1], B.v[J[2] - 1], b2);
    if (OP == BGB_OP_HELMHOLTZ3D_DL) tri_unit_normal(B, nrm);
    if (OP == BGB_OP_HELMHOLTZ3D_DLT) tri_unit_normal(A, nrm);
    // terms of the series: theta <= k times the largest distance of two vertices, truncation below 2^-56
    int nj = 0;
    if (gre == 0.0) {
      float dv[9] = {};  // squared distances between the ends of X and of Y
      for (int c = 0; c < 3; ++c) {
        const float u[3] = {0.f, (float)a1[c], (float)(a1[c] + a2[c])}, v[3] = {0.f, (float)b1[c], (float)(b1[c] + b2[c])};
#pragma unroll
        for (int q = 0; q < 9; ++q) dv[q] = fmaf(u[q / 3] - v[q % 3], u[q / 3] - v[q % 3], dv[q]);
      }
      float d2 = dv[0];
#pragma unroll
      for (int q = 1; q < 9; ++q) d2 = fmaxf(d2, dv[q]);
      const float th = 1.0001f * fabsf((float)gim) * sqrtf(d2);
      if (th <= 3.f) {
        float t = 1.f;
        do {
          ++nj;
          t *= th * th / (float)((2 * nj - 1) * (2 * nj));
        } while (t > 1.3e-17f && nj < BGB_SS_SERIES);
      }
    }
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = 0.0;
    const int cnt = M.cnt[cls];
    const double* __restrict__ tab = pts + M.off[cls];
    for (int idx = lane; idx < cnt; idx += 32) {
      const double al = tab[idx], be = tab[cnt + idx], ga = tab[2 * cnt + idx], de = tab[3 * cnt + idx];
      const double om = tab[4 * cnt + idx];
      double X[3], Y[3], d[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        X[c] = fma(al, a1[c], be * a2[c]);
        Y[c] = fma(ga, b1[c], de * b2[c]);
        d[c] = X[c] - Y[c];
      }
      const double r2 = fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2]));
      const double rinv = rsqrt_newton(r2);
      const double R = r2 * rinv;
      double C[NT], S[NT];  // T_m = C - i S, m = M0 ..
      if (nj > 0) {
        const double th = gim * R, th2 = th * th;
        const double(*__restrict__ ser)[2 * BGB_SS_SERIES] = M.ser[cls];
#pragma unroll
        for (int q = 0; q < NT; ++q) {
          C[q] = ser[q + 1 + M0][2 * nj - 2];
          S[q] = ser[q + 1 + M0][2 * nj - 1];
        }
        for (int k = 2 * nj - 4; k >= 0; k -= 2) {
#pragma unroll
          for (int q = 0; q < NT; ++q) {
            C[q] = fma(C[q], th2, ser[q + 1 + M0][k]);
            S[q] = fma(S[q], th2, ser[q + 1 + M0][k + 1]);
          }
        }
#pragma unroll
        for (int q = 0; q < NT; ++q) S[q] *= th;
      } else {
#pragma unroll
        for (int q = 0; q < NT; ++q) C[q] = S[q] = 0.0;
        for (int l = 0; l < M.n[cls]; ++l) {
          const double xi = M.gx[cls][l];
          double sn = 0.0, cs = 1.0, w = M.gw[cls][l] * xi;
          if (gim != 0.0) sincos(gim * (R * xi), &sn, &cs);
          if (gre != 0.0) w *= exp(-gre * (R * xi));
          if (M0 == 0) w *= xi;
#pragma unroll
          for (int q = 0; q < NT; ++q) {
            C[q] = fma(w, cs, C[q]);
            S[q] = fma(w, sn, S[q]);
            w *= xi;
          }
        }
      }
      const double g = om * rinv;
      if (OP == BGB_OP_MAXWELL3D_DL) {
        // (gamma + 1/(xi R)) T: degree 2 (X x Y): gamma T_1 + T_0 / R; degree 1 (X - Y): gamma T_0 + T_-1 / R
        const double f = g * rinv;
        const double hr2 = f * fma(gre, C[2], fma(gim, S[2], rinv * C[1])), hi2 = f * fma(gim, C[2], -fma(gre, S[2], rinv * S[1]));
        const double hr1 = f * fma(gre, C[1], fma(gim, S[1], rinv * C[0])), hi1 = f * fma(gim, C[1], -fma(gre, S[1], rinv * S[0]));
        const double x[3] = {fma(X[1], Y[2], -X[2] * Y[1]), fma(X[2], Y[0], -X[0] * Y[2]), fma(X[0], Y[1], -X[1] * Y[0])};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          acc[2 * c] = fma(hr2, x[c], acc[2 * c]);
          acc[2 * c + 1] = fma(hi2, x[c], acc[2 * c + 1]);
          acc[6 + 2 * c] = fma(hr1, d[c], acc[6 + 2 * c]);
          acc[6 + 2 * c + 1] = fma(hi1, d[c], acc[6 + 2 * c + 1]);
        }
      } else if (OP == BGB_OP_MAXWELL3D_SL) {
        const double t0r = g * C[0], t0i = -g * S[0], t1r = g * C[1], t1i = -g * S[1];
        const double xy = g * fma(X[0], Y[0], fma(X[1], Y[1], X[2] * Y[2]));
        acc[0] = fma(C[2], xy, acc[0]);
        acc[1] = fma(-S[2], xy, acc[1]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          acc[2 + 2 * c] = fma(t1r, X[c], acc[2 + 2 * c]);
          acc[3 + 2 * c] = fma(t1i, X[c], acc[3 + 2 * c]);
          acc[8 + 2 * c] = fma(t1r, Y[c], acc[8 + 2 * c]);
          acc[9 + 2 * c] = fma(t1i, Y[c], acc[9 + 2 * c]);
        }
        acc[14] += t0r;
        acc[15] += t0i;
      } else {
        double tr[3], ti[3];  // kernel sums of degree 0, 1, 2
        if (ss_double_layer(OP)) {
          // +-(x - y).n (gamma + 1/R) G / R: degree m: rn / R^2 (gamma T_m + T_(m-1) / R)
          double rn = fma(d[0], nrm[0], fma(d[1], nrm[1], d[2] * nrm[2]));
          if (OP == BGB_OP_HELMHOLTZ3D_DLT) rn = -rn;
          const double f = g * rinv * rn;
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            tr[q] = f * fma(gre, C[q + 1], fma(gim, S[q + 1], rinv * C[q]));
            ti[q] = f * fma(gim, C[q + 1], -fma(gre, S[q + 1], rinv * S[q]));
          }
        } else {
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            tr[q] = g * C[q];
            ti[q] = -g * S[q];
          }
        }
        const double p[3] = {1.0, al, be}, q[3] = {1.0, ga, de};
        acc[0] += tr[0];
        acc[1] += ti[0];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int b = 0; b < 3; ++b) {
            if (a + b == 0) continue;
            const int deg = (a > 0) + (b > 0);
            const double pq = a == 0 ? q[b] : (b == 0 ? p[a] : p[a] * q[b]);
            acc[2 * (3 * a + b)] = fma(tr[deg], pq, acc[2 * (3 * a + b)]);
            acc[2 * (3 * a + b) + 1] = fma(ti[deg], pq, acc[2 * (3 * a + b) + 1]);
          }
      }
    }
    // reduction: lane v (and v + 16 when two lanes per value fit) sums row v
#pragma unroll
    for (int k = 0; k < NV; ++k) part[wid][k][lane] = acc[k];
    __syncwarp();
    if (NV <= 16) {
      const int v = lane & 15, h = (lane >> 4) * 16;
      double s = 0.0;
      if (v < NV)
#pragma unroll
        for (int k = 0; k < 16; ++k) s += part[wid][v][h + k];
      s += __shfl_xor_sync(0xffffffffu, s, 16);
      if (lane < NV) red[wid][lane] = s;
    } else if (lane < NV) {
      double s = 0.0, t = 0.0;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        s += part[wid][lane][k];
        t += part[wid][lane][16 + k];
      }
      red[wid][lane] = s + t;
    }
    __syncwarp();
    if (lane < 9) out[e * 9 + lane] = ss_entry<OP>(op, A, B, I, J, red[wid], lane / 3, lane % 3);
    __syncwarp();
  }
}

}  // namespace

// Ray coordinates of the region maps (ss_region): u1 = 1 - xi alpha, u2 = xi beta (test), the same with
// gamma, delta (trial), weight xi^3 omega; q = (alpha, beta, gamma, delta, omega), without the cancellation of
// 1 - u1.
using real = long double;  // the tables' roundings are common to every pair: one each
static void ss_ray(int cls, int r, real h1, real h2, real h3, real q[5]) {
  const real h12 = h1 * h2, h23 = h2 * h3, h123 = h12 * h3;
  real a[2], b[2], w = h1 * h1 * h2;
  bool swap = false;
  auto set = [](real* p, real x, real y) {
    p[0] = x;
    p[1] = y;
  };
  if (cls == BGB_CLASS_CV) {
    w = h2;
    set(a, 1.0, h1);
    set(b, h2, h23);
    swap = r == 1;
  } else if (cls == BGB_CLASS_CE) {
    switch (r) {
      case 0:
      case 2: set(a, 1.0, h1); set(b, 1.0 - h123, h12 * (1.0 - h3)); swap = r == 2; break;
      case 1: set(a, 1.0 - h12, h1 * (1.0 - h2)); set(b, 1.0, h123); break;
      case 3: set(a, 1.0 - h123, h1 * (1.0 - h23)); set(b, 1.0, h12); break;
      default: w = h1 * h1; set(a, 1.0, h1 * h3); set(b, 1.0 - h12, h1 * (1.0 - h2));
    }
  } else {
    swap = (r & 1) != 0;
    switch (r >> 1) {
      case 0: set(a, 1.0, (1.0 - h1) + h12); set(b, 1.0 - h123, 1.0 - h1); break;
      case 1: set(a, 1.0, h1 * ((1.0 - h2) + h23)); set(b, 1.0 - h12, h1 * (1.0 - h2)); break;
      default: set(a, 1.0 - h123, h1 * (1.0 - h23)); set(b, 1.0, h1 * (1.0 - h2));
    }
  }
  const real *t = swap ? b : a, *s = swap ? a : b;
  q[0] = t[0];
  q[1] = t[1];
  q[2] = s[0];
  q[3] = s[1];
  q[4] = w;
}

void build_ss_tables(const QuadSel& qs, std::vector<double>& pts, SsTab64& M) {
  pts.clear();
  M = SsTab64{};
  for (int cls = 1; cls <= 3; ++cls) {
    const int n = qs.ss[cls];
    const int nreg = cls == BGB_CLASS_CV ? 2 : (cls == BGB_CLASS_CE ? 5 : 6);
    const double *gx = qs.gl_x[cls], *gw = qs.gl_w[cls];
    const int cnt = n * n * n * nreg;
    M.off[cls] = (int)pts.size();
    M.cnt[cls] = cnt;
    M.n[cls] = n;
    pts.resize(pts.size() + 5 * (size_t)cnt);
    double* p = pts.data() + M.off[cls];
    int at = 0;
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j)
        for (int k = 0; k < n; ++k)
          for (int r = 0; r < nreg; ++r, ++at) {
            real q[5];
            ss_ray(cls, r, gx[i], gx[j], gx[k], q);
            for (int f = 0; f < 4; ++f) p[f * cnt + at] = (double)q[f];
            p[4 * cnt + at] = (double)((real)gw[i] * gw[j] * gw[k] * q[4]);
          }
    real pw[BGB_MAX_SS];  // w_l xi_l^(1 + p)
    for (int l = 0; l < n; ++l) {
      M.gx[cls][l] = gx[l];
      M.gw[cls][l] = gw[l];
      pw[l] = (real)gw[l] * gx[l];
    }
    real S[2 * BGB_SS_SERIES + 4];  // S_(p - 1)
    for (real& s : S) {
      s = 0.0;
      for (int l = 0; l < n; ++l) {
        s += pw[l];
        pw[l] *= gx[l];
      }
    }
    real f = 1.0;  // n!
    for (int k = 0; k < 2 * BGB_SS_SERIES; ++k) {
      if (k > 1) f *= k;
      for (int m = 0; m < 4; ++m) M.ser[cls][m][k] = (double)(((k >> 1) & 1 ? -1 : 1) * S[m + k] / f);
    }
  }
}

void launch_ss64(int op_kind, const OpParams& op, const OpParams* ops, const int* tri_problem, const SsTab64& M,
                 const double* pts, const Geo64* tg, const Geo64* bg, const int* et, const int* es, const int8_t* ec,
                 const int16_t* emask, int64_t n, double2* out, const volatile int* abort_flag, int num_sms, cudaStream_t st,
                 const int* perm, const int64_t* range) {
  if (n <= 0) return;
  int64_t blocks = (n + kWarps - 1) / kWarps;
  const int64_t cap = (int64_t)num_sms * (perm ? 2 : 32);  // a group: about one wave beside a far kernel
  if (blocks > cap) blocks = cap;
#define BGB_SS64(OPK)                                                                                              \
  case OPK:                                                                                                        \
    k_ss64<OPK><<<(int)blocks, 32 * kWarps, 0, st>>>(op, ops, tri_problem, M, pts, tg, bg, et, es, ec, emask, n, out, \
                                                     abort_flag, perm, range);                                     \
    break
  switch (op_kind) {
    BGB_SS64(BGB_OP_HELMHOLTZ3D_SL);
    BGB_SS64(BGB_OP_MAXWELL3D_SL);
    BGB_SS64(BGB_OP_MAXWELL3D_DL);
    BGB_SS64(BGB_OP_HELMHOLTZ3D_DL);
    BGB_SS64(BGB_OP_HELMHOLTZ3D_DLT);
    BGB_SS64(BGB_OP_HELMHOLTZ3D_HS);
  }
#undef BGB_SS64
}

}  // namespace bgb
