// Singular pairs in double-float arithmetic (mixed-precision path).
//
// The ray form of the Sauter-Schwab rules of bgb_ss64.cu -- x = P0 + xi X, y = P0 + xi Y from the shared
// vertex, R = xi |X - Y|, the sum over xi as the series T_m(theta) -- evaluated with df = float + float
// values on the FP32 pipes instead of native FP64, which runs at 1/62 of the FP32 rate on GB300.  A series
// step costs 12 operations where its term is above 2^-24 of the leading one (the sum's order is known, so a
// fast two-sum does) and one beyond; a ray of n = 4 points takes ~1000 FP32-pipe operations, where a
// sincos and a reciprocal square root per point took ~2800.  Accuracy: ~48-bit operations; local
// matrices agree with the FP64 kernels and the oracle to ~1e-14 relative.  Operators with a lossy wave
// number (Re gamma != 0) and angles k R >= 400 use the FP64 kernel; near pairs and pairs whose
// coincident vertices are not bit-equal stay with k_singular.
//
// Bound by the FP32 pipe's issue.  One warp per pair; the per-lane sums are reduced through shared
// memory (15 df additions per lane instead of 80), and nine lanes each form one entry in df.
#include <cmath>
#include <cstring>
#include <vector>

#include "bgb_df.cuh"
#include "bgb_kernels.cuh"
#include "bgb_ss.cuh"

namespace bgb {

namespace {

constexpr int kWarps = 8;

// Moments (complex): hats 9 (their products); EFIE S, Px, Py, P0; MFIE sum H X x Y, sum H (X - Y).
template <int OP>
struct DfMoments {
  static constexpr int N = OP == BGB_OP_HELMHOLTZ3D_SL ? 9 : (OP == BGB_OP_MAXWELL3D_SL ? 8 : 6);
  static constexpr int M0 = OP == BGB_OP_MAXWELL3D_DL ? -1 : 0;  // lowest T_m used (three of them)
};

__device__ __forceinline__ dfl gdf(const float* p) { return dfl{p[0], p[1]}; }

// a * b, not renormalised (the low part may reach a few units of the high part's last place)
__device__ __forceinline__ dfl df_mulx(dfl a, dfl b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  return {p, __fmaf_rn(a.lo, b.hi, e)};
}
// c + a * b
__device__ __forceinline__ dfl df_macc(dfl c, dfl a, dfl b) { return df_add(c, df_mulx(a, b)); }
__device__ __forceinline__ dfl df_dot(const dfl a[3], const dfl b[3]) {
  return df_macc(df_macc(df_mulx(a[0], b[0]), a[1], b[1]), a[2], b[2]);
}
// 1 / sqrt(s): hardware estimate y and one cubic step y (1 + r (1/2 + 3 r / 8)), r = 1 - s y^2 kept as two floats
__device__ __forceinline__ dfl df_rsqrt_step(dfl s) {
  const float y = rsqrtf(s.hi);
  const float yy = __fmul_rn(y, y);
  const dfl q = df_mulx(s, dfl{yy, __fmaf_rn(y, y, -yy)});
  float rh, rl;
  df_fast_two_sum(__fsub_rn(1.0f, q.hi), -q.lo, rh, rl);
  const float h = 0.5f * y, p = __fmul_rn(h, rh);
  float e = __fmaf_rn(h, rh, -p);
  e = __fmaf_rn(h, rl, e);
  e = __fmaf_rn(__fmul_rn(0.75f * h, rh), rh, e);
  float o, t;
  df_fast_two_sum(y, p, o, t);
  dfl r;
  df_fast_two_sum(o, __fadd_rn(t, e), r.hi, r.lo);
  return r;
}

// Entry (i, j) of the local matrix from the reduced moments (re, im of moment q at v[2 q], v[2 q + 1]).
template <int OP>
__device__ __forceinline__ double2 df_entry(const OpDf& op, const GeoDf& A, const GeoDf& B, const int I[3], const int J[3],
                                            const float2* v, dfl inv4pi, int i, int j) {
  auto m = [&](int q) { return dfl{v[q].x, v[q].y}; };
  const dfl ar = gdf(op.alpha[0]), ai = gdf(op.alpha[1]);
  dfl tr{0.f, 0.f}, ti{0.f, 0.f};
  if (OP == BGB_OP_HELMHOLTZ3D_SL) {
    const int r = I[0] == i + 1 ? 0 : (I[1] == i + 1 ? 1 : 2), c = J[0] == j + 1 ? 0 : (J[1] == j + 1 ? 1 : 2);
    const dfl w = df_mul(df_mulf(df_mul(gdf(A.area), gdf(B.area)), 4.f), inv4pi);
    tr = df_mul(m(2 * (3 * r + c)), w);
    ti = df_mul(m(2 * (3 * r + c) + 1), w);
    const dfl Lr = df_sub(df_mul(ar, tr), df_mul(ai, ti)), Li = df_add(df_mul(ar, ti), df_mul(ai, tr));
    return make_double2(df_to_double(Lr), df_to_double(Li));
  }
  dfl V[3], W[3];
  for (int c = 0; c < 3; ++c) {
    V[c] = df_sub(gdf(A.v[i][c]), gdf(A.v[I[0] - 1][c]));
    W[c] = df_sub(gdf(B.v[j][c]), gdf(B.v[J[0] - 1][c]));
  }
  if (OP == BGB_OP_MAXWELL3D_SL) {
    // (1/(4 A A') of the shapes cancels the Jacobians; the divergences leave 4)
    tr = m(0);
    ti = m(1);
    for (int c = 0; c < 3; ++c) {
      tr = df_sub(tr, df_add(df_mul(V[c], m(8 + 2 * c)), df_mul(W[c], m(2 + 2 * c))));
      ti = df_sub(ti, df_add(df_mul(V[c], m(9 + 2 * c)), df_mul(W[c], m(3 + 2 * c))));
    }
    const dfl vw = df_dot(V, W), pr = m(14), pi = m(15);
    tr = df_mul(df_add(tr, df_mul(vw, pr)), inv4pi);
    ti = df_mul(df_add(ti, df_mul(vw, pi)), inv4pi);
    const dfl i4{4.f * inv4pi.hi, 4.f * inv4pi.lo};
    const dfl br = df_mul(gdf(op.beta[0]), i4), bi = df_mul(gdf(op.beta[1]), i4);
    dfl Lr = df_sub(df_mul(ar, tr), df_mul(ai, ti)), Li = df_add(df_mul(ar, ti), df_mul(ai, tr));
    Lr = df_add(Lr, df_sub(df_mul(br, pr), df_mul(bi, pi)));
    Li = df_add(Li, df_add(df_mul(br, pi), df_mul(bi, pr)));
    return make_double2(df_to_double(Lr), df_to_double(Li));
  }
  // MFIE: (W - V).B + (W x V).E with B = sum H X x Y, E = sum H (X - Y); the sign of H = -(gamma + 1/R) G / R at the end
  const dfl x[3] = {df_sub(df_mul(W[1], V[2]), df_mul(W[2], V[1])), df_sub(df_mul(W[2], V[0]), df_mul(W[0], V[2])),
                    df_sub(df_mul(W[0], V[1]), df_mul(W[1], V[0]))};
  for (int c = 0; c < 3; ++c) {
    const dfl wv = df_sub(W[c], V[c]);
    tr = df_add(tr, df_add(df_mul(wv, m(2 * c)), df_mul(x[c], m(6 + 2 * c))));
    ti = df_add(ti, df_add(df_mul(wv, m(2 * c + 1)), df_mul(x[c], m(7 + 2 * c))));
  }
  tr = df_mul(tr, df_neg(inv4pi));
  ti = df_mul(ti, df_neg(inv4pi));
  const dfl Lr = df_sub(df_mul(ar, tr), df_mul(ai, ti)), Li = df_add(df_mul(ar, ti), df_mul(ai, tr));
  return make_double2(df_to_double(Lr), df_to_double(Li));
}

template <int OP>
__global__ void __launch_bounds__(32 * kWarps, 2) k_singular_df(OpDf op1, const OpDf* __restrict__ ops,
                                                                const int* __restrict__ tri_problem,
                                                                const __grid_constant__ DfTables M,
                                                                const float* __restrict__ tab, const GeoDf* __restrict__ tg,
                                                                const GeoDf* __restrict__ bg, const int* __restrict__ ent_tau,
                                                                const int* __restrict__ ent_sigma,
                                                                const int8_t* __restrict__ ent_cls,
                                                                const int16_t* __restrict__ ent_mask, int64_t n,
                                                                double2* __restrict__ out, const volatile int* abort_flag,
                                                                const int* __restrict__ perm,
                                                                const int64_t* __restrict__ range) {
  constexpr int NA = DfMoments<OP>::N, NV = 2 * NA, M0 = DfMoments<OP>::M0;
  constexpr bool kHat = OP == BGB_OP_HELMHOLTZ3D_SL;
  constexpr int NS = NV <= 16 ? 16 : 32;  // rows of the reduction (two lanes per row when 16 suffice)
  __shared__ float4 trig[128];
  __shared__ float2 part[kWarps][NV][33];
  __shared__ float2 red[kWarps][NV];
  for (int i = threadIdx.x; i < 128; i += blockDim.x) trig[i] = ((const float4*)(tab + M.trig_off))[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  // perm: the entries perm[range[0] .. range[1]) (one output block's group); otherwise 0 .. n
  const int64_t i0 = perm ? range[0] : 0, i1 = perm ? range[1] : n;
  for (int64_t it = i0 + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); it < i1; it += warps) {
    if (abort_flag && *abort_flag) return;
    const int64_t e = perm ? (int64_t)perm[it] : it;
    const int cls = ent_cls[e], mask = ent_mask[e];
    if (cls < BGB_CLASS_CV || cls > BGB_CLASS_CF || (mask & BGB_MASK_INEXACT)) continue;  // k_singular
    if (OP == BGB_OP_MAXWELL3D_DL && cls == BGB_CLASS_CF) {  // vanishes on a flat face
      if (lane < 9) out[e * 9 + lane] = make_double2(0.0, 0.0);
      continue;
    }
    const int tau = ent_tau[e];
    const OpDf& op = ops ? ops[tri_problem[tau]] : op1;  // one instance for both: the same bits
    const GeoDf &A = tg[tau], &B = bg[ent_sigma[e]];
    int I[3], J[3];
    ss_permutation_mask(cls, mask, I, J);
    for (int k = 0; k < 3; ++k) {  // guard against an inconsistent mask
      I[k] = I[k] < 1 ? 1 : (I[k] > 3 ? 3 : I[k]);
      J[k] = J[k] < 1 ? 1 : (J[k] > 3 ? 3 : J[k]);
    }
    dfl a1[3], a2[3], b1[3], b2[3];
    float dv[9] = {};  // squared distances between the ends of X and of Y
    for (int c = 0; c < 3; ++c) {
      a1[c] = df_sub(gdf(A.v[I[2] - 1][c]), gdf(A.v[I[0] - 1][c]));
      a2[c] = df_sub(gdf(A.v[I[1] - 1][c]), gdf(A.v[I[2] - 1][c]));
      b1[c] = df_sub(gdf(B.v[J[2] - 1][c]), gdf(B.v[J[0] - 1][c]));
      b2[c] = df_sub(gdf(B.v[J[1] - 1][c]), gdf(B.v[J[2] - 1][c]));
      const float u[3] = {0.f, a1[c].hi, a1[c].hi + a2[c].hi}, v[3] = {0.f, b1[c].hi, b1[c].hi + b2[c].hi};
#pragma unroll
      for (int q = 0; q < 9; ++q) dv[q] = fmaf(u[q / 3] - v[q % 3], u[q / 3] - v[q % 3], dv[q]);
    }
    const dfl kd = gdf(op.k);
    // terms of the series (theta <= k times the largest distance of two vertices): nd in df, then float ones
    // to 2^-51
    int nd = 0, nj = 0;
    {
      float d2 = dv[0];
#pragma unroll
      for (int q = 1; q < 9; ++q) d2 = fmaxf(d2, dv[q]);
      const float th = 1.0001f * fabsf(kd.hi) * sqrtf(d2);
      if (th <= 3.f) {
        float t = 1.f;
        do {
          ++nj;
          if (t > 6e-8f) nd = nj;
          t *= th * th / (float)((2 * nj - 1) * (2 * nj));
        } while (t > 4e-16f && nj < BGB_SS_SERIES);
      }
    }
    df2 acc[NA];  // (real, imaginary) moments
#pragma unroll
    for (int k = 0; k < NA; ++k) acc[k] = df2{0ull, 0ull};
    const int cnt = M.cnt[cls];
    const float2* __restrict__ pt = (const float2*)(tab + M.ss_off[cls]);
    for (int idx = lane; idx < cnt; idx += 32) {
      const float2 p0 = pt[idx], p1 = pt[cnt + idx], p2 = pt[2 * cnt + idx], p3 = pt[3 * cnt + idx], p4 = pt[4 * cnt + idx];
      const dfl al{p0.x, p0.y}, be{p1.x, p1.y}, ga{p2.x, p2.y}, de{p3.x, p3.y}, om{p4.x, p4.y};
      dfl X[3], Y[3], d[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        X[c] = df_macc(df_mulx(al, a1[c]), be, a2[c]);
        Y[c] = df_macc(df_mulx(ga, b1[c]), de, b2[c]);
        d[c] = df_sub(X[c], Y[c]);
      }
      const dfl r2 = df_dot(d, d);
      const dfl rinv = df_rsqrt_step(r2);
      const dfl th = df_mul(kd, df_mulx(r2, rinv));
      df2 T[3];  // (C, S) of T_m = C - i S, m = M0 .. M0 + 2; hats: T_m with (1 - xi)^2 / xi^2, (1 - xi) / xi, 1 in m = 2
      if (nj > 0) {
        const dfl th2s = df_mul(th, th);
        const df2 th2 = df2_both(th2s);
        auto ser = [&](int q, int k) { return kHat && q < 2 ? M.hat[cls][q][k] : M.ser[cls][q + 1 + M0][k]; };
        unsigned long long t[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) t[q] = 0ull;
        for (int k = nj - 1; k >= nd; --k) {
#pragma unroll
          for (int q = 0; q < 3; ++q) t[q] = fma2(t[q], th2.hi, ser(q, k).hi);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) T[q] = df2{t[q], 0ull};
        for (int k = nd - 1; k >= 1; --k) {
#pragma unroll
          for (int q = 0; q < 3; ++q) T[q] = df2_fma_big(T[q], th2, ser(q, k));
        }
        const df2 one_th = df2_of(dfl{1.f, 0.f}, th);
#pragma unroll
        for (int q = 0; q < 3; ++q)  // the first two terms may be of either order
          T[q] = df2_mul(df2_macc(ser(q, 0), T[q], th2), one_th);
      } else {
#pragma unroll
        for (int q = 0; q < 3; ++q) T[q] = df2{0ull, 0ull};
        for (int l = 0; l < M.n[cls]; ++l) {
          dfl sn, cs;
          const dfl xi = M.gx[cls][l];
          df_sincos(df_mul(th, xi), trig, M.trig, sn, cs);
          const df2 e2 = df2_of(cs, sn);
          dfl w = df_mul(M.gw[cls][l], xi);
          if (M0 == 0) w = df_mul(w, xi);
          const dfl om_xi = df_sub(dfl{1.f, 0.f}, xi);
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            dfl wq = w;
            for (int z = q; kHat && z < 2; ++z) wq = df_mul(wq, om_xi);
            T[q] = df2_macc(T[q], df2_both(wq), e2);
            w = df_mul(w, xi);
          }
        }
      }
      const dfl g = df_mul(om, rinv);
      if (OP == BGB_OP_MAXWELL3D_DL) {
        // (i k + 1/(xi R)) (C - i S): degree 2 (X x Y) from T_1, T_0 / R, degree 1 (X - Y) from T_0, T_-1 / R
        const dfl f = df_mul(g, rinv);
        dfl c0, s0, c1, s1, c2, s2;
        df2_parts(T[0], c0, s0);
        df2_parts(T[1], c1, s1);
        df2_parts(T[2], c2, s2);
        const df2 kk = df2_both(kd), rr = df2_of(rinv, df_neg(rinv)), ff = df2_both(f);
        const df2 h2 = df2_mul(ff, df2_add(df2_mulx(kk, df2_of(s2, c2)), df2_mulx(rr, T[1])));
        const df2 h1 = df2_mul(ff, df2_add(df2_mulx(kk, df2_of(s1, c1)), df2_mulx(rr, T[0])));
        const dfl x[3] = {df_sub(df_mulx(X[1], Y[2]), df_mulx(X[2], Y[1])), df_sub(df_mulx(X[2], Y[0]), df_mulx(X[0], Y[2])),
                          df_sub(df_mulx(X[0], Y[1]), df_mulx(X[1], Y[0]))};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          acc[c] = df2_macc(acc[c], h2, df2_both(x[c]));
          acc[3 + c] = df2_macc(acc[3 + c], h1, df2_both(d[c]));
        }
      } else if (OP == BGB_OP_MAXWELL3D_SL) {
        const df2 gg = df2_of(g, df_neg(g)), t1 = df2_mul(gg, T[1]);
        const dfl xy = df_mul(g, df_dot(X, Y));
        acc[0] = df2_macc(acc[0], df2_of(xy, df_neg(xy)), T[2]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          acc[1 + c] = df2_macc(acc[1 + c], t1, df2_both(X[c]));
          acc[4 + c] = df2_macc(acc[4 + c], t1, df2_both(Y[c]));
        }
        acc[7] = df2_macc(acc[7], gg, T[0]);
      } else {
        const df2 gg = df2_of(g, df_neg(g));
        df2 t[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) t[q] = df2_mul(gg, T[q]);
        // hats of the reordered vertices: (1 - xi) + (1 - alpha) xi, beta xi, (alpha - beta) xi, every term positive:
        // summed as the moments of 1, alpha xi, beta xi, a matrix loses a factor of 2 (1.0e-14 -> 2.0e-14 of its norm)
        const dfl one{1.f, 0.f}, a0 = df_sub(one, al), c0 = df_sub(one, ga);
        const dfl a[2] = {be, df_sub(al, be)}, c[2] = {de, df_sub(ga, de)};
        const df2 v = df2_macc(t[1], t[2], df2_both(a0)), w = df2_macc(t[1], t[2], df2_both(c0));
        acc[0] = df2_add(acc[0], df2_macc(df2_macc(t[0], t[1], df2_both(a0)), v, df2_both(c0)));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          acc[1 + i] = df2_macc(acc[1 + i], v, df2_both(c[i]));
          acc[3 + 3 * i] = df2_macc(acc[3 + 3 * i], w, df2_both(a[i]));
#pragma unroll
          for (int j = 0; j < 2; ++j) acc[4 + 3 * i + j] = df2_macc(acc[4 + 3 * i + j], t[2], df2_both(df_mul(a[i], c[j])));
        }
      }
    }
    // reduction: lane v (and v + 16 when 16 rows suffice) sums row v
#pragma unroll
    for (int k = 0; k < NA; ++k) {
      dfl re, im;
      df2_parts(acc[k], re, im);
      part[wid][2 * k][lane] = make_float2(re.hi, re.lo);
      part[wid][2 * k + 1][lane] = make_float2(im.hi, im.lo);
    }
    __syncwarp();
    {
      const int v = lane & (NS - 1), h = NS == 16 ? (lane >> 4) * 16 : 0;
      dfl s{0.f, 0.f};
      if (v < NV)
        for (int k = 0; k < (NS == 16 ? 16 : 32); ++k) {
          const float2 x = part[wid][v][h + k];
          s = df_add(s, dfl{x.x, x.y});
        }
      if (NS == 16) {
        const dfl o{__shfl_xor_sync(0xffffffffu, s.hi, 16), __shfl_xor_sync(0xffffffffu, s.lo, 16)};
        s = df_add(s, o);
      }
      if (lane < NV) red[wid][lane] = make_float2(s.hi, s.lo);
    }
    __syncwarp();
    if (lane < 9) out[e * 9 + lane] = df_entry<OP>(op, A, B, I, J, red[wid], M.trig.inv4pi, lane / 3, lane % 3);
    __syncwarp();
  }
}

__global__ void k_prepare_geodf(const Geo64* __restrict__ g, int nt, GeoDf* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  GeoDf r;
  for (int a = 0; a < 3; ++a)
    for (int c = 0; c < 3; ++c) {
      const double x = g[t].v[a][c];
      r.v[a][c][0] = (float)x;
      r.v[a][c][1] = (float)(x - (double)r.v[a][c][0]);
    }
  const double A = g[t].area, iA = 1.0 / A;
  r.area[0] = (float)A;
  r.area[1] = (float)(A - (double)r.area[0]);
  r.inv_area[0] = (float)iA;
  r.inv_area[1] = (float)(iA - (double)r.inv_area[0]);
  out[t] = r;
}

void split(double x, float* out) {
  const float hi = (float)x;
  out[0] = hi;
  out[1] = (float)(x - (double)hi);
}

void split_ld(long double x, float* out) {
  const float hi = (float)x;
  out[0] = hi;
  out[1] = (float)(x - (long double)hi);
}

}  // namespace

void build_df_tables(const QuadSel& qs, std::vector<float>& buf, DfTables& M) {
  buf.clear();
  M = DfTables{};
  auto align4 = [&]() {
    while (buf.size() % 4) buf.push_back(0.f);
  };
  std::vector<double> pts;
  SsTab64 T;
  build_ss_tables(qs, pts, T);
  auto df = [](double x) {
    float q[2];
    split(x, q);
    return dfl{q[0], q[1]};
  };
  for (int cls = 1; cls <= 3; ++cls) {
    align4();
    M.ss_off[cls] = (int)buf.size();
    M.cnt[cls] = T.cnt[cls];
    M.n[cls] = T.n[cls];
    for (int i = 0; i < 5 * T.cnt[cls]; ++i) {
      float q[2];
      split(pts[(size_t)T.off[cls] + i], q);
      buf.push_back(q[0]);
      buf.push_back(q[1]);
    }
    for (int l = 0; l < T.n[cls]; ++l) {
      M.gx[cls][l] = df(T.gx[cls][l]);
      M.gw[cls][l] = df(T.gw[cls][l]);
    }
    auto put = [&](double cos_k, double sin_k, df2& out) {
      const dfl c = df(cos_k), s = df(sin_k);
      const float hi[2] = {c.hi, s.hi}, lo[2] = {c.lo, s.lo};
      std::memcpy(&out.hi, hi, sizeof(hi));
      std::memcpy(&out.lo, lo, sizeof(lo));
    };
    for (int m = 0; m < 4; ++m)
      for (int k = 0; k < BGB_SS_SERIES; ++k) put(T.ser[cls][m][2 * k], T.ser[cls][m][2 * k + 1], M.ser[cls][m][k]);
    // as T_0 and T_1, with (1 - xi)^2 in the place of 1 and (1 - xi) xi in the place of xi: sums of positive terms, in
    // double (Arm's long double is software: 1.2 ms of a batch call)
    for (int q = 0; q < 2; ++q) {
      double pw[BGB_MAX_SS], f = 1.0, term[2 * BGB_SS_SERIES];
      for (int l = 0; l < T.n[cls]; ++l) {
        const double xi = T.gx[cls][l], z = 1.0 - xi;
        pw[l] = T.gw[cls][l] * xi * xi * z * (q ? xi : z);
      }
      for (int k = 0; k < 2 * BGB_SS_SERIES; ++k) {
        if (k > 1) f *= k;
        double s = 0.0;
        for (int l = 0; l < T.n[cls]; ++l) {
          s += pw[l];
          pw[l] *= T.gx[cls][l];
        }
        term[k] = ((k >> 1) & 1 ? -1 : 1) * s / f;
      }
      for (int k = 0; k < BGB_SS_SERIES; ++k) put(term[2 * k], term[2 * k + 1], M.hat[cls][q][k]);
    }
  }
  align4();
  M.trig_off = (int)buf.size();
  const long double pi = 3.141592653589793238462643383279502884L;
  for (int j = 0; j < 128; ++j) {
    float e[4];
    split_ld(sinl(pi * j / 64.0L), e);
    split_ld(cosl(pi * j / 64.0L), e + 2);
    buf.insert(buf.end(), e, e + 4);
  }
  const long double step = pi / 64.0L;
  int ex;
  const double mant = frexp((double)step, &ex);
  const float p1 = (float)ldexp(floor(mant * 2048.0) / 2048.0, ex);
  const float p2 = (float)(step - (long double)p1);
  const float p3 = (float)(step - (long double)p1 - (long double)p2);
  M.trig.inv_step = (float)(64.0L / pi);
  M.trig.p1 = p1;
  M.trig.p2 = p2;
  M.trig.p3 = p3;
  float t[2];
  split(-1.0 / 6.0, t);
  M.trig.s3 = dfl{t[0], t[1]};
  split(1.0 / 120.0, t);
  M.trig.s5 = dfl{t[0], t[1]};
  M.trig.s7 = (float)(-1.0 / 5040.0);
  M.trig.c4 = (float)(1.0 / 24.0);
  M.trig.c6 = (float)(-1.0 / 720.0);
  split_ld(1.0L / (4.0L * pi), t);
  M.trig.inv4pi = dfl{t[0], t[1]};
  M.total_floats = (int)buf.size();
}

void launch_prepare_geodf(const Geo64* g, int nt, GeoDf* out, cudaStream_t st) {
  if (nt > 0) k_prepare_geodf<<<(nt + 255) / 256, 256, 0, st>>>(g, nt, out);
}

OpDf make_opdf(const OpParams& op) {
  OpDf r{};
  for (int c = 0; c < 2; ++c) {
    split(op.alpha[c], r.alpha[c]);
    split(op.beta[c], r.beta[c]);
  }
  split(op.gamma[1], r.k);
  r.kind = op.kind;
  r.oscill = op.gamma[1] != 0.0;
  return r;
}

void launch_singular_df(int op_kind, const OpDf& op, const OpDf* opdf_array, const int* tri_problem,
                        const DfTables& M, const float* dtab, const GeoDf* tg, const GeoDf* bg, const int* et,
                        const int* es, const int8_t* ec, const int16_t* emask, int64_t n, double2* out,
                        const volatile int* abort_flag, int num_sms, cudaStream_t st, const int* perm,
                        const int64_t* range) {
  if (n <= 0) return;
  int64_t blocks = (n + 7) / 8;
  const int64_t cap = (int64_t)num_sms * (perm ? 2 : 32);  // a group: about one wave beside a far kernel
  if (blocks > cap) blocks = cap;
#define BGB_LAUNCH_DF(OPK)                                                                                          \
  case OPK:                                                                                                         \
    k_singular_df<OPK><<<(int)blocks, 32 * kWarps, 0, st>>>(op, opdf_array, tri_problem, M, dtab, tg, bg, et, es, ec, \
                                                            emask, n, out, abort_flag, perm, range);                \
    break
  switch (op_kind) {  // other operators take the FP64 kernel (df_singular_ok)
    BGB_LAUNCH_DF(BGB_OP_HELMHOLTZ3D_SL);
    BGB_LAUNCH_DF(BGB_OP_MAXWELL3D_SL);
    BGB_LAUNCH_DF(BGB_OP_MAXWELL3D_DL);
    default: break;
  }
#undef BGB_LAUNCH_DF
}

}  // namespace bgb
