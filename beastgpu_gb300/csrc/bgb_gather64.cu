// The gather half of the plain FP64 far stage: output tiles from the local matrices of a panel.
//
// The plain FP64 path computes the 3x3 local matrix of every triangle pair of a panel (all test
// triangles of the call x the trial triangles of a run of output tiles) once, in k_pair64
// (bgb_far_impl.cuh), into a device workspace; k_place_special replaces those of the singular and near
// pairs, and k_gather64 adds them into the output entries.  The tiles of the fused kernel compute the
// pairs at their rims again (1.5x the pairs for RWG functions in 64-wide tiles, 1.7x for hats in 48-wide
// ones), which on an FP64 pipe at 1/62 of the FP32 rate costs far more than the workspace's traffic:
// 144 B written and ~1.6 x 144 B read per pair, against the ~8 KB that HBM could move in the ~1.1 ns that the
// pipe needs for one pair.
//
// k_gather64: one CTA per output tile.  The local matrices of the next chunk of trial triangles are
// copied to shared memory (cp.async, 16 B) while the current chunk is added into the entries, in the
// order of the fused kernel -- trial triangle ascending, then test triangle ascending -- so the result
// does not depend on tiles or panels.  Bound by its FP64 sums (half of the pipe's cycles) and the panel's reads.
// The copies step through (row, column) without divisions and unit coefficients (hats) cost no product: far
// stage 47.2 -> 44.9 ms (cube of 6,912 triangles, hats), 31.8 -> 30.4 ms (level-4 EFIE).  An odd chunk width keeps the 16-byte
// shared-memory reads of consecutive rows free of bank conflicts (rows are SC * 144 B apart).
#include "bgb_kernels.cuh"

#include <algorithm>

namespace bgb {
namespace {

constexpr int kThreads = 256;  // 384 and 512 are within 0.5%
constexpr int kFetch = kThreads / 9;  // pairs copied per step, nine threads each
constexpr int kUnit = 1 << 30;        // in a support's code: its coefficient is 1

struct GatherSmem {
  double2* L[2];
  double2* Zs;
  double* fcoef;
  double* gsCoef;
  int64_t* rowT;  // workspace offset of a test triangle's row
  int *colB, *fcnt, *fcode, *grpFn, *grpOff, *chGrp, *gsCode;
};

__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline size_t carve64(unsigned char* base, const TilePlan& p, GatherSmem* s) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off = al16(off + bytes);
    return base ? base + o : nullptr;
  };
  const int nch = (p.nmax + p.SC - 1) / p.SC;
  unsigned char* q;
  for (int k = 0; k < 2; ++k) {
    q = take(sizeof(double2) * 9 * (size_t)p.tmax * p.SC);
    if (s) s->L[k] = (double2*)q;
  }
  q = take(sizeof(double2) * (size_t)p.FM * p.FN); if (s) s->Zs = (double2*)q;
  q = take(sizeof(double) * (size_t)p.FM * p.MAXS); if (s) s->fcoef = (double*)q;
  q = take(sizeof(double) * (size_t)p.gsmax); if (s) s->gsCoef = (double*)q;
  q = take(sizeof(int64_t) * p.tmax); if (s) s->rowT = (int64_t*)q;
  q = take(sizeof(int) * p.nmax); if (s) s->colB = (int*)q;
  q = take(sizeof(int) * p.FM); if (s) s->fcnt = (int*)q;
  q = take(sizeof(int) * (size_t)p.FM * p.MAXS); if (s) s->fcode = (int*)q;
  q = take(sizeof(int) * (size_t)p.gmax); if (s) s->grpFn = (int*)q;
  q = take(sizeof(int) * (size_t)(p.gmax + 1)); if (s) s->grpOff = (int*)q;
  q = take(sizeof(int) * (size_t)(nch + 1)); if (s) s->chGrp = (int*)q;
  q = take(sizeof(int) * (size_t)p.gsmax); if (s) s->gsCode = (int*)q;
  return off;
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}

// prow / pcol: workspace row of a test triangle, workspace column of a trial triangle of the panel.
__global__ void __launch_bounds__(kThreads) k_gather64(const TilePlan* __restrict__ plan, int bn0,
                                                       const int* __restrict__ prow, const int* __restrict__ pcol,
                                                       const double2* __restrict__ ws, int ncols,
                                                       const volatile int* abort_flag) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ TilePlan p;
  __shared__ int stop;
  const int tid = threadIdx.x;
  for (int i = tid; i < (int)(sizeof(TilePlan) / 4); i += kThreads) ((int*)&p)[i] = ((const int*)plan)[i];
  if (tid == 0) stop = abort_flag && *abort_flag;
  __syncthreads();
  if (stop) return;
  const int bm = blockIdx.x % p.n_tblocks, bn = bn0 + blockIdx.x / p.n_tblocks;
  GatherSmem s;
  carve64(smem, p, &s);
  const int SC = p.SC, MAXS = p.MAXS;
  const int t0 = p.tb_off[bm], tm = p.tb_off[bm + 1] - t0;
  const int b0 = p.bb_off[bn], nbk = p.bb_off[bn + 1] - b0;
  const int f0 = p.tb_fn_off[bm], fm = p.tb_fn_off[bm + 1] - f0;
  const int g0 = p.bb_fn_off[bn], fn = p.bb_fn_off[bn + 1] - g0;
  for (int i = tid; i < tm; i += kThreads) s.rowT[i] = (int64_t)prow[p.tb_tris[t0 + i]] * ncols * 9;
  for (int i = tid; i < nbk; i += kThreads) s.colB[i] = pcol[p.bb_tris[b0 + i]] * 9;
  __syncthreads();
  // local matrices of chunk c: entry (i, j) of pair (ti, si) at L[(ti * SC + si) * 9 + i * 3 + j]
  // (nine threads per pair, each stepping through the pairs without a division)
  const int fp = tid / 9, fk = tid - 9 * fp, fti = fp / SC, fsi = fp - fti * SC, dti = kFetch / SC, dsi = kFetch - dti * SC;
  auto fetch = [&](int c, double2* dst) {
    const int base = c * SC, scn = min(SC, nbk - base);
    if (fp < kFetch)
      for (int ti = fti, si = fsi; ti < tm; ti += dti) {
        if (si < scn) cp_async16(dst + (ti * SC + si) * 9 + fk, ws + (s.rowT[ti] + s.colB[base + si] + fk));
        si += dsi;
        if (si >= SC) {
          si -= SC;
          ++ti;
        }
      }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const int c0 = p.bb_chunk_off[bn], nch = p.bb_chunk_off[bn + 1] - c0;
  double2* const L0 = s.L[0];
  const int lstep = (int)(s.L[1] - L0);  // the two chunk buffers
  if (nch > 0) fetch(0, L0);
  // supports as offsets into a chunk's matrices
  for (int m = tid; m < fm; m += kThreads) {
    const int a0 = p.fs_off[f0 + m], a1 = p.fs_off[f0 + m + 1];
    const int cnt = min(a1 - a0, MAXS);
    s.fcnt[m] = cnt;
    for (int k = 0; k < cnt; ++k) {
      const int fc = p.fs_code[a0 + k];  // test triangle << 2 | local
      s.fcode[m * MAXS + k] = (fc >> 2) * SC * 9 + (fc & 3) * 3;
      s.fcoef[m * MAXS + k] = p.fs_coef[a0 + k];
    }
  }
  const int gb0 = p.ch_grp_off[c0], gb1 = p.ch_grp_off[c0 + nch];
  const int sb0 = p.grp_sup_off[gb0], sb1 = p.grp_sup_off[gb1];
  for (int i = tid; i < gb1 - gb0; i += kThreads) {
    s.grpFn[i] = p.grp_fn[gb0 + i];
    s.grpOff[i] = p.grp_sup_off[gb0 + i] - sb0;
  }
  if (tid == 0) s.grpOff[gb1 - gb0] = sb1 - sb0;
  for (int i = tid; i <= nch; i += kThreads) s.chGrp[i] = p.ch_grp_off[c0 + i] - gb0;
  for (int i = tid; i < sb1 - sb0; i += kThreads) {
    const int code = p.gs_code[sb0 + i];  // trial slot << 2 | local
    const int slot = code >> 2;
    const double cb = p.gs_coef[sb0 + i];
    s.gsCode[i] = ((slot % SC) * 9 + (code & 3)) | (cb == 1.0 ? kUnit : 0);
    s.gsCoef[i] = cb;
  }
  for (int i = tid; i < fm * fn; i += kThreads) s.Zs[i] = make_double2(0.0, 0.0);
  // gather roles: row m, groups gq + k * gstep (whole warps of rows when that keeps the groups in flight)
  const int FM32 = (p.FM + 31) & ~31;
  const int FMb = kThreads / FM32 == kThreads / p.FM ? FM32 : p.FM;
  const int gstep = kThreads / FMb, gq = tid / FMb, m = tid - gq * FMb;
  const bool on = m < fm && gq < gstep;
  for (int c = 0; c < nch; ++c) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // chunk c is in shared memory, and nobody reads the other buffer any more
    const double2* __restrict__ L = L0 + (c & 1) * lstep;
    if (c + 1 < nch) fetch(c + 1, L0 + ((c + 1) & 1) * lstep);
    if (on) {
      const int gg0 = s.chGrp[c], gg1 = s.chGrp[c + 1];
      const int cnt = s.fcnt[m];
      for (int g = gg0 + gq; g < gg1; g += gstep) {
        double2* z = &s.Zs[s.grpFn[g] * fm + m];
        double2 acc = *z;
        const int q1 = s.grpOff[g + 1];
        for (int q = s.grpOff[g]; q < q1; ++q) {
          const int code = s.gsCode[q], col = code & (kUnit - 1);
          if (code & kUnit) {  // hats: the product of the coefficients is the test side's, an FP64 operation less in three
            for (int a = 0; a < cnt; ++a) {
              const double w = s.fcoef[m * MAXS + a];
              const double2 l = L[s.fcode[m * MAXS + a] + col];
              acc.x = __fma_rn(w, l.x, acc.x);
              acc.y = __fma_rn(w, l.y, acc.y);
            }
          } else {
            const double cb = s.gsCoef[q];
            for (int a = 0; a < cnt; ++a) {
              const double w = __dmul_rn(s.fcoef[m * MAXS + a], cb);
              const double2 l = L[s.fcode[m * MAXS + a] + col];
              acc.x = __fma_rn(w, l.x, acc.x);
              acc.y = __fma_rn(w, l.y, acc.y);
            }
          }
        }
        *z = acc;
      }
    }
  }
  __syncthreads();
  for (int n = tid >> 5; n < fn; n += kThreads / 32) {  // output columns by warps, rows by lanes
    const int64_t col = p.cols[g0 + n] * p.ld;
    for (int mm = tid & 31; mm < fm; mm += 32) {
      const int64_t idx = p.rows[f0 + mm] + col;
      const double2 v = s.Zs[n * fm + mm];
      if (p.out_c64) ((double2*)p.out)[idx] = v;
      else ((float2*)p.out)[idx] = make_float2((float)v.x, (float)v.y);
    }
  }
}

__global__ void k_index_of(const int* __restrict__ list, int n, int* __restrict__ index) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) index[list[i]] = i;
}

// The local matrices of the non-far pairs of the panel (index -1: not in it), 9 threads per entry.
__global__ void k_place_special(const int* __restrict__ tau, const int* __restrict__ sigma, int64_t n,
                                const int* __restrict__ prow, const int* __restrict__ pcol,
                                const double2* __restrict__ L, int ncols, double2* __restrict__ ws) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 9 * n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = i / 9;
    const int r = prow[tau[e]], c = pcol[sigma[e]];
    if (r >= 0 && c >= 0) ws[((int64_t)r * ncols + c) * 9 + (i - 9 * e)] = L[i];
  }
}

}  // namespace

size_t gather64_smem_bytes(const TilePlan& p) { return carve64(nullptr, p, nullptr); }

static int gather64_smem_limit() {
  int dev = 0, v = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, k_gather64) != cudaSuccess) return v;
  return v - (int)fa.sharedSizeBytes;
}

int gather64_occupancy(size_t smem_bytes, int* per_sm) {
  *per_sm = 0;
  const int lim = gather64_smem_limit();
  if (smem_bytes > (size_t)std::max(0, lim)) return 0;
  BGB_CUDA(cudaFuncSetAttribute(k_gather64, cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
  BGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_gather64, kThreads, smem_bytes));
  return 0;
}

int launch_gather64(const TilePlan* plan, int ntiles, int bn0, const int* prow, const int* pcol, const double2* ws,
                    int ncols, size_t smem_bytes, const volatile int* abort_flag, cudaStream_t st) {
  BGB_CUDA(cudaFuncSetAttribute(k_gather64, cudaFuncAttributeMaxDynamicSharedMemorySize, gather64_smem_limit()));
  if (ntiles > 0)
    k_gather64<<<ntiles, kThreads, smem_bytes, st>>>(plan, bn0, prow, pcol, ws, ncols, abort_flag);
  BGB_CUDA(cudaGetLastError());
  return 0;
}

int launch_index_of(const int* list, int n, int* index, int nindex, cudaStream_t st) {
  BGB_CUDA(cudaMemsetAsync(index, 0xff, sizeof(int) * (size_t)nindex, st));
  if (n > 0) k_index_of<<<std::min((n + 255) / 256, 1024), 256, 0, st>>>(list, n, index);
  BGB_CUDA(cudaGetLastError());
  return 0;
}

int launch_place_special(const int* tau, const int* sigma, int64_t n, const int* prow, const int* pcol, const double2* L,
                         int ncols, double2* ws, cudaStream_t st) {
  if (n > 0)
    k_place_special<<<(int)std::min<int64_t>((9 * n + 255) / 256, 8192), 256, 0, st>>>(tau, sigma, n, prow, pcol, L,
                                                                                       ncols, ws);
  BGB_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace bgb
