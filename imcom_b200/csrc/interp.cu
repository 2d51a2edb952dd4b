// interp.cu -- A and B assembly by lookup-table interpolation.
//
// Reference: imcom_lookup_A (imcom_matrix.f90:206-284), imcom_lookup_B
// (:288-357), imcom_interp_lookup (:497-542), imcom_polin2/imcom_polint
// (imcom_proc.f90:351-429).
//
// Per element the reference takes the table window [floor-npm, ceil+npm]
// clipped to [1, L] (8 x 8 points for a non-integer argument, 7 x 7 for an
// integer one), interpolates along y for each window row, then along x.
// The argument, floor/ceiling and window bounds are computed here with the
// same floating-point operations, so they are bit-identical.  The
// interpolating polynomial on those nodes is unique; this kernel evaluates
// it in Lagrange form (weights from prefix/suffix products of (t - x_j) and
// exact integer denominators) instead of Neville's tableau: ~8x fewer flops
// and no divisions, equal to the reference up to rounding (tests bound the
// difference at 1e-13 of the table scale).
//
// Mapping: a CTA computes a 32 x 32 tile into shared memory and writes it
// (and, for A, its mirror) coalesced.  A warp takes 16 elements at a time:
//   weights: lanes 0-15 form the eight x weights of one element each and
//            lanes 16-31 the eight y weights, into shared memory;
//   gather:  eight lanes per element, lane k owning window column x_k: g_k =
//            sum_l wy_l T(x_k, y_l), so a warp load touches 4 elements x 1 row =
//            4 contiguous 64-byte segments; the sums over k of four elements
//            are reduced together.
// Bound by the L1's tag lookups of the gathers (11.5 lines per element) and
// the L2 sectors behind them.  With the weights formed by all eight lanes of
// an element and three shuffle sums per element the kernels were bound by
// instruction issue (79% of the slots): at n = m = 4096 B 2.20 -> 0.74 ms, A
// 1.15 -> 0.41 ms.
#include <cmath>
#include <vector>

#include "common.cuh"

namespace imcom {

int build_tables(imcom_ctx* ctx, int npad, int isB);

namespace {

constexpr int TILE = 32;
constexpr int WARPS = 8;

struct InterpGeom {
  const double* tables;
  long long L;     // table side
  long long L2;    // L * L
  double cent;     // L/2 + 1
  int npm;
};

constexpr int BATCH = 16;       // elements per warp at a time
constexpr int WSTRIDE = 18;     // doubles per element: 8 x weights, 8 y weights, table offset
constexpr int INVD = 9 * 8;     // 1 / prod_{j != k} (k - j) for K nodes: [K][k]

struct InterpSmem {
  double tile[TILE][TILE + 1];
  double w[WARPS][BATCH * WSTRIDE];
  double invd[INVD];
};

__device__ __forceinline__ void fill_invd(double* invd) {
  for (int e = threadIdx.x; e < INVD; e += blockDim.x) {
    const int K = e >> 3, k = e & 7;
    double d = 1.0;
    for (int j = 0; j < K; ++j)
      if (j != k) d *= (double)(k - j);
    invd[e] = 1.0 / d;
  }
}

// Weights of one axis at table argument arg (1-based) into dst[0..7], for
// table nodes b .. b + 7 with b (returned, 0-based) shifted so that all eight
// lie in the table; nodes outside the reference's window weigh nothing.
// *inside is false (and the weights are zero) where the reference returns 0.
__device__ __forceinline__ int axis_weights(const InterpGeom& g, const double* invd, double arg,
                                            bool valid, double* dst) {
  const int L = (int)g.L;
  const double fl = floor(arg);
  const int lo = (int)fl, hi = (int)ceil(arg);
  const bool inside = valid && lo >= 1 && hi <= L;
  const int first = max(1, lo - g.npm), last = min(L, hi + g.npm);
  const int K = inside ? last - first + 1 : 0;
  const int b = inside ? max(1, min(first, L - 7)) : 1;
  const int shift = inside ? first - b : 0;
  double s[8], pre[8];
  // the usual case of a whole warp: a non-integer argument with its window
  // inside the table, so eight nodes and none of them hit (16-byte stores and
  // literal denominators; B at n = m = 4096 0.85 -> 0.74 ms)
  if (__all_sync(0xffffffffu, !valid || (K == 8 && shift == 0))) {
    constexpr double inv[8] = {-1.0 / 5040, 1.0 / 720, -1.0 / 240, 1.0 / 144,
                               -1.0 / 144,  1.0 / 240, -1.0 / 720, 1.0 / 5040};
    const double s0 = K ? arg - (double)first : 0.0;  // exact, and so is every s0 - l
    double acc = 1.0;
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      pre[l] = acc;
      acc *= s0 - (double)l;
    }
    acc = K ? 1.0 : 0.0;
#pragma unroll
    for (int l = 6; l >= 0; l -= 2) {
      double2 w;
      w.y = pre[l + 1] * acc * inv[l + 1];
      acc *= s0 - (double)(l + 1);
      w.x = pre[l] * acc * inv[l];
      acc *= s0 - (double)l;
      *(double2*)(dst + l) = w;
    }
    return b - 1;
  }
  bool node = false;
#pragma unroll
  for (int l = 0; l < 8; ++l) {
    s[l] = (l < K) ? arg - (double)(first + l) : 1.0;
    node |= s[l] == 0.0;
  }
  double acc = 1.0;
#pragma unroll
  for (int l = 0; l < 8; ++l) {
    pre[l] = acc;
    acc *= s[l];
  }
  acc = 1.0;
#pragma unroll
  for (int l = 7; l >= 0; --l) {
    double w = pre[l] * acc * invd[K * 8 + l];
    acc *= s[l];
    if (node) w = (s[l] == 0.0) ? 1.0 : 0.0;
    dst[(l + shift) & 7] = (l < K) ? w : 0.0;
  }
  return b - 1;
}

// Sums of BATCH elements whose weights are in W; lane (grp, k) returns the
// sum of element 4 (k >> 1) + grp (twice).
__device__ __forceinline__ double gather_batch(const InterpGeom& g, const double* W, int k,
                                               int grp) {
  const int L = (int)g.L;
  double v[BATCH / 4];
#pragma unroll
  for (int s = 0; s < BATCH / 4; ++s) {
    const double* we = W + (4 * s + grp) * WSTRIDE;
    const double* col = g.tables + __double_as_longlong(we[16]) + min(k, L - 1);
    const double wx = we[k];
    const double2* wy = (const double2*)(we + 8);
    double gk = 0.0;
#pragma unroll
    for (int l = 0; l < 8; l += 2) {
      const double2 w2 = wy[l / 2];
      gk = fma(w2.x, __ldg(col), gk);
      if (l + 1 < L) col += L;  // a table of fewer than 8 rows: zero weights past it
      gk = fma(w2.y, __ldg(col), gk);
      if (l + 2 < L) col += L;
    }
    v[s] = wx * gk;
  }
  static_assert(BATCH == 16, "transposed reduction of four elements");
  const bool h4 = k & 4, h2 = k & 2;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const double send = h4 ? v[s] : v[s + 2], keep = h4 ? v[s + 2] : v[s];
    v[s] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  const double send = h2 ? v[0] : v[1], keep = h2 ? v[1] : v[0];
  double f = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  return f + __shfl_xor_sync(0xffffffffu, f, 1);
}

// A: upper-triangle tiles (bj >= bi); writes the tile and its mirror.  B(i,
// a): tile of 32 input pixels x 32 output pixels.
template <bool IS_A>
__global__ void __launch_bounds__(WARPS * 32)
lookup_kernel(InterpGeom g, const double* __restrict__ x, const double* __restrict__ y,
              const int* __restrict__ expi, const double* __restrict__ X,
              const double* __restrict__ Y, int n, int m, int psfconst, double npad, double psfx,
              double psfy, double* __restrict__ out, long long ldo) {
  const int bi = blockIdx.x, bj = blockIdx.y;
  if (IS_A && bj < bi) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  InterpSmem& sm = *reinterpret_cast<InterpSmem*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = lane & 7, grp = lane >> 3;
  fill_invd(sm.invd);
  __syncthreads();
  double* W = sm.w[warp];
  // this lane's axis and element within a batch
  const bool ydir = lane >= BATCH;
  const int el = lane & (BATCH - 1);
  const double* pi = ydir ? y : x;
  const double* pj = IS_A ? pi : (ydir ? Y : X);
  const double psf = ydir ? psfy : psfx;
  for (int c = 0; c < TILE / WARPS; ++c) {
    const int jj = warp + WARPS * c, j = bj * TILE + jj;
    for (int h = 0; h < TILE / BATCH; ++h) {
      const int i = bi * TILE + BATCH * h + el;
      const bool valid = i < n && j < m && (!IS_A || j >= i);
      const int ie = valid ? i : 0, je = valid ? j : 0;
      // the reference's argument, operation by operation
      const double d = IS_A ? __dsub_rn(pj[je], pi[ie]) : __dsub_rn(pi[ie], pj[je]);
      const double arg = __dadd_rn(g.cent, __ddiv_rn(__dmul_rn(npad, d), psf));
      const int b = axis_weights(g, sm.invd, arg, valid, W + el * WSTRIDE + (ydir ? 8 : 0));
      const int by = __shfl_down_sync(0xffffffffu, b, BATCH);
      if (!ydir) {
        int t = 0;
        if (psfconst != 1) {
          const int ei = expi[ie];
          t = ei - 1;
          if (IS_A) {
            const int ej = expi[je];
            t += ej * (ej - 1) / 2;
          }
        }
        W[el * WSTRIDE + 16] = __longlong_as_double(t * g.L2 + (long long)by * g.L + b);
      }
      __syncwarp();
      const double f = gather_batch(g, W, k, grp);
      if (!(k & 1)) sm.tile[jj][BATCH * h + 4 * (k >> 1) + grp] = f;
      __syncwarp();
    }
  }
  __syncthreads();
  // A(i, j) for j >= i from the tile; below the diagonal use the mirror.
  for (int e = threadIdx.x; e < TILE * TILE; e += WARPS * 32) {
    const int ii = e & 31, jj = e >> 5;
    const int i = bi * TILE + ii, j = bj * TILE + jj;
    if (i < n && j < m)
      out[(size_t)i + (size_t)j * ldo] =
          (IS_A && bi == bj && jj < ii) ? sm.tile[ii][jj] : sm.tile[jj][ii];
  }
  if (IS_A && bi != bj) {
    // A(j, i) = A(i, j): column i of the mirror block, rows j.
    for (int e = threadIdx.x; e < TILE * TILE; e += WARPS * 32) {
      const int jj = e & 31, ii = e >> 5;
      const int i = bi * TILE + ii, j = bj * TILE + jj;
      if (i < n && j < n) out[(size_t)j + (size_t)i * ldo] = sm.tile[jj][ii];
    }
  }
}

template <bool IS_A>
int launch_lookup(imcom_ctx* ctx, int npad, int npm, int m, const double* X, const double* Y,
                  imcom::DMat& out) {
  const int L = ctx->nps * npad;
  InterpGeom g{ctx->tables, L, (long long)L * L, (double)(L / 2 + 1), npm};
  const dim3 grd((ctx->n + TILE - 1) / TILE, (m + TILE - 1) / TILE);
  IMC_CUDA(cudaFuncSetAttribute(lookup_kernel<IS_A>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(InterpSmem)));
  lookup_kernel<IS_A><<<grd, WARPS * 32, sizeof(InterpSmem), ctx->stream>>>(
      g, ctx->x, ctx->y, ctx->exp_i, X, Y, ctx->n, m, ctx->psfconst, (double)npad, ctx->psfx,
      ctx->psfy, out.p, out.ld);
  IMC_LAUNCH();
  return 0;
}

int check_interp_args(imcom_ctx* ctx, int npoly_in, int npad, int* npm) {
  if (!ctx->have_spectra)
    return set_err(ctx, IMCOM_ERR_STATE, "imcom_gpu_psf_spectra has not run");
  if (ctx->n <= 0) return set_err(ctx, IMCOM_ERR_STATE, "imcom_gpu_set_inputs has not run");
  int npoly = npoly_in;
  if (npoly % 2 == 0) npoly = npoly - 1;  // imcom_matrix.f90:515-519
  if (npoly < 1 || npoly > 7)
    return set_err(ctx, -2, "npoly must be 1..8 (window of at most 8 points)");
  if (npad < 1) return set_err(ctx, -3, "npad must be >= 1");
  *npm = npoly / 2;
  if (ctx->psfconst == 0 && ctx->max_exp > ctx->nexppsf)
    return set_err(ctx, IMCOM_ERR_STATE, "exp_i reaches %d but only %d PSFs were set",
                   ctx->max_exp, ctx->nexppsf);
  return 0;
}

}  // namespace
}  // namespace imcom

using namespace imcom;

extern "C" int imcom_gpu_build_A(imcom_ctx* ctx, int npoly, int npad, double* A_out) {
  if (!ctx) return -1;
  int npm = 0;
  IMC_TRY(check_interp_args(ctx, npoly, npad, &npm));
  cudaSetDevice(ctx->device);
  stage_begin(ctx, ST_A);
  IMC_TRY(build_tables(ctx, npad, 0));
  IMC_TRY(ensure_mat(ctx, ctx->A, ctx->n, ctx->n));
  IMC_TRY(launch_lookup<true>(ctx, npad, npm, ctx->n, ctx->x, ctx->y, ctx->A));
  stage_end(ctx, ST_A);
  ctx->have_A = true;
  ctx->have_QL = false;
  if (A_out) {
    IMC_TRY(download_mat(ctx, ctx->A, A_out));
    IMC_CUDA(cudaStreamSynchronize(ctx->stream));
  }
  return 0;
}

extern "C" int imcom_gpu_build_B(imcom_ctx* ctx, int npoly, int npad, double* B_out) {
  if (!ctx) return -1;
  int npm = 0;
  IMC_TRY(check_interp_args(ctx, npoly, npad, &npm));
  cudaSetDevice(ctx->device);
  stage_begin(ctx, ST_B);
  IMC_TRY(build_tables(ctx, npad, 1));
  IMC_TRY(ensure_mat(ctx, ctx->B, ctx->n, ctx->m));
  IMC_TRY(launch_lookup<false>(ctx, npad, npm, ctx->m, ctx->X, ctx->Y, ctx->B));
  stage_end(ctx, ST_B);
  ctx->have_B = true;
  ctx->have_P = false;
  if (B_out) {
    IMC_TRY(download_mat(ctx, ctx->B, B_out));
    IMC_CUDA(cudaStreamSynchronize(ctx->stream));
  }
  return 0;
}
