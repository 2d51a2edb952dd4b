// eigen_jacobi.cu -- one-sided (Hestenes) Jacobi eigensolver for small
// positive semi-definite systems, batched: one CTA per matrix, with the
// matrix and the accumulated rotations held in shared memory.
//
// The reference calls LAPACK DSYEVR (imcom_matrix.f90:617-643).  IMCOM's A is
// a Gram matrix of PSF overlaps (positive semi-definite) whose eigenvalues
// span many decades, and U and Sigma are set by the smallest of them; Jacobi
// methods compute those to high relative accuracy (Demmel & Veselic, "Jacobi's
// method is more accurate than QR", SIAM J. Matrix Anal. Appl. 13, 1992),
// which a tridiagonal reduction does not promise.
//
// Method (Hestenes 1958; the parallel ordering of Brent & Luk 1985):
//   G = A, V = I.  A sweep visits every column pair (p, q) once, in n'-1
//   rounds of n'/2 disjoint pairs (n' = n rounded up to even; the round-robin
//   "circle" ordering), eight lanes per pair:
//     alpha = g_p.g_p, beta = g_q.g_q, gamma = g_p.g_q;
//     if |gamma| > tol sqrt(alpha beta):
//       zeta = (beta - alpha) / (2 gamma), t = sign(zeta) / (|zeta| + sqrt(1 + zeta^2)),
//       c = 1 / sqrt(1 + t^2), s = c t;
//       (g_p, g_q) <- (c g_p - s g_q, s g_p + c g_q), the same for (v_p, v_q).
//   Sweeps repeat until one rotates nothing (at most max_sweeps; an error
//   status otherwise).  Then G = A V has orthogonal columns; for symmetric A
//   g_i = lambda_i v_i, and lambda_i = v_i.g_i keeps the sign.  The pairs are
//   returned in ascending order of lambda (the caller reverses them, as for
//   the other solvers).
//
// Limits: n <= JAC_MAX (G and V fill the shared memory); eigenvalue pairs
// +lambda, -lambda of an indefinite matrix are not separated (A is positive
// semi-definite here).
#include <cmath>
#include <vector>

#include "common.cuh"
#include "eigen.cuh"

namespace imcom {
namespace {

constexpr int JAC_MAX = IMCOM_JACOBI_MAX_N;
constexpr int JAC_MAX_SWEEPS = 60;

__device__ __forceinline__ double jwarp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Columns in shared memory start 64 bytes apart modulo 128, so that eight rows
// of four consecutive columns take two wavefronts.
__host__ __device__ inline int jac_ld(int n) { return (n + 7) / 16 * 16 + 8; }

// Matrix b of the batch: A_b at A + b strideA (column-major, lda); output
// eigenvectors (ascending) at Q + b strideQ (ldq), eigenvalues at
// L + b strideL.  status[b] = sweeps used, or -1 if it did not converge.
//
// A round is a chain (columns from shared memory, three sums, square roots and
// divisions, columns back), so each pair's work is spread over as few
// instructions as its sums allow: a warp takes four pairs at once, eight lanes
// each, and every lane rows i + 8 a + 32 c, with an accumulator per a.  Adding
// these (0 with 2, 1 with 3) and then lanes is the tree of a whole warp on one
// pair, so the results are the same to the bit.  Columns stay in registers
// between the sums and the rotation, and the rotations' columns are on their way
// while the angle is formed.  The test takes the square root only where the
// squares do not decide it, and lanes that do not rotate divide 1 by 1 (a zero
// or infinite operand sends the whole warp through the division's slow path).
// A call with one system of 75 (20 sweeps of 75 rounds): 5.2 ms with a warp per
// pair, three pairs one after another, 2.0 now; of 112, 64 systems: 19.3 -> 8.4.
template <int C>  // chunks of 32 rows
__global__ void __launch_bounds__(32 * (((C < 4 ? 32 * C : JAC_MAX) + 7) / 8), 1)
jacobi_kernel(const double* __restrict__ A, long long lda, long long strideA, int n,
              double* __restrict__ Q, long long ldq, long long strideQ,
              double* __restrict__ L, long long strideL, int* __restrict__ status) {
  extern __shared__ __align__(16) double jsm[];
  const int ld = jac_ld(n);
  double* G = jsm;                   // n columns, column-major
  double* V = G + (size_t)n * ld;
  double* lam = V + (size_t)n * ld;  // n
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int NT = blockDim.x, NW = NT / 32;
  const double* Ab = A + (size_t)b * strideA;
  for (int idx = tid; idx < n * n; idx += NT) {
    const int r = idx % n, c = idx / n;
    G[r + c * ld] = Ab[r + (long long)c * lda];
    V[r + c * ld] = (r == c) ? 1.0 : 0.0;
  }
  const int np = n + (n & 1);  // players of the round-robin (one idle when n is odd)
  const int m = np - 1;        // rotating players; player m is fixed
  const double tol = 2.0 * 1.1102230246251565e-16 * sqrt((double)n);
  const int k = wid * 4 + (lane >> 3), r0 = lane & 7;
  int sweeps = 0;
  bool converged = (n <= 1);
  __syncthreads();
  while (!converged && sweeps < JAC_MAX_SWEEPS) {
    bool rotated = false;
    // round s: (m, s) and ((s + k) mod m, (s - k) mod m), k = 1 .. np/2 - 1
    int up = k % m, dn = (m - up) % m;
    for (int s = 0; s < m; ++s) {
      const int p = k == 0 ? s : min(up, dn), q = k == 0 ? m : max(up, dn);
      if (++up == m) up = 0;
      if (++dn == m) dn = 0;
      const bool on = k < np / 2 && q < n;  // not the idle player's
      double* gp = G + p * ld + r0;
      double* gq = G + q * ld + r0;
      double x[4 * C], y[4 * C];
#pragma unroll
      for (int e = 0; e < 4 * C; ++e) {
        const bool in = on && (e < 4 * C - 4 || r0 + 8 * e < n);
        x[e] = in ? gp[8 * e] : 0.0;
        y[e] = in ? gq[8 * e] : 0.0;
      }
      double al[4], be[4], ga[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        al[a] = be[a] = ga[a] = 0.0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          al[a] = fma(x[4 * c + a], x[4 * c + a], al[a]);
          be[a] = fma(y[4 * c + a], y[4 * c + a], be[a]);
          ga[a] = fma(x[4 * c + a], y[4 * c + a], ga[a]);
        }
      }
      double sa = (al[0] + al[2]) + (al[1] + al[3]);
      double sb = (be[0] + be[2]) + (be[1] + be[3]);
      double sg = (ga[0] + ga[2]) + (ga[1] + ga[3]);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        sa += __shfl_xor_sync(0xffffffffu, sa, o);
        sb += __shfl_xor_sync(0xffffffffu, sb, o);
        sg += __shfl_xor_sync(0xffffffffu, sg, o);
      }
      // |sg| > tol sqrt(sa sb): by the squares unless they are within 1e-6 or
      // near the ends of the range
      const double pr = sa * sb, lim = (tol * tol) * pr, g2 = sg * sg;
      bool rot = g2 > lim;
      if (on && (!(fabs(g2 - lim) > 1e-6 * lim) || !(pr > 1e-240 && pr < 1e290) || !(g2 < 1e290)))
        rot = sg != 0.0 && fabs(sg) > tol * sqrt(pr);
      rot = rot && on;
      if (__any_sync(0xffffffffu, rot)) {
        double* vp = V + p * ld + r0;
        double* vq = V + q * ld + r0;
        constexpr int H = C < 4 ? 4 * C : 8;  // rows of V held at a time
        double u[H], w[H];
        auto load = [&](int e0) {
#pragma unroll
          for (int e = 0; e < H; ++e) {
            const bool in = rot && (e0 + e < 4 * C - 4 || r0 + 8 * (e0 + e) < n);
            u[e] = in ? vp[8 * (e0 + e)] : 0.0;
            w[e] = in ? vq[8 * (e0 + e)] : 0.0;
          }
        };
        load(0);
        // lanes that do not rotate divide 1 by 1
        const double zeta = (rot ? sb - sa : 1.0) / (rot ? 2.0 * sg : 1.0);
        const double t = copysign(1.0, zeta) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        const double c = 1.0 / sqrt(1.0 + t * t), sn = c * t;
#pragma unroll
        for (int e = 0; e < 4 * C; ++e) {
          if (rot && (e < 4 * C - 4 || r0 + 8 * e < n)) {
            gp[8 * e] = c * x[e] - sn * y[e];
            gq[8 * e] = sn * x[e] + c * y[e];
          }
        }
#pragma unroll
        for (int e0 = 0; e0 < 4 * C; e0 += H) {
          if (e0) load(e0);
#pragma unroll
          for (int e = 0; e < H; ++e) {
            if (rot && (e0 + e < 4 * C - 4 || r0 + 8 * (e0 + e) < n)) {
              vp[8 * (e0 + e)] = c * u[e] - sn * w[e];
              vq[8 * (e0 + e)] = sn * u[e] + c * w[e];
            }
          }
        }
        rotated |= rot;
      }
      __syncthreads();
    }
    ++sweeps;
    converged = !__syncthreads_or(rotated);
  }
  if (tid == 0) status[b] = converged ? sweeps : -1;
  // lambda_i = v_i . g_i
  for (int i = wid; i < n; i += NW) {
    double acc = 0.0;
    for (int r = lane; r < n; r += 32) acc = fma(V[i * ld + r], G[i * ld + r], acc);
    acc = jwarp_sum(acc);
    if (lane == 0) lam[i] = acc;
  }
  __syncthreads();
  // ascending order: the rank of lambda_i (ties by index) is its output slot
  double* Qb = Q + (size_t)b * strideQ;
  double* Lb = L + (size_t)b * strideL;
  for (int i = wid; i < n; i += NW) {
    const double li = lam[i];
    int rank = 0;
    for (int j = lane; j < n; j += 32) {
      const double lj = lam[j];
      rank += (lj < li || (lj == li && j < i)) ? 1 : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (lane == 0) Lb[rank] = li;
    for (int r = lane; r < n; r += 32) Qb[r + (long long)rank * ldq] = V[i * ld + r];
  }
}

size_t jacobi_smem(int n) { return (2 * (size_t)n * jac_ld(n) + n) * sizeof(double); }


int launch_jacobi(imcom_ctx* ctx, const double* A, long long lda, long long strideA, int n,
                  int count, double* Q, long long ldq, long long strideQ, double* L,
                  long long strideL, int* status) {
  if (n > JAC_MAX)
    return set_err(ctx, IMCOM_ERR_STATE,
                   "the Jacobi eigensolver takes n <= %d (shared memory); n = %d", JAC_MAX, n);
  const size_t smem = jacobi_smem(n);
  const int threads = 32 * ((n + 7) / 8);  // four pairs per warp
  auto launch = [&](auto kernel) {
    // the largest size's need: the attribute is process-wide (see usum.cuh)
    IMC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)jacobi_smem(JAC_MAX)));
    kernel<<<count, threads, smem, ctx->stream>>>(A, lda, strideA, n, Q, ldq, strideQ, L, strideL,
                                                  status);
    return 0;
  };
  IMC_TRY(n <= 32   ? launch(jacobi_kernel<1>)
          : n <= 64 ? launch(jacobi_kernel<2>)
          : n <= 96 ? launch(jacobi_kernel<3>)
                    : launch(jacobi_kernel<4>));
  IMC_LAUNCH();
  return 0;
}

int check_jacobi(imcom_ctx* ctx, const int* status_dev, int count, int* sweeps_host) {
  std::vector<int> st((size_t)count);
  IMC_CUDA(cudaMemcpyAsync(st.data(), status_dev, (size_t)count * sizeof(int),
                           cudaMemcpyDeviceToHost, ctx->stream));
  IMC_CUDA(cudaStreamSynchronize(ctx->stream));
  for (int b = 0; b < count; ++b) {
    if (sweeps_host) sweeps_host[b] = st[b];
    if (st[b] < 0)
      return set_err(ctx, IMCOM_ERR_EIGEN, "Jacobi eigensolver: matrix %d did not converge in %d "
                     "sweeps", b, JAC_MAX_SWEEPS);
  }
  return 0;
}

}  // namespace

int eigen_jacobi(imcom_ctx* ctx, const DMat& A, DMat& Q, double* L) {
  const int n = (int)A.rows;
  int* status = ctx->flags + 44;  // one slot: a single matrix
  IMC_TRY(launch_jacobi(ctx, A.p, A.ld, 0, n, 1, Q.p, Q.ld, 0, L, 0, status));
  return check_jacobi(ctx, status, 1, nullptr);
}

}  // namespace imcom

using namespace imcom;

// Batched eigendecomposition of `count` small symmetric positive semi-definite
// matrices (n <= IMCOM_JACOBI_MAX_N) on host arrays; see the header.
extern "C" int imcom_gpu_eigh_jacobi_batched(imcom_ctx* ctx, int n, int count, const double* A,
                                             double* Q, double* L, int* sweeps) {
  if (!ctx) return -1;
  if (n < 1 || n > JAC_MAX) return -2;
  if (count < 1) return -3;
  if (!A) return -4;
  if (!Q) return -5;
  if (!L) return -6;
  cudaSetDevice(ctx->device);
  const size_t nn = (size_t)n * n, mats = nn * (size_t)count;
  const size_t need = (2 * mats + (size_t)n * count) * sizeof(double) + (size_t)count * sizeof(int) +
                      256;
  IMC_TRY(ensure_buf(ctx, &ctx->jac_buf, ctx->jac_bytes, need));
  double* dA = (double*)ctx->jac_buf;
  double* dQ = dA + mats;
  double* dL = dQ + mats;
  int* dst = (int*)(dL + (size_t)n * count);
  IMC_CUDA(cudaMemcpyAsync(dA, A, mats * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  IMC_TRY(launch_jacobi(ctx, dA, n, (long long)nn, n, count, dQ, n, (long long)nn, dL, n, dst));
  IMC_CUDA(cudaMemcpyAsync(Q, dQ, mats * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  IMC_CUDA(cudaMemcpyAsync(L, dL, (size_t)n * count * sizeof(double), cudaMemcpyDeviceToHost,
                           ctx->stream));
  return check_jacobi(ctx, dst, count, sweeps);
}
