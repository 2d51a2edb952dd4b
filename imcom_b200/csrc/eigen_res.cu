// eigen_res.cu -- the last columns of the tridiagonalisation with the whole
// trailing matrix resident in the SMs' shared memory, one exchange per column.
//
// Once the trailing matrix of order S fits the grid's shared memory (S = 2048
// on 148 SMs), a panel column is a chain of latencies: two grid barriers,
// each a store, a fence, an atomic and a poll, and dependent L2 round trips
// between them (8 to 11 us whatever the size).  Here CTA q keeps full
// symmetric rows and every CTA keeps the vectors of the current column,
// redundantly, in registers.  Unblocked LAPACK dsytd2 'L', per column j with
// x = A(j, j+1:) known to everyone:
//   rows:      apply the previous column's update to the own rows and form
//              z_r = A(r, :) x in the same pass over shared memory;
//   exchange:  publish z_r and A(r, j+1) of the own rows;
//   everyone:  the reflector v = scl x + delta e_{j+1} from x alone (while
//              the exchange is in flight), y = A v = scl z + delta A(:, j+1),
//              w = tau y - 1/2 tau^2 (v^T y) v, with v^T y from x^T z, and the
//              next x = A(j+1, :) - w - w_{j+1} v.
// So the only wait of a column is for the published values.  Each is a
// 16-byte {value, column tag} written and read as one 128-bit access: the
// reader polls the data itself, with no fence, flag or barrier.  Two buffers
// by column parity suffice: a CTA publishes column j+2 only after it has read
// every value of column j+1, which each owner wrote after reading column j.
// A CTA whose last row is j+1 owns none of them, so it publishes column j and
// returns without reading it; column j of V, d, e and tau is written by the
// owner of row j+2 (res_rows.h).
// Polls are bounded: a value that does not come sets the error word.
//
// What bounds it: the latency of one exchange (about 1500 cycles for 600
// values, 2100 for 3500) and the in-order issue of two warps per scheduler;
// from S of about 1500 also the shared-memory pass over the rows (16 bytes
// per element at 128 B/clk per SM).  256 threads: the scalars and reductions
// are replicated per warp, and 512 threads were 15-40% slower.  Measured,
// whole tridiagonalisation: n = 300 1.43 -> 0.57 ms, 1000 7.7 -> 2.4 ms,
// 1453 12.0 -> 4.6 ms, 2000 18.0 -> 7.4 ms (before: panels and the cluster
// tail).
#include <algorithm>

#include "common.cuh"
#include "eigen.cuh"
#include "res_rows.h"
#include "tagged.cuh"

namespace imcom {

namespace {


constexpr int RT = 256;      // threads per CTA
constexpr int RW = RT / 32;  // warps

struct ResArgs {
  const double* A;  // lower triangle valid for rows and columns k0 .. n-1
  long long lda;
  double* V;
  long long ldv;
  double *d, *e, *tau;
  int n, k0, nrow;  // nrow: most rows per CTA
  ulonglong2* rec;  // [2][ldS][2] {z_r, tag}, {A(r, j+1), tag}
  int* err;
  long long spin;
  int stall;  // test of the bounded polls: the first column's values never come
};

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of one value per warp.
__device__ __forceinline__ double sum_warps(const double* r) {
  const double2* t = (const double2*)r;
  double2 s = t[0], q = t[1];
#pragma unroll
  for (int u = 2; u < RW / 2; u += 2) {
    const double2 t0 = t[u], t1 = t[u + 1];
    s.x += t0.x;
    s.y += t0.y;
    q.x += t1.x;
    q.y += t1.y;
  }
  return (s.x + s.y) + (q.x + q.y);
}

// Transposed reduction of N slots (a power of two, at most 16) over the warp:
// lane L ends with the sum of slot L / (32 / N).
template <int N>
__device__ __forceinline__ double wsum_slots(double* acc, int lane) {
  int m = 16;
#pragma unroll
  for (int h = N / 2; h >= 1; h >>= 1, m >>= 1) {
    const bool hi = (lane & m) != 0;
#pragma unroll
    for (int u = 0; u < h; ++u) {
      const double send = hi ? acc[u] : acc[u + h];
      const double keep = hi ? acc[u + h] : acc[u];
      acc[u] = keep + __shfl_xor_sync(0xffffffffu, send, m);
    }
  }
  double v = acc[0];
#pragma unroll
  for (; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}

// Scalars of a column, written by the last warp for everyone.
struct ResScal {
  double t, scl, delta;
};

// Place of column c in a row: groups of 64 columns, lane L of the group's warp
// holding columns 16 (L % 2) + L / 2 and 32 more (so that the lanes' records
// are consecutive in memory, see the polls) as a 16-byte pair.
__device__ __forceinline__ int res_pos(int c) {
  return (c & ~63) + 4 * (c & 15) + ((c >> 4) & 1) * 2 + ((c >> 5) & 1);
}

// One pending update and product on the NR rows from own row i: the rows'
// sums per warp go to red.  A warp takes its slots kmin .. kmax-1.
template <int KP, int NR>
__device__ __forceinline__ void res_pass(double* As, int ldS, const double4* xzr, double* red,
                                         const double2* x, const double2* v, const double2* w,
                                         double c1, double c2, double c3, double scl, int i,
                                         int kmin, int kmax) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double acc[NR], vr[NR], wr[NR];
#pragma unroll
  for (int u = 0; u < NR; ++u) {
    const double4 t4 = xzr[i + u];
    vr[u] = scl * t4.x;
    wr[u] = fma(c1, t4.y, fma(c2, t4.z, c3 * t4.x));
    acc[u] = 0.0;
  }
  double2* base = (double2*)(As + (size_t)i * ldS) + tid;
#pragma unroll
  for (int k = 0; k < KP; ++k) {
    if (k < kmin || k >= kmax) continue;
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      double2* p = base + u * (ldS / 2) + RT * k;
      double2 t = *p;
      t.x = fma(-vr[u], w[k].x, fma(-wr[u], v[k].x, t.x));
      t.y = fma(-vr[u], w[k].y, fma(-wr[u], v[k].y, t.y));
      *p = t;
      acc[u] = fma(t.x, x[k].x, fma(t.y, x[k].y, acc[u]));
    }
  }
  const double zc = wsum_slots<NR>(acc, lane);
  constexpr int W = 32 / NR;
  if (lane % W == 0) red[(i + lane / W) * RW + wid] = zc;
}

// KP column pairs per thread (S <= 2 RT KP); rows in blocks of RBLK.
template <int KP>
__global__ void __launch_bounds__(RT, 1) trd_resident_kernel(ResArgs a) {
  const int q = blockIdx.x, G = gridDim.x;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int S = a.n - a.k0, ldS = (S + 63) & ~63, k0 = a.k0;
  // own rows; those past S of the last block are zero
  const ResRows rows(q, G, S, a.nrow);
  const int nrow = rows.nrow;
  const int nblk = (nrow + RBLK - 1) / RBLK;
  extern __shared__ __align__(16) double rsm[];
  double* As = rsm;                                     // [nrow][ldS], columns at res_pos, zero past S
  double* red = As + (size_t)a.nrow * ldS;              // [nrow][RW] row sums per warp
  double4* xzr = (double4*)(red + (size_t)a.nrow * RW);  // [nrow] {x, z, r} of the pending column
  __shared__ __align__(16) double red2[RW], redn[RW];
  __shared__ double s_alpha, s_z1, s_r1;
  __shared__ ResScal s_sc;
  __shared__ int s_fail;

  if (*(volatile int*)a.err) return;  // an earlier step failed
  // rows from the lower triangle: down the column right of the diagonal,
  // across the columns left of it
  const double* A0 = a.A + (long long)k0 * (a.lda + 1);
  for (int i = 0; i < RBLK * nblk; ++i) {
    const int r = rows.row(i);
    for (int c = tid; c < ldS; c += RT) {
      double v = 0.0;
      if (c < S && r < S)
        v = (c >= r) ? A0[c + (long long)r * a.lda] : A0[r + (long long)c * a.lda];
      As[(size_t)i * ldS + res_pos(c)] = v;
    }
    if (tid == 0) xzr[i] = make_double4(r >= 1 && r < S ? A0[r] : 0.0, 0.0, 0.0, 0.0);
  }
  // this thread's columns: the current x, and v, w of the pending update
  double2 x[KP], v[KP], w[KP];
  const int kmax = (ldS / 64 - wid + RW - 1) / RW;  // slots of this warp
  auto col = [&](int k, int h) {
    return 64 * (wid + RW * k) + 32 * h + 16 * (lane & 1) + (lane >> 1);
  };
#pragma unroll
  for (int k = 0; k < KP; ++k) {
    const int ca = col(k, 0), cb = col(k, 1);
    x[k].x = (ca >= 1 && ca < S) ? A0[ca] : 0.0;
    x[k].y = (cb < S) ? A0[cb] : 0.0;
    v[k] = w[k] = make_double2(0.0, 0.0);
  }
  if (tid == 0) {
    s_fail = 0;
    if (q == 0) a.d[k0] = A0[0];
  }
  __syncthreads();

  // of the pending column: w_r = c1 z_r + c2 A(r, j+1) + c3 x_r, v_r = scl x_r
  double c1 = 0.0, c2 = 0.0, c3 = 0.0, scl = 0.0, w1 = 0.0;
  int i0 = 0, r0 = rows.row(0);  // first own row below row j
  for (int j = 0; j < S - 1; ++j) {
    const unsigned tag = (unsigned)(j + 1);
    if (r0 <= j) {
      r0 = rows.after(i0, r0);
      ++i0;
    }
    const bool pub = rows.writes(j, i0, r0);
    const int kmin = (j + 1) / (2 * RT);  // the slots before it are left of column j+1
    const int p1 = res_pos(j + 1);
    const bool at1 = tid + RT * kmin == p1 >> 1;  // holds column j+1, in slot kmin
    // the norm of x below alpha = x(j+1)
    double nrm = 0.0;
#pragma unroll
    for (int k = 0; k < KP; ++k) nrm = fma(x[k].x, x[k].x, fma(x[k].y, x[k].y, nrm));
    if (at1) {
      nrm = 0.0;
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        double x0 = x[k].x, x1 = x[k].y;
        if (k == kmin) {
          s_alpha = (p1 & 1) ? x1 : x0;
          if (p1 & 1) x1 = 0.0;
          else x0 = 0.0;
        }
        nrm = fma(x0, x0, fma(x1, x1, nrm));
      }
    }
    // own rows, whole blocks (the finished rows of the first one and the
    // rows past S come to nothing): the pending update and z = A x
    {
      int i = i0 - i0 % RBLK;
      const int ie = RBLK * nblk;
      for (; KP <= 2 && i + 8 <= ie; i += 8)
        res_pass<KP, 8>(As, ldS, xzr, red, x, v, w, c1, c2, c3, scl, i, kmin, kmax);
      for (; i + 4 <= ie; i += 4)
        res_pass<KP, 4>(As, ldS, xzr, red, x, v, w, c1, c2, c3, scl, i, kmin, kmax);
      if (i < ie) res_pass<KP, 2>(As, ldS, xzr, red, x, v, w, c1, c2, c3, scl, i, kmin, kmax);
    }
    nrm = wsum(nrm);
    if (lane == 0) redn[wid] = nrm;
    __syncthreads();
    // records {z_r, A(r, j+1)} of the own rows, two lanes per row, and the
    // row's {x, z, r} for the next pass
    ulonglong2* rec = a.rec + (size_t)(j & 1) * 2 * ldS;
    for (int t = 2 * i0 + tid; t < 2 * nrow; t += RT) {
      const int i = t >> 1;
      const double rv = As[(size_t)i * ldS + p1], zv = sum_warps(red + i * RW);
      st_tagged(rec + 2 * rows.row(i) + (t & 1), (t & 1) ? rv : zv, tag);
      if (!(t & 1)) {
        const double4 o = xzr[i];  // of column j-1
        const double vr = scl * o.x, wr = fma(c1, o.y, fma(c2, o.z, c3 * o.x));
        xzr[i] = make_double4(j ? fma(-w1, vr, o.z - wr) : o.x, zv, rv, 0.0);
      }
    }
    if (rows.retires(j, i0, r0)) return;
    if (wid == RW - 1) {
      // Householder reflector of x (LAPACK dlarfg), while the records travel
      const double xn2 = sum_warps(redn);
      const double alpha = s_alpha;
      ResScal sc;
      double beta;
      if (xn2 == 0.0) {
        sc.t = 0.0;
        beta = alpha;
        sc.scl = 0.0;
      } else {
        beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
        sc.t = (beta - alpha) / beta;
        sc.scl = 1.0 / (alpha - beta);
      }
      sc.delta = 1.0 - sc.scl * alpha;
      if (lane == 0) {
        s_sc = sc;
        if (pub) {
          a.e[k0 + j] = beta;
          a.tau[k0 + j] = sc.t;
        }
      }
    }
    // poll the values themselves
    double2 z[KP], r[KP];
    {
      const unsigned want = a.stall ? 0xffffffffu : tag;
      // a warp's 64 columns are 128 consecutive records: lane L reads record
      // L of each 32, z (L even) or A(., j+1) (L odd) of row L / 2, and the
      // lane pairs swap what the other one's column needs
      ulonglong2 t[KP][4];
      unsigned miss = 0;
#pragma unroll
      for (int k = 0; k < KP; ++k)
        if (k >= kmin && k < kmax) miss |= 1u << k;
      for (int it = 0; miss;) {
#pragma unroll
        for (int k = 0; k < KP; ++k)
          if (miss & (1u << k)) {
            const ulonglong2* p = rec + 128 * (wid + RW * k) + lane;
#pragma unroll
            for (int u = 0; u < 4; ++u) t[k][u] = ld_tagged(p + 32 * u);
          }
#pragma unroll
        for (int k = 0; k < KP; ++k)
          if (miss & (1u << k)) {
            bool ok = true;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int c = 64 * (wid + RW * k) + 16 * u + (lane >> 1);
              ok = ok && ((unsigned)t[k][u].y == want || c <= j || c >= S);
            }
            if (__all_sync(0xffffffffu, ok)) miss &= ~(1u << k);
          }
        if ((++it & 31) == 0 && miss && (it > a.spin || *(volatile int*)a.err)) {
          if (lane == 0) atomicExch(a.err, 1);
          s_fail = 1;
          break;
        }
      }
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        z[k] = r[k] = make_double2(0.0, 0.0);
        if (k >= kmin && k < kmax) {
          const bool odd = lane & 1;
          const double s0 = __shfl_xor_sync(
              0xffffffffu, __longlong_as_double((long long)(odd ? t[k][0].x : t[k][1].x)), 1);
          const double s1 = __shfl_xor_sync(
              0xffffffffu, __longlong_as_double((long long)(odd ? t[k][2].x : t[k][3].x)), 1);
          const int ca = col(k, 0), cb = col(k, 1);
          if (ca > j && ca < S) {
            z[k].x = odd ? s0 : __longlong_as_double((long long)t[k][0].x);
            r[k].x = odd ? __longlong_as_double((long long)t[k][1].x) : s0;
          }
          if (cb > j && cb < S) {
            z[k].y = odd ? s1 : __longlong_as_double((long long)t[k][2].x);
            r[k].y = odd ? __longlong_as_double((long long)t[k][3].x) : s1;
          }
        }
      }
    }
    double xz = 0.0;  // x^T z
#pragma unroll
    for (int k = 0; k < KP; ++k) xz = fma(x[k].x, z[k].x, fma(x[k].y, z[k].y, xz));
    if (at1) {
#pragma unroll
      for (int k = 0; k < KP; ++k)
        if (k == kmin) {
          s_z1 = (p1 & 1) ? z[k].y : z[k].x;
          s_r1 = (p1 & 1) ? r[k].y : r[k].x;
        }
    }
    xz = wsum(xz);
    if (lane == 0) red2[wid] = xz;
    __syncthreads();
    if (s_fail) return;
    // v^T y = scl^2 x^T A x + 2 scl delta (A x)(j+1) + delta^2 A(j+1, j+1); scl is not
    // squared: that overflows for a column of norm 1e-155 and less
    const double t = s_sc.t, delta = s_sc.delta, z1 = s_z1, r1 = s_r1;
    scl = s_sc.scl;
    xz = sum_warps(red2);
    const double vty = fma(scl, fma(scl, xz, 2.0 * delta * z1), delta * (delta * r1));
    const double a2 = -0.5 * t * t * vty;
    c1 = t * scl;
    c2 = t * delta;
    c3 = a2 * scl;
    w1 = fma(t, fma(scl, z1, delta * r1), a2);  // w(j+1)
    // v and w, and the next x = row j+1 from column j+2 on
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      v[k] = make_double2(scl * x[k].x, scl * x[k].y);
      w[k].x = fma(c1, z[k].x, fma(c2, r[k].x, c3 * x[k].x));
      w[k].y = fma(c1, z[k].y, fma(c2, r[k].y, c3 * x[k].y));
      x[k].x = fma(-w1, v[k].x, r[k].x - w[k].x);
      x[k].y = fma(-w1, v[k].y, r[k].y - w[k].y);
    }
    if (at1) {
#pragma unroll
      for (int k = 0; k < KP; ++k)
        if (k == kmin) {
          if (p1 & 1) x[k].y = 0.0;
          else x[k].x = 0.0;
        }
    }
    if (pub) {
      double* Vj = a.V + (long long)(k0 + j) * a.ldv + k0;
#pragma unroll
      for (int k = 0; k < KP; ++k) {  // 1 at row j+1, 0 above
        const int ca = col(k, 0), cb = col(k, 1);
        if (ca > j && ca < S) Vj[ca] = (ca == j + 1) ? 1.0 : v[k].x;
        if (cb > j && cb < S) Vj[cb] = (cb == j + 1) ? 1.0 : v[k].y;
      }
      if (tid == 0) a.d[k0 + j + 1] = fma(-2.0, w1, r1);
    }
  }
}

// Rows per CTA when S rows go to G CTAs in blocks of RBLK.
int res_rows(int S, int G) { return ((S + RBLK - 1) / RBLK + G - 1) / G * RBLK; }

size_t res_smem(int S, int G) {
  const size_t nrow = res_rows(S, G), ldS = (S + 63) & ~63;
  return nrow * (ldS + RW + 4) * sizeof(double);
}

size_t res_rec_bytes(int S) { return 4 * (size_t)((S + 63) & ~63) * sizeof(ulonglong2); }

size_t res_limit(int dev) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return optin > 2048 ? (size_t)optin - 1024 : 0;  // room for static shared
}

template <int KP>
int launch_res(imcom_ctx* ctx, ResArgs& a, int G, size_t smem) {
  // the limit, not this order's need: the attribute is process-wide, and contexts on
  // other threads must not lower it under one another's launches
  IMC_CUDA(cudaFuncSetAttribute(trd_resident_kernel<KP>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)res_limit(ctx->device)));
  void* args[] = {&a};
  IMC_CUDA(cudaLaunchCooperativeKernel((void*)trd_resident_kernel<KP>, G, RT, args, smem,
                                       ctx->stream));
  IMC_LAUNCH();
  return 0;
}

}  // namespace

size_t resident_bytes(int n) { return res_rec_bytes(std::min(n, RES_TRD_MAX)); }

int resident_max(imcom_ctx* ctx, int sms) {
  const size_t limit = res_limit(ctx->device);
  int S = RES_TRD_MAX;
  while (S > 2 && res_smem(S, sms) > limit) --S;
  return S;
}

int resident_tridiag(imcom_ctx* ctx, const DMat& Aw, DMat& Vall, double* d, double* e, double* tau,
                     int k0, int sms, void* scratch, int* err, long long spin, int stall) {
  const int n = (int)Aw.rows, S = n - k0;
  const int G = std::min((S + RBLK - 1) / RBLK, sms);
  ResArgs a{Aw.p, Aw.ld, Vall.p, Vall.ld, d, e, tau, n, k0, res_rows(S, G),
            (ulonglong2*)scratch, err, spin, stall};
  IMC_CUDA(cudaMemsetAsync(scratch, 0, res_rec_bytes(S), ctx->stream));  // tags of an earlier call
  const size_t smem = res_smem(S, G);
  if (S <= 2 * RT) return launch_res<1>(ctx, a, G, smem);
  if (S <= 4 * RT) return launch_res<2>(ctx, a, G, smem);
  return launch_res<4>(ctx, a, G, smem);
}

}  // namespace imcom
