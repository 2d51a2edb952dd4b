// stacks.cu -- H = T^T I for several image stacks on the FP64 tensor path
// (imcom_build_image, imcom_matrix.f90:754-790, for S stacks that share T).
//
// T (n x m) and the stacks (n x S) are both contiguous along the summed
// dimension.  A CTA owns 32 output pixels and NT stacks; each of its eight warps
// takes an eighth of every 64-deep stage, holding 32 x NT sums in m16n8k4 DMMA
// tiles, and the eight slices are added through shared memory at the end.  So T
// crosses HBM once for up to 64 stacks, the stacks come from L2, and 32 pixels
// per CTA give one CTA per SM at m of about 4700 without splitting the sum; other
// sizes split it over a few CTAs and add the partial sums in a second kernel.
//
// A sum's error grows with its length, and a DMMA adds to its accumulator one
// product at a time.  So each stage's products (8 per slice) are summed by
// themselves and then added to the slice's sum; tiles of more than 48 stacks,
// which have no registers for that, take a depth of 2048 at a time instead.
// Relative error of the result against 128-bit sums, n = m = 4096 (the FMA kernel
// and the GEMM for comparison): 3.1e-16 (4.0e-16) up to 32 stacks, 3.1e-16 (7.3e-16)
// up to 48, 5.5e-16 (7.3e-16) up to 64; one chain per slice: 7.6e-16.
//
// What bounds it: HBM (one read of T) up to about 16 stacks, the FP64 tensor
// pipe and the latency of a stage above.  The 128 x 128 GEMM tile computes 128
// stacks whatever S is, and the FMA kernel (solve.cu) reads T once per eight
// stacks and is bound by its shared-memory reads.  Measured, 48 stacks at 3999 x
// 4225, us: 178 in the GEMM, 74 here (1.6 GFLOP, 45 us at the DGEMM rate; 63 with one
// chain per slice of a 16-deep step and 1.4e-15 of error where the GEMM has 1.1e-15).
// n = m = 4096 in a loop of calls, us a call:
//   S          2     8    16    32    48    64
//   GEMM     169   169   169   169   169   169
//   FMA       52    69   113   190
//   here      39    36    48    71    91   110
#include <algorithm>

#include "common.cuh"
#include "dgemm_tile.cuh"

namespace imcom {

__global__ void splitk_reduce_kernel(const double* __restrict__ part, long long ldp, int splits,
                                     long long M, long long N, double alpha, double beta,
                                     double* __restrict__ C, long long ldc);

namespace {

constexpr int ST_THREADS = 256, ST_BM = 32, ST_BK = 64;
constexpr int ST_WK = 8, ST_MT = 2;        // warps, each an eighth of a stage's depth; its pixel tiles
constexpr int ST_SK = ST_BK + 4;           // shared stride: fragment loads hit distinct banks
constexpr int ST_KW = ST_BK / ST_WK;       // depth per warp and stage

template <int NT>
constexpr int st_stage() {
  return (ST_BM + NT) * ST_SK;
}
// Stages in flight: four, or what fits with the sums' exchange area.
template <int NT>
constexpr int st_stages() {
  return NT <= 32 ? 4 : 3;
}
// Whether each stage's products are summed by themselves first (twice the registers).
template <int NT>
constexpr bool st_staged() {
  return NT <= 48;
}
template <int NT>
constexpr size_t st_smem() {
  const size_t pipe = (size_t)st_stages<NT>() * st_stage<NT>();
  const size_t sums = (size_t)ST_WK * ST_BM * (NT + 1);
  return (pipe > sums ? pipe : sums) * sizeof(double);
}

// Tile (bx, by) of slice bz of nz of the sum.  VI: doubles per copy of the stacks (2
// where their columns are 16-byte aligned, else 1); T's columns always are.
template <int NT, int VI>
__device__ __forceinline__ void stacks_tile(const double* __restrict__ T, long long ldt,
                                            const double* __restrict__ I, long long ldi,
                                            double* __restrict__ H, long long ldh, int n, int m,
                                            int S, int kchunk, int bx, int by, int bz, int nz) {
  extern __shared__ __align__(16) double st_sm[];
  constexpr int STG = st_stages<NT>(), SZ = st_stage<NT>();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int a0 = bx * ST_BM, s0 = by * NT;
  const int kb = bz * kchunk, ke = min(n, kb + kchunk);
  const int nk = (ke - kb + ST_BK - 1) / ST_BK;
  const int na = min(ST_BM, m - a0), ns = min(NT, S - s0);
  T += (long long)a0 * ldt;
  I += (long long)s0 * ldi;
  if (nz > 1) H += (size_t)bz * (size_t)ldh * (size_t)S;  // partial slice

  // Quarter u of stage kt: pixel rows 8 u .. 8 u + 7 of T and every fourth group of
  // the stacks' copies.  Rows past the last one copy it again (their sums are not
  // written), so only the last stage's depth needs a test.
  const int tr = tid / (ST_BK / 2), tk = tid % (ST_BK / 2) * 2;
  const double* tsrc = T + kb + tk;
  double* tdst = st_sm + tr * ST_SK + tk;
  const int ir = tid / (ST_BK / VI), ik = tid % (ST_BK / VI) * VI;
  constexpr int IROWS = ST_THREADS / (ST_BK / VI);  // stacks per group of copies
  const double* isrc = I + kb + ik;
  double* idst = st_sm + (ST_BM + ir) * ST_SK + ik;
  auto load = [&](int kt, int u) {
    const int st = (kt % STG) * SZ, left = ke - kb - kt * ST_BK;
    const double* ts = tsrc + (long long)min(tr + 8 * u, na - 1) * ldt + kt * ST_BK;
    double* td = tdst + st + 8 * u * ST_SK;
    if (left >= ST_BK) gemm::cp_async(td, ts, 16, 2);
    else gemm::cp_async(td, left > tk ? ts : T, 8 * max(0, min(left - tk, 2)), 2);
#pragma unroll
    for (int q = u; q < NT / IROWS; q += 4) {
      const double* is = isrc + (long long)min(ir + IROWS * q, ns - 1) * ldi + kt * ST_BK;
      double* id = idst + st + IROWS * q * ST_SK;
      if (left >= ST_BK) gemm::cp_async(id, is, 8 * VI, VI);
      else gemm::cp_async(id, left > ik ? is : I, 8 * max(0, min(left - ik, VI)), VI);
    }
  };
  static_assert(ST_BM == 16 * ST_MT && ST_THREADS / (ST_BK / 2) == 8 && ST_KW == 8,
                "quarters of a stage, two at each of a warp's two steps");

  // the sums, and those of the current stage
  constexpr int R = st_staged<NT>() ? 1 : 0;
  double sum[1 + R][ST_MT][NT / 8][4];
#pragma unroll
  for (int i = 0; i < ST_MT; ++i)
#pragma unroll
    for (int j = 0; j < NT / 8; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) sum[0][i][j][r] = sum[R][i][j][r] = 0.0;
#pragma unroll
  for (int s = 0; s < STG - 1; ++s) {
    if (s < nk)
      for (int u = 0; u < 4; ++u) load(s, u);
    gemm::cp_commit();
  }
  for (int kt = 0; kt < nk; ++kt) {
    gemm::cp_wait<STG - 2>();
    __syncthreads();
    const double* sa = st_sm + (kt % STG) * SZ + g * ST_SK + warp * ST_KW + t;
    const double* sb = sa + ST_BM * ST_SK;
#pragma unroll
    for (int kk = 0; kk < ST_KW; kk += 4) {
      // the next stage's copies between the products, which leave most issue
      // slots free
      if (kt + STG - 1 < nk) {
        load(kt + STG - 1, kk / 2);
        load(kt + STG - 1, kk / 2 + 1);
      }
      double f[ST_MT][2];
#pragma unroll
      for (int i = 0; i < ST_MT; ++i) {
        f[i][0] = sa[16 * i * ST_SK + kk];
        f[i][1] = sa[(16 * i + 8) * ST_SK + kk];
      }
#pragma unroll
      for (int j = 0; j < NT / 8; ++j) {
        const double b = sb[8 * j * ST_SK + kk];
#pragma unroll
        for (int i = 0; i < ST_MT; ++i) {
          double* c = sum[R][i][j];
          asm volatile(
              "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
              "{%0,%1,%2,%3};\n"
              : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
              : "d"(f[i][0]), "d"(f[i][1]), "d"(b));
        }
      }
    }
    gemm::cp_commit();
    if (R) {
#pragma unroll
      for (int i = 0; i < ST_MT; ++i)
#pragma unroll
        for (int j = 0; j < NT / 8; ++j)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            sum[0][i][j][r] += sum[R][i][j][r];
            sum[R][i][j][r] = 0.0;
          }
    }
  }
  gemm::cp_wait<0>();
  __syncthreads();
  // the depth slices' sums, [slice][pixel][stack]
  double* sums = st_sm + (size_t)warp * ST_BM * (NT + 1);
#pragma unroll
  for (int i = 0; i < ST_MT; ++i)
#pragma unroll
    for (int j = 0; j < NT / 8; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r)
        sums[(16 * i + g + ((r >> 1) ? 8 : 0)) * (NT + 1) + 8 * j + 2 * t + (r & 1)] =
            sum[0][i][j][r];
  __syncthreads();
  for (int e = tid; e < ST_BM * NT; e += ST_THREADS) {
    const int r = e % ST_BM, s = e / ST_BM;
    if (r < na && s < ns) {
      const double* p = st_sm + r * (NT + 1) + s;
      constexpr int Z = ST_BM * (NT + 1);
      H[(a0 + r) + (long long)(s0 + s) * ldh] = ((p[0] + p[Z]) + (p[2 * Z] + p[3 * Z])) +
                                                ((p[4 * Z] + p[5 * Z]) + (p[6 * Z] + p[7 * Z]));
    }
  }
}

template <int NT, int VI>
__global__ void __launch_bounds__(ST_THREADS)
stacks_mma_kernel(const double* __restrict__ T, long long ldt, const double* __restrict__ I,
                  long long ldi, double* __restrict__ H, long long ldh, int n, int m, int S,
                  int kchunk) {
  stacks_tile<NT, VI>(T, ldt, I, ldi, H, ldh, n, m, S, kchunk, blockIdx.x, blockIdx.y, blockIdx.z,
                      gridDim.z);
}

// The same tiles, gx x gy x gz of them, in turn on the CTAs of a share of the SMs.
template <int NT, int VI>
__global__ void __launch_bounds__(ST_THREADS)
stacks_share_kernel(const double* __restrict__ T, long long ldt, const double* __restrict__ I,
                    long long ldi, double* __restrict__ H, long long ldh, int n, int m, int S,
                    int kchunk, int gx, int gy, int gz) {
  for (int b = blockIdx.x; b < gx * gy * gz; b += gridDim.x) {
    __syncthreads();  // every warp is done with the previous tile's shared memory
    stacks_tile<NT, VI>(T, ldt, I, ldi, H, ldh, n, m, S, kchunk, b % gx, b / gx % gy, b / gx / gy,
                        gz);
  }
}

template <int NT>
int launch_nt(imcom_ctx* ctx, int S, const double* dI, long long ldi, double* dH, long long ldh) {
  const int n = ctx->n, m = ctx->m, sms = sm_count(ctx);
  const long long tiles = (long long)((m + ST_BM - 1) / ST_BM) * ((S + NT - 1) / NT);
  // slices of the sum: the fewest rounds of stages per SM, each further slice
  // charged with the second kernel (about 3 us, 12 stages) and its partial
  // sums (about 2 stages per million)
  const int ksteps = (n + ST_BK - 1) / ST_BK;
  int splits = 1;
  double best = 0.0;
  for (int s = 1; s <= 16 && ksteps >= 4 * s; ++s) {
    double cost = (double)((tiles * s + sms - 1) / sms) * ((ksteps + s - 1) / s);
    if (s > 1) cost += 12.0 + 2e-6 * s * (double)m * S;
    if (s == 1 || cost < best) {
      best = cost;
      splits = s;
    }
  }
  // (tiles that do not sum each stage by itself take a depth of 2048 at a time)
  if (!st_staged<NT>()) splits = std::max(splits, (n + 2047) / 2048);
  const int kchunk = (ksteps + splits - 1) / splits * ST_BK;
  splits = (n + kchunk - 1) / kchunk;
  double* out = dH;
  long long ldo = ldh;
  if (splits > 1) {
    ldo = pad_ld(m);
    IMC_TRY(ensure_buf(ctx, &ctx->gemm_ws, ctx->gemm_ws_bytes,
                       (size_t)splits * (size_t)ldo * (size_t)S * sizeof(double)));
    out = (double*)ctx->gemm_ws;
  }
  const bool v2 = ((uintptr_t)dI & 15) == 0 && ldi % 2 == 0;
  const int gx = (m + ST_BM - 1) / ST_BM, gy = (S + NT - 1) / NT;
  const size_t smem = st_smem<NT>();
  // on a share of the SMs, products bound by the tensor pipe keep to it: one CTA per
  // SM, as the GEMM (few stacks are bound by the read of T)
  bool done = false;
  if constexpr (NT > 32) {
    if (ctx->sm_share > 0) {
      auto k = v2 ? stacks_share_kernel<NT, 2> : stacks_share_kernel<NT, 1>;
      IMC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      k<<<(unsigned)std::min<long long>(tiles * splits, sms), ST_THREADS, smem, ctx->stream>>>(
          ctx->T.p, ctx->T.ld, dI, ldi, out, ldo, n, m, S, kchunk, gx, gy, splits);
      done = true;
    }
  }
  if (!done) {
    auto k = v2 ? stacks_mma_kernel<NT, 2> : stacks_mma_kernel<NT, 1>;
    IMC_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k<<<dim3((unsigned)gx, (unsigned)gy, (unsigned)splits), ST_THREADS, smem, ctx->stream>>>(
        ctx->T.p, ctx->T.ld, dI, ldi, out, ldo, n, m, S, kchunk);
  }
  IMC_LAUNCH();
  if (splits > 1) {
    const dim3 g2((unsigned)std::min((m + 255) / 256, 64), (unsigned)S);
    splitk_reduce_kernel<<<g2, 256, 0, ctx->stream>>>(out, ldo, splits, m, S, 1.0, 0.0, dH, ldh);
    IMC_LAUNCH();
  }
  return 0;
}

}  // namespace

int stacks_mma(imcom_ctx* ctx, int S, const double* dI, long long ldi, double* dH,
               long long ldh) {
  // the narrowest tile that takes the stacks in the fewest reads of T
  const int passes = (S + 63) / 64, per = (S + passes - 1) / passes;
  if (per <= 8) return launch_nt<8>(ctx, S, dI, ldi, dH, ldh);
  if (per <= 16) return launch_nt<16>(ctx, S, dI, ldi, dH, ldh);
  if (per <= 24) return launch_nt<24>(ctx, S, dI, ldi, dH, ldh);
  if (per <= 32) return launch_nt<32>(ctx, S, dI, ldi, dH, ldh);
  if (per <= 40) return launch_nt<40>(ctx, S, dI, ldi, dH, ldh);
  if (per <= 48) return launch_nt<48>(ctx, S, dI, ldi, dH, ldh);
  if (per <= 56) return launch_nt<56>(ctx, S, dI, ldi, dH, ldh);
  return launch_nt<64>(ctx, S, dI, ldi, dH, ldh);
}

}  // namespace imcom
