// dgemm_tile.cuh -- the FP64 DMMA GEMM tile (see dgemm.cu), shared by the
// GEMM launchers of dgemm.cu and the grouped divide-and-conquer products of
// eigen_dc.cu.
#pragma once

#include "common.cuh"

namespace imcom {
namespace gemm {

constexpr int BM = 128, BN = 128, BK = 32, STAGES = 3, THREADS = 256;
constexpr int SKC = BK + 4;   // stride of a k-contiguous tile row
constexpr int SMC = BM + 4;   // stride of an m/n-contiguous tile row
constexpr int TILE_DBL = (BM * SKC > BK * SMC) ? BM * SKC : BK * SMC;  // 4608
constexpr int STAGE_DBL = 2 * TILE_DBL;
constexpr size_t SMEM_BYTES = (size_t)STAGES * STAGE_DBL * sizeof(double);

__device__ __forceinline__ void cp_async(double* dst, const double* src, int bytes, int vec) {
  unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  if (vec == 2)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(src), "r"(bytes));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// One operand tile.  KCONTIG: element (r, k) at P[k + r * ld] (r = m or n),
// stored S[r][k] (stride SKC).  Otherwise element (r, k) at P[r + k * ld],
// stored S[k][r] (stride SMC).  Out-of-range elements are zero-filled.  The
// copies of a stage come in BK / 4 pieces, which the main loop issues between
// its products; piece q of thread t is row (or k) t / PER + ROWS q.
template <bool KCONTIG, int VEC>
struct TileLoad {
  static constexpr int PER = (KCONTIG ? BK : BM) / VEC;  // copies per row (or k)
  static constexpr int ROWS = THREADS / PER;             // rows (or k) per round of copies
  static constexpr int ROUNDS = (KCONTIG ? BM : BK) / ROWS;
  static constexpr int PIECE = ROUNDS / (BK / 4);        // rounds per piece
  static_assert(THREADS % PER == 0 && ROUNDS % (BK / 4) == 0, "pieces of a stage");
  const double* base;  // this thread's first element of stage 0
  const double* P;
  long long ld;
  int dst, i0, o0, nrow;  // offset in the tile; own row (or k) and k (or row); rows in range

  __device__ __forceinline__ TileLoad(const double* P_, long long ld_, long long r0, long long k0,
                                      long long R) {
    P = P_;
    ld = ld_;
    i0 = threadIdx.x / PER;
    o0 = threadIdx.x % PER * VEC;
    dst = i0 * (KCONTIG ? SKC : SMC) + o0;
    base = KCONTIG ? P + (k0 + o0) + (r0 + i0) * ld : P + (r0 + o0) + (k0 + i0) * ld;
    nrow = (int)min((long long)BM, R - r0);
  }
  // piece q of the stage at depth kt BK, with `left` = K minus that depth
  __device__ __forceinline__ void piece(double* S, int kt, int left, int q) const {
    const double* src = base + (long long)kt * BK * (KCONTIG ? 1 : ld);
#pragma unroll
    for (int u = 0; u < PIECE; ++u) {
      const int i = (q * PIECE + u) * ROWS;
      const int v = KCONTIG ? (i0 + i < nrow ? min(VEC, left - o0) : 0)
                            : (i0 + i < left ? min(VEC, nrow - o0) : 0);
      cp_async(S + dst + i * (KCONTIG ? SKC : SMC), v > 0 ? src + i * ld : P, 8 * max(v, 0), VEC);
    }
  }
};

// LOWER: only output tiles with a row on or below the diagonal (row >= col)
// are computed; tiles strictly above it are left as they are (the symmetric
// rank-2k update of a matrix kept in its lower triangle, LAPACK dsyr2k 'L').
// One 128 x 128 output tile (rows m0.., columns n0..) of the K slice kz of
// nkz (split-K: partial sums go to slice kz of C when nkz > 1).
template <bool AK, bool BKC, int VEC, bool LOWER = false>
__device__ __forceinline__ void dgemm_tile(long long M, long long N, long long K, double alpha,
                                           const double* __restrict__ A, long long lda,
                                           const double* __restrict__ B, long long ldb,
                                           double beta, double* __restrict__ C, long long ldc,
                                           long long kchunk, long long m0, long long n0, int kz,
                                           int nkz) {
  extern __shared__ __align__(16) double smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp & 1, wn = warp >> 1;  // 2 x 4 warps
  const int g = lane >> 2, t = lane & 3;
  if (LOWER && m0 + BM <= n0) return;
  // split-K: this CTA covers k in [kb, ke); partial sums go to slice z of C
  const long long kb = (long long)kz * kchunk;
  const long long ke = min(K, kb + kchunk);
  if (nkz > 1) C += (size_t)kz * (size_t)ldc * (size_t)N;
  const int nk = ke > kb ? (int)((ke - kb + BK - 1) / BK) : 0;

  double acc[4][4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;
  // beta C is added in the epilogue.  Its tile is prefetched into L2 now (a
  // hint, no registers held), so the epilogue's loads hit L2 and the HBM
  // reads overlap the main loop instead of holding up the first MMA.
  const bool readc = nkz == 1 && beta != 0.0;
  if (readc) {
    // 128 columns x 128 rows: 8 lines of 128 bytes per column, 4 per thread
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int line = threadIdx.x + q * THREADS;
      const long long col = n0 + (line >> 3), row = m0 + (line & 7) * 16;
      if (row < M && col < N)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(C + row + col * ldc));
    }
  }

  auto stageA = [&](int s) { return smem + s * STAGE_DBL; };
  auto stageB = [&](int s) { return smem + s * STAGE_DBL + TILE_DBL; };

  const TileLoad<AK, VEC> la(A, lda, m0, kb, M);
  const TileLoad<BKC, VEC> lb(B, ldb, n0, kb, N);
  const int klen = (int)(ke - kb);
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) {
#pragma unroll 1
      for (int q = 0; q < BK / 4; ++q) {
        la.piece(stageA(s), s, klen - s * BK, q);
        lb.piece(stageB(s), s, klen - s * BK, q);
      }
    }
    cp_commit();
  }

  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    const double* As = stageA(kt % STAGES);
    const double* Bs = stageB(kt % STAGES);
    double* An = stageA((kt + STAGES - 1) % STAGES);
    double* Bn = stageB((kt + STAGES - 1) % STAGES);
    const bool more = kt + STAGES - 1 < nk;
    const int lnext = klen - (kt + STAGES - 1) * BK;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      // a piece of the next stage's copies between the products: issued all
      // together after them they cost a tenth of the main loop (both warps of
      // a scheduler leave the tensor pipe idle meanwhile)
      if (more) {
        la.piece(An, kt + STAGES - 1, lnext, kk / 4);
        lb.piece(Bn, kt + STAGES - 1, lnext, kk / 4);
      }
      double af[4][2], bf[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        int mr = wm * 64 + i * 16 + g;
        if (AK) {
          af[i][0] = As[mr * SKC + kk + t];
          af[i][1] = As[(mr + 8) * SKC + kk + t];
        } else {
          af[i][0] = As[(kk + t) * SMC + mr];
          af[i][1] = As[(kk + t) * SMC + mr + 8];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int nc = wn * 32 + j * 8 + g;
        bf[j] = BKC ? Bs[nc * SKC + kk + t] : Bs[(kk + t) * SMC + nc];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          asm volatile(
              "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
              "{%0,%1,%2,%3};\n"
              : "+d"(acc[i][j][0]), "+d"(acc[i][j][1]), "+d"(acc[i][j][2]), "+d"(acc[i][j][3])
              : "d"(af[i][0]), "d"(af[i][1]), "d"(bf[j]));
    }
    cp_commit();
  }
  cp_wait<0>();

  // one 16-row band at a time: its 16 C values are loaded together, then
  // combined and stored
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    double cv[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const long long row = m0 + wm * 64 + i * 16 + g + ((r >> 1) ? 8 : 0);
        const long long col = n0 + wn * 32 + j * 8 + 2 * t + (r & 1);
        cv[j][r] = (readc && row < M && col < N) ? C[row + col * ldc] : 0.0;
      }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const long long row = m0 + wm * 64 + i * 16 + g + ((r >> 1) ? 8 : 0);
        const long long col = n0 + wn * 32 + j * 8 + 2 * t + (r & 1);
        if (row < M && col < N)
          C[row + col * ldc] = readc ? fma(beta, cv[j][r], alpha * acc[i][j][r])
                                     : alpha * acc[i][j][r];
      }
  }
}

template <bool AK, bool BKC, int VEC, bool LOWER = false>
__global__ void __launch_bounds__(THREADS, 1)
dgemm_kernel(long long M, long long N, long long K, double alpha, const double* __restrict__ A,
             long long lda, const double* __restrict__ B, long long ldb, double beta,
             double* __restrict__ C, long long ldc, long long kchunk) {
  dgemm_tile<AK, BKC, VEC, LOWER>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, kchunk,
                                  (long long)blockIdx.x * BM, (long long)blockIdx.y * BN,
                                  (int)blockIdx.z, (int)gridDim.z);
}

// The same gm x gn x nkz tiles from a grid of at most a context's SM share:
// CTA b takes tiles b, b + gridDim.x, ... (row blocks fastest), so a context
// that shares the GPU with others keeps to about its share of the SMs.
template <bool AK, bool BKC, int VEC>
__global__ void __launch_bounds__(THREADS, 1)
dgemm_persist_kernel(long long M, long long N, long long K, double alpha,
                     const double* __restrict__ A, long long lda, const double* __restrict__ B,
                     long long ldb, double beta, double* __restrict__ C, long long ldc,
                     long long kchunk, int gm, int gn, int nkz) {
  const long long total = (long long)gm * gn * nkz;
  for (long long tile = blockIdx.x; tile < total; tile += gridDim.x) {
    __syncthreads();  // every warp is done with the previous tile's shared stages
    const long long xy = tile % ((long long)gm * gn);
    dgemm_tile<AK, BKC, VEC, false>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, kchunk,
                                    (xy % gm) * BM, (xy / gm) * BN,
                                    (int)(tile / ((long long)gm * gn)), nkz);
  }
}

// Products whose 128 x 128 tiles leave most SMs idle: 32 x 32 tiles of 4 warps
// (2 x 2, a warp 16 x 16), three stages of 32 deep, up to four CTAs per SM.  The sum
// over k runs in the same order as above, so without split-K the results are the
// same to the bit.
constexpr int SBM = 32, SSTRIDE = SBM + 4, STHREADS = 128, SSTAGES = 3;
static_assert(BK == SBM, "either order of a tile has 32 lines of 32");
constexpr int SSTAGE_DBL = 2 * SBM * SSTRIDE;
constexpr size_t SSMEM_BYTES = (size_t)SSTAGES * SSTAGE_DBL * sizeof(double);

// Microseconds of a product in small tiles (a step of 32 deep costs 0.7 us with
// one CTA on an SM, 0.42 per CTA with more) and in large ones (per step of 32, waves
// x depth).
inline double small_tiles_us(long long tiles, long long K, int sms) {
  const double per = 0.42 * (double)((tiles + sms - 1) / sms);
  return 2.5 + (double)((K + BK - 1) / BK) * (per > 0.7 ? per : 0.7);
}
inline double large_tiles_us(double steps) { return 3.0 + 0.14 * BK * steps; }

template <bool AK, bool BKC, int VEC>
__device__ __forceinline__ void dgemm_small_tile(int M, int N, int K, double alpha,
                                                 const double* __restrict__ A, long long lda,
                                                 const double* __restrict__ B, long long ldb,
                                                 double beta, double* __restrict__ C,
                                                 long long ldc, int m0, int n0) {
  extern __shared__ __align__(16) double smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = (warp & 1) * 16, wn = (warp >> 1) * 16, g = lane >> 2, t = lane & 3;
  constexpr int PER = SBM / VEC, LINES = STHREADS / PER;
  const int li = tid / PER, lo = tid % PER * VEC;
  // lines of a tile: rows of k if k is contiguous, else k of rows
  auto load = [&](double* S, const double* P, long long ld, bool kc, int r0, int R, int k0) {
#pragma unroll
    for (int i = li; i < SBM; i += LINES) {
      const int r = r0 + (kc ? i : lo), k = k0 + (kc ? lo : i);
      const int v = kc ? (r < R ? min(VEC, K - k) : 0) : (k < K ? min(VEC, R - r) : 0);
      cp_async(S + i * SSTRIDE + lo, v > 0 ? (kc ? P + k + r * ld : P + r + k * ld) : P,
               8 * max(v, 0), VEC);
    }
  };
  const int nk = (K + BK - 1) / BK;
  double acc[2][4] = {};
#pragma unroll
  for (int s = 0; s < SSTAGES - 1; ++s) {
    if (s < nk) {
      load(smem + s * SSTAGE_DBL, A, lda, AK, m0, M, s * BK);
      load(smem + s * SSTAGE_DBL + SSTAGE_DBL / 2, B, ldb, BKC, n0, N, s * BK);
    }
    cp_commit();
  }
  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<SSTAGES - 2>();
    __syncthreads();
    const int nx = kt + SSTAGES - 1;
    if (nx < nk) {
      double* Sn = smem + nx % SSTAGES * SSTAGE_DBL;
      load(Sn, A, lda, AK, m0, M, nx * BK);
      load(Sn + SSTAGE_DBL / 2, B, ldb, BKC, n0, N, nx * BK);
    }
    cp_commit();
    const double* As = smem + kt % SSTAGES * SSTAGE_DBL;
    const double* Bs = As + SSTAGE_DBL / 2;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      const int k = kk + t;
      const double a0 = AK ? As[(wm + g) * SSTRIDE + k] : As[k * SSTRIDE + wm + g];
      const double a1 = AK ? As[(wm + g + 8) * SSTRIDE + k] : As[k * SSTRIDE + wm + g + 8];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int nc = wn + 8 * j + g;
        const double b = BKC ? Bs[nc * SSTRIDE + k] : Bs[k * SSTRIDE + nc];
        asm volatile(
            "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
            "{%0,%1,%2,%3};\n"
            : "+d"(acc[j][0]), "+d"(acc[j][1]), "+d"(acc[j][2]), "+d"(acc[j][3])
            : "d"(a0), "d"(a1), "d"(b));
      }
    }
  }
  cp_wait<0>();
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = m0 + wm + g + ((r >> 1) ? 8 : 0), col = n0 + wn + 8 * j + 2 * t + (r & 1);
      if (row < M && col < N) {
        double* c = C + row + col * ldc;
        *c = beta != 0.0 ? fma(beta, *c, alpha * acc[j][r]) : alpha * acc[j][r];
      }
    }
}

// CTA b takes tiles b, b + gridDim.x, ... (a context on a share of the SMs has fewer
// CTAs than tiles).
template <bool AK, bool BKC, int VEC>
__global__ void __launch_bounds__(STHREADS)
dgemm_small_kernel(int M, int N, int K, double alpha, const double* __restrict__ A, long long lda,
                   const double* __restrict__ B, long long ldb, double beta,
                   double* __restrict__ C, long long ldc) {
  const int gm = (M + SBM - 1) / SBM, total = gm * ((N + SBM - 1) / SBM);
  for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
    __syncthreads();  // every warp is done with the previous tile's shared stages
    dgemm_small_tile<AK, BKC, VEC>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, tile % gm * SBM,
                                   tile / gm * SBM);
  }
}

}  // namespace gemm
}  // namespace imcom
