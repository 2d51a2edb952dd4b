// eigen_panel.cu -- one panel (32 columns) of the Householder
// tridiagonalisation (LAPACK dlatrd, lower) in one cooperative kernel.
//
// Per column j every row of the trailing matrix needs z = A22 x for the raw
// column x = A(j+1:n, j), with A22 as it was at the panel's start, and the
// panel's corrections.  Two exchanges of tagged records (tagged.cuh) replace
// grid barriers:
//   stream:  every CTA sums its share of the lower triangle's tiles, TR rows
//            by CW columns, through registers: row sums sum_c A(r, c) x(c)
//            and column sums sum_{r > c} A(r, c) x(r);
//   exchange 1: the row sums (added over the CTA) and each tile's column sums
//            go out as records; the CTA that owns row r collects the records
//            that cover it;
//   rows:    the owner forms w(r) and the next column's x(r) = A(r, j+1) -
//            V W^T - W V^T, with y0 = A22 v = scl z + delta A22(:, j+1) for v =
//            scl x + delta e_{j+1};
//   exchange 2: x(r) goes out; every CTA stages the whole of it in shared
//            memory for the next column's stream.
// What the rows step needs of all rows arrives beside that: x^T A22 x (one
// record per CTA, published with exchange 1), row j+1 of V and W (from its
// owner) and the dot products of x with the panel's V and W and its norm
// (per CTA, summed by one CTA each while the others stream).  The eighth warp
// collects these and forms the reflector's scalars beside the stream and
// exchange 1.  Sums are taken in a fixed order, so results do not depend on
// timing.
//
// Records carry the column's number and alternate between two buffers: a
// buffer is written again two columns later, by a CTA that has since read a
// record of every other CTA, each of which was published after its own reads
// of the older column.  Polls are bounded and set the error word.
//
// What bounds it: the stream, from L2 up to about 5400 rows (9.2 TB/s alone at
// 4096 rows, 7.3 us) and from HBM above (6.6 TB/s, 41 us at 8192), and about 6 us
// per column of exchanges and sums.  Microseconds per column with the trailing
// update, before (grid barriers, tiles through shared memory) and now: from
// 8192 to 2048 rows 43.8 -> 32.9, from 4096 18.5 -> 12.6, from 3000 19.1 -> 11.0,
// from 1453 down 8.5 -> 7.4, from 512 down 8.1 either way (8.0 to 8.2 by machine; 16 to
// 32 CTAs there instead of all: 7.9).  Row sums that wait for the
// reflector's scalars before they go out cost 1.2 us per column more; dots
// laid out by sum and not by CTA (lines that eight CTAs write), 0.6; fewer rows
// per owner than a warp has lanes (16 at 2100 rows), 0.5.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "eigen.cuh"
#include "tagged.cuh"

namespace imcom {

namespace {

constexpr int TR = 128, CW = 8;        // rows and columns of a tile
constexpr int CPB = TR / CW;           // column chunks per row block along the diagonal
constexpr int NWK = 7;                 // worker warps
constexpr int PT = 32 * (NWK + 1);     // threads: the workers and the service warp
constexpr int NB = TRD_NB;
constexpr int HP = (NB + NWK - 1) / NWK;  // panel columns per worker warp
constexpr int NDOT = 72;               // records per CTA: 2 NB dots, the norm, padding
constexpr int DOT_NRM = 2 * NB;

struct PanelArgs {
  double* A;
  long long lda;
  double* V;  // n x n: column j holds v_j (zero above row j+1, 1 at row j+1)
  long long ldv;
  double* W;  // n x NB panel
  long long ldw;
  double *d, *e, *tau;
  ulonglong2* xrec;    // [2][ldr] x
  ulonglong2* colrec;  // [2][rbmax][ldr] column sums of a row block
  ulonglong2* rowrec;  // [2][rbmax + G][TR] row sums of a CTA in a row block
  ulonglong2* vtyrec;  // [2][G] x^T A22 x
  ulonglong2* dotrec;  // [2][G][NDOT] dots of the own rows: x W_p, x V_p, x x
  ulonglong2* sumrec;  // [2][NDOT] their sums
  ulonglong2* vwrec;   // [2][2 NB] row j+1: V, W
  int* err;
  int n, k, b, rp, nseg;
  long long ldr, rbmax;
  long long spin;
  int stall;  // test of the bounded polls: the first x never comes
};

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ double ld_cg(const double* p) { return __ldcg(p); }

// Kept where it stands: a tile's loads are issued before the products of the
// tile before it.
__device__ __forceinline__ double2 ld2_now(const double* p) {
  double2 v;
  asm volatile("ld.global.cg.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

template <int ID, int N>
__device__ __forceinline__ void bar() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}

// Tiles of the trailing matrix of column j, on or below the diagonal, counted
// row block by row block.  Row block rb is the TR rows from base + rb TR, at or
// above j + 1, so that the row blocks end at n rounded up to 8 and none is ragged
// (rows n and up are zero in the working matrix, x is zero up to row j); base is
// j + 1 rounded down to 8 where that would start above the matrix.  It has the
// column chunks ch0 <= ch < end(rb), counted from base.  CTA q of G takes the
// tiles floor(q nt / G) .. floor((q + 1) nt / G) - 1 (G at most nt).
struct Tiles {
  int base, ch0, RB, NC, rbc, tri, nt, G;
  __device__ __forceinline__ Tiles(int n, int j, int ctas) {
    const int n8 = (n + 7) & ~7;
    base = n8 - (n8 - (j + 1) + TR - 1) / TR * TR;
    if (base < 0) base = (j + 1) & ~7;
    ch0 = (j + 1 - base) / CW;
    const int R = n - base;
    RB = (R + TR - 1) / TR;
    NC = (R + CW - 1) / CW;
    rbc = min(RB, max(0, (NC - 1) / CPB));  // row blocks with CPB (rb + 1) chunks
    tri = CPB * rbc * (rbc + 1) / 2 - ch0 * rbc;
    nt = tri + (RB - rbc) * (NC - ch0);
    G = min(ctas, nt);
  }
  __device__ __forceinline__ int end(int rb) const { return min(NC, CPB * (rb + 1)); }  // one past the last chunk
  __device__ __forceinline__ int first(int rb) const {
    return rb <= rbc ? CPB * rb * (rb + 1) / 2 - ch0 * rb : tri + (rb - rbc) * (NC - ch0);
  }
  __device__ __forceinline__ int start(int q) const {
    if (q >= G) return nt;
    return nt < 10000000 ? (int)((unsigned)q * (unsigned)nt / (unsigned)G)
                         : (int)((long long)q * nt / G);
  }
  __device__ __forceinline__ int cta(int tile) const {
    return nt < 10000000 ? (int)((((unsigned)tile + 1) * (unsigned)G - 1) / (unsigned)nt)
                         : (int)((((unsigned long long)tile + 1) * G - 1) / (unsigned)nt);
  }
  __device__ __forceinline__ void decode(int tile, int& rb, int& ch) const {
    if (tile < tri) {
      const float h = (float)(CPB / 2 - ch0);
      int q = (int)((sqrtf(h * h + (float)(2 * CPB) * (float)tile) - h) / (float)CPB);
      q = max(0, min(q, rbc - 1));
      while (first(q + 1) <= tile) ++q;
      while (first(q) > tile) --q;
      rb = q;
      ch = ch0 + tile - first(q);
    } else {
      rb = rbc + (tile - tri) / (NC - ch0);
      ch = ch0 + (tile - tri) % (NC - ch0);
    }
  }
};

// A warp's tiles of one column: the next one to sum and the end.
struct Walk {
  int tile, end, rb, ch;
  __device__ __forceinline__ Walk(const Tiles& tl, int q, int w) {
    const int T0 = tl.start(q), T1 = tl.start(q + 1);
    tile = T0 + (T1 - T0) * w / NWK;
    end = T0 + (T1 - T0) * (w + 1) / NWK;
    rb = ch = 0;
    if (tile < end) tl.decode(tile, rb, ch);
  }
};

// MODE 0: the column's x and the own rows of V and W are kept in shared
// memory; 1: x only; 2: neither (x is read from its records).
template <int MODE>
__global__ void __launch_bounds__(PT, 1) trd_panel_kernel(PanelArgs a) {
  constexpr bool XS = MODE <= 1, VS = MODE == 0;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int q = blockIdx.x, G = gridDim.x;
  const int n = a.n, k = a.k, rp = a.rp;
  const long long lda = a.lda;
  double* A = a.A;
  const bool service = wid == NWK;
  // own rows r0 .. r0 + nr - 1, in rounds of 32 (a lane each), a round per worker
  // warp at a time; the CTAs that own any
  const int r0 = k + q * rp, nr = max(0, min(rp, n - r0));
  const int rounds = (rp + 31) / 32, nown = (n - k + rp - 1) / rp;
  const bool owner = nr > 0;
  extern __shared__ __align__(16) double psm[];
  double* xs = psm;                                                 // x from row base
  double* rs = xs + (XS ? n - k + 3 * TR : 0) / 2 * 2;         // [NWK][nseg][TR]
  const int held = min(rounds, NWK);
  double* sm_y = rs + (size_t)NWK * a.nseg * TR;                    // [held][NWK][32]
  double* sm_c = sm_y + (size_t)held * NWK * 32;
  double* sm_u = sm_c + (size_t)held * NWK * 32;
  double* sm_a = sm_u + (size_t)held * NWK * 32;                    // [rounds][32] next x
  double* sm_V = sm_a + rounds * 32;                                // [rounds 32][NB + 1]
  double* sm_W = sm_V + (VS ? rounds * 32 * (NB + 1) : 0);
  __shared__ double s_p[NB], s_q[NB], s_rowV[NB], s_rowW[NB];  // W^T v, V^T v, row j+1
  __shared__ double s_t, s_scl, s_delta, s_al2, s_w1;
  __shared__ double s_vty[NWK];
  __shared__ int s_rb0[NWK], s_ns[NWK];  // row blocks of the warps' tiles
  // a poll failed: [2] between a column's barriers 1 and 2 of all warps, [parity]
  // before barrier 1; read only after a barrier past which it is not set
  __shared__ int s_fail[3];
  auto own_V = [&](int l, int p) {
    return VS ? sm_V[l * (NB + 1) + p] : ld_cg(a.V + (r0 + l) + (long long)(k + p) * a.ldv);
  };
  auto own_W = [&](int l, int p) {
    return VS ? sm_W[l * (NB + 1) + p] : ld_cg(a.W + (r0 + l) + (long long)p * a.ldw);
  };
  auto fail = [&](int which) { s_fail[which] = 1; };
  if (*(volatile int*)a.err) return;  // an earlier panel failed
  if (tid == 0) {
    s_fail[0] = s_fail[1] = s_fail[2] = 0;
    if (q == 0) a.d[k] = A[(long long)k * (lda + 1)];
  }
  // column k as the first x, and its norm below row k+1
  if (wid == 0) {
    double nrm = 0.0;
    for (int rd = 0; rd < rounds; ++rd) {
      const int l = 32 * rd + lane, r = r0 + l;
      if (l < nr && r > k) {
        const double v = ld_cg(A + r + (long long)k * lda);
        st_tagged(a.xrec + r, v, (unsigned)(k + 1));
        if (r >= k + 2) nrm += v * v;
      }
    }
    nrm = wsum(nrm);
    if (lane == 0 && owner) st_tagged(a.dotrec + (size_t)q * NDOT + DOT_NRM, nrm, (unsigned)(k + 1));
  }
  __syncthreads();
  // The workers and the service warp run the same columns and meet at three
  // barriers in each (one in a CTA that owns no rows).
  if (service) {
    for (int i = 0; i < a.b; ++i) {
      const int j = k + i, par = i & 1;
      const unsigned tag = (unsigned)(j + 1);
      const ulonglong2* xrec = a.xrec + par * a.ldr;
      const ulonglong2* colrec = a.colrec + par * a.rbmax * a.ldr;
      const ulonglong2* rowrec = a.rowrec + par * (a.rbmax + G) * TR;
      const Tiles cur(n, j, G);
      double sc_t = 0, sc_scl = 0, sc_delta = 0, a11 = 0, qp = 0, corr1 = 0;
      if (i > 0 && owner) {
        // this column's dots with W and V over the own rows, a lane per panel
        // column, and its norm
        double sw = 0.0, sv = 0.0, nrm = 0.0;
        const int p = min(lane, i - 1);
#pragma unroll 8
        for (int l = 0; l < nr; ++l) {
          const double am = sm_a[l];
          sw = fma(am, own_W(l, p), sw);
          sv = fma(am, own_V(l, p), sv);
          nrm = fma(am, am, nrm);
        }
        ulonglong2* dr = a.dotrec + (size_t)(par * G + q) * NDOT;
        if (lane < i) {
          st_tagged(dr + 2 * lane, sw, tag);
          st_tagged(dr + 2 * lane + 1, sv, tag);
        }
        if (lane == 0) st_tagged(dr + DOT_NRM, nrm, tag);
      }
      // this CTA's share of the dots' sums (per owner, in order): a lane per owner,
      // with few owners several sums at a time
      const ulonglong2* drec = a.dotrec + (size_t)par * G * NDOT;
      auto sum_of = [&](int e) { return e < 2 * i ? e : DOT_NRM; };
      if (nown > 16) {
        for (int e = q; e <= 2 * i; e += G) {
          double s = 0.0;
          for (int c = lane; c < nown; c += 160) {
            double v[5];
            if (!poll_records<5>([&](int u) { return drec + (size_t)(c + 32 * u) * NDOT + sum_of(e); },
                                 [&](int u) { return c + 32 * u < nown; }, tag, v, a.spin, a.err))
              fail(par);
#pragma unroll
            for (int u = 0; u < 5; ++u) s += v[u];
          }
          s = wsum(s);
          if (lane == 0) st_tagged(a.sumrec + par * NDOT + sum_of(e), s, tag);
        }
      } else {
        const int gw = nown > 8 ? 16 : nown > 4 ? 8 : nown > 2 ? 4 : nown;
        const int c = lane & (gw - 1);
        for (int e0 = q; e0 <= 2 * i; e0 += G * (32 / gw) * 5) {
          const int e = e0 + G * (lane / gw), step = G * (32 / gw);
          double v[5];
          if (!poll_records<5>(
                  [&](int u) { return drec + (size_t)c * NDOT + sum_of(e + step * u); },
                  [&](int u) { return c < nown && e + step * u <= 2 * i; }, tag, v, a.spin, a.err))
            fail(par);
#pragma unroll
          for (int u = 0; u < 5; ++u) {
            for (int o = gw / 2; o > 0; o >>= 1) v[u] += __shfl_xor_sync(0xffffffffu, v[u], o);
            if (c == 0 && e + step * u <= 2 * i)
              st_tagged(a.sumrec + par * NDOT + sum_of(e + step * u), v[u], tag);
          }
        }
      }
      if (owner) {
        a11 = ld_cg(A + (long long)(j + 1) * (lda + 1));
        // sums, row j+1 of V and W, the norm and alpha = x(j+1)
        double v[6];
        const ulonglong2* sr = a.sumrec + par * NDOT;
        const ulonglong2* vw = a.vwrec + par * 2 * NB;
        if (!poll_records<6>(
                [&](int u) {
                  return u == 0   ? sr + 2 * lane
                         : u == 1 ? sr + 2 * lane + 1
                         : u == 2 ? vw + 2 * lane
                         : u == 3 ? vw + 2 * lane + 1
                         : u == 4 ? sr + DOT_NRM
                                  : xrec + j + 1;
                },
                [&](int u) { return u >= 4 || lane < i; }, tag, v, a.spin, a.err))
          fail(par);
        // Householder reflector of x (LAPACK dlarfg)
        const double alpha = v[5], xn2 = v[4];
        double beta;
        if (xn2 == 0.0) {
          sc_t = 0.0;
          beta = alpha;
          sc_scl = 0.0;
        } else {
          beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
          sc_t = (beta - alpha) / beta;
          sc_scl = 1.0 / (alpha - beta);
        }
        sc_delta = 1.0 - sc_scl * alpha;
        const double p = v[3] + sc_scl * v[0], qv = v[2] + sc_scl * v[1];
        s_rowV[lane] = v[2];
        s_rowW[lane] = v[3];
        s_p[lane] = p;
        s_q[lane] = qv;
        qp = wsum(p * qv);
        corr1 = wsum(v[2] * p + v[3] * qv);
        if (lane == 0) {
          s_t = sc_t;
          s_scl = sc_scl;
          s_delta = sc_delta;
          if (q == 0) {
            a.e[j] = beta;
            a.tau[j] = sc_t;
          }
        }
      }
      bar<2, PT>();
      if (s_fail[par]) return;
      if (!owner) continue;
      // x^T A22 x and (A22 x)(j+1); then alpha2 = -1/2 tau^2 v^T y and w(j+1), with
      // v^T y = v^T y0 - 2 (V^T v).(W^T v) and v^T y0 = scl^2 x^T A22 x + 2 scl delta
      // (A22 x)(j+1) + delta^2 A(j+1, j+1) (scl is not squared: that overflows for a
      // column of norm 1e-155 and less)
      double xax = 0.0, y1 = 0.0;
      const int nrun = cur.cta(cur.end(0) - cur.ch0 - 1) + 1, tot = nrun + cur.RB;
      for (int m = lane; m < max(G, tot); m += 160) {
        double v[10];
        if (!poll_records<10>(
                [&](int u) {
                  const int e = m + 32 * (u % 5);
                  return u < 5      ? a.vtyrec + par * G + e
                         : e < nrun ? rowrec + (size_t)e * TR + (j + 1 - cur.base)
                                    : colrec + (long long)(e - nrun) * a.ldr + (j + 1);
                },
                [&](int u) { return m + 32 * (u % 5) < (u < 5 ? G : tot); }, tag, v, a.spin,
                a.err))
          fail(2);
        xax += ((v[0] + v[1]) + (v[2] + v[3])) + v[4];
        y1 += ((v[5] + v[6]) + (v[7] + v[8])) + v[9];
      }
      xax = wsum(xax);
      y1 = wsum(y1);
      const double y1v = sc_scl * y1 + sc_delta * a11;
      const double vty = sc_scl * (sc_scl * xax + 2.0 * sc_delta * y1) + sc_delta * sc_delta * a11;
      const double al2 = -0.5 * sc_t * sc_t * (vty - 2.0 * qp);
      if (lane == 0) {
        s_al2 = al2;
        s_w1 = sc_t * (y1v - corr1) + al2;
      }
      bar<2, PT>();
      if (s_fail[2]) return;
      bar<3, PT>();  // the next column's dots read the rows' results
    }
    return;
  }

  // the first tile of a column is on its way before the column's x: lane (lr,
  // lc) of 8 x 4 holds rows 16 h + 2 lr, + 1 of columns lc + 4 u, so a load
  // touches four whole lines
  const int lr = lane & 7, lc = lane >> 3;
  double2 nx[16];  // [h][u]
  const int n8 = (n + 7) & ~7;  // rows n .. n8 - 1 are zero
  auto tile_at = [&](const Tiles& tl, int rb, int ch) {
    return A + (tl.base + rb * TR + 2 * lr) + (long long)(tl.base + ch * CW + lc) * lda;
  };
  auto issue = [&](const Tiles& tl, const Walk& w) {
    if (w.tile >= w.end) return;
    const double* p = tile_at(tl, w.rb, w.ch);
    const int r = tl.base + w.rb * TR + 2 * lr, c = tl.base + w.ch * CW + lc;
#pragma unroll
    for (int h = 0; h < 8; ++h)
#pragma unroll
      for (int u = 0; u < 2; ++u)
        nx[2 * h + u] = (r + 16 * h < n8 && c + 4 * u < n)
                            ? __ldcg((const double2*)(p + 16 * h + (long long)(4 * u) * lda))
                            : make_double2(0.0, 0.0);
  };
  Tiles cur(n, k, G);
  Walk wk(cur, q, wid);
  issue(cur, wk);
  for (int i = 0; i < a.b; ++i) {
    const int j = k + i, par = i & 1;
    const unsigned tag = (unsigned)(j + 1);
    const bool next = i + 1 < a.b;
    const ulonglong2* xrec = a.xrec + par * a.ldr;
    ulonglong2* colrec = a.colrec + par * a.rbmax * a.ldr;
    ulonglong2* rowrec = a.rowrec + par * (a.rbmax + G) * TR;
    // exchange 2: x, zero up to row j and past row n
    {
      const unsigned want = (a.stall && i == 0) ? 0xffffffffu : tag;
      constexpr int N = 10;
      for (int m = j + 1 + tid; m < n; m += 32 * NWK * N) {
        unsigned miss = 0;
#pragma unroll
        for (int u = 0; u < N; ++u)
          if (m + 32 * NWK * u < n) miss |= 1u << u;
        for (int it = 0; miss;) {
          ulonglong2 t[N];
#pragma unroll
          for (int u = 0; u < N; ++u)
            if (miss & (1u << u)) t[u] = ld_tagged(xrec + m + 32 * NWK * u);
#pragma unroll
          for (int u = 0; u < N; ++u)
            if ((miss & (1u << u)) && (unsigned)t[u].y == want) {
              if (XS)
                xs[m + 32 * NWK * u - cur.base] = __longlong_as_double((long long)t[u].x);
              miss &= ~(1u << u);
            }
          if (miss && !poll_again(it, a.spin, a.err)) {
            fail(par);
            break;
          }
        }
      }
    }
    if (XS) {
      if (tid <= j - cur.base) xs[tid] = 0.0;
      for (int r = n + tid; r < cur.base + cur.RB * TR + CW; r += 32 * NWK) xs[r - cur.base] = 0.0;
    }
    bar<1, 32 * NWK>();
    // ---- stream ----
    auto x1 = [&](int r) {
      if (XS) return xs[r - cur.base];
      return (r > j && r < n) ? __longlong_as_double((long long)ld_tagged(xrec + r).x) : 0.0;
    };
    auto x2 = [&](int r) {
      if (XS) return *(const double2*)(xs + (r - cur.base));
      return make_double2(x1(r), x1(r + 1));
    };
    double racc[16], vty = 0.0;
#pragma unroll
    for (int e = 0; e < 16; ++e) racc[e] = 0.0;
    int seg = 0;
    const int rb_first = wk.rb;
    while (wk.tile < wk.end) {
      const int rb = wk.rb, ch = wk.ch;
      const int r = cur.base + rb * TR + 2 * lr, c = cur.base + ch * CW + lc;
      if (++wk.ch == cur.end(rb)) {
        wk.ch = cur.ch0;
        ++wk.rb;
      }
      const bool more = ++wk.tile < wk.end;
      const double xc0 = x1(c), xc1 = x1(c + 4);
      double z0 = 0.0, z1 = 0.0;
      // Each pair makes room for the next tile's as it is used.  masked: A(r, c)
      // with r < c leaves the row sums, r <= c the column sums; edge: the
      // next tile may reach past the matrix, or there is none.
      const double* pn = tile_at(cur, wk.rb, wk.ch);
      auto sum_tile = [&](auto masked, auto edge) {
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          const double2 xr = x2(r + 16 * h);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            double2 v = nx[2 * h + u];
            const double* src = pn + 16 * h + (long long)(4 * u) * lda;
            if (!decltype(edge)::value) {
              nx[2 * h + u] = ld2_now(src);
            } else {
              const int rn = cur.base + wk.rb * TR + 2 * lr + 16 * h;
              const int cn = cur.base + wk.ch * CW + lc + 4 * u;
              if (more && rn < n8 && cn < n) nx[2 * h + u] = ld2_now(src);
              else nx[2 * h + u] = make_double2(0.0, 0.0);
            }
            const double xc = u ? xc1 : xc0;
            const int dr = r + 16 * h - (c + 4 * u);
            if (decltype(masked)::value) {
              if (dr < 0) v.x = 0.0;
              if (dr + 1 < 0) v.y = 0.0;
            }
            racc[2 * h] = fma(v.x, xc, racc[2 * h]);
            racc[2 * h + 1] = fma(v.y, xc, racc[2 * h + 1]);
            if (decltype(masked)::value) {
              if (dr == 0) v.x = 0.0;
              if (dr + 1 == 0) v.y = 0.0;
            }
            double& z = u ? z1 : z0;
            z = fma(v.x, xr.x, fma(v.y, xr.y, z));
          }
        }
      };
      const bool inner =
          more && cur.base + wk.rb * TR + TR <= n8 && cur.base + wk.ch * CW + CW <= n;
      if (!inner) sum_tile(std::true_type{}, std::true_type{});
      else if (rb * TR >= ch * CW + CW)
        sum_tile(std::false_type{}, std::false_type{});
      else sum_tile(std::true_type{}, std::false_type{});
      // column sums over the eight row lanes: lanes lr < 4 end with column lc,
      // the others with lc + 4
      {
        const bool h4 = lr & 4;
        double zc = (h4 ? z1 : z0) + __shfl_xor_sync(0xffffffffu, h4 ? z0 : z1, 4);
        zc += __shfl_xor_sync(0xffffffffu, zc, 2);
        zc += __shfl_xor_sync(0xffffffffu, zc, 1);
        const int cz = c + (h4 ? 4 : 0);
        if (!(lr & 3) && cz < n) {
          st_tagged(colrec + rb * a.ldr + cz, zc, tag);
          vty = fma(h4 ? xc1 : xc0, zc, vty);
        }
      }
      if (!more || wk.rb != rb) {
        // the row sums over the four column lanes: lane lc ends with the four
        // rows of h = 2 lc, 2 lc + 1
        const bool h16 = lane & 16, h8 = lane & 8;
        double o[4];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const double send = h16 ? racc[e] : racc[8 + e];
          racc[e] = (h16 ? racc[8 + e] : racc[e]) + __shfl_xor_sync(0xffffffffu, send, 16);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const double send = h8 ? racc[e] : racc[4 + e];
          o[e] = (h8 ? racc[4 + e] : racc[e]) + __shfl_xor_sync(0xffffffffu, send, 8);
        }
        double* dst = rs + (size_t)(wid * a.nseg + seg) * TR + 32 * lc + 2 * lr;
        *(double2*)dst = make_double2(o[0], o[1]);
        *(double2*)(dst + 16) = make_double2(o[2], o[3]);
        const int rr = cur.base + rb * TR + 32 * lc + 2 * lr;
        const double2 xa = x2(rr), xb = x2(rr + 16);
        vty += xa.x * o[0] + xa.y * o[1] + xb.x * o[2] + xb.y * o[3];
        ++seg;
#pragma unroll
        for (int e = 0; e < 16; ++e) racc[e] = 0.0;
      }
    }
    vty = wsum(vty);
    if (lane == 0) {
      s_vty[wid] = vty;
      s_rb0[wid] = rb_first;
      s_ns[wid] = seg;
    }
    bar<1, 32 * NWK>();
    // exchange 1: the CTA's row sums and its part of x^T A22 x (a CTA's last warp
    // has a tile if any has)
    int rbf = s_rb0[NWK - 1];
#pragma unroll
    for (int w = NWK - 2; w >= 0; --w)
      if (s_ns[w] > 0) rbf = s_rb0[w];
    for (int e = tid; e < (s_rb0[NWK - 1] + s_ns[NWK - 1] - rbf) * TR; e += 32 * NWK) {
      const int b_ = rbf + e / TR, l = e % TR;
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < NWK; ++w) {
        const int sg = b_ - s_rb0[w];
        if (sg >= 0 && sg < s_ns[w]) s += rs[(size_t)(w * a.nseg + sg) * TR + l];
      }
      if (cur.base + b_ * TR + l < n) st_tagged(rowrec + (size_t)(b_ + q) * TR + l, s, tag);
    }
    if (tid == 0) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < NWK; ++w) s += s_vty[w];
      st_tagged(a.vtyrec + par * G + q, s, tag);
    }
    if (!owner) {
      bar<2, PT>();
      if (s_fail[par]) return;
      cur = Tiles(n, next ? j + 1 : j, G);
      wk = Walk(cur, q, wid);
      if (next) issue(cur, wk);
      continue;
    }
    for (int g0 = 0; g0 < rounds; g0 += NWK) {
      double aold = 0.0;  // A(r, j+1) of the row this lane finishes (round g0 + wid)
      if (g0 + wid < rounds) {
        const int l = 32 * (g0 + wid) + lane, r = r0 + l;
        if (l < nr && r > j) aold = ld_cg(A + r + (long long)(j + 1) * lda);
      }
      for (int rd = g0; rd < min(rounds, g0 + NWK); ++rd) {
        const int l = 32 * rd + lane, r = r0 + l;
        const bool valid = l < nr && r > j;
        // the records that cover row r: those of the CTAs in its row block,
        // then the row blocks that cover column r
        const int rbr = valid ? (r - cur.base) / TR : 0;
        const int t0 = cur.first(rbr), cf = cur.cta(t0);
        const int nrun = cur.cta(t0 + cur.end(rbr) - cur.ch0 - 1) - cf + 1;
        const int rb0 = valid ? (r - cur.base) / CW / CPB : 0;
        const int tot = valid ? nrun + cur.RB - rb0 : 0;
        double ys = 0.0;
        for (int m = wid; __any_sync(0xffffffffu, m < tot); m += 8 * NWK) {
          double v[8];
          if (!poll_records<8>(
                  [&](int u) {
                    const int e = m + NWK * u;
                    return e < nrun ? rowrec + (size_t)(rbr + cf + e) * TR + (r - cur.base - rbr * TR)
                                    : colrec + (long long)(rb0 + e - nrun) * a.ldr + r;
                  },
                  [&](int u) { return m + NWK * u < tot; }, tag, v, a.spin, a.err))
            fail(g0 == 0 ? par : par ^ 1);
          ys += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        }
        sm_y[((rd - g0) * NWK + wid) * 32 + lane] = ys;
      }
      if (g0 == 0) {
        bar<2, PT>();  // barrier 1: the reflector's scalars
        if (s_fail[par]) return;
      }
      for (int rd = g0; rd < min(rounds, g0 + NWK); ++rd) {
        const int l = 32 * rd + lane;
        double cs = 0.0, us = 0.0;
#pragma unroll
        for (int h = 0; h < HP; ++h) {
          const int p = wid + NWK * h;
          if (l < nr && r0 + l > j && p < i) {
            const double vp = own_V(l, p), wp = own_W(l, p);
            cs += vp * s_p[p] + wp * s_q[p];
            us += vp * s_rowW[p] + wp * s_rowV[p];
          }
        }
        const int o = ((rd - g0) * NWK + wid) * 32 + lane;
        sm_c[o] = cs;
        sm_u[o] = us;
      }
      if (g0 == 0) {
        if (next) {
          const Tiles nxt(n, j + 1, G);
          wk = Walk(nxt, q, wid);
          issue(nxt, wk);
        }
        bar<2, PT>();  // barrier 2: alpha2 and w(j+1)
        if (s_fail[2]) return;
      } else {
        bar<1, 32 * NWK>();
      }
      // ---- rows: w, the next column and what the others need of it ----
      const int rd = g0 + wid;
      if (rd < rounds) {
        ulonglong2* xnext = a.xrec + (par ^ 1) * a.ldr;
        const double t = s_t, scl = s_scl, delta = s_delta, al2 = s_al2, w1 = s_w1;
        const int l = 32 * rd + lane, r = r0 + l;
        const bool valid = l < nr && r > j;
        double ys = 0.0, corr = 0.0, upd = 0.0;
#pragma unroll
        for (int w = 0; w < NWK; ++w) {
          const int o = (wid * NWK + w) * 32 + lane;
          ys += sm_y[o];
          corr += sm_c[o];
          upd += sm_u[o];
        }
        double xr = 0.0;
        if (valid)
          xr = XS ? xs[r - cur.base] : __longlong_as_double((long long)ld_tagged(xrec + r).x);
        const double vr = (r == j + 1) ? 1.0 : xr * scl;
        const double wr = t * ((scl * ys + delta * aold) - corr) + al2 * vr;
        double am = 0.0;
        if (next && valid) {
          const double anew = aold - (upd + vr * w1 + wr);
          if (r >= j + 2) st_tagged(xnext + r, anew, tag + 1);
          if (r == j + 1) a.d[j + 1] = anew;
          if (r >= j + 3) am = anew;
        }
        if (valid) {
          a.V[r + (long long)j * a.ldv] = vr;
          a.W[r + (long long)i * a.ldw] = wr;
        }
        sm_a[l] = am;
        if (VS) {
          sm_V[l * (NB + 1) + i] = valid ? vr : 0.0;
          sm_W[l * (NB + 1) + i] = valid ? wr : 0.0;
        }
        // row j+2 of V and W for the next column
        if (next && j + 2 >= r0 + 32 * rd && j + 2 < min(r0 + 32 * rd + 32, r0 + nr)) {
          const int src = j + 2 - (r0 + 32 * rd), ls = j + 2 - r0;
          const double vn = __shfl_sync(0xffffffffu, vr, src), wn = __shfl_sync(0xffffffffu, wr, src);
          if (lane <= i) {
            ulonglong2* vw = a.vwrec + ((par ^ 1) * NB + lane) * 2;
            st_tagged(vw, lane == i ? vn : own_V(ls, lane), tag + 1);
            st_tagged(vw + 1, lane == i ? wn : own_W(ls, lane), tag + 1);
          }
        }
      }
      if (g0 + NWK < rounds) bar<1, 32 * NWK>();
    }
    cur = Tiles(n, next ? j + 1 : j, G);
    bar<3, PT>();  // the service warp's dots read the rows' results
  }
}

// Tiles per worker warp at most, and the row blocks they can touch: the
// smallest s whose first s blocks hold as many, and one more.
int panel_segments(int R, int G) {
  const long long rb = (R + 7 + 2 * TR - 1) / TR, nt = CPB * rb * (rb + 1) / 2;
  const long long per = (nt / std::max(1, G) + 2) / NWK + 2;
  int s = 1;
  while ((long long)CPB * s * (s + 1) / 2 < per) ++s;
  return s + 1;
}

struct PanelShape {
  int rp, nseg;
  size_t smem[3];  // by MODE
};

PanelShape panel_shape(int R, int G) {
  PanelShape p;
  // at least a row per lane: with fewer owners each record line has one poller
  // less; records of four rows fill 64 bytes
  p.rp = std::max(32, ((R + G - 1) / G + 3) / 4 * 4);
  p.nseg = panel_segments(R, G);
  const size_t rounds = (p.rp + 31) / 32;
  p.smem[2] = ((size_t)NWK * p.nseg * TR + std::min<size_t>(rounds, NWK) * 32 * 3 * NWK +
               rounds * 32) * sizeof(double);
  p.smem[1] = p.smem[2] + (size_t)(R + 3 * TR + 1) * sizeof(double);
  p.smem[0] = p.smem[1] + rounds * 32 * 2 * (NB + 1) * sizeof(double);
  return p;
}

size_t panel_limit(int dev) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return optin > 4096 ? (size_t)optin - 4096 : 0;  // room for static shared
}

long long panel_ldr(int n) { return (n + 15) / 8 * 8; }
long long panel_rbmax(int n) { return (n + 7) / TR + 3; }

}  // namespace

size_t panel_bytes(int n, int G) {
  const size_t ldr = panel_ldr(n), rb = panel_rbmax(n);
  return sizeof(ulonglong2) * 2 *
         (ldr * (rb + 1) + (rb + G) * TR + G + (size_t)G * NDOT + NDOT + 2 * NB);
}

int panel_grid(imcom_ctx* ctx, int n) {
  const int all = device_sm_count(ctx->device);
  int G = std::min(sm_count(ctx), all);
  while (G < all && panel_shape(n, G).smem[2] > panel_limit(ctx->device)) ++G;
  return G;
}

int panel_prepare(imcom_ctx* ctx) {
  const size_t limit = panel_limit(ctx->device);
  const void* kernels[] = {(void*)trd_panel_kernel<0>, (void*)trd_panel_kernel<1>,
                           (void*)trd_panel_kernel<2>};
  int per = 1;
  for (const void* f : kernels) {
    int p = 0;
    IMC_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
    IMC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, f, PT, limit));
    per = std::min(per, p);
  }
  if (per < 1) return set_err(ctx, IMCOM_ERR_CUDA, "panel kernel does not fit on an SM");
  return 0;
}

int panel_launch(imcom_ctx* ctx, const DMat& Aw, DMat& Vall, double* W, long long ldw, double* d,
                 double* e, double* tau, int k, int b, int G, void* scratch, int* err,
                 long long spin, int stall) {
  const int n = (int)Aw.rows;
  const PanelShape sh = panel_shape(n - k, G);
  const size_t limit = panel_limit(ctx->device);
  PanelArgs a{};
  a.A = Aw.p;
  a.lda = Aw.ld;
  a.V = Vall.p;
  a.ldv = Vall.ld;
  a.W = W;
  a.ldw = ldw;
  a.d = d;
  a.e = e;
  a.tau = tau;
  a.ldr = panel_ldr(n);
  a.rbmax = panel_rbmax(n);
  ulonglong2* p = (ulonglong2*)scratch;
  auto take = [&](size_t count) {
    ulonglong2* r = p;
    p += 2 * count;
    return r;
  };
  a.xrec = take(a.ldr);
  a.colrec = take(a.ldr * a.rbmax);
  a.rowrec = take((a.rbmax + G) * TR);
  a.dotrec = take((size_t)G * NDOT);
  a.sumrec = take(NDOT);
  a.vwrec = take(2 * NB);
  a.vtyrec = take(G);
  a.err = err;
  a.n = n;
  a.k = k;
  a.b = b;
  a.rp = sh.rp;
  a.nseg = sh.nseg;
  a.spin = spin;
  a.stall = stall;
  const int mode = sh.smem[0] <= limit ? 0 : sh.smem[1] <= limit ? 1 : 2;
  const size_t smem = sh.smem[mode];
  if (smem > limit)
    return set_err(ctx, IMCOM_ERR_EIGEN, "order %d is too large for %d SMs' panels", n, G);
  void* args[] = {&a};
  IMC_CUDA(cudaLaunchCooperativeKernel(mode == 0   ? (void*)trd_panel_kernel<0>
                                       : mode == 1 ? (void*)trd_panel_kernel<1>
                                                   : (void*)trd_panel_kernel<2>,
                                       G, PT, args, smem, ctx->stream));
  IMC_LAUNCH();
  return 0;
}

}  // namespace imcom
