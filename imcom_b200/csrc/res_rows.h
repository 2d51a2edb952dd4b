// res_rows.h -- which rows a CTA of the resident tridiagonalisation owns, when it
// has published its last one, and which CTA writes a column's results
// (eigen_res.cu; plain C++, so that a model of the exchange can be run on the CPU).
#pragma once

#ifdef __CUDACC__
#define RES_FN __host__ __device__ __forceinline__
#else
#define RES_FN inline
#endif

namespace imcom {

// Rows go to the CTAs in pairs: a pair's records are 64 consecutive bytes,
// written by one store instruction.  (Measured on an exchange alone, 148 CTAs
// publishing 1776 16-byte values: 8000 cycles when every value is its own
// store into a line shared with 7 other CTAs, 2190 with 64 bytes per store,
// 2100 with whole 128-byte lines.)
constexpr int RBLK = 2;

// CTA q of G for S rows; own rows i = 0, 1, .. in ascending order.
struct ResRows {
  int q, G, S, nrow;
  RES_FN ResRows(int q_, int G_, int S_, int most) : q(q_), G(G_), S(S_), nrow(most) {
    while (nrow > 0 && row(nrow - 1) >= S) --nrow;
  }
  RES_FN int row(int i) const { return RBLK * (q + G * (i / RBLK)) + i % RBLK; }
  // row(i + 1) from r = row(i)
  RES_FN int after(int i, int r) const {
    return r + ((i + 1) % RBLK ? 1 : 1 + RBLK * (G - 1));
  }
  // Column j, own row i = row r the first one below row j.  Whether this CTA
  // publishes its last value in it and returns without reading the column: nobody
  // waits for it in column j + 1, so by then its buffer may be written again.
  RES_FN bool retires(int j, int i, int r) const {
    return i == nrow - 1 && r == j + 1 && r < S - 1;
  }
  // Whether it writes column j's reflector and diagonal: the owner of row j + 2,
  // which reads column j (of row S - 1 in the last column).
  RES_FN bool writes(int j, int i, int r) const {
    const int w = j + 2 < S - 1 ? j + 2 : S - 1;
    return r == w || (i + 1 < nrow && after(i, r) == w);
  }
};

}  // namespace imcom
