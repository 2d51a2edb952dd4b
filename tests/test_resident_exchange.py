"""The exchange of the resident tridiagonalisation (csrc/eigen_res.cu) as an event
model: CTAs that publish tagged values into two buffers by column parity and read
them back, with any delays.  The rules of the rows come from csrc/res_rows.h, compiled
here; the rest follows the kernel: in column j a CTA publishes its rows below j,
returns if it retires, reads every row below j, and may write the column's results.
No value may be overwritten before every reader has it, and every column is written
once, by a CTA that has read it.  The model finds the loss where a retiring CTA
reads its last column instead (the last check of the program)."""
import os
import subprocess

SRC = r"""
#include <cstdio>
#include <vector>
#include <algorithm>
#include "res_rows.h"
using namespace imcom;

static int rows_of(int S, int G) { return ((S + RBLK - 1) / RBLK + G - 1) / G * RBLK; }

struct Cta {
  ResRows rows;
  int j = 0, i0 = 0, r0, phase = 0, got = 0;  // phase 0: publish, 1: read row by row
  bool done = false;
  Cta(int q, int G, int S) : rows(q, G, S, rows_of(S, G)), r0(rows.row(0)) {}
};

// 0: every value arrived; 1: one was lost; 2: stuck; 3: a column not written once
struct Model {
  int S, G;
  bool stay;  // the retiring CTA reads its last column
  std::vector<Cta> c;
  std::vector<int> buf[2], wrote;
  Model(int S_, int G_, bool stay_) : S(S_), G(G_), stay(stay_) {
    for (int q = 0; q < G; ++q) c.emplace_back(q, G, S);
    buf[0].assign(S, 0);
    buf[1].assign(S, 0);
    wrote.assign(S, 0);
  }
  // one step of CTA q: 1 it moved, 0 it waits, -1 a value it wants is gone
  int step(int q) {
    Cta& x = c[q];
    if (x.done) return 0;
    std::vector<int>& b = buf[x.j & 1];
    if (x.phase == 0) {
      if (x.r0 <= x.j) {
        x.r0 = x.rows.after(x.i0, x.r0);
        ++x.i0;
      }
      if (x.i0 >= x.rows.nrow) {
        x.done = true;
        return 1;
      }
      for (int i = x.i0; i < x.rows.nrow; ++i) b[x.rows.row(i)] = x.j + 1;
      if (!stay && x.rows.retires(x.j, x.i0, x.r0)) {
        x.done = true;
        return 1;
      }
      x.phase = 1;
      x.got = x.j + 1;
      return 1;
    }
    if (b[x.got] > x.j + 1) return -1;
    if (b[x.got] < x.j + 1) return 0;
    if (++x.got < S) return 1;
    if (x.rows.writes(x.j, x.i0, x.r0)) ++wrote[x.j];
    x.phase = 0;
    if (++x.j == S - 1) x.done = true;
    return 1;
  }
  int finish() {
    for (const Cta& x : c)
      if (!x.done) return 2;
    if (!stay)
      for (int j = 0; j < S - 1; ++j)
        if (wrote[j] != 1) return 3;
    return 0;
  }
};

// CTA q stops before its step number `at` until the others have gone as far as they can
static int frozen(int S, int G, bool stay, int q, int at) {
  Model m(S, G, stay);
  int taken = 0;
  bool thawed = false;
  for (;;) {
    bool moved = false;
    for (int p = 0; p < G; ++p) {
      if (p == q && !thawed && taken >= at) continue;
      const int r = m.step(p);
      if (r < 0) return 1;
      if (r > 0) {
        moved = true;
        if (p == q) ++taken;
      }
    }
    if (!moved) {
      if (thawed) break;
      thawed = true;
    }
  }
  return m.finish();
}

static int shuffled(int S, int G, bool stay, unsigned seed) {
  Model m(S, G, stay);
  unsigned s = seed * 2654435761u + 1;
  for (int idle = 0; idle < 64 * G;) {
    s ^= s << 13; s ^= s >> 17; s ^= s << 5;
    int q = (s >> 8) % G, burst = 1 + (s >> 3) % (2 * S);
    int any = 0;
    while (burst-- > 0) {
      const int r = m.step(q);
      if (r < 0) return 1;
      if (r == 0) break;
      any = 1;
    }
    idle = any ? 0 : idle + 1;
  }
  return m.finish();
}

int main() {
  int lost = 0;
  for (int S = 2; S <= 19; ++S)
    for (int sms = 1; sms <= 9; ++sms) {
      const int G = std::min((S + RBLK - 1) / RBLK, sms);
      for (int q = 0; q < G; ++q)
        for (int at = 0; at < S * (S + 2); ++at) {
          const int r = frozen(S, G, false, q, at);
          if (r) return std::printf("S %d G %d CTA %d stopped at %d: %d\n", S, G, q, at, r), 1;
          if (G > 2 && S < 12) lost += frozen(S, G, true, q, at) == 1;
        }
      for (unsigned seed = 1; seed <= 40; ++seed) {
        const int r = shuffled(S, G, false, seed);
        if (r) return std::printf("S %d G %d seed %u: %d\n", S, G, seed, r), 1;
      }
    }
  return lost ? 0 : 2;
}
"""


def test_no_value_is_lost(tmp_path):
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imcom_b200",
                        "csrc")
    src = tmp_path / "m.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "m")
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-I" + csrc, str(src), "-o",
                    exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
