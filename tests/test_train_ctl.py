"""The training calls' check for a timed-out barrier (csrc/train_ctl.h) on a thread
that treats denormals as zero: the device writes the whole number 1, whose bits are
a denormal float."""
import os
import subprocess

SRC = r"""
#include <string.h>
#include <xmmintrin.h>
#include "train_ctl.h"
int main() {
  _mm_setcsr(_mm_getcsr() | 0x8040);  // denormals are zero, in and out
  imcom::TrainCtl c[3];
  memset(c, 0, sizeof c);
  if (imcom::train_failed(c, 3)) return 1;
  const int one = 1;
  memcpy((char*)&c[2] + 8, &one, 4);  // the third word, as the device writes it
  if (!imcom::train_failed(c, 3)) return 2;
  return imcom::train_failed(c, 2) ? 3 : 0;
}
"""


def test_failed_flag_with_denormals_as_zero(tmp_path):
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imcom_b200",
                        "csrc")
    src = tmp_path / "t.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-I" + csrc, str(src), "-o", exe],
                   check=True)
    assert subprocess.run([exe]).returncode == 0


def test_callers_read_the_words_through_it():
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imcom_b200",
                        "csrc", "kappa.cu")
    text = open(path).read()
    train = text[text.index("imcom_gpu_mlp_train("):]
    # the check comes before the caller's parameters are written
    assert 0 < train.index("train_failed(") < train.index("cudaMemcpyAsync(params,")
