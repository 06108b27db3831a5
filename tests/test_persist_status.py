"""The status word of the one-kernel CG (hpccg_persist.cuh): blocks report in no order, and a
wait that ran out in any of them has to stand.  The rule is host code too, so it is
compiled for the host here and run over every order of the reports; no GPU."""
import itertools
import os
import subprocess

from conftest import PKG, ROOT

import hpccg_b200 as hp

PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "hpccg_persist.cuh"
struct Word {
  int v;
  void set(int s) { v = s; }
  void set_if_ok(int s) { if (v == HPCCG_OK) v = s; }
};
int main(int argc, char **argv) {  // lead ok status, per report
  Word w{HPCCG_OK};
  for (int i = 1; i + 2 < argc; i += 3)
    hpccg::persist_report(w, atoi(argv[i]) != 0, atoi(argv[i + 1]) != 0, atoi(argv[i + 2]));
  printf("%d", w.v);
}
"""


def test_an_expired_wait_stands_in_every_order(tmp_path):
    src, exe = tmp_path / "status.cu", tmp_path / "status"
    src.write_text(PROGRAM)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(ROOT, "include"),
                    str(src), "-o", str(exe)], check=True, capture_output=True, timeout=300)

    def word(reports):
        args = [str(int(v)) for r in reports for v in r]
        return int(subprocess.run([str(exe), *args], capture_output=True, text=True, check=True, timeout=60).stdout)

    for how in (hp.HPCCG_OK, hp.HPCCG_ERR_BREAKDOWN):
        lead, rest, late = (True, True, how), (False, True, how), (False, False, how)
        for order in itertools.permutations([lead, rest, rest]):
            assert word(order) == how
        for order in itertools.permutations([lead, rest, late]):
            assert word(order) == hp.HPCCG_ERR_TIMEOUT, order
    assert word([(False, True, 0), (True, False, 0)]) == hp.HPCCG_ERR_TIMEOUT
