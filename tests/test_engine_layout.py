"""Sizes and offsets the N4 engine works with, from its own header: a small host
program that includes csrc/n4_engine.cuh prints what its functions return."""
import os
import subprocess

import pytest

from conftest import ROOT
from n4b200.build import nvcc

MAIN = r"""
#include <cstdio>
#include <cstring>
#include <cstdlib>
#include "n4_engine.cuh"
int main(int argc, char **argv) {
  char what[32];
  long long a, b, c;
  while (std::scanf("%31s %lld %lld %lld", what, &a, &b, &c) == 4) {
    if (!std::strcmp(what, "axis")) {   // voxels, control points of the finest level, of this level
      const n4::EAxis e = n4::eaxis_at(0, (int)a, (int)c, n4::kWeightTail);
      std::printf("%d %d %d %d %d %d %d %d %zu\n", e.o_w, e.o_p, e.o_q, e.o_tail, e.o_s, e.o_lo, e.o_hi,
                  n4::kWeightTail, n4::eaxis_bytes((int)a, (int)b - 3, n4::kWeightTail));
    }
  }
}
"""


@pytest.fixture(scope="module")
def engine(tmp_path_factory):
    d = tmp_path_factory.mktemp("layout")
    (d / "main.cu").write_text(MAIN)
    exe = str(d / "main")
    subprocess.run([nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O0", "-cudart", "shared",
                    "-I", os.path.join(ROOT, "cuda-n4_b200", "csrc"), "-o", exe, str(d / "main.cu")], check=True)

    def ask(lines):
        out = subprocess.run([exe], input="".join(" ".join(map(str, x)) + "\n" for x in lines), text=True,
                             capture_output=True, check=True).stdout
        return [[int(v) for v in row.split()] for row in out.splitlines()]
    return ask


def test_every_weight_read_lies_in_a_table_or_its_zero_tail(engine):
    """The z contraction reads the numerator weights and the denominator weights
    in steps of 8 voxels (four lanes per span, from a start of at most Z - 1), of
    2, 3 or 4 (one lane) or of 2 that are 1, 2, 4 or 8 voxels apart (a span's
    lanes on the whole-GPU path), pass A the cubic weights in steps of 2.  What a step
    holds past the row has to be one of the tables (filled for every voxel) or
    the zero entries behind them."""
    ask = [("axis", Z, nc, lv) for Z in range(1, 200) for nc, lv in ((4, 4), (5, 4), (11, 4), (19, 7), (64, 64))]
    for (_, Z, _, lv), (ow, op, oq, ot, os_, olo, ohi, tail, size) in zip(ask, engine(ask)):
        written = set(range(ow, ow + 16 * Z, 16)) | set(range(op, op + 16 * Z, 16)) | set(range(oq, oq + 16 * Z, 16))
        assert len(written) == 3 * Z   # no two of them overlap
        written |= set(range(ot, ot + 16 * tail, 16))
        last = set()
        for start in range(Z):
            last.add(start + 7)                          # quad_rows: min(a + q, Z - 1) + 7
            last.update(start + u - 1 for u in (2, 3, 4))   # SpanSums::add
            last.update(start + d for d in (1, 2, 4, 8))    # its lanes on the whole-GPU path
        reads = {o + 16 * z for o in (op, oq) for z in range(max(last) + 1)}
        reads |= {ow + 16 * z for z in range(Z + 1)}     # pass A
        assert reads <= written
        assert max(written) + 16 <= os_ and os_ + 4 * Z <= olo and olo + 4 * (lv - 3) == ohi and ohi + 4 * (lv - 3) <= size
