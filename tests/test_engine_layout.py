"""Sizes and offsets the N4 engine works with, from its own header: a small host
program that includes csrc/n4_engine.cuh prints what its functions return."""
import os
import subprocess

import numpy as np
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
    } else if (!std::strcmp(what, "share")) {   // rows, voxels of a row, CTAs
      std::printf("%d %lld %lld\n", n4::grid_row_overhead((int)b), n4::grid_rows_bound(a, (int)b, (int)c),
                  n4::grid_voxels_bound(a, (int)b, (int)c));
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


def shares(lens, K, c):
    """First row of each CTA's share, as the whole-GPU path deals rows out whose
    masked ranges are `lens` voxels long (0: none): a row weighs its range and c,
    the CTAs add up even shares of the rows, and a CTA's share begins at the
    first row with its part of the total before it."""
    w = np.where(lens > 0, lens + c, 0).astype(np.int64)
    n = w.size
    cut = [n * k // K for k in range(K + 1)]
    before = np.concatenate(([0], np.cumsum(w)))

    def boundary(target):
        k = max(q for q in range(K) if before[cut[q]] <= target)
        rows = np.arange(cut[k], cut[k + 1])
        hit = rows[before[rows] >= target]
        return int(hit[0]) if hit.size else cut[k + 1]

    return [boundary(int(before[-1]) * r // K) for r in range(K)] + [n], w


@pytest.mark.parametrize("seed", range(24))
def test_shares_of_the_rows_lie_within_their_buffers(engine, seed):
    """The row list and the slab of a CTA are sized by grid_rows_bound and
    grid_voxels_bound of the code and filled without further checks."""
    rng = np.random.default_rng(seed)
    Z = int(rng.choice([1, 2, 5, 31, 32, 33, 60, 160, 181, 700, 1024]))
    n, K = int(rng.integers(1, 4000)), int(rng.choice([1, 7, 148]))
    lens = rng.integers(0, Z + 1, n)
    kind = seed % 4
    if kind == 1:
        lens[rng.random(n) < 0.95] = 0
    if kind == 2:
        lens = np.where(rng.random(n) < 0.5, 1, Z)              # short rows beside full ones
    if kind == 3:
        lens = np.where(np.arange(n) < n // 2, 1, Z)            # all short ones first
    ((c, rows_bound, voxels_bound),) = engine([("share", n, Z, K)])
    b, w = shares(lens, K, c)
    assert not w[:b[0]].any() and all(x <= y for x, y in zip(b, b[1:]))   # every row once
    for r in range(K):
        part = lens[b[r]:b[r + 1]]
        assert (part > 0).sum() <= rows_bound and part.sum() <= voxels_bound
