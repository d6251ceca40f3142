"""The digit-pair MMAs of the tensor-core contractions, as they are issued for every
number of digits, columns and K steps in use: each pair once, into the accumulator of
its weight; each accumulator begun by its first MMA; and all MMAs into an accumulator
over the same columns, since the order of two of them is given only for the same
accumulator and shape.  The list comes from the function that the kernels issue by,
compiled for the host."""
import subprocess

import pytest

from mocca_gb300.build import CSRC, nvcc

# digits, columns, K steps: derivatives (both forms), overlaps and gaps, applies
SHAPES = ([(8, 16, 1), (8, 32, 2), (6, 32, 1), (6, 64, 2), (6, 96, 3)]
          + [(6, n, 2) for n in (16, 32, 48, 64, 80)] + [(8, n, 2) for n in (32, 48, 64)]
          + [(6, n, n // 16) for n in (16, 32, 48, 64, 80)]
          + [(8, n, n // 16) for n in (32, 48, 64)])

MAIN = """
#include <cstdint>
#include <cstdio>
#include <cmath>
#include <cstring>
#include "df.cuh"
#include "tc.cuh"
#include "ozaki.cuh"
template <int ND, int COLS, int KS> void list() {
    printf("shape %%d %%d %%d %%d\\n", ND, COLS, KS, mg::oz::stack_zeros(ND, COLS));
    mg::oz::stacked_pairs<ND, COLS, KS>([](int a, int b, int ks, int acc, int count, bool first) {
        printf("%%d %%d %%d %%d %%d %%d\\n", a, b, ks, acc, count, (int)first);
    });
}
int main() { %s }
"""


@pytest.fixture(scope="module")
def issued(tmp_path_factory):
    d = tmp_path_factory.mktemp("mma")
    calls = "\n".join(f"list<{nd}, {c}, {k}>();" for nd, c, k in sorted(set(SHAPES)))
    (d / "main.cu").write_text(MAIN % calls)
    subprocess.run([nvcc(), "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_103a,code=sm_103a", "-I", str(CSRC), "-o", str(d / "main"),
                    str(d / "main.cu")], check=True, capture_output=True)
    out, lists = subprocess.run([str(d / "main")], check=True, capture_output=True, text=True), {}
    for line in out.stdout.splitlines():
        if line.startswith("shape"):
            *key, zeros = map(int, line.split()[1:])
            now = lists[tuple(key)] = (zeros, [])
        else:
            now[1].append(tuple(map(int, line.split())))
    return lists


@pytest.mark.parametrize("shape", sorted(set(SHAPES)))
def test_issue(issued, shape):
    nd, cols, ksteps = shape
    zeros, mmas = issued[shape]
    own = 8 if nd == 8 else 3            # accumulators of one weight
    seen, columns = set(), {}
    for a, b, ks, acc, count, first in mmas:
        assert count * cols <= 256 and (count * cols) % 16 == 0
        assert -zeros <= b and b + count <= nd
        for k in range(count):
            group = columns.setdefault(acc + k, (acc, count))
            assert group == (acc, count), "an accumulator in MMAs of two shapes"
            begun = any(s[3] == acc + k for s in seen)
            assert bool(first) == (not begun)
            if b + k < 0:
                continue                 # a plane of zeros
            weight = a + b + k
            assert acc + k == min(weight, own)
            assert (a, b + k, ks) not in {s[:3] for s in seen}
        for k in range(count):
            seen.add((a, b + k, ks, acc + k))
    pairs = {(a, b, ks) for a, b, ks, _ in seen if b >= 0}
    assert pairs == {(a, b, ks) for a in range(nd) for b in range(nd - a) for ks in range(ksteps)}
