"""The rules that choose a step's launch shapes from its sizes
(channel_gb300/csrc/launch_rules.h), compiled as host code: what an ensemble's
members cost together, and that a lone handle's choices are its own."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "channel_gb300" / "csrc"
NSM = 152
PROGRAM = """
#include <cstdio>
#include <cstring>
#include "launch_rules.h"
int main() {
  char what[8];
  int modes, ny, nsm;
  double together;
  while (std::scanf("%7s %d %d %d %lf", what, &modes, &ny, &nsm, &together) == 5) {
    const chgpu::RhsCost c = !std::strcmp(what, "fp64") ? chgpu::kRhsCostFP64 : !std::strcmp(what, "fp64dd") ? chgpu::kRhsCostDD : chgpu::kRhsCostFP32;
    std::printf("%d %d %d\\n", chgpu::rhs_rows(c, modes, ny, nsm, together), chgpu::default_solve_form(modes, nsm), chgpu::solve_in_four_parts(modes, nsm, together));
  }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(PROGRAM)
    exe = d / "rules"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(CSRC), str(d / "rules.cpp"), "-o", str(exe)], check=True)

    def ask(rows):
        text = "".join(f"{w} {m} {ny} {n} {t}\n" for w, m, ny, n, t in rows)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(int(v) for v in line.split()) for line in out.splitlines()]

    return ask


def loaded(rb, ny):
    """Rows that k_rhs loads for the ny - 1 rows of one column of modes: each thread its rows and four more."""
    return sum(min(rb, ny - 1 - r) + 4 for r in range(0, ny - 1, rb))


@pytest.mark.parametrize("prec", ["fp64", "fp64dd", "mixed"])
def test_members_of_a_full_ensemble_take_long_row_runs(rules, prec):
    """64 members load at most half a row more than they produce; with each member's rows chosen as if it had the GPU to
    itself, 1.1 to 1.7 more."""
    sizes = [(nx, ny, nz) for nx in (16, 24, 32) for ny in (48, 64, 96) for nz in (16, 24, 32)]
    modes = [(nx + 1) * (2 * nz + 1) for nx, _, nz in sizes]
    total = 64 / len(sizes) * sum(modes)
    got = rules([(prec, m, ny, NSM, total / m) for m, (_, ny, _) in zip(modes, sizes)])
    assert sum(loaded(g[0], ny) for g, (_, ny, _) in zip(got, sizes)) <= 1.5 * sum(ny - 1 for _, ny, _ in sizes)


def test_solve_shapes(rules):
    """Eight threads per pair up to one wave of blocks, four below 65 536 pairs; four parts up to two blocks per SM
    of all members."""
    assert [r[1] for r in rules([("mixed", n, 64, NSM, 1.0) for n in (9728, 9729, 65535, 65536)])] == [5, 3, 3, 1]
    blocks = [(304, 1.0), (305, 1.0), (76, 4.0), (77, 4.0)]
    assert [r[2] for r in rules([("mixed", b, 64, NSM, t) for b, t in blocks])] == [1, 0, 1, 0]
