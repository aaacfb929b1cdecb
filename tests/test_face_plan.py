"""The split of the reference profiles' face passes into launches (CPU)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cylinder-flow_gb300", "csrc")

PROG = r"""
#include <cstdio>
#include <cstdlib>
#include "face_plan.hpp"
// nops ndir limit cells...: per launch, per (pass, population): launch pass population cells
int main(int argc, char **argv) {
  cflbm::FaceOps ops{};
  ops.n = std::atoi(argv[1]);
  long long cells[6];
  for (int q = 0; q < ops.n; ++q) {
    ops.op[q].ndir = std::atoi(argv[2]);
    cells[q] = std::atoll(argv[4 + q]);
  }
  const long long limit = std::atoll(argv[3]) ? std::atoll(argv[3]) : cflbm::FACE_THREADS;
  int p = 0, k = 0, launch = 0;
  do {
    if (!cflbm::next_faces(ops, cells, limit, p, k)) { std::printf("beyond\n"); return 0; }
    if (ops.start[0] != 0 || ops.start[ops.n] > limit) return 1;
    for (int q = 0; q < ops.n; ++q) {
      if ((ops.start[q + 1] - ops.start[q]) % cells[q]) return 2;
      for (int j = 0; j < (ops.start[q + 1] - ops.start[q]) / cells[q]; ++j)
        std::printf("%d %d %d\n", launch, q, ops.first[q] + j);
    }
    ++launch;
  } while (p < ops.n);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "p.cpp").write_text(PROG)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(d / "p.cpp"), "-o", str(d / "p")], check=True)

    def run(nops, ndir, limit, cells):
        out = subprocess.run([str(d / "p"), *map(str, (nops, ndir, limit, *cells))], check=True, text=True,
                             capture_output=True).stdout
        return [tuple(map(int, line.split())) if line[0].isdigit() else line for line in out.splitlines()]
    return run


def faces(nx, ny, nz):
    xy, xz, yz = (nx + 2) * (ny + 2), (nx + 2) * (nz + 2), (ny + 2) * (nz + 2)
    return [xy, xy, xz, xz, yz, yz]


@pytest.mark.parametrize("shape,launches", [((257, 97, 97), 1), ((11000, 11000, 4), 3), ((17000, 17000, 4), 6)])
def test_every_population_of_every_pass_once(plan, shape, launches):
    got = plan(6, 9, 0, faces(*shape))
    assert [g[1:] for g in got] == [(q, k) for q in range(6) for k in range(9)]
    assert [g[0] for g in got] == sorted(g[0] for g in got) and got[-1][0] == launches - 1


@pytest.mark.parametrize("limit", [100, 101, 299, 300, 10 ** 6])
def test_split_at_any_limit(plan, limit):
    got = plan(4, 3, limit, [100, 100, 33, 7])
    assert [g[1:] for g in got] == [(q, k) for q in range(4) for k in range(3)]


def test_no_passes_and_a_plane_beyond_the_limit(plan):
    assert plan(0, 9, 0, []) == []
    assert plan(4, 3, 99, [100, 100, 33, 7]) == ["beyond"]
