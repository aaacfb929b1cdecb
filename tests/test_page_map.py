"""Mapping of a buffer's pages ahead of copies into it (CPU)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cylinder-flow_gb300", "csrc")

PROG = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "page_map.hpp"
using cflbm::PageMapper;
// mode offset: what the mapper did with a 24 MB buffer (+ offset) and whether its bytes kept
int main(int argc, char **argv) {
  const char *mode = argv[1];
  const size_t off = std::atoll(argv[2]), page = sysconf(_SC_PAGESIZE), n = (24u << 20) + 1234, all = n + off + page;
  const bool ro = !std::strcmp(mode, "readonly");
  char *m = (char *)mmap(nullptr, all, ro ? PROT_READ : PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  char *p = m + off;
  if (!std::strcmp(mode, "resident")) std::memset(m, 7, all);
  if (!std::strcmp(mode, "part")) for (size_t o = 0; o < n; o += 1000003) p[o] = (char)(o % 251 + 1);
  if (!std::strcmp(mode, "hole")) munmap(m + all / 2 / page * page, page);
  bool did;
  {
    PageMapper map;
    did = map.start(p, n);
    map.wait(n);
    if (did && !ro) {  // every page is there
      char *b = p - (size_t)p % page;
      std::vector<unsigned char> v((p + n - b + page - 1) / page);
      if (mincore(b, p + n - b, v.data())) return 2;
      for (unsigned char c : v) if (!(c & 1)) return 3;
    }
  }
  bool kept = true;
  if (!std::strcmp(mode, "part")) for (size_t o = 0; o < n; o += 1000003) kept = kept && p[o] == (char)(o % 251 + 1);
  if (!std::strcmp(mode, "resident")) for (size_t o = 0; o < n; o += 997) kept = kept && p[o] == 7;
  std::printf("%d %d\n", did, kept);
}
"""


@pytest.fixture(scope="module")
def prog(tmp_path_factory):
    d = tmp_path_factory.mktemp("pages")
    (d / "p.cpp").write_text(PROG)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, str(d / "p.cpp"), "-o", str(d / "p")], check=True)
    return str(d / "p")


@pytest.mark.parametrize("offset", [0, 8, 4096 - 8])
@pytest.mark.parametrize("mode,did", [("fresh", "1"), ("part", "1"), ("resident", "0"), ("hole", "0"),
                                      ("readonly", None)])
def test_maps_only_what_is_missing_and_keeps_bytes(prog, mode, did, offset):
    r = subprocess.run([prog, mode, str(offset)], text=True, capture_output=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
    got = r.stdout.split()
    assert got[1] == "1" and (did is None or got[0] == did)
