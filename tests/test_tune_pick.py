"""The autotuners' choice among measured candidates (csrc/tune_pick.h), compiled for the host."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "csmv-gpu-stm_gb300" / "csrc"
MAIN = """#include "tune_pick.h"
#include <cstdio>
int main() {
  size_t n, k;
  if (scanf("%zu %zu", &n, &k) != 2) return 1;
  std::vector<double> ms(n);
  std::vector<size_t> again(k);
  for (double& x : ms) if (scanf("%lf", &x) != 1) return 1;
  for (size_t& i : again) if (scanf("%zu", &i) != 1) return 1;
  printf("%zu", csmv::tune_pick(again, ms));
}
"""


@pytest.fixture(scope="module")
def pick(tmp_path_factory):
    d = tmp_path_factory.mktemp("tune_pick")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", str(d / "main.cpp"), "-o", str(d / "pick")], check=True)

    def run(ms, again):
        text = " ".join(map(str, [len(ms), len(again), *ms, *again]))
        return int(subprocess.run([str(d / "pick")], input=text, capture_output=True, text=True, check=True).stdout)

    return run


@pytest.mark.parametrize("ms,again,want", [
    ([3, 2, 1, 4], [2, 1], 2),
    ([3, 2, 1, 2], [1, 3, 0], 1),
    ([3, 2, 1, 2], [3, 1, 0], 1),         # equal times, the other way round in the first runs
    ([5, 1e30, 5, 7], [1, 2, 0], 0),      # a candidate whose run failed
    ([1, 9, 9], [2, 1], 1),               # the fastest first run was not measured again
])
def test_equal_times_go_to_the_lowest_candidate(pick, ms, again, want):
    assert pick(ms, again) == want
