"""The rule that decides which levels of a search run the dominance reductions."""
import itertools
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
DRIVER = r"""
#include <cstdio>
#include "search_rules.hpp"
int main() {
  int mode, word, bounded, pressure; double seconds, dropped, rest; unsigned parents; unsigned long long rows;
  while (std::scanf("%d %d %d %d %lf %lf %u %llu %lf", &mode, &word, &bounded, &pressure, &seconds, &dropped, &parents,
                    &rows, &rest) == 9) {
    sw::Reduction last; last.seconds = seconds; last.dropped = dropped; last.parents = parents;
    const sw::LevelRule r = sw::reductions_of_level(mode, word, bounded, pressure, last, rows, rest);
    std::printf("%d%d\n", (int)r.reduce, (int)r.left_out);
  }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_rule(tmp_path):
    (tmp_path / "rule.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'include'}", f"-I{ROOT / 'synchrowords_gb300' / 'csrc'}",
                    str(tmp_path / "rule.cpp"), "-o", str(tmp_path / "rule")], check=True)
    auto, always, memory = 0, 1, 2  # SW_REDUCE_*
    cases = list(itertools.product((auto, always, memory), (0, 1), (0, 1), (0, 1), (1e-3,), (0.0, 0.2), (0, 1000),
                                   (1000, 50000), (0.0, 1e-4, 10.0)))
    out = subprocess.run([str(tmp_path / "rule")], input="".join(" ".join(map(str, c)) + "\n" for c in cases),
                         capture_output=True, text=True, check=True).stdout.split()
    assert len(out) == len(cases)
    seen = set()
    for (mode, word, bounded, pressure, seconds, dropped, parents, rows, rest), got in zip(cases, out):
        wanted = mode == always or (mode == auto and word)
        dear = parents > 0 and rest > 0 and seconds * (rows / max(parents, 1)) ** 2 > 1.4 * dropped * rest
        left_out = wanted and mode == auto and bool(bounded) and dear and not pressure
        # only the checks' cost leaves them out: not a plan without them, nor memory bringing them on
        assert got == f"{int(bool(pressure) or wanted and not left_out)}{int(left_out)}"
        seen.add((got, mode, pressure))
    assert ("00", memory, 0) in seen and ("10", auto, 1) in seen and ("01", auto, 0) in seen


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_lists_stay_small(tmp_path):
    (tmp_path / "small.cpp").write_text("#include <cstdio>\n#include \"search_rules.hpp\"\nint main() {\n"
                                        "  double b, m; unsigned long long l;\n"
                                        "  while (std::scanf(\"%lf %llu %lf\", &b, &l, &m) == 3)\n"
                                        "    std::printf(\"%d\", (int)sw::lists_stay_small(b, l, m));\n}\n")
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'include'}", f"-I{ROOT / 'synchrowords_gb300' / 'csrc'}",
                    str(tmp_path / "small.cpp"), "-o", str(tmp_path / "small")], check=True)
    cases = [(b, l, m) for b in (1e6, 1e8, 1e9) for l in (0, 1, 5, 20) for m in (4e6, 1e9, 12e9)]
    out = subprocess.run([str(tmp_path / "small")], input="".join(f"{b} {l} {m}\n" for b, l, m in cases),
                         capture_output=True, text=True, check=True).stdout
    assert out == "".join(str(int(4 * b * 1.3 ** l <= m)) for b, l, m in cases)
