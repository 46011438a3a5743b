"""Rules that the kernels and the host share as plain functions (stage_program.h), evaluated over all their arguments."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "souffle_models_b200", "csrc")


def _run(tmp_path, body):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    (tmp_path / "t.cpp").write_text('#include <cstdio>\n#include "stage_program.h"\nusing namespace souffle;\n'
                                    "#define CHECK(c) do { if (!(c)) { printf(\"line %d: %s\\n\", __LINE__, #c); return 1; } } while (0)\n"
                                    "int main() {\n" + body + "  return 0;\n}\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    run = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


def test_row_statistics_lie_in_a_box_of_a_warp_with_the_same_rows(tmp_path):
    """The two warps that meet over a quarter's statistics are the only ones that write the box these lie in."""
    _run(tmp_path, """
  for (int q = 0; q < 4; ++q)
    for (int w = 2; w < 10; ++w) {
      const bool owner = ln_stats_box(q) >= epi_box(w) && ln_stats_box(q) < epi_box(w) + 2;
      CHECK(owner == (w == epi_warp(q, 1)));
      if (owner) CHECK(epi_quarter(w) == q && epi_part(w) == 1 && ln_stats_box(q) == epi_box(w) + 1);
    }
  for (int w = 2; w < 10; ++w) CHECK(epi_warp(epi_quarter(w), epi_part(w)) == w);
""")


def test_a_late_cta_reads_the_number_of_its_own_launch(tmp_path):
    """Whichever other CTAs of a launch have left before it starts; and the next launch's number is the next one."""
    _run(tmp_path, """
  for (uint32_t ctas = 1; ctas <= kLaunchSteps; ++ctas) {
    uint32_t all = 0;
    for (uint32_t c = 0; c < ctas; ++c) all += launch_step(c, ctas);
    CHECK(all == kLaunchSteps);
    for (uint32_t late = 0; late < ctas; ++late) CHECK(launch_step(late, ctas) >= 1 && all - launch_step(late, ctas) < kLaunchSteps);
  }
""")
