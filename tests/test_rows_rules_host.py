"""Which of two forms a many-row launch takes (csrc/sz_rows_rules.cuh), compiled for the host: at sizes where both were measured, the one that
was sooner."""
import os
import subprocess

import pytest

from tests.util import ROOT

CSRC = os.path.join(ROOT, "shadow-engine_b200", "csrc")


def ask(tmp_path, expr):
    src = tmp_path / "rule.cpp"
    src.write_text('#include <cstdio>\n#include "sz_rows_rules.cuh"\nint main() { std::printf("%%d", (int)(%s)); }\n' % expr)
    exe = str(tmp_path / "rule")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wno-unused-function", "-I", CSRC, str(src), "-o", exe], check=True)
    return int(subprocess.run([exe], check=True, capture_output=True, text=True).stdout)


# (rows, columns, experts a row) -> a warp a (row, 128 outputs), or a warp a rank
@pytest.mark.parametrize("live,hidden,top_k,by_warp", [(504, 2048, 10, 1), (256, 2048, 10, 1), (208, 2048, 10, 1), (256, 2048, 16, 1), (136, 4096, 10, 1), (504, 1024, 10, 1), (136, 2048, 10, 1), (128, 2048, 16, 1), (288, 1024, 10, 1),
                                                       (1, 2048, 10, 0), (8, 2048, 16, 0), (80, 2048, 10, 0), (192, 2048, 10, 0), (160, 2048, 10, 0), (136, 2048, 8, 0), (136, 1024, 10, 0), (352, 1024, 10, 0), (320, 512, 10, 0),
                                                       (504, 2048, 8, 0), (256, 4096, 8, 0), (256, 2048, 2, 0)])
def test_combine(tmp_path, live, hidden, top_k, by_warp):
    assert ask(tmp_path, "sz_rows_combine_by_warp(%d, %d, %d, 148)" % (live, hidden, top_k)) == by_warp
