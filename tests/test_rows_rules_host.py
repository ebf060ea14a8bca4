"""Which of two forms a many-row launch takes (csrc/sz_rows_rules.cuh), compiled for the host: at sizes where both were measured, the one that
was sooner."""
import os
import subprocess

import pytest

from tests.test_gpu_rows_forms import ROUTES
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


# (router rows, rows, columns) -> the form: where the router rows are few a verify pass's kernel, however many rows
@pytest.mark.parametrize("route_rows,rows,hidden,form", [(513, 128, 2048, "PASS"), (513, 136, 2048, "PASS"), (513, 176, 2048, "16x16"), (513, 256, 2048, "32x32"), (513, 504, 2048, "32x64"),
                                                         (17, 504, 2048, "PASS"), (65, 504, 2048, "PASS"), (129, 256, 2048, "PASS"), (257, 136, 2048, "PASS"), (257, 304, 2048, "16x16"),
                                                         (1001, 400, 2048, "16x16"), (17, 256, 4096, "PASS"), (65, 256, 4096, "PASS"), (129, 256, 4096, "16x16"), (513, 136, 4096, "16x16"),
                                                         (17, 504, 1024, "PASS"), (65, 256, 512, "PASS"), (513, 136, 1024, "16x16"), (513, 504, 512, "16x16")])
def test_router(tmp_path, route_rows, rows, hidden, form):
    assert ask(tmp_path, "sz_route_rows_form(%d, %d, %d, %d, 148) == SZ_ROUTE_%s" % (route_rows, rows, rows, hidden, form))


@pytest.mark.parametrize("hidden,n_expert,top_k,shared,rows,form", ROUTES)
def test_the_gpu_tests_reach_the_routers_forms(tmp_path, hidden, n_expert, top_k, shared, rows, form):
    assert ask(tmp_path, "sz_route_rows_form(%d, %d, %d, %d, 148) == %s" % (n_expert + shared, rows, rows, hidden, form))


# blocks with positions: one, two and three sequences at 8,000 (2 KV heads x 32 splits each), 32 at 200
@pytest.mark.parametrize("blocks,four", [(64, 0), (128, 0), (148, 0), (192, 1), (256, 1), (4096, 1)])
def test_attention_of_a_step(tmp_path, blocks, four):
    assert ask(tmp_path, "sz_attn_four_warps(%d, 148)" % blocks) == four


# (matrix rows, rows, columns) -> warps, groups of 8 rows, blocks that share the columns
@pytest.mark.parametrize("out,rows,cols,form", [(12352, 80, 2048, (8, 4, 1)), (9216, 8, 2048, (4, 1, 2)), (9216, 16, 2048, (4, 2, 2)), (12352, 16, 2048, (4, 2, 2)),
                                                (2048, 8, 4096, (4, 1, 4)), (2048, 24, 4096, (4, 1, 4)), (2048, 64, 4096, (4, 2, 2)), (2048, 80, 4096, (4, 2, 2)), (4096, 32, 1024, (4, 2, 2)),
                                                (2048, 8, 768, (4, 1, 2)), (8192, 8, 512, (4, 2, 1)), (1024, 32, 512, (4, 1, 4)), (12352, 16, 512, (4, 2, 1)), (12352, 24, 2048, (4, 2, 1))])
def test_projections(tmp_path, out, rows, cols, form):
    f = "sz_dense_rows_form(%d, %d, %d, 148)" % (out // 16, rows, cols)
    assert ask(tmp_path, "%s.warps * 100 + %s.groups * 10 + %s.share" % (f, f, f)) == form[0] * 100 + form[1] * 10 + form[2]
