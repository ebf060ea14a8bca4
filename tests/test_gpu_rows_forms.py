"""The forms of a many-row launch that only some sizes take (csrc/sz_rows_rules.cuh), each against the passes whose bits it gives.  Which form a case
of ROUTES takes on 148 multiprocessors is checked on the host (test_rows_rules_host.py)."""
import numpy as np
import pytest
import torch

from tests.util import pkg

szlib, synth, md, moe = pkg.lib, pkg.synth, pkg.model, pkg.moe

pytestmark = pytest.mark.gpu

#: hidden, experts, of them a row, a shared one, rows, form: tiles that end in both directions, columns that end inside a part's second half (1,536), 17 ranks
ROUTES = [(2048, 1000, 16, True, 248, "SZ_ROUTE_32x64"), (1536, 500, 6, False, 248, "SZ_ROUTE_32x32"), (2048, 500, 10, True, 232, "SZ_ROUTE_32x32"),
          (2048, 500, 10, True, 200, "SZ_ROUTE_16x16"), (1024, 500, 6, True, 200, "SZ_ROUTE_16x16"), (4096, 200, 4, False, 248, "SZ_ROUTE_16x16"),
          (2048, 64, 8, True, 248, "SZ_ROUTE_PASS"), (4096, 16, 3, False, 256, "SZ_ROUTE_PASS"), (512, 20, 4, True, 136, "SZ_ROUTE_PASS")]


def layer(hidden, n_expert, top_k, shared, seed):
    L = synth.make_moe_layer(hidden, n_expert, top_k, 128, 128 if shared else 0, szlib.TYPE_EXL3(2), szlib.TYPE_EXL3(2), seed=seed)
    L["router"][1::3] = L["router"][0]      # ties, chosen by index
    return moe.MoeLayer(L, "cuda:0")


@pytest.mark.parametrize("hidden,n_expert,top_k,shared,rows,form", ROUTES)
def test_the_routers_forms_over_many_rows_are_the_passes(hidden, n_expert, top_k, shared, rows, form):
    ml = layer(hidden, n_expert, top_k, shared, 31)
    x = synth.normal((rows, hidden), 1.0, 33, "rows.forms").cuda()
    x[5::17] = 0.0
    y, ridx, rw = ml.moe_rows(x, want_routing=True)
    assert ml.moe_rows_status(rows) == 0
    for c in range(0, rows, 8):
        yc, ic, wc = ml.moe_batch(x[c:c + 8].contiguous(), want_routing=True)
        assert torch.equal(ridx[c:c + 8], ic) and torch.equal(rw[c:c + 8].view(torch.int64), wc.view(torch.int64)), "rows %d.." % c
        assert torch.equal(y[c:c + 8].view(torch.int32), yc.view(torch.int32)), "rows %d.." % c


# the kernel that chooses, behind tiles of every size: rows whose logits are not numbers, infinite either way or of both kinds, and their neighbours
@pytest.mark.parametrize("hidden,n_expert,top_k,rows", [(1024, 500, 10, 200), (2048, 500, 10, 232), (2048, 1000, 16, 248)])
def test_rows_that_are_not_numbers_are_routed_as_in_the_passes(hidden, n_expert, top_k, rows):
    ml = layer(hidden, n_expert, top_k, True, 35)
    x = synth.normal((rows, hidden), 1.0, 37, "rows.nan").cuda()
    x[3, 5] = float("nan")
    x[10, 700] = float("inf")
    x[77, 9] = float("-inf")
    x[rows - 1, 3], x[rows - 1, 900] = float("inf"), float("-inf")
    x[40] = 3e38                             # logits beyond f32
    y, ridx, rw = ml.moe_rows(x, want_routing=True)
    assert ml.moe_rows_status(rows) == 0
    for c in range(0, rows, 8):
        yc, ic, wc = ml.moe_batch(x[c:c + 8].contiguous(), want_routing=True)
        assert torch.equal(ridx[c:c + 8], ic), "rows %d.." % c
        for a, b in ((rw[c:c + 8], wc), (y[c:c + 8], yc)):
            assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(0.0, 1.0, -1.0), b.nan_to_num(0.0, 1.0, -1.0)), "rows %d.." % c
