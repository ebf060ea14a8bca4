"""Many-row dense projections on tcgen05 (`sz_mma_cols`) against the restated arithmetic of the reference's `mma_cols_<type>` family."""
import numpy as np
import pytest
import torch

from oracle import binding as ob
from tests.util import pkg

szlib, synth, mc = pkg.lib, pkg.synth, pkg.mma_cols

pytestmark = pytest.mark.gpu


def make(rows, cols, seed):
    w = synth.normal((rows, cols), 0.02, seed, "mma_cols.w")
    return synth.quantize_q8_0(w)


@pytest.mark.parametrize("rows,cols,m", [(128, 256, 16), (128, 256, 1), (200, 512, 100), (512, 2048, 256), (384, 2048, 300), (96, 4096, 64),
                                         (1024, 2048, 700)])
def test_rows_of_many_tokens_match_the_f16_restatement(rows, cols, m):
    wb = make(rows, cols, 5)
    x = synth.normal((m, cols), 1.0, 7, "mma_cols.x")
    op = mc.MmaCols(wb, rows, cols, m)
    y = op(x.cuda())
    assert op.status() == 0
    want, mag = ob.mma_cols_q8(wb.numpy(), rows, cols, x.numpy())
    got = y.cpu().numpy().astype(np.float64)
    # f32 accumulation of `cols` products: each partial sum is off by at most 2^-23 of the magnitudes summed so far
    bound = cols * 2.0 ** -23 * mag + 1e-30
    worst = float(np.max(np.abs(got - want) / bound))
    assert worst < 1.0, "distance / bound = %g" % worst
    # and against the exact f32 weights and inputs the mode is the reference's "inexact" one: about 1e-3 of the magnitudes
    exact = x.numpy().astype(np.float64) @ ob.dequant(ob.Q8_0, wb.numpy()).reshape(rows, cols).astype(np.float64).T
    assert float(np.max(np.abs(got - exact) / mag)) < 2e-3


def test_strided_rows_and_a_second_call_reuse_the_scratch():
    rows, cols, m = 256, 1024, 40
    wb = make(rows, cols, 11)
    xbig = synth.normal((m, cols + 64), 1.0, 13, "mma_cols.xs").cuda()
    x = xbig[:, :cols]                                 # row stride cols + 64 floats
    ybig = torch.full((m, rows + 32), -7.0, device="cuda")
    op = mc.MmaCols(wb, rows, cols, 64)
    op(x, out=ybig[:, :rows])
    a = ybig[:, :rows].clone()
    assert bool((ybig[:, rows:] == -7.0).all())        # nothing written past the rows
    op(x[:9], out=ybig[:9, :rows])                     # fewer tokens: another tile width
    assert op.status() == 0
    assert torch.equal(ybig[:9, :rows], a[:9])         # a token's result does not depend on how many tokens share the tile
    want, mag = ob.mma_cols_q8(wb.numpy(), rows, cols, x.cpu().numpy())
    assert float(np.max(np.abs(a.cpu().numpy() - want) / (cols * 2.0 ** -23 * mag))) < 1.0


# Every form of the kernel: one row tile without parts of K (one and several units a block), two row tiles, K in 2, 3 and 4 parts (and
# a tile narrower than 256 tokens); two calls in a burst write to buffers of their own, so that the second starts under the first.
@pytest.mark.parametrize("rows,cols,m,calls", [(12288, 2048, 256, 2000), (2600, 512, 2000, 2000), (3000, 768, 2049, 2000), (12288, 2048, 4093, 400),
                                               (8192, 2048, 256, 2000), (385, 3328, 40, 2000), (2048, 4096, 256, 2000), (512, 2048, 17, 2000)])
def test_thousands_of_calls_give_the_same_bits(rows, cols, m, calls):
    wb = make(rows, cols, 31)
    x = synth.normal((m, cols), 1.0, 33, "mma_cols.x").cuda()
    op = mc.MmaCols(wb, rows, cols, m)
    first = op(x).clone()
    w16 = torch.from_numpy(ob.dequant(ob.Q8_0, wb.numpy()).reshape(rows, cols)).cuda().half().double()
    for t in range(0, m, 512):     # against the f64 product of the f16 operands, within f32 accumulation
        x16 = x[t:t + 512].half().double()
        bound = cols * 2.0 ** -23 * (x16.abs() @ w16.abs().T) + 1e-30
        assert float(((first[t:t + 512].double() - x16 @ w16.T).abs() / bound).max()) < 1.0, "tokens %d.." % t
    ys = [torch.empty_like(first) for _ in range(4 if first.numel() < 1 << 24 else 2)]
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    seen = torch.empty_like(first)
    for _ in range(calls // len(ys)):
        for y in ys:
            op(x, out=y)
        for y in ys:
            off = torch.any(y.view(torch.int32) != first.view(torch.int32))
            seen = torch.where(off, y, seen)
            bad += off
    assert op.status() == 0
    if int(bad):
        at = (seen.view(torch.int32) != first.view(torch.int32)).nonzero()
        tok, row = at[:, 0].unique().tolist(), at[:, 1].unique().tolist()     # one row, all tokens: the weights' side; one token, 128 rows: the tokens'
        pytest.fail("%d of %d calls differ; in the last of them %d tokens (%s ..) and %d rows (%s ..)" % (int(bad), calls, len(tok), tok[:8], len(row), row[:8]))


def test_arguments_are_checked():
    wb = make(128, 256, 3)
    op = mc.MmaCols(wb, 128, 256, 16)
    with pytest.raises(szlib.SzError):
        mc.MmaCols(make(128, 96, 3), 128, 96, 16)      # cols not a multiple of 256
    bad = pkg.model.Tensor(14, 0, op.w.data_ptr(), 128, 256)
    import ctypes as C
    rc = op.lib.sz_mma_cols(C.byref(bad), 256, 256, 256, 128, 1, op.scratch.data_ptr(), op.scratch.numel(), 0)
    assert rc == szlib.E_TYPE if hasattr(szlib, "E_TYPE") else rc != 0


@pytest.mark.parametrize("rows,cols,m", [(200, 1024, 3830), (200, 1024, 3850), (130, 256, 513)])
def test_token_tiles_either_side_of_the_deep_rings_rule(rows, cols, m):
    # K in two parts: 15 token tiles take the deep ring, 16 the shallow one; 256 columns are one turn of the deep ring
    wb = make(rows, cols, 31)
    x = synth.normal((m, cols), 1.0, 33, "mma_cols.x")
    op = mc.MmaCols(wb, rows, cols, m)
    y = op(x.cuda())
    assert op.status() == 0
    w16 = torch.from_numpy(ob.dequant(ob.Q8_0, wb.numpy()).reshape(rows, cols)).half().double()
    x16 = x.half().double()
    want, mag = x16 @ w16.T, x16.abs() @ w16.abs().T
    # (f32 accumulation of `cols` products: each partial sum is off by at most 2^-23 of the magnitudes summed so far)
    assert float(((y.cpu().double() - want).abs() / (cols * 2.0 ** -23 * mag + 1e-30)).max()) < 1.0
