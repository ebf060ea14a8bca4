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


SLICE = dict(n_layer=4, hidden=2048, streams=4, hc_rank=256, vocab=4096, n_head=16, n_kv_head=2, head_dim=256, rope_dims=64, n_expert=512, n_expert_used=10, expert_ff=512,
             shared_ff=512, ssm_k_heads=16, ssm_v_heads=32, ssm_head_dim=128, conv_k=4, attn_interval=4, eps=1e-6, rope_theta=1e7)


@pytest.fixture(scope="module")
def slice4():
    return md.DeviceModel(md.make_model(SLICE, dense_type=szlib.TYPE_Q8_0, expert_type=szlib.TYPE_EXL3(3), seed=5, device="cuda"))


# histories of less than a chunk of 64 positions, of one, of many chunks a split and of many splits, at and beside their edges.  Five sequences in blocks of
# four warps, two chunks and more each; one and two (at most 128 blocks with positions) in blocks of eight
@pytest.mark.parametrize("lengths", [(70, 700, 1333, 3001, 5000), (2045, 4096, 8100, 61, 2048), (64, 7000), (6000,)])
def test_attention_of_a_step_over_long_histories_is_the_passes(slice4, lengths):
    n, ctx = len(lengths), 8192
    rng = np.random.default_rng(41)
    batch = md.Batch(slice4, n, ctx)
    alone = [md.Session(slice4, ctx, kv_q8=True, lean=True) for _ in range(n)]
    for b, length in enumerate(lengths):
        batch.sessions[b].fill_synthetic(length, seed=50 + b)
        alone[b].fill_synthetic(length, seed=50 + b)
    for step in range(2):                # (the second one stands on the first one's rows)
        rows = [[int(t) for t in rng.integers(0, SLICE["vocab"], 3 + (b + step) % 2)] for b in range(n)]
        batch.verify(rows)
        for b in range(n):
            got = batch.sessions[b].result(logits=True)[2].view(np.uint32)
            batch.sessions[b].commit(len(rows[b]))
            alone[b].verify(rows[b])
            want = alone[b].result(logits=True)[2].view(np.uint32)
            alone[b].commit(len(rows[b]))
            assert np.array_equal(got, want), "step %d, history %d" % (step, lengths[b])


# the projections of 9,216 and 12,352 outputs of 2,048 columns and of 2,048 of 4,096 at 8, 16, 24, 40, 64 and 80 rows: every form of their kernel
@pytest.mark.parametrize("ms", [(5,), (8, 3), (8, 8, 2), (8,) * 4 + (3,), (8,) * 8, (8,) * 9 + (5,)])
def test_projections_of_few_rows_are_the_passes(slice4, ms):
    rng = np.random.default_rng(43)
    batch = md.Batch(slice4, len(ms), 16)
    rows = [[int(t) for t in rng.integers(0, SLICE["vocab"], m)] for m in ms]
    batch.verify(rows)
    for b, r in enumerate(rows):
        s = md.Session(slice4, 16, kv_q8=True, lean=True)
        s.verify(r)
        assert np.array_equal(batch.sessions[b].result(logits=True)[2].view(np.uint32), s.result(logits=True)[2].view(np.uint32)), "sequence %d" % b


def fed_alone(dm, ctx, prompt):
    """A session that took the prompt in passes of up to 8 rows; the last one is pending."""
    s = md.Session(dm, ctx, kv_q8=True, lean=True)
    for c in range(0, len(prompt), 8):
        s.verify(prompt[c:c + 8])
        if c + 8 < len(prompt):
            s.result()
            s.commit(8)
    return s


# the scan's instances for more blocks than two a multiprocessor, with more stages of 8 rows than its ring has: prompts fed together, each one's last pass beside its
# chunk.  Some of the last pass is kept, and the next pass stands on the chunk's state and the kept rows'.
@pytest.mark.parametrize("d,lens", [(128, (75, 33, 41, 66)), (128, (17, 24, 57)), (64, (75, 40, 33, 64, 49, 9))])
def test_the_scan_of_many_sequences_chunks_is_the_passes(d, lens):
    cfg = dict(md.TINY, vocab=2048, n_expert=16, n_expert_used=4, shared_ff=256, n_layer=4, ssm_head_dim=d, ssm_k_heads=16, ssm_v_heads=32)
    dm = md.DeviceModel(md.make_model(cfg, expert_type=szlib.TYPE_EXL3(3), seed=24))
    prompts = [md.make_prompt(n, cfg["vocab"], seed=120 + n) for n in lens]
    batch = md.Batch(dm, len(lens), 128)
    batch.prefill(prompts)
    for b, p in enumerate(prompts):
        s, f = fed_alone(dm, 128, p), batch.sessions[b]
        keep = ((len(p) - 1) % 8 + 1 + 1) // 2
        for q in (s, f):
            q.first = q.result(logits=True)[2].view(np.uint32)
            q.commit(keep)
            q.verify([7, 8, 9, 10])
            q.second = q.result(logits=True)[2].view(np.uint32)
        assert len(f) == len(s) and np.array_equal(f.first, s.first) and np.array_equal(f.second, s.second), "prompt %d" % b


# a prompt's chunk at the shapes of the benchmark's layers: the router's 32 x 64 tiles, the combine a warp a row, the scan of one sequence, rows of two query tiles at its end
@pytest.mark.parametrize("n", [507, 268])
def test_a_long_chunk_at_the_benchmarks_layers_is_the_passes(slice4, n):
    prompt = md.make_prompt(n, SLICE["vocab"], seed=n)
    a, b = md.Session(slice4, 560, kv_q8=True), fed_alone(slice4, 560, prompt)
    a.prefill(prompt)
    for s in (a, b):
        s.first = s.result(logits=True)
        s.commit(2)
        s.verify([5, 6, 7])
        s.second = s.result(logits=True)
    assert np.array_equal(a.first[2].view(np.uint32), b.first[2].view(np.uint32)) and np.array_equal(a.first[1], b.first[1])
    assert np.array_equal(a.second[2].view(np.uint32), b.second[2].view(np.uint32)) and np.array_equal(a.second[1], b.second[1])
