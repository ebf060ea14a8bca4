"""The forms that take many rows at once, at the sizes where they could go wrong: one row more or less than a tile, a chunk, a block's
group; the smallest and largest of their ranges.  A session's rows are bit for bit those of passes of up to 8 rows; a block-format expert
layer and the tensor-core projections are held against the CPU restatement."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from oracle import binding as ob
from tests.test_gpu_batch import CFG
from tests.test_gpu_mma_cols import make
from tests.test_gpu_moe import run_case
from tests.util import pkg

szlib, synth, md, moe = pkg.lib, pkg.synth, pkg.model, pkg.moe

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dm():
    return md.DeviceModel(md.make_model(CFG, expert_type=szlib.TYPE_EXL3(3), seed=4, cycle_alpha=0.9, cycle_beta=0.5))


# the scan's stages of 8 rows: two, three, more than its ring; states of 64 and of 128 rows; value heads that share a key head
@pytest.mark.parametrize("n,d,kh,vh", [(17, 128, 4, 4), (25, 128, 2, 4), (66, 128, 1, 3), (41, 64, 2, 4)])
def test_the_scan_of_a_chunk_equals_the_scans_of_passes(n, d, kh, vh):
    cfg = dict(CFG, n_layer=2, ssm_head_dim=d, ssm_k_heads=kh, ssm_v_heads=vh)
    dm = md.DeviceModel(md.make_model(cfg, expert_type=szlib.TYPE_EXL3(3), seed=14))
    prompt = md.make_prompt(n, cfg["vocab"], seed=n)
    a, b = md.Session(dm, 160, kv_q8=True), md.Session(dm, 160, kv_q8=True)
    a.prefill(prompt)
    for c in range(0, n, 8):
        rows = prompt[c:c + 8]
        b.verify(rows)
        if c + 8 < n:
            b.result()
            b.commit(len(rows))
    _, top, lg = a.result(logits=True)
    _, top2, lg2 = b.result(logits=True)
    assert np.array_equal(lg.view(np.uint32), lg2.view(np.uint32)) and np.array_equal(top, top2)


# the rows of a prompt's last pass go with its last chunk: 1 and 8 of them; two chunks; a full room, where they do not fit; a session with
# no position to spare.  Then some of them are kept, and the next pass stands on chunk and pass.
@pytest.mark.parametrize("n,keep,ctx", [(17, 1, 64), (24, 3, 64), (31, 7, 64), (67, 0, 128), (48, 8, 48), (512, 5, 560), (520, 2, 560), (525, 4, 560)])
def test_a_prompts_last_pass_beside_its_last_chunk(dm, n, keep, ctx):
    prompt = md.make_prompt(n, CFG["vocab"], seed=90 + n)
    a, b = md.Session(dm, ctx, kv_q8=True), md.Session(dm, ctx, kv_q8=True)
    a.prefill(prompt)
    for c in range(0, n, 8):
        rows = prompt[c:c + 8]
        b.verify(rows)
        if c + 8 < n:
            b.result()
            b.commit(len(rows))
    for s in (a, b):
        s.first = s.result(logits=True)
        s.commit(keep)
    assert a.first[2].shape == b.first[2].shape and np.array_equal(a.first[2].view(np.uint32), b.first[2].view(np.uint32)) and np.array_equal(a.first[1], b.first[1])
    assert len(a) == len(b) == (n - 1) // 8 * 8 + keep
    if len(a) + 4 > ctx:
        return
    for s in (a, b):
        s.verify([7, 8, 9, 10])
        s.second = s.result(logits=True)
    assert np.array_equal(a.second[2].view(np.uint32), b.second[2].view(np.uint32)) and np.array_equal(a.second[1], b.second[1])


# 16 rows: the fewest that go as a chunk; 128 / 136: where the reads change their form; 512 / 520: one chunk, two
@pytest.mark.parametrize("n", [16, 17, 25, 129, 137, 145, 265, 513, 521, 529])
def test_a_prompt_in_chunks_equals_passes_of_eight_rows(dm, n):
    prompt = md.make_prompt(n, CFG["vocab"], seed=60 + n)
    a, b = md.Session(dm, 560, kv_q8=True), md.Session(dm, 560, kv_q8=True)
    a.prefill(prompt)
    for c in range(0, n, 8):
        rows = prompt[c:c + 8]
        b.verify(rows)
        _, top2, lg2 = b.result(logits=True)
        if c + 8 < n:
            b.commit(len(rows))
    _, top, lg = a.result(logits=True)
    assert np.array_equal(lg.view(np.uint32), lg2.view(np.uint32)) and np.array_equal(top, top2)
    for s in (a, b):
        s.commit((n - 1) % 8 + 1)
        s.verify([5, 6, 7])
    assert np.array_equal(a.result(logits=True)[2].view(np.uint32), b.result(logits=True)[2].view(np.uint32))


# the reads' many-row kernels (rank 256): 48 rows are the last without tiles, 56 the first; tiles of 32 rows and what is over them.  scale: the
# norm weights' - sums of 64 columns beyond 2^11 take the other way to fixed point, in both forms.  hidden 1,024: the columns in two parts (201 rows),
# in one wave of blocks (289) and in three parts in two waves (297 and 385).
@pytest.mark.parametrize("n,scale,hidden", [(49, 1.0, 0), (57, 1.0, 0), (65, 1.0, 0), (73, 1.0, 0), (137, 1.0, 0), (513, 1.0, 0), (65, 20000.0, 0),
                                            (201, 1.0, 1024), (289, 1.0, 1024), (297, 1.0, 1024), (385, 1.0, 1024)])
def test_the_reads_of_a_chunk_in_tiles_equal_the_passes(n, scale, hidden):
    M = md.make_model(dict(CFG, hc_rank=256, hidden=hidden or CFG["hidden"]), expert_type=szlib.TYPE_EXL3(3), seed=6)
    for k, t in M["tensors"].items():
        if k.endswith("hc_attn_norm.weight") or k.endswith("hc_ffn_norm.weight"):
            t[3].mul_(scale)
    dm = md.DeviceModel(M)
    prompt = md.make_prompt(n, CFG["vocab"], seed=n)
    a, b = md.Session(dm, 560, kv_q8=True), md.Session(dm, 560, kv_q8=True)
    a.prefill(prompt)
    for c in range(0, n, 8):
        b.verify(prompt[c:c + 8])
        _, top2, lg2 = b.result(logits=True)
        if c + 8 < n:
            b.commit(8)
    _, top, lg = a.result(logits=True)
    assert np.isfinite(lg).all() and np.array_equal(lg.view(np.uint32), lg2.view(np.uint32)) and np.array_equal(top, top2)


@pytest.mark.parametrize("n_expert,top_k,rows", [(16, 1, 8), (16, 16, 24), (16, 2, 256), (64, 4, 248), (512, 10, 136)])
def test_groups_of_many_and_of_few_rows_an_expert(n_expert, top_k, rows):
    """16 experts of 256 rows: more rows an expert than a group takes; 512 of 136: most experts have two or three; 16 of 16: all."""
    ty = szlib.TYPE_EXL3(3)
    ml = moe.MoeLayer(synth.make_moe_layer(512, n_expert, top_k, 256, 256, ty, ty, seed=7), "cuda:0")
    x = synth.normal((rows, 512), 1.0, 9, "rows.edges").cuda()
    y = ml.moe_rows(x)
    assert ml.moe_rows_status(rows) == 0
    for c in range(0, rows, 8):
        yc = ml.moe_batch(x[c:c + 8].contiguous())
        assert torch.equal(y[c:c + 8].view(torch.int32), yc.view(torch.int32)), "rows %d.." % c


# the shared expert in both launches of the routed ones, in the first only (another width), in none (another type), absent
@pytest.mark.parametrize("ff,sf,ety,sty,m", [(256, 256, "iq3", "iq3", 8), (256, 512, "iq3", "iq3", 3), (512, 512, "q8", "q8", 8), (256, 256, "iq3", "q8", 5),
                                             (512, 0, "iq3", "iq3", 4), (1024, 1024, "iq3", "iq3", 8), (256, 256, "q8", "q8", 1)])
def test_block_format_experts_with_and_without_the_shared_one_beside_them(ff, sf, ety, sty, m):
    ty = {"iq3": szlib.TYPE_IQ3_S, "q8": szlib.TYPE_Q8_0}
    run_case(512, 32, 4, ff, sf, ty[ety], ty[sty], m, seed=40)


# K in 2, 3 and 4 parts (3 of unequal length), two row tiles a block with a ragged last one, several units a block, one token a tile; either
# side of the line between the two rings of stages with K in 1, 2 and 4 parts
@pytest.mark.parametrize("rows,cols,m", [(130, 1024, 1), (300, 1024, 70), (385, 3328, 40), (129, 2304, 257), (512, 2048, 17), (3000, 768, 2049), (2600, 512, 2000),
                                         (1024, 3072, 1676), (1024, 3072, 1870), (1024, 3072, 2840), (256, 8192, 1438), (256, 8192, 1870)])
def test_projections_split_along_k_and_over_row_tiles(rows, cols, m):
    wb = make(rows, cols, 21)
    x = synth.normal((m, cols), 1.0, 23, "mma_cols.x")
    op = pkg.mma_cols.MmaCols(wb, rows, cols, m)
    y = torch.full((m + 1, rows + 5), -7.0, device="cuda")
    op(x.cuda(), out=y[:m, :rows])
    assert op.status() == 0 and bool((y[m] == -7.0).all()) and bool((y[:, rows:] == -7.0).all())
    w16 = torch.from_numpy(ob.dequant(ob.Q8_0, wb.numpy()).reshape(rows, cols)).half().double()
    x16 = x.half().double()
    want, mag = x16 @ w16.T, x16.abs() @ w16.abs().T
    assert float(((y[:m, :rows].cpu().double() - want).abs() / (cols * 2.0 ** -23 * mag + 1e-30)).max()) < 1.0


@pytest.mark.parametrize("lens,which", [([75, 3, 80, 200, 8, 9], None), ([300, 290], None), ([25, 75, 16], [1, 2])])
def test_prompts_of_a_batch_in_one_sessions_room_or_in_the_scratch(dm, lens, which):
    """One session of a batch has room for steps of 512 rows; without it (the others alone) the steps are the scratch's."""
    prompts = [md.make_prompt(n, CFG["vocab"], seed=80 + i) for i, n in enumerate(lens)]
    which = which if which is not None else list(range(len(lens)))
    batch = md.Batch(dm, len(lens), 320)
    batch.prefill([prompts[b] for b in which], which=which)
    for b in which:
        alone = md.Session(dm, 320, kv_q8=True, lean=True)
        alone.prefill(prompts[b])
        for s in (alone, batch.sessions[b]):
            s.top = s.result(logits=True)
            s.commit((lens[b] - 1) % 8 + 1)
            s.verify([5, 6, 7])
        assert np.array_equal(batch.sessions[b].top[2].view(np.uint32), alone.top[2].view(np.uint32)), "prompt %d" % b
        assert np.array_equal(batch.sessions[b].result(logits=True)[2].view(np.uint32), alone.result(logits=True)[2].view(np.uint32)), "after prompt %d" % b


def raise_error(dm, mem, addr, size):
    """Sets the error word of a room for up to 256 rows that ends `size` bytes after `addr` (its MoE scratch lies last: 64 bytes of
    counters a block of 8 rows, then the word), as an expert kernel whose wait ran out would."""
    n = C.c_int64()
    szlib.check(szlib.load().sz_moe_rows_scratch_bytes(C.byref(dm.model.layers[0].moe), 256, C.byref(n)))
    at = addr - mem.data_ptr() + size - n.value + 64 * (256 // 8) + 4
    word = mem[at:at + 4].view(torch.int32)
    assert int(word) == 0
    word.fill_(1)
    torch.cuda.synchronize()
    return word


def make_room(dm, rows, stream):
    lib, n, h = szlib.load(), C.c_int64(), C.c_void_p()
    szlib.check(lib.sz_room_bytes(C.byref(dm.model), rows, C.byref(n)))
    mem = torch.empty(n.value + 256, dtype=torch.uint8, device="cuda")
    addr = mem.data_ptr() + (-mem.data_ptr()) % 256
    torch.cuda.synchronize()
    szlib.check(lib.sz_room_create(C.byref(dm.model), rows, addr, n.value, stream, C.byref(h)))
    torch.cuda.synchronize()
    return h, mem, addr, n.value


def test_a_wait_that_ran_out_in_a_prompts_chunk_is_reported(dm):
    s = md.Session(dm, 128, kv_q8=True, lean=True)
    room, mem, addr, size = make_room(dm, 64, s.stream)
    szlib.check(s.lib.sz_session_use_room(s.h, room))
    word = raise_error(dm, mem, addr, size)
    s.prefill(md.make_prompt(60, CFG["vocab"], seed=90))
    with pytest.raises(szlib.SzError) as e:
        s.result()
    assert e.value.code == szlib.E_DEVICE
    assert int(word) == 0            # the session's now, until it is reset
    s.reset()
    s.prefill(md.make_prompt(60, CFG["vocab"], seed=90))
    s.result()
    s.lib.sz_room_destroy(room)


@pytest.mark.parametrize("shared", ["1", "0"])
def test_a_wait_that_ran_out_in_a_step_is_reported_by_every_sequence(dm, monkeypatch, shared):
    monkeypatch.setenv("SZ_BATCH_SHARED", shared)
    batch = md.Batch(dm, 3, 64)
    word = raise_error(dm, batch.mem, batch.scratch, batch.scratch_bytes)
    batch.verify([[1, 2], [3], [4, 5, 6]])
    for s in batch.sessions:
        with pytest.raises(szlib.SzError) as e:
            s.result()
        assert e.value.code == szlib.E_DEVICE
        s.reset()
    assert int(word) == 0
    batch.verify([[1, 2], [3], [4, 5, 6]])
    for s in batch.sessions:
        s.result()


@pytest.mark.parametrize("kind", ["shared", "own", "small"])
def test_sessions_of_several_threads_feed_their_prompts_through_a_room(dm, kind):
    """Four sessions, a thread and a stream each: the model's room, rooms of their own, one room of 16 rows (many chunks)."""
    prompts = [[md.make_prompt(n, CFG["vocab"], seed=200 + 10 * t + i) for i, n in enumerate((70, 17, 150))] for t in range(4)]
    room = None
    sessions = []
    for _ in prompts:
        s = md.Session(dm, 320, kv_q8=True, room=kind == "own", lean=kind == "small")
        if kind == "small":
            room = room or make_room(dm, 16, s.stream)
            szlib.check(s.lib.sz_session_use_room(s.h, room[0]))
        sessions.append(s)
    if room:
        sessions[0].lib.sz_room_destroy(room[0])      # (the sessions keep it)
    got = [[] for _ in prompts]

    def feed(t):
        s = sessions[t]
        for p in prompts[t]:
            s.reset()
            s.prefill(p)
            got[t].append(s.result(logits=True)[2])
            s.commit((len(p) - 1) % 8 + 1)
            s.verify([5, 6, 7])
            got[t].append(s.result(logits=True)[2])

    threads = [threading.Thread(target=feed, args=(t,)) for t in range(len(prompts))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    alone = md.Session(dm, 320, kv_q8=True, lean=True)       # in passes of 8
    for t, ps in enumerate(prompts):
        for i, p in enumerate(ps):
            alone.reset()
            alone.prefill(p)
            assert np.array_equal(alone.result(logits=True)[2].view(np.uint32), got[t][2 * i].view(np.uint32)), "thread %d, prompt %d" % (t, i)
            alone.commit((len(p) - 1) % 8 + 1)
            alone.verify([5, 6, 7])
            assert np.array_equal(alone.result(logits=True)[2].view(np.uint32), got[t][2 * i + 1].view(np.uint32)), "after prompt %d of thread %d" % (i, t)


def session_bytes(m, flags):
    n = C.c_int64()
    szlib.check(szlib.load().sz_session_bytes(C.byref(m.model), 320, flags, C.byref(n)))
    return n.value


def test_a_session_has_room_for_chunks_only_where_it_was_asked_for(dm):
    lib = szlib.load()
    n, small = C.c_int64(), C.c_int64()
    szlib.check(lib.sz_room_bytes(C.byref(dm.model), 512, C.byref(n)))
    szlib.check(lib.sz_room_bytes(C.byref(dm.model), 16, C.byref(small)))
    assert n.value > small.value > 0
    assert session_bytes(dm, 1) == session_bytes(dm, 1 | 4) == session_bytes(dm, 1 | 4 | 8)
    assert session_bytes(dm, 1 | 8) == session_bytes(dm, 1) + n.value
    assert session_bytes(dm, 8) == session_bytes(dm, 0)                                  # an f32 cache: prompts go in passes
    for rows in (0, 8, 20, 520):
        assert lib.sz_room_bytes(C.byref(dm.model), rows, C.byref(n)) == szlib.E_ARG
    h = C.c_void_p()
    assert lib.sz_room_create(C.byref(dm.model), 16, 4100, 1 << 40, 0, C.byref(h)) == szlib.E_ARG
    assert lib.sz_room_create(C.byref(dm.model), 16, 4096, small.value - 1, 0, C.byref(h)) == szlib.E_SCRATCH
    assert lib.sz_session_use_room(None, None) == szlib.E_ARG
    other = md.Session(md.DeviceModel(md.make_model(CFG, expert_type=szlib.TYPE_EXL3(3), seed=5)), 64, lean=True)
    room = md.Room(dm, other.stream, rows=16)
    assert lib.sz_session_use_room(other.h, room.h) == szlib.E_ARG       # another model's


def test_a_model_whose_prompts_go_in_passes_needs_no_room():
    lib = szlib.load()
    q8 = md.DeviceModel(md.make_model(md.TINY, seed=1))                  # Q8_0 experts
    n = C.c_int64(-1)
    szlib.check(lib.sz_room_bytes(C.byref(q8.model), 512, C.byref(n)))
    assert n.value == 0 and session_bytes(q8, 1 | 8) == session_bytes(q8, 1)
    h = C.c_void_p()
    assert lib.sz_room_create(C.byref(q8.model), 512, 4096, 1 << 40, 0, C.byref(h)) == szlib.E_TYPE
