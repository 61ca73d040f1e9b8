"""Kernels at the sizes where they can go wrong -- edges of tiles and groups, remainders, the
smallest and largest of a range -- against the CPU oracle. Sets of edges: every comparison is exact."""
import ctypes

import numpy as np
import pytest

import grg_gen as G
from test_csr5 import pack_csr5

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv", [1, 31, 32, 33, 193, 1000, 40_000])
def test_counts_and_hash_by_row_groups(grg_mod, oracle_mod, nv):
    """Counts, degrees and the hash are summed over groups of 1 to 32 rows a warp (fewer in small
    graphs); ranges that start and end inside a group add up to the whole."""
    w = G.alias(seed=nv, num_vars=nv, num_base_edges=3 * nv, block=min(nv, 300)) if nv > 1 else None
    if w is None:                                   # one vertex with a loop of each label
        src, dst, lab = np.zeros(3, np.uint32), np.zeros(3, np.uint32), np.arange(1, 4, dtype=np.uint8)
        rules, nl = np.array([[1, 1, 1], [2, 3, 1]], np.int32), 3
    else:
        src, dst, lab, rules, nl = w.src, w.dst, w.lab, w.rule_ids(), w.num_labels
    r = oracle_mod.closure(nv, rules, nl, 0, src, dst, lab)
    ctx, st = grg_mod.run_closure(nv, rules, nl, 0, src, dst, lab)
    counts = r.label_counts().tolist()
    assert ctx.label_counts().tolist() == counts and ctx.set_hash() == r.set_hash
    deg = ctx.degree()
    e, el = r.degree()
    assert np.array_equal(deg[0], e) and np.array_equal(deg[3], el)
    cuts = [0, nv // 3, nv // 3 + 1, nv - nv // 5, nv]
    parts = [ctx.range_counts(a, b) for a, b in zip(cuts, cuts[1:])]
    assert np.sum([p[0] for p in parts], axis=0).tolist() == counts
    assert sum(p[1] for p in parts) % (1 << 64) == r.set_hash
    ctx.close()


@pytest.mark.parametrize("nv,block,density", [(40, 40, 3), (700, 129, 4), (9_000, 1000, 4), (30_000, 383, 3),
                                              (3_500, 0, 2), (60_000, 1100, 2), (24_000, 1000, 4)])
def test_tiled_joins(grg_mod, oracle_mod, nv, block, density):
    """Grammars with a derivable second symbol join tiles of neighbouring rows. Blocks of a few ids,
    of more ids than one window of 8 elements holds (unconfined rows and their further windows), and
    of fewer records than a tile pays for give the oracle's closure, whole, alone and in a batch."""
    w = G.alias(seed=nv + block, num_vars=nv, num_base_edges=density * nv, block=block or None)
    r = oracle_mod.closure(nv, w.rule_ids(), w.num_labels, 0, w.src, w.dst, w.lab)
    want = (r.label_counts().tolist(), r.set_hash)
    for dev in (True, False):
        ctx = grg_mod.Context(0)
        ctx.set_device_rounds(dev)
        ctx.transfer_rules(w.rule_ids(), w.num_labels)
        ctx.load_edges(nv, w.src, w.dst, w.lab)
        ctx.closure(0)
        assert (ctx.label_counts().tolist(), ctx.set_hash()) == want
        ctx.close()
    ctx = grg_mod.Context(0)
    b = grg_mod.Batch(ctx, 2 * nv, 2, [(w.rules, w.labels)], 0)
    for j in (0, 1):
        b.admit(j, j * nv, 0, nv, w.src, w.dst, w.lab)
    b.step(0)
    for j in (0, 1):
        c, h = b.result(j, 0)
        assert (c.tolist(), h) == want
    ctx.close()


@pytest.mark.parametrize("kind,nv,block,ne,f", [
    ("small", 50, 0, 120, 0),            # one element a row
    ("small", 3_000, 0, 9_000, 0),       # 16 elements a row: two runs a batch, one window of 96
    ("small", 19_500, 0, 40_000, 0),     # rows of more elements than the widest window
    ("blocks", 64, 500, 1500, 1),        # narrow rows, and exits that reach five blocks
    ("blocks", 40, 1001, 3003, 0),
])
def test_row_joins(grg_mod, oracle_mod, kind, nv, block, ne, f):
    """Grammars with static right-hand rows: every window width, rows wider than all of them, small
    rounds cut into sub-records, and pools small enough that inserts fail and run again."""
    w = (G.dataflow_small(seed=nv, num_vars=nv, num_edges=ne) if kind == "small"
         else G.dataflow_blocks(seed=nv, num_blocks=nv, block=block, num_edges=ne * nv, seed_n=f == 1))
    r = oracle_mod.closure(w.num_vars, w.rule_ids(), w.num_labels, f, w.src, w.dst, w.lab)
    want = (r.label_counts().tolist(), r.set_hash)
    for dev, pool in ((True, 0), (False, 0), (True, 1 << 18)):
        ctx = grg_mod.Context(0)
        ctx.set_device_rounds(dev)
        ctx.transfer_rules(w.rule_ids(), w.num_labels)
        ctx.allocate_pool(pool)
        ctx.load_edges(w.num_vars, w.src, w.dst, w.lab)
        st = ctx.closure(f)
        assert (ctx.label_counts().tolist(), ctx.set_hash()) == want
        ctx.close()


@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("ne,fill", [(1, 0), (15, 0), (17, 0), (64, 1), (4_095, 0), (4_096, 1), (4_097, 0), (20_001, 1)])
def test_stream_edges_of_tiles(grg_mod, ne, fill, shift):
    """Streams of about a tile of 4,096 edges, of one full element (fill) and sparse ones, read from the
    device at an odd address too and written back as they were."""
    import torch

    rng = np.random.default_rng(ne + fill)
    V = 5_000
    src = rng.integers(0, V, ne) if not fill else rng.integers(0, 1 + ne // 700, ne) * 31
    dst = rng.integers(0, V if not fill else 400, ne)
    if fill:                                             # one element with all of its 192 ids
        src, dst = np.append(src, np.full(192, V - 1)), np.append(dst, np.arange(384, 576))
    lab = rng.integers(1, 3, len(src))
    e = np.unique(np.stack([src, lab, dst], 1), axis=0)
    want, deg = pack_csr5(e[:, 0], e[:, 2], e[:, 1], 0, V)
    buf = torch.zeros(len(want) + shift, dtype=torch.uint8, device="cuda")
    buf[shift:] = torch.from_numpy(want).cuda()
    ddeg = torch.from_numpy(deg.view(np.int32)).cuda()
    torch.cuda.synchronize()
    ctx = grg_mod.Context(0)
    ctx.transfer_rules(np.array([[1, 2, 1]], np.int32), 2)
    ctx._check(ctx._L.grg_load_csr5(ctx._h, V, 0, V, ctypes.c_void_p(ddeg.data_ptr()), len(e),
                                    ctypes.c_void_p(buf.data_ptr() + shift), 1), "load_csr5")
    assert [int(x) for x in ctx.label_counts()] == [int((e[:, 1] == k).sum()) for k in (1, 2)]
    for lo, hi in ((0, V), (0, V - 1)):
        got, gdeg = ctx.export_csr5(lo, hi)
        w, d = pack_csr5(e[:, 0], e[:, 2], e[:, 1], lo, hi)
        assert np.array_equal(got, w) and np.array_equal(gdeg, d)
    ctx.close()


@pytest.mark.parametrize("device_rounds", [True, False])
def test_joins_by_rows_are_reported(grg_mod, oracle_mod, device_rounds):
    """A closure that joins by rows times no window and no item form of the plain join and reports none;
    one that measures them (mode 3) may keep either kernel and says which; fixed ones run the plain join."""
    w = G.dataflow_blocks(seed=31, num_blocks=70 + 65 * device_rounds, block=1000, num_edges=210_000 + 195_000 * device_rounds)
    # a grammar of its own (X ::= N e beside N ::= N e): no other test has measured it in this process
    n, e = w.labels.index("N") + 1, w.labels.index("e") + 1
    rules, nl = np.array([[n, n, e], [w.num_labels + 1, n, e]], np.int32), w.num_labels + 1
    r = oracle_mod.closure(w.num_vars, rules, nl, w.filter_flag, w.src, w.dst, w.lab)
    want = (r.label_counts().tolist(), r.set_hash)
    rows = []
    for window, items in ((2, 2), (3, 3), (2, 2), (1, 1)):
        with grg_mod.Context(0) as ctx:
            ctx.set_device_rounds(device_rounds)
            ctx.set_join_window(window)
            ctx.set_join_items(items)
            ctx.transfer_rules(rules, nl)
            ctx.load_edges(w.num_vars, w.src, w.dst, w.lab)
            st = ctx.closure(w.filter_flag)
            assert (ctx.label_counts().tolist(), ctx.set_hash()) == want
            j = ctx.last_joins()
        assert (j["tiles"], j["tile_left"]) == (0, 0)
        if j["rows"]:
            assert st["wide_window"] == 0 and st["join_elements"] == 0
        rows.append((j["rows"], st["window_tuned"], st["window_trial_ms"]))
    assert rows[0] == (1, 0, [0.0, 0.0])                  # nothing to choose, nothing timed
    assert rows[1][1] == 1 and min(rows[1][2]) > 0
    assert rows[2] == (rows[1][0], 2, [0.0, 0.0])         # the measured choice holds for later closures
    assert rows[3][:2] == (0, 0)


def test_join_launches_are_those_with_records(grg_mod):
    """A round of few records is joined in one launch, whether the host or the device drives it."""
    w = G.alias(seed=8, num_vars=300, num_base_edges=900, block=100)
    for dev in (True, False):
        with grg_mod.Context(0) as ctx:
            ctx.set_device_rounds(dev)
            ctx.transfer_rules(w.rule_ids(), w.num_labels)
            ctx.load_edges(w.num_vars, w.src, w.dst, w.lab)
            st = ctx.closure(0)
            assert st["retry_records"] == 0 and ctx.last_joins()["tiles"] == 0
            assert st["join_launches"] == st["rounds"]


def test_partitions_keep_the_row_join(grg_mod, oracle_mod):
    """Runs of a partitioned graph choose their joins as a single closure does: none of them fixes the window
    of the plain join for the runs after it."""
    w = G.dataflow_blocks(seed=12, num_blocks=160, block=1000, num_edges=480_000)
    r = oracle_mod.closure(w.num_vars, w.rule_ids(), w.num_labels, w.filter_flag, w.src, w.dst, w.lab)
    with grg_mod.Context(0) as ctx:
        ctx.transfer_rules(w.rule_ids(), w.num_labels)
        p = grg_mod.Partitioned(ctx, w.num_vars, 2)
        p.load_edges(w.src, w.dst, w.lab)
        assert p.run(w.filter_flag)["runs"] >= 2
        counts, h = p.label_counts()
        p.close()
        assert (counts.tolist(), h) == (r.label_counts().tolist(), r.set_hash)
        assert ctx.last_joins()["rows"] == 1


@pytest.mark.parametrize("device_rounds", [True, False])
def test_closure_without_room_for_tile_lists(grg_mod, oracle_mod, monkeypatch, device_rounds):
    """The tile lists are memory a closure can do without: where they cannot be had, at all or past a size,
    the rounds run without tiles and the closure is the same."""
    w = G.alias(seed=9_000, num_vars=9_000, num_base_edges=36_000, block=1000)
    r = oracle_mod.closure(w.num_vars, w.rule_ids(), w.num_labels, 0, w.src, w.dst, w.lab)
    want = (r.label_counts().tolist(), r.set_hash)
    tiles = []
    for room in (None, "0", "40000"):
        if room is not None:
            monkeypatch.setenv("GRG_TILE_ROOM", room)
        with grg_mod.Context(0) as ctx:
            ctx.set_device_rounds(device_rounds)
            ctx.transfer_rules(w.rule_ids(), w.num_labels)
            for _ in range(2):
                ctx.load_edges(w.num_vars, w.src, w.dst, w.lab)
                ctx.closure(0)
                assert (ctx.label_counts().tolist(), ctx.set_hash()) == want
            tiles.append(ctx.last_joins()["tiles"])
    assert tiles[0] > 0 and tiles[1] == 0 and tiles[2] < tiles[0]


@pytest.mark.parametrize("local,device_rounds", [(True, True), (True, False), (False, True), (False, False)])
def test_row_joins_of_rows_wider_than_the_window(grg_mod, local, device_rounds):
    """Rows of more elements than the row join's whole window (96): records of local graphs keep their
    destinations in windows of their own, others in one a row. Compared with the plain join: the same
    closure, fewer destinations outside the windows."""
    if local:
        w = G.dataflow_small(seed=30, num_vars=30_000, num_edges=90_000)
        V, src, dst, lab = w.num_vars, w.src, w.dst, w.lab
    else:
        w = G.dataflow_small(seed=30, num_vars=100, num_edges=300)
        rng = np.random.default_rng(30)
        V = 40_000
        src, dst = rng.integers(0, V, (2, 60_000)).astype(np.uint32)
        lab = np.full(len(src), w.labels.index("e") + 1, np.uint8)
    got = []
    for window, items in ((2, 2), (1, 0)):
        with grg_mod.Context(0) as ctx:
            ctx.set_device_rounds(device_rounds)
            ctx.set_join_window(window)
            ctx.set_join_items(items)
            ctx.transfer_rules(w.rule_ids(), w.num_labels)
            ctx.load_edges(V, src, dst, lab)
            st = ctx.closure(0)
            got.append((ctx.label_counts().tolist(), ctx.set_hash(), st["window_out_elems"], ctx.last_joins()["rows"]))
    assert got[0][:2] == got[1][:2] and (got[0][3], got[1][3]) == (1, 0)
    assert 0 < got[0][2] < (0.3 if local else 0.7) * got[1][2]


def _wide(nv, rows, kblocks, bits, deg, seed=0):
    """A ::= B C over rows 0..rows-1 of B with `bits` intermediates in each of the first `kblocks` blocks of
    192 ids, and `deg` destinations of C for each of these (-deg: in the first 8 blocks); B and C are derived,
    so C is joined old-left too."""
    span, deg = (nv if deg > 0 else 8 * 192), abs(deg)
    rng = np.random.default_rng(seed + nv + kblocks + deg)
    k = np.concatenate([b * 192 + np.argsort(rng.random((rows, 192)), axis=1)[:, :bits] for b in range(kblocks)], axis=1)
    bsrc, bdst = np.repeat(np.arange(rows), kblocks * bits), k.ravel()
    esrc, edst = np.repeat(np.arange(kblocks * 192), deg), rng.integers(0, span, kblocks * 192 * deg)
    src, dst = np.concatenate([bsrc, esrc]).astype(np.uint32), np.concatenate([bdst, edst]).astype(np.uint32)
    lab = np.repeat(np.array([4, 5], np.uint8), [len(bsrc), len(esrc)])
    return nv, np.array([[2, 4, 0], [3, 5, 0], [1, 2, 3]], np.int32), 5, 0, src, dst, lab


@pytest.mark.parametrize("nv,rows,kblocks,bits,deg,left", [
    (20_000, 4000, 4, 50, 2000, "none"),     # right rows of 105 elements, dense: 14 windows
    (20_000, 4000, 4, 50, 150, "none"),      # the same, 79 of 105 elements in a row
    (200_000, 4000, 4, 50, 3, "all"),        # 3 elements a right row, anywhere in 1,042: given up after 8 windows
    (20_000, 3000, 40, 40, 5, "some"),       # more blocks of intermediates than a tile's table holds (32)
    (20_000, 3000, 50, 40, 4, "whole"),      # more leftovers than are cut: joined as they are
    (20_000, 4000, 100, 60, 4, "whole"),
    (20_000, 3000, 50, 40, -4, "whole"),     # (destinations in 8 blocks)
    (20_000, 1200, 36, 40, -4, "split"),     # leftovers cut by bitmap word (32,768 to 131,072 of them)
    (20_000, 300, 36, 40, -4, "parts"),      # fewer: cut into parts of 8 bits
])
def test_tiles_of_wide_rows(grg_mod, oracle_mod, nv, rows, kblocks, bits, deg, left):
    """Tiles at their limits: windows, blocks of intermediates, and the sizes of the list they leave (rows of
    more than 12 elements outgrow their tables, which then lie in any order: their own records make no tiles)."""
    w = _wide(nv, rows, kblocks, bits, deg)
    r = oracle_mod.closure(*w)
    want = (r.label_counts().tolist(), r.set_hash)
    for dev in (True, False):
        with grg_mod.Context(0) as ctx:
            ctx.set_device_rounds(dev)
            ctx.transfer_rules(w[1], w[2])
            ctx.load_edges(w[0], *w[4:])
            ctx.closure(0)
            assert (ctx.label_counts().tolist(), ctx.set_hash()) == want
            j = ctx.last_joins()
        assert j["tiles"] > 0
        lo, hi = {"none": (0, 0), "all": (8 * rows, None), "some": (1, None), "parts": (1, 32_767),
                  "split": (32_768, 131_071), "whole": (131_072, None)}[left]
        assert lo <= j["tile_left"] and (hi is None or j["tile_left"] <= hi)


@pytest.mark.parametrize("room", [None, "16"])
def test_tile_rows_that_outgrow_their_tables(grg_mod, oracle_mod, monkeypatch, room):
    """Rows of tiles whose inserts fail are joined again after their tables grow, or (more failures than the
    retry list holds) the whole round is."""
    if room:
        monkeypatch.setenv("GRG_RETRY_ROOM", room)
    w = _wide(20_000, 4000, 4, 50, 150)
    r = oracle_mod.closure(*w)
    for dev in (True, False):
        with grg_mod.Context(0) as ctx:
            ctx.set_device_rounds(dev)
            ctx.transfer_rules(w[1], w[2])
            ctx.load_edges(w[0], *w[4:])
            st = ctx.closure(0)
            assert (ctx.label_counts().tolist(), ctx.set_hash()) == (r.label_counts().tolist(), r.set_hash)
            assert ctx.last_joins()["tiles"] > 0 and st["retry_records"] > 0 and st["grow_rows"] >= 4000


def _chains(nv, length):
    """A ::= e, A ::= A A over chains of `length` vertices."""
    src = np.arange(nv - 1, dtype=np.uint32)
    src = src[(src + 1) % length != 0]
    return nv, np.array([[1, 2, 0], [1, 1, 1]], np.int32), 2, 0, src, src + 1, np.full(len(src), 2, np.uint8)


@pytest.mark.parametrize("nv,length,tiled", [(60_000, 20, False), (6_000, 24, False), (150_000, 30, False),
                                             (60_000, 400, True)])
def test_sparse_rounds_join_without_tiles(grg_mod, oracle_mod, nv, length, tiled):
    """Rounds whose records hold few intermediates run without tiles, however many they are."""
    w = _chains(nv, length)
    r = oracle_mod.closure(*w)
    for dev in (True, False):
        with grg_mod.Context(0) as ctx:
            ctx.set_device_rounds(dev)
            ctx.transfer_rules(w[1], w[2])
            ctx.load_edges(w[0], *w[4:])
            ctx.closure(0)
            assert (ctx.label_counts().tolist(), ctx.set_hash()) == (r.label_counts().tolist(), r.set_hash)
            assert (ctx.last_joins()["tiles"] > 0) == tiled


@pytest.mark.parametrize("w", [_chains(6_000, 24), _chains(6_000, 3_000), "alias"], ids=["sparse", "dense", "alias"])
def test_static_scratch_above_the_split_line(grg_mod, oracle_mod, w):
    """The allocation-free closure with rounds of more records than it cuts: with tiles and without."""
    import torch

    if w == "alias":
        a = G.alias(seed=9, num_vars=3_000, num_base_edges=12_000, block=1000)
        w = a.num_vars, a.rule_ids(), a.num_labels, 0, a.src, a.dst, a.lab
    nv, rules, nl, f, src, dst, lab = w
    r = oracle_mod.closure(*w)
    d = [torch.from_numpy(x).cuda() for x in (src.view(np.int32), dst.astype(np.uint32).view(np.int32), lab)]
    counts = torch.full((nl,), -1, dtype=torch.int64, device="cuda")
    h = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ptr = [ctypes.c_void_p(x.data_ptr()) for x in (*d, counts, h)]
    rules = np.ascontiguousarray(rules, np.int32).reshape(-1)
    rounds = ctypes.c_uint64()
    st = grg_mod.load_library().grg_closure_noalloc(0, None, len(rules) // 3, ctypes.c_void_p(rules.ctypes.data), nl, f,
                                                    nv, len(src), *ptr, ctypes.byref(rounds))
    assert st == grg_mod.OK
    got = counts.cpu().numpy().view(np.uint64).tolist(), int(h.cpu().numpy().view(np.uint64)[0])
    assert got == (r.label_counts().tolist(), r.set_hash)


@pytest.mark.parametrize("direct", ["0", "1"])
@pytest.mark.parametrize("room", [None, "16"])
@pytest.mark.parametrize("nv,ne", [(400, 900), (4_000, 5_200), (40_000, 30_000)])
def test_row_joins_of_several_rules(grg_mod, oracle_mod, monkeypatch, nv, ne, room, direct):
    """Two right-hand labels and unary rules through the row join, in a pool that leaves no room to presize
    rows: inserts of the join and of k_apply fail, tables grow, and the failed records (or, past the retry
    list, the whole pass) run again."""
    if room:
        monkeypatch.setenv("GRG_RETRY_ROOM", room)
    monkeypatch.setenv("GRG_DIRECT_INSERTS", direct)
    rng = np.random.default_rng(nv)
    src, dst = rng.integers(0, nv, (2, ne)).astype(np.uint32)
    lab = rng.integers(2, 4, ne).astype(np.uint8)
    rules = np.array([[1, 2, 0], [1, 1, 2], [1, 1, 3], [4, 1, 2], [4, 4, 3], [5, 4, 0]], np.int32)
    r = oracle_mod.closure(nv, rules, 5, 0, src, dst, lab)
    want = (r.label_counts().tolist(), r.set_hash)
    for dev in (True, False):
        with grg_mod.Context(0) as ctx:
            ctx.set_device_rounds(dev)
            ctx.transfer_rules(rules, 5)
            ctx.set_pool_limit(95 * nv * 65)              # slots of 65 bytes; presized rows take half of 96 nv
            ctx.load_edges(nv, src, dst, lab)
            st = ctx.closure(0)
            assert (ctx.label_counts().tolist(), ctx.set_hash()) == want
            assert ctx.last_joins()["rows"] == 1 and st["direct_inserts"] == int(direct)
            assert st["retry_records"] > 0 and st["grow_rows"] > 0


def test_window_tuned_for_the_plain_join(grg_mod, oracle_mod):
    """With the item form fixed the plain join runs, and the window that was measured for it is the one that
    later closures of the input report and use."""
    w = G.dataflow_blocks(seed=77, num_blocks=140, block=1000, num_edges=420_000)
    r = oracle_mod.closure(w.num_vars, w.rule_ids(), w.num_labels, w.filter_flag, w.src, w.dst, w.lab)
    seen = []
    for mode in (3, 2):
        with grg_mod.Context(0) as ctx:
            ctx.set_join_window(mode)
            ctx.set_join_items(1)
            ctx.transfer_rules(w.rule_ids(), w.num_labels)
            ctx.load_edges(w.num_vars, w.src, w.dst, w.lab)
            st = ctx.closure(w.filter_flag)
            assert (ctx.label_counts().tolist(), ctx.set_hash()) == (r.label_counts().tolist(), r.set_hash)
            assert ctx.last_joins()["rows"] == 0 and st["join_elements"] == 1
            seen.append((st["window_tuned"], st["wide_window"], min(st["window_trial_ms"]) > 0))
    assert seen == [(1, seen[0][1], True), (2, seen[0][1], False)]
