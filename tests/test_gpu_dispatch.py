"""The branches that the update's kernels choose by size, each at the sizes where it can go wrong,
against the oracle bit for bit:

  - near-far steps that a block continues by itself: short frontiers of light rows, the hand-over
    back to the grid, a chain longer than the claims' generations last;
  - threshold raises that find nothing below the new threshold and skip to the next distance;
  - relocated rows around the length above which a row moves in chunks, and rows around the length
    above which the index build and the compaction cut them;
  - host batches around the size that comes over with the control block;
  - the subtree walk that an update without a schedule tries when few tree edges changed: its
    limits in roots, batch, depth and width;
  - pointer jumping on either side of the size up to which it starts without a seeding pass, and
    on a graph that fills its vertex capacity.
"""
import numpy as np
import pytest

import dyng_b200 as D
from oracle import oracle as O
from tests.helpers import random_batch

pytestmark = pytest.mark.gpu

MOVE_CHUNK = 512          # slots of a row that move as one piece
LONG_ROW = 1024           # slots of a row that the storage passes take as one piece
PJ_SHORT = 1 << 18        # vertices up to which pointer jumping starts from the tree itself
STAGED_VALUES = 64 * 1024 // 4  # values of a host batch that come over with the control block


def _both(n, src, dst, w, props=None, oprops=None):
    g = D.Graph.from_edges(src, dst, w, n, props)
    og = O.Graph.from_edges(n, src, dst, w, 1, oprops)
    t = D.sssp.compute(g, 0)
    ot, _ = O.compute(og, 0, rule=1)
    _same(t, ot, "compute")
    return g, og, t, ot


def _same(t, ot, label):
    np.testing.assert_array_equal(t.distances, ot.distances, err_msg=label)
    np.testing.assert_array_equal(t.parents, ot.parents, err_msg=label)


def _update(g, og, t, ot, b, label, schedule=None):
    st = D.sssp.update(g, D.EdgeBatch.from_arrays(b["ins_src"], b["ins_dst"], b["ins_w"],
                                                  b["del_src"], b["del_dst"]), t, schedule)
    ost, osm = O.update(og, O.Batch(b["ins_src"], b["ins_dst"], b["ins_w"], b["del_src"],
                                    b["del_dst"]), ot)
    _same(t, ot, label)
    assert (st.invalidated, st.affected) == (ost["invalidated"], ost["affected"]), label
    assert st.batch.inserted_edges == osm["inserted_edges"], label
    assert st.batch.deleted_edges == osm["deleted_edges"], label
    return st


def _csr_same(g, og):
    csr, want = g.to_csr(), og.to_csr()
    np.testing.assert_array_equal(csr.row_ptr, want["row_ptr"])
    np.testing.assert_array_equal(csr.col_ind, want["col"])
    np.testing.assert_array_equal(csr.weights, want["w"])


def _i32(*a):
    return [np.asarray(x, np.int32) for x in a]


def _grid(side, rng, w_max):
    v = np.arange(side * side)
    x, y = v % side, v // side
    right, down = v[x + 1 < side], v[y + 1 < side]
    src = np.concatenate([right, right + 1, down, down + side])
    dst = np.concatenate([right + 1, right, down + side, down])
    return side * side, *_i32(src, dst, rng.integers(1, w_max, src.size, endpoint=True))


@pytest.mark.parametrize("side,delta", [(3, 0), (33, 1), (90, 0), (200, 0), (200, 1 << 40)])
@pytest.mark.parametrize("small", [0, -1, 1, 100000])
def test_short_frontiers_of_light_rows(side, delta, small):
    rng = np.random.default_rng(side)
    n, src, dst, w = _grid(side, rng, 50)
    g, og, t, ot = _both(n, src, dst, w)
    for step in range(3):
        b = random_batch(rng, n, src, dst, max(4, n // 20), tree_parents=ot.parents)
        _update(g, og, t, ot, b, f"step {step}", D.sssp.Schedule(delta=delta, small_frontier=small))


def test_repeated_updates_of_one_grid_keep_the_same_tree():
    # the same batch and its inverse again and again: a lost or doubled list entry anywhere shows
    # as another tree sooner or later
    rng = np.random.default_rng(8)
    n, src, dst, w = _grid(160, rng, 40)
    g, og, t, ot = _both(n, src, dst, w)
    pick = rng.choice(src.size, 900, replace=False)
    there = dict(ins_src=src[:0], ins_dst=dst[:0], ins_w=w[:0], del_src=src[pick], del_dst=dst[pick])
    back = dict(ins_src=src[pick], ins_dst=dst[pick], ins_w=w[pick], del_src=src[:0], del_dst=dst[:0])
    _update(g, og, t, ot, there, "there")
    want = ot.distances.copy(), ot.parents.copy()
    _update(g, og, t, ot, back, "back")
    home = ot.distances.copy(), ot.parents.copy()
    for i in range(400):
        for b, (d, p) in ((there, want), (back, home)):
            D.sssp.update(g, D.EdgeBatch.from_arrays(*b.values()), t)
            np.testing.assert_array_equal(t.distances, d, err_msg=str(i))
            np.testing.assert_array_equal(t.parents, p, err_msg=str(i))


def test_a_chain_longer_than_the_claims_generations():
    # 2^21 + 4096 dependent rounds in one call; then an update whose claims start over
    n = (1 << 21) + 4096
    src = np.arange(n - 1, dtype=np.int32)
    w = np.ones(n - 1, np.int32)
    g = D.Graph.from_edges(src, src + 1, w, n)
    t, st = D.sssp.compute(g, 0, stats=True)
    assert st.iterations >= n - 1
    np.testing.assert_array_equal(t.distances, np.arange(n))
    cut = n - 1000
    D.sssp.update(g, D.EdgeBatch(insert=([0], [cut], [5]), delete=([cut - 1], [cut])), t)
    want = np.arange(n)
    want[cut:] = 5 + np.arange(n - cut)
    np.testing.assert_array_equal(t.distances, want)


@pytest.mark.parametrize("gap", [1, 7, 1 << 20, 2**31 - 1])
def test_threshold_raises_over_gaps(gap):
    # chains whose edges weigh 1 or `gap`: with width 1 most raises find nothing
    rng = np.random.default_rng(3)
    n = 300
    src = np.concatenate([np.arange(n - 1), rng.integers(0, n, 60)])
    dst = np.concatenate([np.arange(1, n), rng.integers(0, n, 60)])
    w = np.where(rng.random(src.size) < 0.1, gap, 1)
    src, dst, w = _i32(src, dst, w)
    g, og, t, ot = _both(n, src, dst, w)
    for step in range(3):
        b = random_batch(rng, n, src, dst, 20, tree_parents=ot.parents)
        _update(g, og, t, ot, b, f"step {step}", D.sssp.Schedule(delta=1))


@pytest.mark.parametrize("kind", ["sorted", "append", "undirected", "multi"])
@pytest.mark.parametrize("length", [1, MOVE_CHUNK - 1, MOVE_CHUNK, MOVE_CHUNK + 1,
                                    2 * MOVE_CHUNK + 3, 5 * MOVE_CHUNK])
def test_relocated_rows_around_the_chunk_length(kind, length):
    # two hubs of `length` out-edges (and one of `length` in-edges) lose a third of their edges,
    # which leaves tombstones in every chunk, and take enough new ones to move
    rng = np.random.default_rng(length)
    n = 6 * MOVE_CHUNK + 64
    props = dict(sorted=kind in ("sorted", "undirected"), allow_multi=kind == "multi",
                 directed=kind != "undirected")
    far = 10 + rng.permutation(n - 10)[:length]
    src = np.concatenate([np.zeros(length), np.ones(length), far])
    dst = np.concatenate([far, far, np.full(length, 2)])
    src, dst = _i32(np.append(src, [0, 0]), np.append(dst, [1, 2]))
    w = rng.integers(1, 100, src.size).astype(np.int32)
    g, og, t, ot = _both(n, src, dst, w, D.GraphProperties(**props), O.default_props(
        directed=int(props["directed"]), sorted=int(props["sorted"]),
        allow_multi=int(props["allow_multi"])))
    gone = rng.random(src.size) < 1 / 3
    extra = 10 + rng.permutation(n - 10)[:length // 2 + 8]
    ins_src = np.concatenate([np.zeros(extra.size), np.ones(extra.size), extra])
    ins_dst = np.concatenate([extra, extra, np.full(extra.size, 2)])
    b = dict(zip(("ins_src", "ins_dst", "ins_w", "del_src", "del_dst"),
                 _i32(ins_src, ins_dst, rng.integers(1, 100, ins_src.size), src[gone], dst[gone])))
    _update(g, og, t, ot, b, "move")
    _csr_same(g, og)
    # the moved edges are found again (the edge index followed them)
    again = dict(ins_src=src[:0], ins_dst=dst[:0], ins_w=w[:0], del_src=src[~gone], del_dst=dst[~gone])
    _update(g, og, t, ot, again, "delete the moved edges")
    _csr_same(g, og)


@pytest.mark.parametrize("kind", ["sorted", "append", "multi"])
def test_index_build_and_compaction_of_long_rows(kind):
    # hubs with rows around one, two and five pieces on either side, churned until the abandoned
    # slots pass half the edges and the next overflow compacts: a third of every hub's edges go and
    # as many come, so its row holds tombstones in every piece when the pass reads it
    rng = np.random.default_rng(17)
    n = 5 * LONG_ROW + 200
    lengths = [1, 31, LONG_ROW - 1, LONG_ROW, LONG_ROW + 1, LONG_ROW + 32, 2 * LONG_ROW - 1,
               2 * LONG_ROW, 2 * LONG_ROW + 1, 5 * LONG_ROW]
    hubs = 2 + np.arange(len(lengths))
    far = [100 + rng.permutation(n - 100)[:size] for size in lengths]
    src = np.concatenate([[0] * hubs.size, *[np.full(f.size, h) for h, f in zip(hubs, far)],
                          *[f for f in far]])
    dst = np.concatenate([hubs, *far, *[np.full(f.size, 50 + h) for h, f in zip(hubs, far)]])
    src, dst, w = _i32(src, dst, rng.integers(1, 100, src.size))
    props = dict(sorted=kind == "sorted", allow_multi=kind == "multi")
    g, og, t, ot = _both(n, src, dst, w, D.GraphProperties(**props), O.default_props(
        sorted=int(props["sorted"]), allow_multi=int(props["allow_multi"])))
    builds = g.storage()["index_builds"]
    for step in range(60):
        gone = [f[rng.random(f.size) < 1 / 3] for f in far]
        come = [100 + rng.permutation(n - 100)[:x.size + 8] for x in gone]
        far = [np.unique(np.concatenate([np.setdiff1d(f, x), c])) for f, x, c in zip(far, gone, come)]
        pairs = lambda lists: (  # noqa: E731
            np.concatenate([*[np.full(x.size, h) for h, x in zip(hubs, lists)], *lists]),
            np.concatenate([*lists, *[np.full(x.size, 50 + h) for h, x in zip(hubs, lists)]]))
        i, j = pairs(come)
        b = dict(zip(("ins_src", "ins_dst", "ins_w", "del_src", "del_dst"),
                     _i32(i, j, rng.integers(1, 100, i.size), *pairs(gone))))
        _update(g, og, t, ot, b, f"step {step}")
        if g.storage()["compactions"] >= 2:
            break
    st = g.storage()
    assert st["compactions"] >= 2, st
    assert kind == "multi" or st["index_builds"] > builds
    _csr_same(g, og)
    # every edge is found through the rebuilt index
    csr = og.to_csr()
    rows = np.repeat(np.arange(n), np.diff(csr["row_ptr"]))
    some = rng.permutation(rows.size)[:4000]
    b = dict(zip(("ins_src", "ins_dst", "ins_w", "del_src", "del_dst"),
                 _i32([], [], [], rows[some], np.asarray(csr["col"])[some])))
    _update(g, og, t, ot, b, "delete")
    _csr_same(g, og)


@pytest.mark.parametrize("values", [2, STAGED_VALUES - 1, STAGED_VALUES, STAGED_VALUES + 1])
def test_host_batches_around_the_staged_size(values):
    # an insertion is three values of a host batch, a deletion two
    rng = np.random.default_rng(values)
    n = 4000
    src, dst = rng.integers(0, n, (2, 6 * n)).astype(np.int32)
    w = rng.integers(1, 100, src.size).astype(np.int32)
    g, og, t, ot = _both(n, src, dst, w)
    deletions = next(d for d in range(3) if (values - 2 * d) % 3 == 0)
    inserts = (values - 2 * deletions) // 3
    for step in range(2):
        pick = rng.integers(0, src.size, deletions)
        i, j = rng.integers(0, n, (2, inserts)).astype(np.int32)
        b = dict(ins_src=i, ins_dst=j, ins_w=rng.integers(1, 100, inserts).astype(np.int32),
                 del_src=src[pick], del_dst=dst[pick])
        _update(g, og, t, ot, b, f"step {step}")
    _csr_same(g, og)


@pytest.mark.parametrize("roots", [1, 31, 32, 33, 200])
@pytest.mark.parametrize("depth", [1, 5, 7, 60])
def test_few_changed_tree_edges(roots, depth):
    # a shallow dense part (six edges per vertex) with chains of `depth` below it: deleting the
    # chains' first edges invalidates them; the walk reaches them or leaves the rest to the rounds
    rng = np.random.default_rng(100 * roots + depth)
    core = 3000
    chains = 220
    n = core + chains * depth
    src = [rng.integers(0, core, 8 * n)]
    dst = [rng.integers(0, core, 8 * n)]
    w = [rng.integers(1, 50, 8 * n)]
    heads = rng.choice(core, chains, replace=False)
    first = core + np.arange(chains) * depth
    src.append(heads), dst.append(first), w.append(np.ones(chains))
    for k in range(1, depth):
        src.append(first + k - 1), dst.append(first + k), w.append(np.ones(chains))
    src, dst, w = _i32(np.concatenate(src), np.concatenate(dst), np.concatenate(w))
    g, og, t, ot = _both(n, src, dst, w)
    pick = rng.choice(chains, roots, replace=False)
    empty = src[:0]
    b = dict(ins_src=empty, ins_dst=empty, ins_w=empty,
             del_src=heads[pick].astype(np.int32), del_dst=first[pick].astype(np.int32))
    st = _update(g, og, t, ot, b, "cut")
    assert st.invalidated == roots * depth
    assert st.invalidation == (1 if roots <= 32 and depth <= 5 else 0)
    back = dict(ins_src=b["del_src"], ins_dst=b["del_dst"], ins_w=np.full(roots, 3, np.int32),
                del_src=empty, del_dst=empty)
    _update(g, og, t, ot, back, "mend")


@pytest.mark.parametrize("n", [9000, 60_000])
def test_a_cut_edge_above_most_of_the_tree_is_not_walked(n):
    # the source reaches a hub, and the hub nearly every vertex: its row is wider than a level of
    # the walk may be (32 slots per warp of 24 and 157 blocks), so nothing of it is walked
    rng = np.random.default_rng(n)
    v = np.arange(2, n)
    far = rng.integers(2, n, (2, 8 * n))
    src = np.concatenate([[0, 0], np.ones(n - 2), far[0]])
    dst = np.concatenate([[1, 2], v, far[1]])
    w = np.concatenate([[1, 10**6], rng.integers(1, 9, n - 2), rng.integers(10, 1000, 8 * n)])
    src, dst, w = _i32(src, dst, w)
    g, og, t, ot = _both(n, src, dst, w)
    cut = dict(zip(("ins_src", "ins_dst", "ins_w", "del_src", "del_dst"), _i32([], [], [], [0], [1])))
    st = _update(g, og, t, ot, cut, "cut")
    rows = st.work[D.sssp.Stats.WORK_NAMES.index("walk_rows")]
    assert st.invalidated >= n - 2
    assert st.invalidation == 0 and rows == 0


@pytest.mark.parametrize("roots,pairs", [(64, 2048), (65, 2048), (64, 2049), (20, 900)])
def test_the_walks_limits_on_a_large_graph(roots, pairs):
    # 2^20 vertices, one root per 16,384 allowed: leaves cut off, with other changes around them
    rng = np.random.default_rng(roots)
    n, leaves = 1 << 20, 100
    core = n - leaves
    src = np.concatenate([rng.integers(0, core, 7 * n), rng.integers(0, core, leaves)])
    dst = np.concatenate([rng.integers(0, core, 7 * n), np.arange(core, n)])
    w = rng.integers(1, 1000, src.size)
    src, dst, w = _i32(src, dst, w)
    g, og, t, ot = _both(n, src, dst, w)
    assert (ot.parents[core:] >= 0).sum() >= roots
    cut = core + np.nonzero(ot.parents[core:] >= 0)[0][:roots]
    other = rng.choice(core, pairs - roots, replace=False)  # heavy loops: no tree edge changes
    loop = np.full(other.size, 10**6)
    b = dict(zip(("ins_src", "ins_dst", "ins_w", "del_src", "del_dst"),
                 _i32(other, other, loop, ot.parents[cut], cut)))
    st = _update(g, og, t, ot, b, "cut")
    assert st.invalidated == roots
    assert st.invalidation == (1 if roots <= 64 and pairs <= 2048 else 0)


@pytest.mark.parametrize("depth", [1, 2, 3, 4, 40, 3000])
@pytest.mark.parametrize("n", [PJ_SHORT - 1, PJ_SHORT, PJ_SHORT + 1, PJ_SHORT + 5])
def test_pointer_jumping_around_the_seeded_size(n, depth):
    # chains of `depth` below the source (sparse: no walk), cut at random places, the last vertex
    # among them; every vertex keeps a heavy edge from the source
    rng = np.random.default_rng(n + depth)
    v = np.arange(1, n)
    src = np.concatenate([np.where((v - 1) % depth == 0, 0, v - 1), np.zeros(n - 1)])
    dst = np.concatenate([v, v])
    w = np.concatenate([rng.integers(1, 9, n - 1), np.full(n - 1, 10 * depth)])
    keep = (src[: n - 1] != 0).tolist() + [True] * (n - 1)  # one edge from the source per vertex
    src, dst, w = _i32(src[keep], dst[keep], w[keep])
    g, og, t, ot = _both(n, src, dst, w)
    cut = np.append(rng.choice(np.arange(1, n - 1), 60, replace=False), n - 1).astype(np.int32)
    empty = cut[:0]
    b = dict(ins_src=empty, ins_dst=empty, ins_w=empty, del_src=ot.parents[cut], del_dst=cut)
    st = _update(g, og, t, ot, b, "cut")
    assert st.invalidation == 0 and (depth < 3 or st.invalidated >= cut.size)


@pytest.mark.parametrize("blocks", [444, 300, 7, 0])
def test_pointer_jumping_of_a_graph_at_its_vertex_capacity(blocks):
    # 1,000 vertices leave room for 1,024 + 62 more; one batch brings them all.  A chain of `length`
    # leaves about as many survivors after round 0: 1,720 deal four entries a block where the
    # regions are five apart, so the last regions lie past the last vertex
    for length in (1723, 1600, 900, 2080):
        n0, n = 1000, 2086
        v = np.arange(1, n)
        parent = np.where((v > 1) & (v <= length), v - 1, 0)
        w = np.full(n - 1, 2)
        old = v < n0
        src, dst, w = _i32(parent, v, w)
        res = D.Resources()
        g = D.Graph.from_edges(src[old], dst[old], w[old], n0, resources=res)
        og = O.Graph.from_edges(n0, src[old], dst[old], w[old], 1)
        t = D.sssp.compute(g, 0)
        ot, _ = O.compute(og, 0, rule=1)
        empty = src[:0]
        grow = dict(ins_src=src[~old], ins_dst=dst[~old], ins_w=w[~old], del_src=empty, del_dst=empty)
        _update(g, og, t, ot, grow, "grow")
        cut = np.asarray([length - 3, length // 2, n - 1])
        b = dict(ins_src=empty, ins_dst=empty, ins_w=empty, del_src=parent[cut - 1].astype(np.int32),
                 del_dst=cut.astype(np.int32))
        _update(g, og, t, ot, b, "cut", D.sssp.Schedule(grid_blocks=blocks))
        back = dict(ins_src=b["del_src"], ins_dst=b["del_dst"], ins_w=np.full(cut.size, 3, np.int32),
                    del_src=empty, del_dst=empty)
        _update(g, og, t, ot, back, "mend", D.sssp.Schedule(grid_blocks=blocks))


def test_the_grid_follows_the_edges_and_the_batch():
    # 600 vertices with 180,000 edges are as much work as a sparse graph of many more vertices; a
    # batch that brings most of the graph, or names one far vertex, sizes the grid for what it leaves
    rng = np.random.default_rng(2)
    n = 600
    src, dst = rng.integers(0, n, (2, 300 * n)).astype(np.int32)
    w = rng.integers(1, 1000, src.size).astype(np.int32)
    g, og, t, ot = _both(n, src, dst, w)
    full = D.sssp.update(g, D.EdgeBatch(), t, D.sssp.Schedule(grid_blocks=1 << 20)).grid_blocks
    O.update(og, O.Batch(*_i32([], [], [], [], [])), ot)
    st = _update(g, og, t, ot, random_batch(rng, n, src, dst, 50, tree_parents=ot.parents), "dense")
    assert min(full, _edges(g) // 5000) <= st.grid_blocks <= full
    assert D.sssp.compute(g, 0, stats=True)[1].grid_blocks >= st.grid_blocks
    chain = np.arange(99, dtype=np.int32)
    for bring in (40_000, 1):
        g, og, t, ot = _both(100, chain, chain + 1, np.ones(99, np.int32))
        top = 200_000
        src, dst = rng.integers(0, top, (2, bring)).astype(np.int32)
        src[0], dst[0] = 99, top - 1
        empty = src[:0]
        b = dict(ins_src=src, ins_dst=dst, ins_w=rng.integers(1, 9, bring).astype(np.int32),
                 del_src=empty, del_dst=empty)
        st = _update(g, og, t, ot, b, "grow")
        assert st.grid_blocks >= min(full, top // 400)


def _edges(g):
    return int(g.to_csr().row_ptr[-1])


@pytest.mark.parametrize("delta", [1, 700, 0])
def test_heads_that_do_not_improve_start_the_threshold_at_their_distance(delta):
    # a tree kept as it was imported (not canonical): its insertion heads are pulled and pushed even
    # if the inserted edge brings them nothing; the first threshold lies above the smallest of them
    n = 400
    v = np.arange(1, n, dtype=np.int32)
    w = np.full(n - 1, 1000, np.int32)
    g, og, _, _ = _both(n, v - 1, v, w)
    t = D.sssp.Result.from_arrays(g, 0, np.arange(n) * 1000, np.arange(-1, n - 1), canonicalize=False)
    heads = np.asarray([310, 200, 350], np.int32)
    far = np.full(3, 2**30, np.int32)
    b = D.EdgeBatch.from_arrays(np.zeros(3, np.int32), heads, far, [], [])
    st = D.sssp.update(g, b, t, D.sssp.Schedule(delta=delta))
    np.testing.assert_array_equal(t.distances, np.arange(n) * 1000)
    np.testing.assert_array_equal(t.parents, np.arange(-1, n - 1))
    assert st.affected == 0
    width = st.delta
    raises = 0 if width > 150_000 else 4  # the other heads lie 110 and 150 edges on
    assert st.epochs <= raises
    assert st.trace[0][0] > 0  # the nearest head is pushed by the first step, without a raise
