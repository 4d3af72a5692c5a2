"""Kernel variants chosen by size, at the edges of their ranges, against the oracle."""
import ctypes

import numpy as np
import pytest
import scipy.sparse.csgraph
import torch

import pyoracle as po
import graphbrew_gb300 as gb
from graphbrew_gb300 import graphgen as gg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    assert torch.cuda.is_available(), "GPU tests need CUDA"
    c = gb.Context(0)
    yield c
    c.close()


def _communities(sizes, seed):
    """Communities of the given sizes on shuffled ids: random edges inside, a hub
    joined to every second member, a few edges across, members without an edge inside."""
    rng = np.random.default_rng(seed)
    n = int(sum(sizes))
    order = rng.permutation(n)
    edges, memb, at = [], np.zeros(n, dtype=np.uint32), 0
    for c, size in enumerate(sizes):
        ids = order[at:at + size]
        at += size
        memb[ids] = c
        live = ids[: max(2, size - size // 8)]
        u, v = rng.choice(live, 3 * size), rng.choice(live, 3 * size)
        edges += [(int(a), int(b)) for a, b in zip(u, v)]
        edges += [(int(ids[0]), int(b)) for b in ids[1::2]]
    u, v = rng.integers(0, n, n // 4 + 8), rng.integers(0, n, n // 4 + 8)
    edges += [(int(a), int(b)) for a, b in zip(u, v)]
    rp, col = gg.from_edges(n, edges)
    return rp.numpy(), col.numpy(), memb


@pytest.mark.parametrize("window", [1, 2, 8, 100])
@pytest.mark.parametrize("sizes", [
    (4, 5, 31, 32, 33, 34, 127, 128, 129, 514),
    (1023, 1024, 1025, 2048, 4096, 4097),
    (16383, 16384, 16385, 33),
])
def test_gorder_by_community_size(ctx, sizes, window):
    rp, col, memb = _communities(sizes, seed=sum(sizes) + window)
    recipe = gb.DEFAULT_RECIPE.replace("gw8", f"gw{window}").replace("gordf5000", "gordf100000")
    ids, st = ctx.order_compose(rp, col, memb, recipe)
    expect, ost = po.compose(rp, col, memb, gorder_window=window, gorder_fallback=100000)
    np.testing.assert_array_equal(ids, expect)
    assert [st["gorder_communities"], st["gorder_vertices"], st["gorder_max_community"]] == \
        [ost.gorder_communities, ost.gorder_vertices, ost.gorder_max_community]


@pytest.mark.parametrize("form", ["loops", "directed", "both"])
@pytest.mark.parametrize("window", [1, 8])
@pytest.mark.parametrize("sizes", [(20, 32, 33, 300, 1024), (1025, 4097, 16384), (16385, 40)])
def test_gorder_with_loops_and_directed_rows(ctx, sizes, window, form):
    # Rows that the input check lets through: every third vertex and each hub its own
    # neighbour, every fifth entry without its reverse.
    rp, col, memb = _communities(sizes, seed=sum(sizes) + window)
    n = len(rp) - 1
    src = np.repeat(np.arange(n), np.diff(rp))
    dst = col.astype(np.int64)
    if form != "loops":
        keep = (src * 7 + dst * 3) % 5 != 0
        src, dst = src[keep], dst[keep]
    if form != "directed":
        loops = np.union1d(np.arange(0, n, 3), np.argsort(np.diff(rp))[-2 * len(sizes):])
        src, dst = np.concatenate([src, loops]), np.concatenate([dst, loops])
    order = np.lexsort((dst, src))
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int64)
    col = dst[order].astype(np.int32)
    recipe = gb.DEFAULT_RECIPE.replace("gw8", f"gw{window}").replace("gordf5000", "gordf100000")
    ids, _ = ctx.order_compose(rp, col, memb, recipe)
    expect, _ = po.compose(rp, col, memb, gorder_window=window, gorder_fallback=100000)
    np.testing.assert_array_equal(ids, expect)


def _kernel_graph(kind, size):
    if kind == "star":        # one row at the edge of the segmented rows, and a path hanging off it
        edges = [(0, i) for i in range(1, size + 1)] + [(size + i, size + i + 1) for i in range(40)]
        return gg.from_edges(size + 60, edges)
    if kind == "stars":       # several long rows and bridges between them
        edges = [(h * size, h * size + i) for h in range(4) for i in range(1, size)]
        return gg.from_edges(4 * size + 3, edges + [(size - 1, size), (3 * size, 2 * size + 5)])
    if kind == "path":        # as many levels as vertices
        return gg.from_edges(size, [(i, i + 1) for i in range(size - 1)])
    if kind == "grid":        # frontiers on both sides of the one-CTA limit
        return gg.grid(size, 60000 // size + 3, 0.02, seed=size)
    return gg.uniform(size, 8, seed=size)


@pytest.mark.parametrize("kind,size", [("star", 7), ("star", 8), ("star", 9), ("star", 64), ("star", 65),
                                       ("star", 1023), ("star", 1024), ("star", 1025), ("star", 40000),
                                       ("stars", 2049), ("stars", 9000), ("path", 2), ("path", 33), ("path", 3001),
                                       ("grid", 3), ("grid", 245), ("uniform", 5), ("uniform", 13), ("uniform", 17)])
def test_kernels_by_row_length_and_frontier(ctx, kind, size):
    rp, col = (t.numpy() for t in _kernel_graph(kind, size))
    n = len(rp) - 1
    for source in {0, n // 2, int(np.argmax(np.diff(rp)))}:
        np.testing.assert_array_equal(ctx.bfs(rp, col, source)[0], po.bfs_depths(rp, col, source))
    np.testing.assert_array_equal(ctx.connected_components(rp, col)[0], po.cc_min_labels(rp, col))
    # Seven Jacobi sweeps in float64.  A float32 row sum of d terms in lanes and a
    # tree has a relative error below (d / 256 + 10) 2^-24 for the longest rows
    # here (40,000: 1e-5), and a sweep passes 0.85 of the error on.
    score = np.full(n, 1.0 / n)
    degree = np.diff(rp)
    row = np.repeat(np.arange(n), degree)
    for _ in range(7):
        share = np.where(degree > 0, score / np.maximum(degree, 1), 0.0)
        score = 0.15 / n + 0.85 * np.bincount(row, weights=share[col], minlength=n)
    got, sweeps, _ = ctx.pagerank(rp, col, max_iters=7, epsilon=0.0)
    assert sweeps == 7
    np.testing.assert_allclose(got, score, rtol=6e-5)
    # A converged run stops at the sweep whose change is below epsilon.
    _, stop, _ = ctx.pagerank(rp, col, max_iters=100, epsilon=1e-3)
    _, one_less, _ = ctx.pagerank(rp, col, max_iters=max(1, stop - 1), epsilon=1e-3)
    assert stop <= 100 and one_less == max(1, stop - 1)


def _spread(log_n, degree, gaps):
    """A uniform graph whose ids leave out `gaps` ranges: (first id moved, by how much)."""
    rp, col = gg.uniform(log_n, degree, seed=log_n, device="cuda")
    src = torch.repeat_interleave(torch.arange(rp.numel() - 1, device="cuda"), rp[1:] - rp[:-1])
    ids = torch.arange(1 << log_n, device="cuda")
    for first, by in gaps:
        ids[first:] += by
    return gg.squish(ids[src], ids[col.long()], int(ids[-1]) + 1 + (3 if gaps else 0))


def _float64_pagerank(rp, col, sweeps):
    rp, col = rp.cpu().numpy(), col.cpu().numpy()
    n, degree = len(rp) - 1, np.diff(rp)
    row, score = np.repeat(np.arange(n), degree), np.full(n, 1.0 / n)
    for _ in range(sweeps):
        share = np.where(degree > 0, score / np.maximum(degree, 1), 0.0)
        score = 0.15 / n + 0.85 * np.bincount(row, weights=share[col], minlength=n)
    return score


def _least(call, runs=5):
    return min(call() for _ in range(runs))


# Ranges of isolated ids before, inside and behind a chunk of 4,096 entries.
_GAPS = [((1000, 4096), (5000, 70000)), ((0, 300), (1, 255), (30000, 257)), ((30000, 1 << 22),),
         tuple((16 * k, 600) for k in range(1, 4000))]


@pytest.mark.parametrize("gaps", _GAPS)
def test_pagerank_with_gaps_in_the_ids(ctx, gaps):
    rp, col = _spread(16, 8, gaps)
    got, sweeps, _ = ctx.pagerank(rp, col, max_iters=7, epsilon=0.0)
    assert sweeps == 7
    np.testing.assert_allclose(got.cpu().numpy(), _float64_pagerank(rp, col, 7), rtol=6e-5)
    # The ids without entries cost their share of a few passes over the offsets: 4.2 M
    # of them are 34 MB, 5 us a pass.  Twenty such passes and as much again allowed.
    dense = _spread(16, 8, ())
    assert _least(lambda: ctx.pagerank(rp, col, max_iters=7, epsilon=0.0)[2]) <= \
        5 * _least(lambda: ctx.pagerank(*dense, max_iters=7, epsilon=0.0)[2]) + 0.2


@pytest.mark.parametrize("gaps", _GAPS + [((9000, 65000),), ((9000, 65536), (20000, 65300))])
def test_components_with_gaps_in_the_ids(ctx, gaps):
    rp, col = _spread(16, 1, gaps)   # some of its vertices isolated, many small components
    got, _ = ctx.connected_components(rp, col)
    rp_h, col_h = rp.cpu().numpy(), col.cpu().numpy()
    n = len(rp_h) - 1
    graph = scipy.sparse.csr_matrix((np.ones(len(col_h), dtype=np.int8), col_h, rp_h), shape=(n, n))
    _, label = scipy.sparse.csgraph.connected_components(graph, directed=False)
    first = np.full(n, n, dtype=np.int64)
    np.minimum.at(first, label, np.arange(n))
    np.testing.assert_array_equal(got.cpu().numpy(), first[label])
    # Seven passes over the vertices, 17 MB of parents each for 4.2 M ids: 20 us in all,
    # and as much for the offsets; ten times that allowed.
    dense = _spread(16, 1, ())
    assert _least(lambda: ctx.connected_components(rp, col)[1]) <= \
        5 * _least(lambda: ctx.connected_components(*dense)[1]) + 0.4


def test_input_check_of_one_long_row(ctx):
    # Every call checks its graph.  A row of 32 M entries is noted in 8,192 chunks: by a
    # warp 256 steps, 0.1 ms at most; a quarter of the call and twice that allowed beside a
    # path of the same size.
    def call_ms(u, v, n):
        rp, col = gg.squish(u, v, n)

        def once():
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            begin.record()
            ids, _ = ctx.dbg_mapping(rp, col)
            end.record()
            torch.cuda.synchronize()
            return begin.elapsed_time(end)
        return _least(once)

    leaves = torch.arange(1, (1 << 25) + 1, device="cuda")
    star = call_ms(torch.zeros_like(leaves), leaves, len(leaves) + 1)
    path = call_ms(leaves - 1, leaves, len(leaves) + 1)
    assert star <= 1.25 * path + 0.2
    for offsets in ([0, 40000, 0, 40000, 40000], [0, 50000, 40000], [0, 30000, 60000, 40000], [-5, 20000, 40000]):
        with pytest.raises(ValueError, match="row offsets"):
            ctx.dbg_mapping(torch.tensor(offsets, device="cuda"), torch.zeros(40000, dtype=torch.int32, device="cuda"))


def _bfs_levels(rp, col, source):
    """BFS depths, a level at a time over whole arrays."""
    depth = torch.full((len(rp) - 1,), -1, dtype=torch.int32, device=rp.device)
    depth[source] = 0
    front, level = torch.tensor([source], device=rp.device), 0
    while len(front):
        degree = rp[front + 1] - rp[front]
        first = torch.repeat_interleave(rp[front] - torch.cumsum(degree, 0) + degree, degree)
        reached = col[first + torch.arange(len(first), device=rp.device)].long()
        front = torch.unique(reached[depth[reached] < 0])
        level += 1
        depth[front] = level
    return depth


def _layers(width, fan, count):
    """Layers of `width` vertices, each joined to `fan` random ones of the next."""
    i = torch.arange(width * (count - 1), device="cuda").repeat_interleave(fan)
    rng = np.random.default_rng(width + fan)
    j = (i // width + 1) * width + torch.from_numpy(rng.integers(0, width, len(i))).cuda()
    return gg.squish(i, j, width * count)


@pytest.mark.parametrize("width,fan,count,most_us", [
    # Levels of the one-CTA kernel: rows on both sides of 8 entries, frontiers on both
    # sides of 2,048 vertices (4,096 above 1,310,720 vertices), 4,096 and 32,768 entries.
    (1, 1, 60, 0), (3, 7, 60, 0), (40, 40, 40, 0), (512, 4, 60, 0), (513, 4, 60, 0), (1025, 2, 60, 0),
    (2048, 8, 40, 0), (2049, 7, 40, 0), (1024, 16, 40, 0), (1024, 18, 40, 0), (33, 31, 60, 0),
    # A level of some 30,000 entries takes 34 us as two launches and a look at the
    # counters, and no longer by one CTA.
    (1900, 8, 500, 34), (1900, 8, 720, 34)])
def test_bfs_of_small_frontiers(ctx, width, fan, count, most_us):
    rp, col = _layers(width, fan, count)
    for source in {0, (width * count) // 2}:
        assert torch.equal(ctx.bfs(rp, col, source)[0], _bfs_levels(rp, col, source))
    if most_us:
        assert _least(lambda: ctx.bfs(rp, col, 0)[1]) <= 1e-3 * most_us * count


@pytest.mark.parametrize("intra", ["intra_bfs", "intra_rcm"])
def test_orders_of_long_paths_beside_a_hub(ctx, intra):
    # One community: a hub of 4 M leaves, 40 of which begin a path of 1,500 vertices, and a
    # uniform graph.  The levels along the paths cost what they do without the rest, but
    # for some dozen levels of the uniform graph's 67 M entries (a millisecond each).
    def order_ms(leaves, *extra):
        p, i = torch.arange(60000, device="cuda"), torch.arange(1, leaves + 1, device="cuda")
        u = [torch.zeros_like(i), torch.where(p % 1500 == 0, 1 + p // 1500, leaves + p)]
        v, n = [i, leaves + 1 + p], leaves + 60001
        if extra:
            rp, col = gg.uniform(*extra, seed=5, device="cuda")
            u += [torch.repeat_interleave(torch.arange(len(rp) - 1, device="cuda"), rp[1:] - rp[:-1]) + n]
            v += [col.long() + n]
            u, v, n = u + [torch.tensor([0], device="cuda")], v + [torch.tensor([n], device="cuda")], n + len(rp) - 1
        rp, col = gg.squish(torch.cat(u), torch.cat(v), n)
        memb = torch.zeros(n, dtype=torch.int32, device="cuda")
        recipe = gb.DEFAULT_RECIPE.replace("intra_gorder", intra)
        return _least(lambda: ctx.order_compose(rp, col, memb, recipe)[1]["intra_ms"], 3)

    alone = order_ms(40)
    assert order_ms(1 << 22, 21, 16) <= 1.25 * alone + (60 if intra == "intra_rcm" else 15)


@pytest.mark.parametrize("rows,in_dim,batch", [(1, 1, 1), (7, 12, 8), (9, 12, 8), (64, 3, 64), (129, 12, 128),
                                               (300, 32, 256), (513, 12, 100), (300, 33, 256), (300, 12, 257)])
def test_training_by_batch_and_inputs(ctx, rows, in_dim, batch):
    # One launch per epoch up to 32 inputs and minibatches of 256 rows, one per
    # kernel above: two epochs of Adam against float64 steps on the same shuffle.
    rng = np.random.default_rng(rows * 1000 + in_dim)
    count = ctx.mlp_param_count(in_dim)
    start = rng.normal(0, 0.3, count).astype(np.float32)
    x = rng.normal(0, 1, (rows, in_dim)).astype(np.float32)
    t = rng.normal(0, 1, (rows, 3)).astype(np.float32)
    seed, mask = 11, (1 << 64) - 1
    got, loss = ctx.mlp_train(start, x, t, epochs=2, batch=batch, lr=1e-3, seed=seed)
    p, m, v = start.astype(np.float64), np.zeros(count), np.zeros(count)
    order, word, step = list(range(rows)), (seed ^ 0x9E3779B97F4A7C15) & mask, 0
    for _ in range(2):
        for i in range(rows - 1, 0, -1):
            word = (word + 0x9E3779B97F4A7C15) & mask
            z = ((word ^ (word >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            order[i], order[j] = order[j], order[i]
        losses = []
        for at in range(0, rows, batch):
            pick = order[at:at + batch]
            l, g, _ = po.mlp_loss_grad(p, x[pick].astype(np.float64), t[pick].astype(np.float64))
            losses.append(l)
            step += 1
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            p = p - 1e-3 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    # Adam's step is at most lr whatever the gradient's size, so a gradient near
    # the rounding of its own sum can move a parameter by up to lr either way a
    # step; the others agree to the gradients' 1e-4.
    assert np.abs(got - p).max() <= 2 * step * 1e-3
    assert np.mean(np.abs(got - p) > 2e-3 * 1e-3 * step) < 0.02
    np.testing.assert_allclose(loss, np.mean(losses), rtol=1e-3)


@pytest.mark.parametrize("rows,in_dim", [(1, 1), (2, 32), (7, 12), (8, 12), (9, 12), (15, 1), (63, 31), (65, 12),
                                         (100, 12), (128, 12), (129, 32), (255, 12), (256, 1), (256, 32)])
def test_training_epoch_kernel_equals_the_launches(ctx, rows, in_dim):
    # A minibatch of all rows: `batch` up to 256 takes the one-launch epoch, 257 the
    # kernels one by one.  The same sums in the same order: equal to the last bit.
    rng = np.random.default_rng(rows * 1000 + in_dim)
    start = rng.normal(0, 0.3, ctx.mlp_param_count(in_dim)).astype(np.float32)
    x = rng.normal(0, 1, (rows, in_dim)).astype(np.float32)
    t = rng.normal(0, 1, (rows, 3)).astype(np.float32)
    expect, expect_loss = ctx.mlp_train(start, x, t, epochs=4, batch=257, lr=1e-3, seed=5)
    for batch in {rows, 256}:
        got, loss = ctx.mlp_train(start, x, t, epochs=4, batch=batch, lr=1e-3, seed=5)
        np.testing.assert_array_equal(got, expect)
        assert loss == expect_loss


def _fmaf(a, b, c):
    """a * b + c of float32 values, rounded once: the product is exact in float64, and
    the sum's rounding error turns it to the odd neighbour before the last rounding."""
    p, c = a.astype(np.float64) * b.astype(np.float64), c.astype(np.float64)
    s = p + c
    t = s - p
    err = (p - (s - t)) + (c - t)
    even = (s.view(np.int64) & 1) == 0
    return np.where((err != 0) & even, np.nextafter(s, np.copysign(np.inf, err)), s).astype(np.float32)


@pytest.mark.parametrize("rows,in_dim,batch", [(10, 12, 4), (129, 12, 64), (300, 12, 128), (300, 32, 256),
                                               (300, 33, 128)])
def test_training_steps_in_float32(ctx, rows, in_dim, batch):
    # Two epochs of several minibatches: the gradients of the kernels one by one and
    # Adam in float32, with its two fused multiply-adds.
    powf = ctypes.CDLL("libm.so.6").powf
    powf.restype, powf.argtypes = ctypes.c_float, [ctypes.c_float, ctypes.c_float]
    rng = np.random.default_rng(rows * 1000 + in_dim)
    p = rng.normal(0, 0.3, ctx.mlp_param_count(in_dim)).astype(np.float32)
    x = rng.normal(0, 1, (rows, in_dim)).astype(np.float32)
    t = rng.normal(0, 1, (rows, 3)).astype(np.float32)
    seed, mask, f = 11, (1 << 64) - 1, np.float32
    got, loss = ctx.mlp_train(p, x, t, epochs=2, batch=batch, lr=1e-3, seed=seed)
    m, v = np.zeros_like(p), np.zeros_like(p)
    b1, b2, one = f(0.9), f(0.999), f(1)
    order, word, step = list(range(rows)), (seed ^ 0x9E3779B97F4A7C15) & mask, 0
    for _ in range(2):
        for i in range(rows - 1, 0, -1):
            word = (word + 0x9E3779B97F4A7C15) & mask
            z = ((word ^ (word >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            order[i], order[j] = order[j], order[i]
        losses = []
        for at in range(0, rows, batch):
            pick = order[at:at + batch]
            g, l = ctx.mlp_gradient(p, x[pick], t[pick])
            losses.append(l)
            step += 1
            c1, c2 = one - f(powf(float(b1), step)), one - f(powf(float(b2), step))
            m = _fmaf(np.full_like(m, b1), m, (one - b1) * g)
            v = _fmaf(np.full_like(v, b2), v, (one - b2) * g * g)
            p = p - f(1e-3) * (m / c1) / (np.sqrt(v / c2) + f(1e-8))
    np.testing.assert_array_equal(got, p)
    assert f(loss) == f(np.sum(np.array(losses, dtype=np.float64)) / len(losses))


@pytest.mark.parametrize("lengths", [(0, 1, 2, 7, 8, 9, 31, 32, 33), (63, 64, 65, 127, 128, 129, 255, 256, 257),
                                     (511, 512, 513, 1023, 1024, 1025), (2047, 2048, 2049)])
def test_relabel_by_row_length(ctx, lengths):
    rng = np.random.default_rng(sum(lengths))
    n, hubs = 6000, 4 * len(lengths)
    edges = []
    for h in range(hubs):
        edges += [(h, int(w)) for w in hubs + rng.choice(n - hubs, lengths[h % len(lengths)], replace=False)]
    rp, col = (t.numpy() for t in gg.from_edges(n, edges))
    assert set(np.diff(rp)[:hubs]) == set(lengths)
    ids = rng.permutation(n).astype(np.int32)
    new_rp, new_col, old = ctx.relabel_by_mapping(rp, col, ids)
    expect_rp, expect_col = po.relabel(rp, col, ids)
    np.testing.assert_array_equal(new_rp, expect_rp)
    np.testing.assert_array_equal(new_col, expect_col)
    np.testing.assert_array_equal(ids[old], np.arange(n))


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 64, 65, 2047, 2048, 2049, 4095, 4096, 4097, 8192, 8193, 32767, 32768,
                               32769])
def test_sorts_and_scans_by_length(ctx, n):
    # DBG is one stable sort of n small keys; the rebuilt offsets are one scan.
    rp, col = (t.numpy() for t in _kernel_graph("stars", max(1, n // 4)) if n > 8) if n > 8 else \
        (t.numpy() for t in gg.from_edges(n, [(i, i + 1) for i in range(n - 1)]))
    n = len(rp) - 1
    degree = np.diff(rp)
    limits = (len(col) // n) * np.array([1, 2, 4, 8, 16, 32, 64]) // 2
    order = np.argsort(-np.searchsorted(limits, degree, side="left"), kind="stable")
    expect = np.empty(n, dtype=np.int32)
    expect[order] = np.arange(n, dtype=np.int32)
    ids, _ = ctx.dbg_mapping(rp, col)
    np.testing.assert_array_equal(ids, expect)
    new_rp, _, _ = ctx.relabel_by_mapping(rp, col, ids)
    np.testing.assert_array_equal(new_rp, np.concatenate([[0], np.cumsum(degree[order])]))


def _clustered_graph(kind, blocks, size):
    """Blocks whose super-nodes have tied (cliques), nearly tied (copies with a few
    extra edges) or many (a hub block) neighbours."""
    rng = np.random.default_rng(blocks * 1000 + size)
    edges = []
    for b in range(blocks):
        at = b * size
        edges += [(at + i, at + j) for i in range(size) for j in range(i)]
    between = [(b, (b + step) % blocks) for b in range(blocks) for step in (1, 2, 3)]
    if kind == "hub":
        between += [(0, b) for b in range(1, blocks)]
    for a, b in between:
        count = size if kind != "near" else size + int(rng.integers(0, 2))
        edges += [(a * size + int(i), b * size + int(j))
                  for i, j in zip(rng.permutation(size)[:count], rng.permutation(size)[:count])]
    if kind == "near":
        edges += [(int(a), int(b)) for a, b in rng.integers(0, blocks * size, (blocks // 3 + 1, 2)) if a != b]
    return gg.from_edges(blocks * size, edges)


@pytest.mark.parametrize("resolution", [1e-6, 0.3, 1.0, 1.7])
@pytest.mark.parametrize("kind,blocks,size", [("ties", 9, 5), ("ties", 1500, 4), ("near", 40, 6), ("near", 1500, 4),
                                              ("hub", 100, 5), ("hub", 300, 5), ("hub", 3000, 3)])
def test_super_moves_with_close_candidates(ctx, kind, blocks, size, resolution):
    rp, col = (t.numpy() for t in _clustered_graph(kind, blocks, size))
    memb, st = ctx.run_graphbrew(rp, col, gb.DEFAULT_RECIPE, resolution)
    expect, ost = po.leiden(rp, col, resolution)
    np.testing.assert_array_equal(np.asarray(memb).view(np.uint32), expect)
    assert [st["passes"], st["iterations"]] == [ost.passes, ost.iterations]


@pytest.mark.parametrize("sizes", [(1, 7, 8, 15), (16, 17, 18, 31, 32, 33), (48, 49, 63, 64, 65, 66),
                                   (127, 128, 129, 511, 512, 513, 1024), (2048, 2049, 4100, 40, 40),
                                   (20000, 33, 17, 300), (70000, 16, 65)])
def test_local_moving_by_moves_per_community(ctx, sizes):
    # Stars whose leaves join the centre's community in one window, the leaves'
    # ids shuffled; every fifth leaf also sees a leaf of the next star.
    rng = np.random.default_rng(sum(sizes))
    copies = max(1, 400 // sum(sizes))
    stars = [k for k in sizes for _ in range(copies)]
    n = sum(stars) + len(stars)
    ids = np.concatenate([np.arange(len(stars)), len(stars) + rng.permutation(sum(stars))])
    at, leaves, edges = len(stars), [], []
    for c, k in enumerate(stars):
        leaves.append(ids[at:at + k])
        at += k
        edges += [(c, int(v)) for v in leaves[-1]]
    for c in range(len(stars)):
        nxt = leaves[(c + 1) % len(stars)]
        edges += [(int(v), int(nxt[i % len(nxt)])) for i, v in enumerate(leaves[c][::5])]
    rp, col = (t.numpy() for t in gg.from_edges(n, [e for e in edges if e[0] != e[1]]))
    for resolution in (0.1, 1.0):
        memb, st = ctx.run_graphbrew(rp, col, gb.DEFAULT_RECIPE, resolution)
        expect, ost = po.leiden(rp, col, resolution)
        np.testing.assert_array_equal(np.asarray(memb).view(np.uint32), expect)
        assert [st["passes"], st["iterations"]] == [ost.passes, ost.iterations]


@pytest.mark.parametrize("parts", [("grid", "uniform", "grid"), ("uniform", "grid", "uniform")])
def test_local_moving_window_grows_and_shrinks(ctx, parts):
    # Consecutive id ranges that commit a window at once and in many rounds.
    at, edges = 0, []
    for i, kind in enumerate(parts):
        rp_t, col_t = gg.grid(300, 300, 0.05, seed=50 + i) if kind == "grid" else gg.uniform(17, 8, seed=50 + i)
        rp, col = rp_t.numpy(), col_t.numpy()
        src = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
        keep = src < col
        edges.append(np.stack([src[keep], col[keep]], axis=1) + at)
        if at:
            edges.append(np.array([[at - 1, at]]))
        at += len(rp) - 1
    e = np.concatenate(edges)
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.lexsort((dst, src))
    rp = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=at))]).astype(np.int64)
    col = dst[order].astype(np.int32)
    memb, st = ctx.run_graphbrew(rp, col, gb.DEFAULT_RECIPE, 1.0)
    expect, ost = po.leiden(rp, col, 1.0)
    np.testing.assert_array_equal(np.asarray(memb).view(np.uint32), expect)
    assert [st["passes"], st["iterations"]] == [ost.passes, ost.iterations]


def test_launch_count_of_sorts(ctx):
    # One community: the vertices' sort is one launch up to 4,096 of them, and above that
    # a histogram, a scan and a scatter for its one digit; the call's other kernels are the
    # same (scans of up to 32,768 values are one launch).
    def launches(n):
        rp, col = (t.numpy() for t in gg.from_edges(n, [(i, i + 1) for i in range(n - 1)]))
        recipe = gb.DEFAULT_RECIPE.replace("gordf5000", "gordf100000")
        return ctx.order_compose(rp, col, np.zeros(n, dtype=np.uint32), recipe)[1]["kernel_launches"]

    assert launches(4096) == launches(4095)
    assert launches(4097) == launches(4096) + 2


@pytest.mark.parametrize("n", [63, 64, 65, 2047, 2048, 2049, 4095, 4096, 4097, 8192, 8193, 12288, 32767, 32768, 32769])
def test_sorts_and_scans_of_exact_lengths(ctx, n):
    # Stars, a path over some of their leaves and isolated vertices up to n of them.
    rng = np.random.default_rng(n)
    size = max(2, n // 5)
    edges = [(h * size, h * size + i) for h in range(3) for i in range(1, size)]
    edges += [(int(i), int(i) + 1) for i in rng.choice(3 * size - 1, size // 2, replace=False)]
    rp, col = (t.numpy() for t in gg.from_edges(n, edges))
    assert len(rp) - 1 == n
    degree = np.diff(rp)
    limits = (len(col) // n) * np.array([1, 2, 4, 8, 16, 32, 64]) // 2
    order = np.argsort(-np.searchsorted(limits, degree, side="left"), kind="stable")
    ids, _ = ctx.dbg_mapping(rp, col)
    np.testing.assert_array_equal(ids[order], np.arange(n))
    new_rp, _, _ = ctx.relabel_by_mapping(rp, col, ids)
    np.testing.assert_array_equal(new_rp, np.concatenate([[0], np.cumsum(degree[order])]))


@pytest.mark.parametrize("order", ["super-rcm", "super-rabbit", "hilbert"])
@pytest.mark.parametrize("pairs", [1, 2, 4095, 4096, 4097, 8191, 8192, 8193, 12288])
def test_sorts_of_pairs_of_exact_lengths(ctx, pairs, order):
    # Every vertex a community and every edge a pair of them: the super-graph's sorts, of
    # 64-bit keys with and without values and three digits long, have `pairs` of them.
    rng = np.random.default_rng(pairs)
    n = 2000
    pick = rng.choice(n * (n - 1) // 2, pairs, replace=False)
    hi = ((1 + np.sqrt(1 + 8.0 * pick)) // 2).astype(np.int64)
    rp, col = (t.numpy() for t in gg.from_edges(n, np.stack([hi, pick - hi * (hi - 1) // 2], axis=1).tolist()))
    assert len(col) == 2 * pairs
    memb = np.arange(n, dtype=np.uint32)
    name = {"super-rcm": "sg_super_rcm", "super-rabbit": "sg_super_rabbit", "hilbert": "sg_hilbert"}[order]
    recipe = f"leiden:compose:{name}:comm_size_desc:intra_bfs:cd_serial:norefine:2:2"
    ids, _ = ctx.order_compose(rp, col, memb, recipe)
    np.testing.assert_array_equal(ids, po.compose(rp, col, memb, "size-desc", "bfs", super_order=order)[0])


@pytest.mark.parametrize("kind", ["grid", "grid above", "uniform", "rmat"])
def test_bfs_on_both_sides_of_the_bitmap(ctx, kind):
    # Shared memory holds the visited bitmap of 1,310,720 vertices; more of them take the
    # plain one-CTA levels, with frontiers that outgrow it and come back.
    rp, col = {"grid": lambda: gg.grid(1280, 1024, 0.1, seed=1, device="cuda"),
               "grid above": lambda: gg.grid(1280, 1025, 0.1, seed=2, device="cuda"),
               "uniform": lambda: gg.uniform(21, 2, seed=3, device="cuda"),
               "rmat": lambda: gg.rmat(21, 8, seed=4, device="cuda")}[kind]()
    degree = rp[1:] - rp[:-1]
    for source in {int(torch.argmax(degree)), int(torch.nonzero(degree == 1)[0])}:
        assert torch.equal(ctx.bfs(rp, col, source)[0], _bfs_levels(rp, col, source))
