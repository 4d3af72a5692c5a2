"""Kernel variants chosen by size, at the edges of their ranges, against the oracle."""
import numpy as np
import pytest
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
