"""Hashing with a Poseidon2 state spread over four threads (small launches of both fields) and tree
levels computed a subtree per block: against the oracle, bit for bit, at every height where a run of
levels, a block's subtree or a warp's eight states ends, with padded layers (heights that are no
power of two), injections between runs, and rows of different widths in one warp."""
import numpy as np
import pytest

import ziros_b200 as Z
from conftest import BB_P, GL_P, rand_field

pytestmark = pytest.mark.gpu

FORMS = [(Z.BABYBEAR, 16), (Z.GOLDILOCKS, 16), (Z.GOLDILOCKS, 12)]


def _edges(field, m):
    m = m.copy()
    m[0] = 0
    m[-1] = (BB_P if field == Z.BABYBEAR else GL_P) - 1
    return m


def _check(oracle, field, width, mats, seed=5):
    root, tree = Z.CudaMerkleTreeMmcs(field, seed, width).commit(mats)
    want = oracle.mmcs_commit(oracle.hasher(field, seed, width), mats)
    got = tree.digest_layers()
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert (a == b).all()
    assert (root == want[-1][0]).all()


@pytest.mark.parametrize("field,width", FORMS)
@pytest.mark.parametrize("height", [1, 2, 3, 7, 8, 9, 31, 33, 255, 256, 257, 511, 513, 1000, 4099, 16384, 16385])
def test_trees(oracle, field, width, height):
    _check(oracle, field, width, [_edges(field, rand_field(field, (height, 1 + height % 19), height))])


@pytest.mark.parametrize("field,width", FORMS)
def test_injections_between_runs(oracle, field, width):
    rnd = lambda h, w: _edges(field, rand_field(field, (h, w), h + w))  # noqa: E731
    _check(oracle, field, width, [rnd(4096, 3), rnd(512, 9), rnd(256, 8), rnd(2, 1), rnd(1, 12)])
    _check(oracle, field, width, [rnd(3000, 5), rnd(1500, 4), rnd(94, 10), rnd(24, 2)])


@pytest.mark.parametrize("field,width", FORMS)
def test_batch_of_uneven_traces(field, width):
    shapes = [(1 << 5, 3), (1, 9), (1 << 9, 17), (1 << 3, 40), (1 << 6, 1), (2, 8), (1 << 10, 5), (1 << 4, 24)]
    traces = [_edges(field, rand_field(field, s, 60 + i)) for i, s in enumerate(shapes)]
    pcs = Z.CudaTwoAdicPcs(field, 42, 1, width)
    b = Z.BatchCommit(shapes, field=field, p2_width=width, autotune=False)
    for i, t in enumerate(traces):
        b.copy_in(i, t)
    b.run()
    roots = b.roots()
    for i, t in enumerate(traces):
        root, tree = pcs.commit(t)
        assert (roots[i] == root).all()
        assert all((x == y).all() for x, y in zip(b.tree(i).digest_layers(), tree.digest_layers()))


@pytest.mark.parametrize("field", [Z.BABYBEAR, Z.GOLDILOCKS])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 1000, 16384, 16385])
def test_batch_permutation(oracle, field, n):
    st = _edges(field, rand_field(field, (n, 16), n))
    rc, ne, ni = Z.round_constants(field, 7)
    want = np.asarray(oracle.permute(field, st, rc, ne, ni)).reshape(n, 16)
    pos = Z.CudaPoseidon2.new()
    assert (pos.batch_permute_babybear if field == Z.BABYBEAR else pos.batch_permute_goldilocks)(st.reshape(-1), rc, ne, ni)
    assert (st == want).all()
