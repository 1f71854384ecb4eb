"""Goldilocks hashing with the permutation's linear layers on the tensor cores (both widths, launches
of 8,192 rows or more): leaf digests, compressions, injections, the batch permutation and a batched
plan against the oracle, bit for bit, at heights around a multiple of 128, widths that end in a partial
chunk (alone, and after full ones), and all-zero, all-(p-1) and near-2^32 words."""
import numpy as np
import pytest

import ziros_b200 as Z
from conftest import GL_P, rand_field

pytestmark = pytest.mark.gpu


def _edges(m):
    m = m.copy()
    m[0] = 0
    m[1] = GL_P - 1
    m[2] = 0xFFFFFFFF
    m[3] = 0xFFFFFFFF00000000
    m[-1] = GL_P - 1
    m[-2, ::2] = 1 << 32
    return m


def _waits_ok():
    from ziros_b200 import _native as N

    assert N.ntt_tile_load_errors() == 0


def _check(oracle, width, mats, seed=42):
    root, tree = Z.CudaMerkleTreeMmcs(Z.GOLDILOCKS, seed, width).commit(mats)
    want = oracle.mmcs_commit(oracle.hasher(Z.GOLDILOCKS, seed, width), mats)
    got = tree.digest_layers()
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert (a == b).all()
    assert (root == want[-1][0]).all()
    _waits_ok()


@pytest.mark.parametrize("hasher", [12, 16])
@pytest.mark.parametrize("height,width", [(8191, 9), (8192, 9), (8193, 8), (19000, 24), (32769, 8), (65537, 1), (40000, 7), (50001, 13), (65536, 16),
                                          (75777, 18)])
def test_trees(oracle, hasher, height, width):
    _check(oracle, hasher, [_edges(rand_field(Z.GOLDILOCKS, (height, width), height + width))], seed=width)


@pytest.mark.parametrize("hasher", [12, 16])
def test_several_matrices_and_injection(oracle, hasher):
    rnd = lambda h, w: _edges(rand_field(Z.GOLDILOCKS, (h, w), h + w))  # noqa: E731
    _check(oracle, hasher, [rnd(131072, 3), rnd(65536, 5), rnd(131072, 6), rnd(65536, 4), rnd(64, 9)])


@pytest.mark.parametrize("n", [8191, 8192, 18945, 66000])
def test_batch_permutation(oracle, n):
    st = _edges(rand_field(Z.GOLDILOCKS, (n, 16), n))
    rc, ne, ni = Z.round_constants(Z.GOLDILOCKS, 7)
    want = np.asarray(oracle.permute(Z.GOLDILOCKS, st, rc, ne, ni)).reshape(n, 16)
    assert Z.CudaPoseidon2.new().batch_permute_goldilocks(st.reshape(-1), rc, ne, ni)
    assert (st == want).all()
    _waits_ok()


@pytest.mark.parametrize("hasher", [12, 16])
def test_batch_plan_of_mixed_widths(hasher):
    shapes = [(1 << 14, 7), (1 << 13, 8), (1 << 12, 33), (1 << 14, 20), (1 << 7, 3)]
    traces = [_edges(rand_field(Z.GOLDILOCKS, s, 100 + i)) for i, s in enumerate(shapes)]
    pcs = Z.CudaTwoAdicPcs(Z.GOLDILOCKS, 42, 1, hasher)
    b = Z.BatchCommit(shapes, field=Z.GOLDILOCKS, p2_width=hasher, autotune=False)
    for i, t in enumerate(traces):
        b.copy_in(i, t)
    b.run()
    roots = b.roots()
    for i, t in enumerate(traces):
        assert (roots[i] == pcs.commit(t)[0]).all()
    _waits_ok()
