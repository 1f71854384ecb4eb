"""Hashing kernels whose permutations run their linear layers on the tensor cores (BabyBear width
16, launches of more than 18,944 rows): leaf digests, compressions, injections, the
alpha-reduction, column slabs, FRI layers and the batch permutation against the oracle, bit for
bit, at the sizes where a tile, a chunk or a block ends: heights one past a multiple of 128, widths
that end in a partial chunk, rows that are not 16-byte aligned, all-zero and all-(p-1) rows."""
import numpy as np
import pytest

import ziros_b200 as Z
from conftest import BB_P, rand_field

pytestmark = pytest.mark.gpu


def _edges(m):
    m = m.copy()
    m[0] = 0
    m[1] = BB_P - 1
    m[-1] = BB_P - 1
    m[-2, ::2] = 0
    return m


def _waits_ok():
    from ziros_b200 import _native as N

    assert N.ntt_tile_load_errors() == 0


def _check_layers(oracle, mats, seed=42):
    root, tree = Z.CudaMerkleTreeMmcs(Z.BABYBEAR, seed).commit(mats)
    want = oracle.mmcs_commit(oracle.hasher(Z.BABYBEAR, seed), mats)
    got = tree.digest_layers()
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert (a == b).all()
    assert (root == want[-1][0]).all()
    _waits_ok()


@pytest.mark.parametrize("height,width", [(18944, 11), (18945, 11), (37889, 3), (47361, 1), (65537, 7), (65536, 8), (60000, 9), (100001, 12), (94721, 31),
                                          (131072, 40), (47488, 66)])
def test_trees(oracle, height, width):
    _check_layers(oracle, [_edges(rand_field(Z.BABYBEAR, (height, width), height + width))], seed=width)


def test_several_matrices_and_injection(oracle):
    rnd = lambda h, w: _edges(rand_field(Z.BABYBEAR, (h, w), h + w))  # noqa: E731
    _check_layers(oracle, [rnd(262144, 3), rnd(131072, 5), rnd(262144, 6), rnd(65536, 17), rnd(131072, 1), rnd(64, 9)])
    _check_layers(oracle, [rnd(200001, 5), rnd(100001, 4), rnd(50001, 10)])


@pytest.mark.parametrize("height,width", [(65536, 24), (50001, 13)])
def test_reduction_fused_into_the_leaves(oracle, height, width):
    import torch

    m = _edges(rand_field(Z.BABYBEAR, (height, width), 5))
    alpha = rand_field(Z.BABYBEAR, 4, 6)
    d = torch.from_numpy(m.view(np.int32)).cuda()
    cw = torch.empty((height, 4), dtype=torch.int32, device="cuda")
    root, _ = Z.CudaMerkleTreeMmcs(Z.BABYBEAR, 42).commit_reduce_dev(d, alpha, cw)
    want = oracle.mmcs_commit(oracle.hasher(Z.BABYBEAR, 42), [m])
    assert (root == want[-1][0]).all()
    assert (cw.cpu().numpy().view(np.uint32) == oracle.combine_columns_ext4(m, alpha)).all()
    _waits_ok()


@pytest.mark.parametrize("width,transcript", [(128, False), (203, False), (200, True)])
def test_host_slabs_equal_the_oracle(oracle, width, transcript):
    t = _edges(rand_field(Z.BABYBEAR, (1 << 15, width), 9))
    alpha = rand_field(Z.BABYBEAR, 4, 10)
    pcs = Z.CudaTwoAdicPcs(Z.BABYBEAR, 42, 1)
    root, tree, pf = pcs.commit_fri(t, alpha, 8, 5, 1, 2, transcript=transcript)
    lde = oracle.coset_lde(Z.BABYBEAR, t, 1)
    want = oracle.mmcs_commit(oracle.hasher(Z.BABYBEAR, 42), [lde])
    assert (root == want[-1][0]).all()
    assert all((a == b).all() for a, b in zip(tree.digest_layers(), want))
    if not transcript:
        f = oracle.fri_commit_ext4(oracle.combine_columns_ext4(lde, alpha), 8, 42, 1, 5, 2)
        assert (pf.roots == f["roots"]).all() and (pf.final == f["final"]).all()
    _waits_ok()


def test_fri_layers(oracle):
    cw = _edges(rand_field(Z.BABYBEAR, (1 << 18, 4), 3))
    pf = Z.CudaFriProver(42, 8, 9, 7, 11).commit(cw)
    want = oracle.fri_commit_ext4(cw, 8, 42, 7, 9, 11)
    assert (pf.roots == want["roots"]).all() and (pf.final == want["final"]).all()
    _waits_ok()


@pytest.mark.parametrize("n", [18944, 18945, 47361, 120000])
def test_batch_permutation(oracle, n):
    import torch

    st = _edges(rand_field(Z.BABYBEAR, (n, 16), n))
    rc, ne, ni = Z.round_constants(Z.BABYBEAR, 7)
    want = oracle.permute(Z.BABYBEAR, st, rc, ne, ni)
    pos = Z.CudaPoseidon2.new()
    got = st.copy()
    assert pos.batch_permute_babybear(got.reshape(-1), rc, ne, ni)
    assert (got == np.asarray(want).reshape(n, 16)).all()
    # states that start off a 16-byte boundary
    buf = torch.empty(n * 16 + 1, dtype=torch.int32, device="cuda")
    off = buf[1:]
    off.copy_(torch.from_numpy(st.reshape(-1).view(np.int32)))
    pos.batch_permute_dev(Z.BABYBEAR, off, rc, ne, ni)
    assert (off.cpu().numpy().view(np.uint32).reshape(n, 16) == got).all()
    _waits_ok()


def test_batch_plan_of_mixed_widths():
    shapes = [(1 << 14, 7), (1 << 15, 8), (1 << 13, 33), (1 << 14, 20), (1 << 7, 3), (1 << 15, 5)]
    traces = [_edges(rand_field(Z.BABYBEAR, s, 100 + i)) for i, s in enumerate(shapes)]
    pcs = Z.CudaTwoAdicPcs(Z.BABYBEAR, 42, 1)
    b = Z.BatchCommit(shapes, autotune=False)
    for i, t in enumerate(traces):
        b.copy_in(i, t)
    b.run()
    roots = b.roots()
    for i, t in enumerate(traces):
        assert (roots[i] == pcs.commit(t)[0]).all()
    _waits_ok()
