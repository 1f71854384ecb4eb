"""Batch permutations by their form: quads of threads for few states, one state a thread for more and
for numbers of rounds that the tensor-core kernels are not built for, the tensor-core kernel by the
number of 128-state tiles an SM."""
import numpy as np
import pytest
import torch

import ziros_b200 as Z
from conftest import rand_field

pytestmark = pytest.mark.gpu


def _constants(field, ext, internal):
    return rand_field(field, ext * 16 + internal, 1000 * ext + internal)


# around the sizes at which the form changes, a ragged last block, more states than the grid has threads
@pytest.mark.parametrize("field,ext,internal", [(Z.BABYBEAR, 8, 14), (Z.BABYBEAR, 2, 0), (Z.GOLDILOCKS, 8, 21),
                                                (Z.GOLDILOCKS, 6, 22)])
@pytest.mark.parametrize("n", [5, 18944, 18945, 19077, 65535, 65536, 65537, 303105])
def test_equals_the_oracle(oracle, field, ext, internal, n):
    rc = _constants(field, ext, internal)
    st = rand_field(field, (n, 16), n)
    dev = torch.from_numpy(st.view(np.int32 if field == Z.BABYBEAR else np.int64)).cuda()
    Z.CudaPoseidon2().batch_permute_dev(field, dev, rc, ext, internal)
    got = dev.cpu().numpy().view(st.dtype)
    # states are independent of one another: a sample, the ends included
    pick = np.unique(np.r_[0, n - 1, np.random.default_rng(n).integers(0, n, 1500)])
    want = np.asarray(oracle.permute(field, st[pick].copy(), rc, ext, internal)).reshape(-1, 16)
    assert (got[pick] == want).all()


# the standard instance, around the sizes at which 148 SMs get one tile more
@pytest.mark.parametrize("n", [18944, 18945, 37888, 37889, 94720, 94721, 246272, 246273])
def test_tiles_per_sm(oracle, n):
    test_equals_the_oracle(oracle, Z.BABYBEAR, 8, 13, n)


def test_large_batches_do_not_run_as_quads():
    """2^20 BabyBear states with one partial round more than the standard instance: 1.3 times its time
    with one state a thread, 1.9 times as quads."""

    def us(ext, internal):
        x = torch.randint(0, 0x78000001, (1 << 20, 16), dtype=torch.int32, device="cuda")
        rc = _constants(Z.BABYBEAR, ext, internal)
        best = 1e9
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            Z.CudaPoseidon2().batch_permute_dev(Z.BABYBEAR, x, rc, ext, internal)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
        return best

    assert us(8, 14) < 1.6 * us(8, 13)
