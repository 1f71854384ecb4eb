"""The row permutation behind the natural-order transforms: blocks of 32 to 1,024 rows by the width."""
import ctypes as C

import numpy as np
import pytest
import torch

import ziros_b200 as Z
from ziros_b200 import _native as N
from conftest import rand_field

pytestmark = pytest.mark.gpu


# widths around those at which a block's number of rows changes; heights of less than a block, one
# block, more
@pytest.mark.parametrize("field", [Z.BABYBEAR, Z.GOLDILOCKS])
@pytest.mark.parametrize("width", [1, 2, 3, 5, 8, 9, 16, 17, 31, 32, 33, 70])
def test_transforms_in_natural_order(oracle, field, width):
    dft = Z.CudaDft(field)
    for log_h in (1, 4, 5, 6, 9, 10, 11):
        x = rand_field(field, (1 << log_h, width), 100 * log_h + width)
        assert (dft.dft_batch(x) == oracle.dft_batch(field, x)).all(), log_h
        assert (dft.idft_batch(oracle.dft_batch(field, x)) == x).all(), log_h
    x = rand_field(field, (1 << 10, width), width)
    lde = dft.coset_lde_batch(x, 1)
    rev = dft.coset_lde_batch(x, 1, bit_reverse_rows=True)
    order = np.array([int(f"{i:011b}"[::-1], 2) for i in range(1 << 11)])
    assert (lde[order] == rev).all()


def _permutation_us(log_h, width):
    lib = N.load()
    x = torch.randint(0, 0x78000001, (1 << log_h, width), dtype=torch.int32, device="cuda")
    stats = (N.KernelStat * 64)()

    def transform():
        N.check(lib.zkb_dft_batch_dev(Z.BABYBEAR, C.c_void_p(x.data_ptr()), log_h, width, 0, None))

    transform()
    lib.zkb_profile_start()
    for _ in range(20):
        transform()
    torch.cuda.synchronize()
    n = lib.zkb_profile_stop(stats, 64)
    got = [s for s in stats[:n] if s.name == b"bitrev_rows"]
    return got[0].total_ms / got[0].launches * 1e3


def test_a_narrow_matrix_takes_no_more_blocks_than_a_wide_one():
    """2^22 words as one column against sixteen: the writes of single words cost about twice as much
    (29 us and 14 on a B200); blocks that are mostly idle would make it five times."""
    assert _permutation_us(22, 1) < 3.5 * _permutation_us(18, 16)
