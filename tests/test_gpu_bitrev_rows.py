"""The row permutation behind the natural-order transforms: rows per block by the width and the height,
and rows written in runs of eight where single ones would share their sectors."""
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


# runs from 48 MB on for rows that are not whole sectors: both sides of the line in bytes and in the width
@pytest.mark.parametrize("field,log_n,width", [
    (Z.BABYBEAR, 20, 1), (Z.BABYBEAR, 19, 3), (Z.BABYBEAR, 20, 11), (Z.BABYBEAR, 20, 12), (Z.BABYBEAR, 20, 16), (Z.BABYBEAR, 21, 8),
    (Z.BABYBEAR, 18, 63), (Z.BABYBEAR, 18, 64), (Z.BABYBEAR, 18, 65), (Z.GOLDILOCKS, 19, 2), (Z.GOLDILOCKS, 20, 5),
    (Z.GOLDILOCKS, 20, 6), (Z.GOLDILOCKS, 18, 32), (Z.GOLDILOCKS, 18, 33), (Z.GOLDILOCKS, 17, 63), (Z.GOLDILOCKS, 17, 65)])
def test_natural_order_is_the_bit_reversed_one_permuted(field, log_n, width):
    dft = Z.CudaDft(field)
    dt = torch.int32 if field == Z.BABYBEAR else torch.int64
    x = torch.randint(0, 0x78000001, (1 << (log_n - 1), width), dtype=dt, device="cuda")
    nat, rev = (torch.empty((1 << log_n, width), dtype=dt, device="cuda") for _ in range(2))
    dft.coset_lde_batch_dev(x, 1, nat, bit_reverse_rows=False)
    dft.coset_lde_batch_dev(x, 1, rev)
    i = torch.arange(1 << log_n, device="cuda")
    order = torch.zeros_like(i)
    for b in range(log_n):
        order |= ((i >> b) & 1) << (log_n - 1 - b)
    assert torch.equal(nat[order], rev)


def _permutation_us(log_h, width, field=Z.BABYBEAR):
    lib = N.load()
    dt = torch.int32 if field == Z.BABYBEAR else torch.int64
    x = torch.randint(0, 0x78000001, (1 << log_h, width), dtype=dt, device="cuda")
    stats = (N.KernelStat * 64)()

    def transform():
        N.check(lib.zkb_dft_batch_dev(field, C.c_void_p(x.data_ptr()), log_h, width, 0, None))

    transform()
    lib.zkb_profile_start()
    for _ in range(20):
        transform()
    torch.cuda.synchronize()
    n = lib.zkb_profile_stop(stats, 64)
    got = [s for s in stats[:n] if s.name == b"bitrev_rows"]
    return got[0].total_ms / got[0].launches * 1e3


def test_a_narrow_matrix_takes_no_more_blocks_than_a_wide_one():
    """2^22 words as one column against sixteen (16 us and 12 on a B200); blocks that are mostly idle
    would make it five times."""
    assert _permutation_us(22, 1) < 3.5 * _permutation_us(18, 16)


def test_rows_of_partial_sectors_are_written_together():
    """2^21 x 9 Goldilocks words (72-byte rows) against 2^21 x 8: rows written one at a time would read and
    write their shared sectors again, 2.6 times as long."""
    assert _permutation_us(21, 9, Z.GOLDILOCKS) < 1.8 * _permutation_us(21, 8, Z.GOLDILOCKS)
