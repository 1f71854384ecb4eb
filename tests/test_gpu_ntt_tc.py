"""Goldilocks NTT passes and the fused LDE middle with their small DFTs on the tensor cores: every pass
size they exist for (6, 7 and 8 bits), from the smallest launch that takes them, with full and ragged last
chunks of columns, against the oracle; larger ones against the butterfly kernels (register tile
loads), bit for bit."""
import numpy as np
import pytest

import ziros_b200 as Z
from conftest import GL_P, rand_field
from ziros_b200 import _native as N

pytestmark = pytest.mark.gpu


def _edges(m):
    m = m.copy()
    m[0] = GL_P - 1
    m[1] = 0
    m[2] = 0xFFFFFFFF
    m[3] = 0xFFFFFFFF00000000
    m[-1] = GL_P - 1
    return m


@pytest.mark.parametrize("log_h,width,log_b", [(12, 32, 1), (12, 30, 2), (13, 32, 1), (13, 62, 1), (14, 16, 2), (15, 8, 1),
                                               (15, 22, 1), (16, 8, 1), (16, 14, 3), (17, 6, 1), (18, 2, 1), (18, 10, 1)])
def test_lde(oracle, log_h, width, log_b):
    t = _edges(rand_field(Z.GOLDILOCKS, (1 << log_h, width), log_h * width))
    for rev in (True, False):
        got = Z.CudaDft(Z.GOLDILOCKS).coset_lde_batch(t, log_b, bit_reverse_rows=rev)
        assert (got == oracle.coset_lde(Z.GOLDILOCKS, t, log_b, bitrev=rev)).all()
    assert N.ntt_tile_load_errors() == 0


def test_other_shift(oracle):
    t = _edges(rand_field(Z.GOLDILOCKS, (1 << 14, 16), 5))
    got = Z.CudaDft(Z.GOLDILOCKS).coset_lde_batch(t, 1, shift=123456789012345, bit_reverse_rows=True)
    assert (got == oracle.coset_lde(Z.GOLDILOCKS, t, 1, shift=123456789012345)).all()


@pytest.mark.parametrize("log_h,width", [(12, 32), (13, 30), (14, 16), (15, 12), (16, 8), (18, 4)])
def test_dft_both_ways(oracle, log_h, width):
    d = Z.CudaDft(Z.GOLDILOCKS)
    t = _edges(rand_field(Z.GOLDILOCKS, (1 << log_h, width), log_h))
    f = d.dft_batch(t)
    assert (f == oracle.dft_batch(Z.GOLDILOCKS, t)).all()
    assert (d.idft_batch(f) == t).all()
    assert N.ntt_tile_load_errors() == 0


@pytest.mark.parametrize("log_h,width,log_b", [(20, 24, 1), (21, 10, 1), (22, 4, 1)])
def test_equals_the_butterfly_kernels(log_h, width, log_b):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(log_h)
    t = torch.randint(0, 0xFFFFFFFF, (1 << log_h, width), dtype=torch.int64, device="cuda", generator=g) << 32
    t |= torch.randint(0, 1 << 32, t.shape, dtype=torch.int64, device="cuda", generator=g)
    out = [torch.empty((1 << (log_h + log_b), width), dtype=torch.int64, device="cuda") for _ in range(2)]
    lib, d = N.load(), Z.CudaDft(Z.GOLDILOCKS)
    d.coset_lde_batch_dev(t, log_b, out[0])
    N.check(lib.zkb_set_ntt_tile_loads(0))
    try:
        d.coset_lde_batch_dev(t, log_b, out[1])
    finally:
        N.check(lib.zkb_set_ntt_tile_loads(1))
    assert torch.equal(out[0], out[1])
    assert N.ntt_tile_load_errors() == 0
