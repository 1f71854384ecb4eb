"""LDE widths that no column chunk divides: the columns left over go either into a last chunk that is
not full or into a launch of their own, by the number of rows; both against the oracle, for strides
that allow tensor-copy tiles and strides that do not, in bit-reversed and natural order."""
import numpy as np
import pytest

import ziros_b200 as Z
from conftest import rand_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", [Z.BABYBEAR, Z.GOLDILOCKS])
@pytest.mark.parametrize("width", [2, 3, 5, 7, 9, 12, 15, 17, 20, 28, 31, 33])
def test_small_heights(oracle, field, width):
    for log_h, log_b in ((1, 1), (6, 2), (11, 1)):
        t = rand_field(field, (1 << log_h, width), 10 * width + log_h)
        for rev in (True, False):
            got = Z.CudaDft(field).coset_lde_batch(t, log_b, bit_reverse_rows=rev)
            assert (got == oracle.coset_lde(field, t, log_b, bitrev=rev)).all()


@pytest.mark.parametrize("field,log_h,width", [(Z.BABYBEAR, 17, 17), (Z.BABYBEAR, 16, 20), (Z.BABYBEAR, 18, 2),
                                               (Z.GOLDILOCKS, 15, 9), (Z.GOLDILOCKS, 16, 10), (Z.GOLDILOCKS, 14, 15)])
def test_both_sides_of_the_rule(oracle, field, log_h, width):
    t = rand_field(field, (1 << log_h, width), width)
    assert (Z.CudaDft(field).coset_lde_batch(t, 1, bit_reverse_rows=True) == oracle.coset_lde(field, t, 1)).all()


@pytest.mark.parametrize("field", [Z.BABYBEAR, Z.GOLDILOCKS])
@pytest.mark.parametrize("width", [3, 11, 21])
def test_dft_both_ways(oracle, field, width):
    d = Z.CudaDft(field)
    t = rand_field(field, (1 << 12, width), width)
    f = d.dft_batch(t)
    assert (f == oracle.dft_batch(field, t)).all()
    assert (d.idft_batch(f) == t).all()


@pytest.mark.parametrize("field,log_h,width", [(Z.GOLDILOCKS, 8, 1024), (Z.GOLDILOCKS, 12, 64), (Z.BABYBEAR, 12, 8)])
@pytest.mark.parametrize("rev", [True, False])
def test_trace_inside_the_output(field, log_h, width, rev):
    """Two-pass plans read the trace before they write the output; heights of one 8-bit pass keep two."""
    import torch
    h = 1 << log_h
    t = rand_field(field, (h, width), width)
    d = Z.CudaDft(field)
    want = d.coset_lde_batch(t, 1, bit_reverse_rows=rev)
    for row0 in (0, h // 2, h):
        out = torch.zeros((2 * h, width), dtype=torch.int32 if field == Z.BABYBEAR else torch.int64, device="cuda")
        trace = out[row0:row0 + h]
        trace.copy_(torch.from_numpy(t.view(np.int32 if field == Z.BABYBEAR else np.int64)))
        d.coset_lde_batch_dev(trace, 1, out, bit_reverse_rows=rev)
        torch.cuda.synchronize()
        assert (out.cpu().numpy().view(t.dtype) == want).all()
