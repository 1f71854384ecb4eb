"""Natural-order LDEs whose output cannot hold the coefficients (it contains the trace, or is not
16-byte aligned): a second scratch buffer when there is room for it, one when there is not.  The
missing room is a reported out-of-memory of the first allocation, made on the host."""
import numpy as np
import pytest
import torch

import ziros_b200 as Z
from ziros_b200 import _native as N
from conftest import rand_field

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def nothing_injected():
    yield
    N.inject_fault(1, 0)


def _words(a):
    return torch.from_numpy(a.view(np.int32 if a.dtype == np.uint32 else np.int64))


@pytest.mark.parametrize("room", [True, False])
@pytest.mark.parametrize("field,log_h,width", [(Z.BABYBEAR, 11, 5), (Z.BABYBEAR, 12, 8), (Z.GOLDILOCKS, 8, 64),
                                               (Z.GOLDILOCKS, 13, 30), (Z.GOLDILOCKS, 15, 16)])
def test_trace_inside_or_output_unaligned(oracle, field, log_h, width, room):
    dft = Z.CudaDft(field)
    t = rand_field(field, (1 << log_h, width), log_h)
    want = oracle.coset_lde(field, t, 1, bitrev=False)
    rows = 2 << log_h
    inside = torch.empty((rows, width), dtype=_words(t).dtype, device="cuda")
    inside[: 1 << log_h] = _words(t).cuda()
    unaligned = torch.empty(rows * width + 1, dtype=inside.dtype, device="cuda")[1:].view(rows, width)
    apart = _words(t).cuda()
    dft.coset_lde_batch_dev(apart, 1, torch.empty_like(inside), bit_reverse_rows=False)  # the tables
    for trace, out in ((inside[: 1 << log_h], inside), (apart, unaligned)):
        if not room:
            N.inject_fault(1, 1)
        dft.coset_lde_batch_dev(trace, 1, out, bit_reverse_rows=False)
        N.inject_fault(1, 0)
        assert (out.cpu().numpy().view(t.dtype) == want).all()


def test_without_room_for_the_one_buffer_it_fails_before_anything_is_written():
    t = _words(rand_field(Z.BABYBEAR, (1 << 12, 8), 3)).cuda()
    out = torch.full((1 << 13, 8), 7, dtype=torch.int32, device="cuda")
    N.inject_fault(1, 1)
    with pytest.raises(Z.ZkbError) as e:
        Z.CudaDft(Z.BABYBEAR).coset_lde_batch_dev(t, 1, out, bit_reverse_rows=False)
    assert e.value.code == N.ERR_OOM
    assert (out == 7).all()
