"""A bounded wait inside a kernel that gives up is an error of the next call that waits for the
device, never a wrong root.  The wait is one for a product that nothing issues, with a short limit;
the kernel ends by itself and the context stays usable."""
import numpy as np
import pytest
import torch

import ziros_b200 as Z
from ziros_b200 import _native as N
from conftest import rand_field

pytestmark = pytest.mark.gpu

POLLS = 64  # about 0.3 ms


@pytest.fixture(autouse=True)
def nothing_pending():
    N.circuit_reset()
    yield
    N.circuit_reset()
    N.ntt_tile_load_errors()


def _expire():
    N.debug_wait_expiry(POLLS)
    torch.cuda.synchronize()


def _calls():
    trace = rand_field(Z.BABYBEAR, (1 << 10, 16), 1)
    pcs = Z.CudaTwoAdicPcs(Z.BABYBEAR, 42, 1)
    batch = Z.BatchCommit([(1 << 8, 8)], autotune=False)
    batch.copy_in(0, trace[:1 << 8, :8].copy())

    def roots():
        batch.run()
        return batch.roots()

    eng = Z.CommitEngine(slots=1)
    cw = rand_field(Z.BABYBEAR, (1 << 10, 4), 2)
    return {
        "commit": lambda: pcs.commit(trace)[0],
        "commit_fri": lambda: pcs.commit_fri(trace, (1, 2, 3, 4), 2, 3, transcript=True)[0],
        "fri": lambda: Z.CudaFriProver(42, 2, 3).commit(cw).roots,
        "lde": lambda: Z.CudaDft(Z.BABYBEAR).coset_lde_batch(trace, 1),
        "batch": roots,
        "engine": lambda: eng.wait(eng.submit(trace))[0],
    }


def test_every_waiting_call_reports_it_and_recovers():
    for name, call in _calls().items():
        want = call()
        _expire()
        with pytest.raises(Z.ZkbError) as e:
            call()
        assert e.value.code == N.ERR_TIMEOUT and "gave up" in str(e.value), name
        is_open, why = N.circuit_open()
        assert is_open and "gave up" in why, name
        N.circuit_reset()
        assert np.array_equal(call(), want), name


def test_the_count_is_read_once_and_acknowledges():
    call = _calls()["commit"]
    want = call()
    N.ntt_tile_load_errors()
    _expire()
    # each thread of the one block once, though it has two layers; the other block once
    assert N.ntt_tile_load_errors() == 129
    assert N.ntt_tile_load_errors() == 0
    assert np.array_equal(call(), want)


def test_poll_limits_are_checked():
    for polls in (0, 4097):
        with pytest.raises(Z.ZkbError):
            N.debug_wait_expiry(polls)
