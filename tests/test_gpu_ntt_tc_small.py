"""Goldilocks transforms around the sizes from which a pass, or the fused middle, runs on the tensor
cores: against the oracle on both sides, and the kernels that ran."""
import ctypes as C

import numpy as np
import pytest
import torch

import ziros_b200 as Z
from ziros_b200 import _native as N
from conftest import rand_field

pytestmark = pytest.mark.gpu


def _kernels(call):
    lib, stats = N.load(), (N.KernelStat * 64)()
    lib.zkb_profile_start()
    call()
    torch.cuda.synchronize()
    n = lib.zkb_profile_stop(stats, 64)
    return {s.name.decode() for s in stats[:n]}


# 6-bit passes take 2,048 tiles of 16 columns, 7-bit ones 256
@pytest.mark.parametrize("log_h,width,tc", [(12, 496, False), (12, 512, True), (12, 64, False), (14, 16, False), (14, 32, True)])
def test_passes(oracle, log_h, width, tc):
    x = rand_field(Z.GOLDILOCKS, (1 << log_h, width), width)
    x[0], x[-1] = 0xFFFFFFFF00000000, 0
    d = torch.from_numpy(x.view(np.int64)).cuda()
    run = lambda: N.check(N.load().zkb_dft_batch_dev(Z.GOLDILOCKS, C.c_void_p(d.data_ptr()), log_h, width, 0, None))
    assert ("ntt_pass_tc" in _kernels(run)) == tc
    assert (d.cpu().numpy().view(np.uint64) == oracle.dft_batch(Z.GOLDILOCKS, x)).all()


# the fused middle of 6 bits takes 384 tiles, of 7 bits 128
@pytest.mark.parametrize("log_h,width,tc", [(12, 80, False), (12, 96, True), (13, 32, False), (13, 48, True), (14, 16, True)])
def test_fused_middle(oracle, log_h, width, tc):
    x = rand_field(Z.GOLDILOCKS, (1 << log_h, width), width)
    d = torch.from_numpy(x.view(np.int64)).cuda()
    out = torch.empty((2 << log_h, width), dtype=torch.int64, device="cuda")
    run = lambda: Z.CudaDft(Z.GOLDILOCKS).coset_lde_batch_dev(d, 1, out)
    assert ("lde_fused_tc" in _kernels(run)) == tc
    assert (out.cpu().numpy().view(np.uint64) == oracle.coset_lde(Z.GOLDILOCKS, x, 1)).all()
