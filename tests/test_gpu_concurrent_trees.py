"""Trees of many matrices built by two host threads at once, above the tensor-core sizes.

The many-tree kernels take shared memory for their tables and one word a tree, so two threads whose
calls have different numbers of trees launch the same kernel with different sizes.  Every result equals
the thread's own first one, and the first one is checked elsewhere against the oracle."""
import threading

import numpy as np
import pytest
import torch

import ziros_b200 as Z

pytestmark = pytest.mark.gpu


def _uniform(field, shape, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if field == Z.BABYBEAR:
        return torch.randint(0, 0x78000001, shape, dtype=torch.int32, device="cuda", generator=g)
    return torch.randint(0, 1 << 62, shape, dtype=torch.int64, device="cuda", generator=g)


def _both(calls, reps):
    """Runs each call `reps` times in a thread of its own, all at once; the calls' errors."""
    errors, gate = [], threading.Barrier(len(calls))

    def work(call):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                want = call()
                gate.wait(60)
                for _ in range(reps):
                    got = call()
                    assert all(np.array_equal(a, b) for a, b in zip(got, want))
        except BaseException as e:  # noqa: BLE001 - reported below
            gate.abort()
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def test_fri_commits_with_different_numbers_of_rounds():
    def job(log_n, seed):
        cw = _uniform(Z.BABYBEAR, (1 << log_n, 4), seed)
        prover = Z.CudaFriProver(42, 2, 4, challenge_seed=seed, query_seed=seed + 1)

        def call():
            pf = prover.commit_dev(cw)
            return pf.roots, pf.query_rows, pf.query_siblings

        return call

    assert _both([job(16, 1), job(17, 2), job(18, 3)], 500) == []


@pytest.mark.parametrize("field,p2", [(Z.BABYBEAR, 16), (Z.GOLDILOCKS, 16), (Z.GOLDILOCKS, 12)])
def test_batch_plans_with_different_numbers_of_traces(field, p2):
    def job(count, seed):
        shapes = [(1 << 12, 8)] * count
        plan = Z.BatchCommit(shapes, field=field, p2_width=p2, autotune=False, use_graph=False)
        for i, s in enumerate(shapes):
            plan.copy_in(i, _uniform(field, s, seed + i))
        torch.cuda.synchronize()

        def call():
            s = torch.cuda.current_stream().cuda_stream
            for _ in range(10):
                plan.run(s)
            return (plan.roots(s),)

        return call

    assert _both([job(5, 10), job(16, 50), job(7, 90)], 150) == []


def test_a_captured_plan_outlives_a_smaller_one():
    """A plan's graph holds launches of the size it was captured with; a plan of fewer traces made
    later changes nothing for it."""
    shapes = [(1 << 12, 8)] * 16
    plan = Z.BatchCommit(shapes, autotune=False)
    for i, s in enumerate(shapes):
        plan.copy_in(i, _uniform(Z.BABYBEAR, s, i))
    plan.run()
    want = plan.roots()
    small = Z.BatchCommit(shapes[:5], autotune=False)
    small.run()
    plan.run()
    assert (plan.roots() == want).all()


@pytest.mark.parametrize("field,p2,log_h", [(Z.BABYBEAR, 16, 20), (Z.GOLDILOCKS, 12, 18)])
def test_levels_of_fewer_trees_in_one_capture(field, p2, log_h):
    """One tall trace among small ones: the small trees end while the tall one's levels still take the
    tensor-core form, so one graph holds launches of many trees and of one."""
    shapes = [(1 << log_h, 4)] + [(1 << 3, 4)] * 20
    plan = Z.BatchCommit(shapes, field=field, p2_width=p2, autotune=False)
    traces = [_uniform(field, s, i) for i, s in enumerate(shapes)]
    for i, t in enumerate(traces):
        plan.copy_in(i, t)
    pcs = Z.CudaTwoAdicPcs(field, 42, 1, p2)
    want = np.stack([pcs.commit_dev(t)[0] for t in traces])
    for _ in range(2):
        plan.run()
        assert (plan.roots() == want).all()
