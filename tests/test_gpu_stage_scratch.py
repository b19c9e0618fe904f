"""Stage calls hold one of a few scratch slots each: more calls at once than
slots, from threads with streams of their own, do not disturb each other."""
import threading

import numpy as np
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


def test_stage_calls_from_many_threads(cuda, st, oracle):
    torch = cuda
    jobs = [(16 + 8 * (k % 3), 400 + 37 * k, 0.2 + 0.05 * k, 50 + k) for k in range(10)]

    def work(L, R, beta, seed):
        g = st.ssc_init(L, R, seed=seed)
        E, M = st.ssc_sweep_bits(g, L, 3, beta, seed=seed)
        roff, offs, src, lnq, q, rn = st.resample_plan(E, None, pa.SSC, R, R, 2 * R, beta, beta + 0.02, float(E.min()),
                                                       pa.WEIGHTS_FP32, seed, 7)
        new = st.ssc_resample(g, L, src, rn)
        return [x.cpu().numpy() for x in (g, E, M, roff, offs, src[:rn], new)] + [lnq, q, rn]

    alone = [work(*j) for j in jobs]
    got, errors = [None] * len(jobs), []

    def run(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(5):
                    got[k] = work(*jobs[k])
        except Exception as ex:  # noqa: BLE001
            errors.append(ex)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(jobs))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors
    for a, b in zip(alone, got):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))


def test_engines_of_different_shared_memory_in_turn(cuda):
    """A handle launched without a graph after another one, of smaller units,
    was set up: the kernels' shared-memory limit is common to both."""
    for kw in (dict(coding="msc", sweep_variant=1), dict(coding="ssc", sweep_variant=1), dict(coding="msc", sweep_variant=2)):
        with pa.Engine(L=128, R=64, sweeps=1, dbeta=0.5, seed=1, graph=False, **kw) as big:
            with pa.Engine(L=16, R=64, sweeps=1, dbeta=0.5, seed=1, graph=False, **kw) as small:
                small.run()
                big.run()
                got = big.rows(0)
        with pa.Engine(L=128, R=64, sweeps=1, dbeta=0.5, seed=1, **kw) as alone:
            alone.run()
            assert np.array_equal(alone.rows(0), got)
