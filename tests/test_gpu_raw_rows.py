"""Graph runs that leave their rows raw until the end (FP32 weights, resampling
in one launch, nothing recorded) give the same rows, bit for bit, as runs whose
steps are launched and finished one by one."""
import numpy as np
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


def rows(pops, graph, times=1, **kw):
    with (pa.Engine(**pops[0], graph=graph, **kw) if len(pops) == 1 else
          pa.Engine.batch([dict(p) for p in pops], graph=graph, **kw)) as e:
        for _ in range(times):
            e.run()
        return [e.rows(k) for k in range(e.num_sets())]


@pytest.mark.parametrize("kw", [
    dict(pops=[dict(L=16, R=300, sweeps=2, dbeta=0.1, seed=1)], coding="ssc"),
    dict(pops=[dict(L=8, R=90, sweeps=1, dbeta=0.002, seed=2)], coding="msc"),              # 501 rows: two rounds of 256
    dict(pops=[dict(L=8, R=90, sweeps=1, dbeta=1.0 / 256, seed=2)], coding="msc"),          # 257 rows
    dict(pops=[dict(L=16, R=9000, sweeps=2, dbeta=0.2, seed=3)], coding="msc", runs=3),     # a cluster resamples
    dict(pops=[dict(L=16, R=400, sweeps=2, dbeta=0.3, beta_final=0.2, seed=4)], coding="ssc"),
    dict(pops=[dict(L=16, R=700, sweeps=2, dbeta=0.25, beta_final=0.5, seed=5),
               dict(L=32, R=500, sweeps=3, dbeta=0.05, seed=6),
               dict(L=10, R=33, sweeps=1, dbeta=0.5, beta_final=0.5, seed=7)], coding="msc"),  # schedules of unlike length
    dict(pops=[dict(L=8, R=64, sweeps=2, dbeta=0.25, seed=8)], coding="msc", rng="reference"),
], ids=lambda k: f"{k['coding']}-{len(k['pops'])}-{k['pops'][0]['L']}-{k['pops'][0]['dbeta']:.4f}")
def test_rows_left_raw_equal_rows_of_single_steps(cuda, kw):
    kw = dict(kw)
    pops = kw.pop("pops")
    kw.setdefault("capacity", 2.0)  # large steps of beta
    a, b = rows(pops, True, times=2, **kw), rows(pops, False, times=2, **kw)
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert x.shape == y.shape and np.array_equal(x, y)


def test_failed_population_keeps_its_rows(cuda):
    """A population that outgrows its buffer is reported, and the populations
    beside it finish with their rows, with or without a graph."""
    out = []
    for graph in (True, False):
        pops = [dict(L=16, R=1000, sweeps=1, dbeta=0.9, beta_final=0.9, seed=11), dict(L=16, R=400, sweeps=2, dbeta=0.3, seed=12)]
        with pa.Engine.batch(pops, coding="msc", graph=graph, capacity=1.02) as e:
            try:
                e.run()
                out.append((0, e.rows(1)))
            except pa.PaisingError as ex:
                out.append((ex.status, e.rows(1)))
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
