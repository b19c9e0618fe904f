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


@pytest.mark.parametrize("coding,dbeta,seed,beside", [
    ("ssc", 0.02, 2, 400), ("ssc", 0.02, 3, 400), ("ssc", 0.02, 4, 5000), ("msc", 0.1, 2, 400), ("msc", 0.1, 2, 5000)])
def test_extinct_population_beside_another(cuda, coding, dbeta, seed, beside):
    """Two replicas over many small steps die out in some runs of the handle
    (the others draw on from where the last run ended): with rows left raw (one
    CTA or a cluster per population) and finished step by step the same runs
    fail, and the runs that do not have the same rows."""
    out = []
    for graph in (True, False):
        pops = [dict(L=8, R=2, sweeps=1, dbeta=dbeta, seed=seed), dict(L=16, R=beside, sweeps=2, dbeta=0.3, seed=12)]
        with pa.Engine.batch(pops, coding=coding, rng="reference", graph=graph, capacity=2.0) as e:
            runs = []
            for _ in range(8):
                try:
                    e.run()
                    runs.append([e.rows(0), e.rows(1), e.population(0), e.population(1)])
                except pa.PaisingError as ex:
                    assert ex.status == 4  # PA_ERR_EXTINCT
                    runs.append(None)
            out.append(runs)
    assert [r is None for r in out[0]] == [r is None for r in out[1]]
    failed = [k for k, r in enumerate(out[0]) if r is None]
    assert failed and failed[0] < 7 and any(r is not None for r in out[0][failed[0]:])
    for a, b in zip(*out):
        assert (a is None and b is None) or all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("graph", [True, False])
def test_runs_before_an_extinct_one_keep_their_rows(cuda, oracle, graph):
    """Sequential runs of one handle: the first ends, the second dies out; the
    first one's rows are there and are the oracle's, the second one's are not."""
    with pa.Engine(L=8, R=2, sweeps=1, dbeta=0.02, seed=4, runs=3, coding="ssc", rng="reference", graph=graph,
                   capacity=2.0) as e:
        with pytest.raises(pa.PaisingError) as err:
            e.run()
        assert err.value.status == 4 and e.num_sets() == 3
        got = e.rows(0)
        with pytest.raises(pa.PaisingError):
            e.rows(1)
    ref, _ = oracle.anneal("ssc", 8, 2, 1, 0.02, 1.0, 1, 4)
    assert np.array_equal(got[:, 8], ref[0][:, 8])
    assert np.allclose(got, ref[0], rtol=1e-5, atol=1e-5)  # FP32 weights against FP64
