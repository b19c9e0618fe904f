"""Batches of hundreds of populations: what a step launches for each of them."""
import numpy as np
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


def us_per_launch(profile, name):
    launches, ms = profile[name]
    return ms / launches * 1e3


@pytest.mark.parametrize("npop", [17, 200, 600])
def test_heavy_replicas_of_many_populations(cuda, npop):
    """Copies of replicas with more than 1024 of them are written by as many
    blocks as the batch leaves to a population (30, 2 and 1): each population
    equals its own run to the last bit, the one by 32 blocks."""
    pops = [dict(L=32, R=2500 + k % 7, sweeps=1, dbeta=1.0, seed=900 + k) for k in range(npop)]
    kw = dict(coding="msc", rng="reference", weights="fp64", capacity=1.5)
    with pa.Engine.batch(pops, **kw) as e:
        e.run()
        got = [(e.rows(k), e.population(k)) for k in range(npop)]
    for k in (0, 1, npop // 2, npop - 1):
        with pa.Engine(**pops[k], **kw) as e:
            e.run()
            assert np.array_equal(got[k][0], e.rows(0))
            assert np.array_equal(got[k][1], e.population())


def test_plan_of_many_populations_starts_few_blocks(cuda):
    """Plan launch of 1000 populations resampled in several launches: 10 us
    where it starts a block or two for each, 102 with 33."""
    pops = [dict(L=8, R=2500, sweeps=1, dbeta=0.05, seed=k) for k in range(1000)]
    with pa.Engine.batch(pops, coding="msc", weights="fp64", capacity=1.6, graph=False) as e:
        e.profile()
        assert us_per_launch(e.profile(), "plan") < 50.0


@pytest.mark.parametrize("weights,R,npop,one", [
    ("fp64", 300, 15, True), ("fp64", 300, 16, False), ("fp64", 300, 1000, False), ("fp32", 300, 1000, True),
    ("fp32", 1300, 25, True), ("fp32", 1300, 26, False), ("fp32", 2500, 1000, False), ("fp32", 20000, 100, True)])
def test_route_of_the_resampling_plan(cuda, weights, R, npop, one):
    """The plan as one launch where that is the faster: clusters of eight CTAs
    per population lose to separate launches in large batches of small
    populations (1000 populations of 300 with FP64 weights 0.63 ms per
    temperature against 1.43)."""
    pops = [dict(L=8, R=R, sweeps=1, dbeta=0.2, seed=k) for k in range(npop)]
    with pa.Engine.batch(pops, coding="msc", weights=weights, capacity=1.6, graph=False) as e:
        p = e.profile()
    assert ("resample_plan" in p) == one and ("copy_numbers" in p) != one


@pytest.mark.parametrize("coding", ["ssc", "msc"])
@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("weights,R,npop", [("fp64", 900, 16), ("fp32", 1300, 26)])
def test_batches_past_the_line_equal_their_own_runs(cuda, coding, graph, weights, R, npop):
    """Batches just too large for the one launch against each population's own
    run, which takes it."""
    pops = [dict(L=8, R=R - 5 * k, sweeps=1 + k % 2, dbeta=(0.05, 0.1)[k % 2], seed=70 + k) for k in range(npop)]
    kw = dict(coding=coding, rng="reference", weights=weights, graph=graph, capacity=1.6)
    with pa.Engine.batch(pops, **kw) as e:
        e.run()
        got = [(e.rows(k), e.population(k)) for k in range(npop)]
    for k in (0, 1, npop - 1):
        with pa.Engine(**pops[k], **kw) as e:
            e.run()
            assert np.array_equal(got[k][0], e.rows(0))
            assert np.array_equal(got[k][1], e.population())
