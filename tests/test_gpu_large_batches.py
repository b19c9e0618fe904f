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
