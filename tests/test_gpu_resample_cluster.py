"""The resampling plan by a cluster of eight CTAs (FP32 weights, 2049 to 65536
slots) with the weights an anneal has: the same anneal, bit for bit, as by the
separate launches that a larger replica buffer takes."""
import numpy as np
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])  # rows left raw for the next plan, or finished step by step
@pytest.mark.parametrize("coding", ["ssc", "msc"])
@pytest.mark.parametrize("R", [2100, 5000, 20001])
def test_cluster_equals_separate_launches(cuda, coding, R, graph):
    out = []
    for cap in (1.4, 66000.0 / R):  # slots within one launch's range, and beyond it
        with pa.Engine(L=16, R=R, sweeps=2, dbeta=0.05, seed=R, coding=coding, weights="fp32", graph=graph,
                       capacity=cap) as e:
            e.run()
            out.append((e.rows(0), e.population()))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
