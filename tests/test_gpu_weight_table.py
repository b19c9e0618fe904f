"""FP64 weights of populations well above the number of energy levels come from
tables by level: the anneal equals the oracle's, whose weights and copy numbers
are formed replica by replica (population sizes exactly), on both sides of the
size from which the tables are used and for steps that kill most replicas."""
import pytest

import paising_gb300 as pa
from conftest import compare_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coding,L,R,dbeta", [("msc", 8, 98304 + 63, 0.2), ("msc", 8, 98304 + 64, 0.2),
                                              ("msc", 10, 120001, 0.5), ("ssc", 8, 98304 + 64, 0.25)])
def test_anneal_with_weights_by_level(cuda, oracle, coding, L, R, dbeta):
    seed = R
    with pa.Engine(L=L, R=R, sweeps=1, dbeta=dbeta, beta_final=1.0, seed=seed, coding=coding, weights="fp64",
                   capacity=1.5) as e:
        tile = e.sweep_form(0)["tile"]
        e.run()
        got = e.rows(0)
    if coding == "msc":
        ref = oracle.anneal_msc_native(L, R, 1, dbeta, 1.0, 1, seed, seed, oracle.NATIVE_TAG_MSC, 256, tile, 1)
    else:
        ref = oracle.anneal_ssc_bits_native(L, R, 1, dbeta, 1.0, 1, seed, seed, oracle.NATIVE_TAG_SSC, tile)
    compare_rows(got, ref[0], rtol=2e-10)
