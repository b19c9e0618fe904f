"""pa_autotune keeps the form that it measured to be the faster one."""
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta_final,ctas", [(0.1, (1,)), (1.0, (2, 4))])
def test_form_of_a_population_of_one_wave(cuda, beta_final, ctas):
    """94 groups of L = 64, a unit per SM.  At the hot end one CTA per group
    takes 4% less time than clusters of 2 (470 against 490 us at 100 sweeps)
    and is kept; over a schedule to beta = 1 clusters of 2 take 2% less."""
    with pa.Engine(L=64, R=3000, sweeps=100, dbeta=0.02, beta_final=beta_final, seed=664, coding="msc") as e:
        e.autotune()
        assert e.sweep_form(0)["cluster_ctas"] in ctas
