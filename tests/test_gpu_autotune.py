"""pa_autotune keeps the form that it measured to be the faster one."""
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,R,beta_final,ctas", [(56, 4800, 0.08, (1,)), (64, 40000, 0.08, (1,)), (64, 3000, 1.0, (2, 4))])
def test_form_by_the_schedule(cuda, L, R, beta_final, ctas):
    """At the hot end one CTA per group takes less time than the faster cluster
    and is kept (50 sweeps, us a launch: L = 56, 4800 replicas 260 against 272;
    L = 64, 40000 1390 against 1472).  Over a schedule to beta = 1 94 groups of
    L = 64 take 483 against 471 (100 sweeps), and clusters are kept."""
    with pa.Engine(L=L, R=R, sweeps=100 if beta_final == 1.0 else 50, dbeta=0.02, beta_final=beta_final, seed=664,
                   coding="msc") as e:
        e.autotune()
        assert e.sweep_form(0)["cluster_ctas"] in ctas
