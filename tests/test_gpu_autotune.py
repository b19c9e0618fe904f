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


def test_tiles_of_a_mixed_batch_are_timed_in_its_kernel(cuda):
    """Kernels hold the forms of a launch's lattice sizes, and a form's time
    depends on the kernel: L = 48 alone is fastest one group at a time, in a
    kernel with code for its remainder rows, but beside L = 96 in stacks.  64
    uneven populations tuned size by size in kernels of their own took 2% more
    than with the built-in tiles."""
    def device_ms(tune):
        pops = [dict(L=L, R=6000 + 500 * k, sweeps=20, dbeta=0.1, seed=40 + k)
                for k, L in enumerate((16, 32, 48, 64, 96, 128) * 6)]
        with pa.Engine.batch(pops, coding="msc", capacity=1.6) as e:
            if tune:
                e.autotune()
            times = []
            for _ in range(4):
                e.run()
                times.append(e.timing()[0])
        return min(times)

    assert device_ms(True) < 1.005 * device_ms(False)
