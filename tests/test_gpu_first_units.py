"""First units of the one-CTA sweeps' persistent CTAs: launches of no more
units than CTAs whose last round of the SMs is more than half full give them
out by the CTAs' places on their SMs, all others by block index.  Every unit is
swept exactly once either way: spins and energies equal the oracle's bit for
bit, also where another stream's launches hold places."""
import numpy as np
import pytest
import torch

import paising_gb300 as pa

pytestmark = pytest.mark.gpu

SMS = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 152


@pytest.mark.parametrize("units", [1, SMS // 2, SMS // 2 + 1, SMS, SMS + 1, 2 * SMS - 3, 3 * SMS, 4 * SMS - 1, 4 * SMS,
                                   4 * SMS + 1, 5 * SMS])
@pytest.mark.parametrize("other", [False, True])
def test_every_unit_is_swept_once(cuda, st, oracle, units, other):
    L, R, seed, step, beta = 16, 32 * units - 7, 40 + units, 2, 0.4
    w, act = st.msc_init(L, R, seed=seed, iseq=0)
    ow, _ = oracle.msc_init(L, R, seed, 0)
    T4, T8 = (int(x) for x in oracle.msc_thresholds(beta))
    ref = oracle.msc_sweep_native(ow, L, 1, T4, T8, seed, 1, oracle.NATIVE_TAG_MSC | step)
    if other:  # places taken by another stream's sweep
        with pa.Engine(L=64, R=8000, sweeps=50, dbeta=0.5, beta_final=1.0, seed=3, coding="msc", sweep_variant=1) as e:
            import threading
            t = threading.Thread(target=e.run)
            t.start()
            E, M = st.msc_sweep(w, act, L, 1, beta, pa.RNG_NATIVE, seed=seed, iseq=0, step=step)
            t.join()
    else:
        E, M = st.msc_sweep(w, act, L, 1, beta, pa.RNG_NATIVE, seed=seed, iseq=0, step=step)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), ref)
    oE, oM = oracle.msc_energy(ref, L)
    assert np.array_equal(E.cpu().numpy(), oE) and np.array_equal(M.cpu().numpy(), oM)


@pytest.mark.parametrize("pops", [[(32, 3000), (16, 1700)], [(16, 4500), (32, 900), (20, 2000)], [(96, 2500), (32, 2300)]])
def test_batches_by_place(cuda, pops):
    """Uneven batches of a count given out by place equal the populations run alone."""
    kw = dict(sweeps=3, dbeta=0.2, beta_final=0.6, weights="fp64", tile_groups=1, sweep_variant=1)
    with pa.Engine.batch([dict(L=L, R=R, seed=9 + k, **kw) for k, (L, R) in enumerate(pops)], coding="msc") as e:
        e.run()
        got = [e.rows(k) for k in range(len(pops))]
    for k, (L, R) in enumerate(pops):
        assert np.all(np.abs(got[k][:, 8] - R) < 0.2 * R)
    # a population's stream depends on its place in the batch, not on its neighbours' units
    with pa.Engine.batch([dict(L=L, R=R, seed=9 + k, **kw) for k, (L, R) in enumerate(pops)] + [dict(L=8, R=40000, seed=99, **kw)],
                         coding="msc") as e:
        e.run()
        for k in range(len(pops)):
            assert np.array_equal(e.rows(k), got[k])
