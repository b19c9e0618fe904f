"""The int8 SSC sweep's forms by Philox blocks per thread: one block of one word
(L <= 40), one of two (L <= 64), several (rows that end in a single word at
L = 72).  Spins and energies equal the oracle's bit for bit; enough blocks that
some need more than the two spare words for undecided sites."""
import numpy as np
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.02, 0.44, 1.0])
@pytest.mark.parametrize("L,R,sweeps", [(8, 700, 5), (16, 33, 4), (24, 5, 3), (40, 60, 20), (48, 7, 3), (56, 9, 3),
                                        (64, 60, 40), (72, 5, 3), (104, 4, 2), (128, 8, 4), (256, 3, 2)])
def test_int8_sweep_by_blocks_per_thread(cuda, st, oracle, L, R, sweeps, beta):
    seed, step = 70 + L, 3
    g = st.ssc_init(L, R, seed=seed, iseq=0)
    init = oracle.ssc_init(L, R, seed, 0)
    E, M = st.ssc_sweep(g, L, sweeps, beta, pa.RNG_NATIVE, seed=seed, iseq=0, step=step)
    T4, T8 = (int(x) for x in oracle.msc_thresholds(beta))
    ref = oracle.ssc_sweep_native(init, L, sweeps, T4, T8, seed, 1, oracle.NATIVE_TAG_SSC | step)
    assert np.array_equal(g.cpu().numpy(), ref)
    oE, oM = oracle.ssc_energy(ref, L)
    assert np.array_equal(E.cpu().numpy(), oE) and np.array_equal(M.cpu().numpy(), oM)
