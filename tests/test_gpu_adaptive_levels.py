"""The adaptive step over the population's energy levels, against the same
search restated over its energies: few levels in a shared-memory histogram,
few of a histogram too large for it, and more levels than its list holds."""
import numpy as np
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


def _next_step(E, beta, db, beta_final, rinit, lo, hi):
    E = E.astype(np.float64)
    R, Em = len(E), E.mean()

    def overlap(d):
        lnq = -d * Em + np.log(np.exp(-d * (E - Em)).sum()) - np.log(R)
        return np.minimum(1.0, rinit / R * np.exp(-d * E - lnq)).sum() / R

    top, bottom = db, 0.0
    while True:
        ov = overlap(top)
        if not (ov >= hi and beta + top < beta_final):
            break
        top *= 1.1
    if ov >= lo:
        mean = top
    else:
        for _ in range(200):
            mean = 0.5 * (bottom + top)
            ov = overlap(mean)
            if ov < lo:
                top = mean
            elif ov >= hi:
                bottom = mean
            else:
                break
    return beta_final - beta if beta < beta_final and beta + mean > beta_final else mean


@pytest.mark.parametrize("L,R,wide", [(32, 400, False), (64, 300, False), (128, 3000, True)])
def test_adaptive_schedule_restated(cuda, L, R, wide):
    rng = np.random.default_rng(L)
    N = L * L
    spins = rng.choice(np.array([-1, 1], dtype=np.int8), size=(R, N))
    if wide:  # from disordered to ordered: nearly every replica has a level of its own
        p = np.linspace(0.5, 1.0, R)[:, None]
        spins = np.where(rng.random((R, N)) < p, 1, -1).astype(np.int8)
    bfin, db0 = (0.004, 1e-5) if wide else (0.12, 0.01)
    with pa.Engine(L=L, R=R, sweeps=0 if wide else 2, dbeta=db0, beta_final=bfin, coding="ssc", adaptive=True,
                   store_energies=True, capacity=2.0, seed=3) as e:
        e.set_population(spins)
        e.run()
        beta = e.rows(0)[:, 0]
        energies = [e.energies(0, i) for i in range(len(beta))]
    assert len(beta) > 4
    if wide:
        assert len(np.unique(energies[1])) > 2048
    db = db0
    for i in range(1, len(beta) - 1):
        db = _next_step(energies[i], beta[i], db, bfin, R, 0.85, 0.87)
        assert beta[i + 1] == pytest.approx(beta[i] + db, rel=1e-12), i
