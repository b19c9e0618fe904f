"""Ancestors carried by the native stream's MSC gather, families counted beside
the records: few families left after large steps (groups gathered bit by bit,
broadcast pairs), a last group partly empty, with and without an energy
histogram.  Checked against ancestors observed in the lattices, which without
sweeps are copies of the initial ones."""
import numpy as np
import pytest

import paising_gb300 as pa
from test_gpu_family import _family_stats_of, _replica_lattices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,dB,mhr", [(33, 0.4, False), (2999, 0.05, True), (2999, 0.6, False), (20000, 0.3, True)])
def test_ancestors_carried_by_the_gather(cuda, R, dB, mhr):
    L, N = 8, 64
    rng = np.random.default_rng(R)
    init = rng.integers(0, 2**32, ((R + 31) // 32, N), dtype=np.uint32)
    with pa.Engine(L=L, R=R, sweeps=0, dbeta=dB, beta_final=2.5 * dB, seed=R, coding="msc", family=True, mhr=mhr,
                   capacity=3.0) as e:
        e.set_population(init)
        e.run()
        rows, fam, pop = e.rows(0), e.family_rows(0), e.population()
    first = _replica_lattices("msc", init, R, L)
    index = {row.tobytes(): i for i, row in enumerate(first)}
    assert len(index) == R
    anc = np.array([index[row.tobytes()] for row in _replica_lattices("msc", pop, int(rows[2, 8]), L)])
    nf, rho, sf = _family_stats_of(np.bincount(anc))
    assert fam[2, 0] == nf < R
    assert fam[2, 1] == pytest.approx(rho, rel=1e-12) and fam[2, 2] == pytest.approx(sf, rel=1e-12, abs=1e-12)
