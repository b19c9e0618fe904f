"""Replicas with very many copies (a large dbeta against the energy spread) in
populations resampled in several launches: offsets and the gather map equal
those of the copy numbers, through the stage call and the engine alike."""
import numpy as np
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coding", [pa.SSC, pa.MSC])
@pytest.mark.parametrize("R,dbeta", [(70000, 0.01), (70000, 0.4), (70001, 3.0), (300000, 0.15), (300000, 0.08)])
def test_map_of_populations_with_heavy_replicas(cuda, st, coding, R, dbeta):
    torch = cuda
    gen = torch.Generator(device="cuda").manual_seed(R)
    slots = R if coding == pa.SSC else (R + 31) // 32 * 32
    E = (4 * torch.round(torch.randn(slots, generator=gen, device="cuda") * 15 - 300)).to(torch.int32).clamp(-2048, 2048)
    E[1234] = E[1235] = E[R - 1] = -2000  # three of one tile or none: nearly all copies at the large steps
    act = None
    if coding == pa.MSC:
        act = torch.zeros(slots, dtype=torch.uint8, device="cuda")
        act[:R] = 1
    roff, offs, src, lnq, q, rn = st.resample_plan(E, act, coding, R, R, 2 * R, 0.1, 0.1 + dbeta, float(E[:R].min()),
                                                   pa.WEIGHTS_FP32, 77, 7)
    r = roff.cpu().numpy().astype(np.int64)
    want = np.repeat(np.arange(slots), r)
    assert rn == r.sum() > 0
    assert np.array_equal(offs.cpu().numpy().astype(np.int64), np.cumsum(r) - r)
    assert np.array_equal(src[:rn].cpu().numpy().astype(np.int64), want)
    if dbeta > 0.05:
        assert r.max() > 2 * max(1024, 2 * R // 512)  # the heavy path ran


@pytest.mark.parametrize("weights", ["fp32", "fp64"])
def test_anneal_with_heavy_replicas(cuda, weights):
    """The engine's launches (the work plan finishing the scatter) against the
    same anneal stepped on the host without a graph."""
    out = []
    for graph in (True, False):
        with pa.Engine(L=32, R=140000, sweeps=2, dbeta=0.3, seed=3, coding="msc", weights=weights, graph=graph,
                       capacity=2.0) as e:
            e.run()
            out.append((e.rows(0), e.population()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert np.all(np.abs(out[0][0][:, 8] - 140000) < 0.5 * 140000)
