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


@pytest.mark.parametrize("weights", [pa.WEIGHTS_FP32, pa.WEIGHTS_FP64])
@pytest.mark.parametrize("coding,R,dbeta", [("ssc", 60000, 0.4), ("msc", 60000, 0.4), ("msc", 300001, 0.15)])
def test_engine_copies_heavy_replicas(cuda, st, coding, R, dbeta, weights):
    """One step without sweeps from a given population, whose copies the engine
    writes beside its work plan: replica by replica the initial population
    repeated by the copy numbers, which the stage call gives."""
    torch = cuda
    L, seed, msc = 16, 5, coding == "msc"
    if msc:
        init, act = st.msc_init(L, R, 31)
        E, _ = st.msc_sweep(init, act, L, 0, 0.0, pa.RNG_NATIVE, 1)
        groups, drawn = init.shape[0], init.shape[0]
    else:
        init, act = st.ssc_init(L, R, 31), None
        E, _ = st.ssc_sweep(init, L, 0, 0.0, pa.RNG_NATIVE, 1)
        drawn = R
    e_ref = 0.0 if weights == pa.WEIGHTS_FP64 else float((E[:R]).min())
    roff, _, _, _, _, rn = st.resample_plan(E, act, pa.MSC if msc else pa.SSC, R, R, 2 * R, 0.0, dbeta, e_ref, weights,
                                            seed, 128 * drawn)
    r = roff.cpu().numpy().astype(np.int64)
    assert r.max() > max(1024, 2 * R // 512)  # the heavy path runs
    host = init.cpu().numpy()
    with pa.Engine(L=L, R=R, sweeps=0, dbeta=dbeta, beta_final=dbeta, seed=seed, coding=coding, capacity=2.0,
                   weights="fp64" if weights == pa.WEIGHTS_FP64 else "fp32") as e:
        e.set_population(host.ctypes.data)
        e.run()
        assert int(e.rows(0)[1, 8]) == rn == r.sum()
        got = e.population()
    if msc:  # bit k of group g = replica 32 g + k
        bits = np.unpackbits(host.view(np.uint8), axis=1, bitorder="little").reshape(groups, L * L, 32)
        lattices = bits.transpose(0, 2, 1).reshape(groups * 32, L * L)
        gb = np.unpackbits(np.ascontiguousarray(got).view(np.uint8), axis=1, bitorder="little").reshape(len(got), L * L, 32)
        got, host = gb.transpose(0, 2, 1).reshape(len(got) * 32, L * L)[:rn], lattices
    assert np.array_equal(got, np.repeat(host[:len(r)], r, axis=0))
