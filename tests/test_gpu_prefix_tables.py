"""The sweeps' Philox prefix tables (first rounds of a block formed once per
temperature, in shared memory beside the lattice): both tables, the chains'
alone, or none, by lattice size.  Every choice draws the same native stream,
so spins and energies equal the oracle's restatement bit for bit."""
import numpy as np
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.05, 0.8])
@pytest.mark.parametrize("L", [8, 18, 46, 48, 56, 62, 66, 68, 70, 72, 82, 84, 88, 90, 96, 100, 102, 104, 126, 128])
def test_one_cta_sweep_at_the_table_limits(cuda, st, oracle, L, beta):
    """One group per CTA: both tables up to L = 82, the chains' up to 102,
    none from 104 on; rows that do not fill the last batch of four (one, two
    and three rows left: L = 48, 82, 72), and a second group with two replicas."""
    R, seed, step = 34, 60 + L, 2
    w, act = st.msc_init(L, R, seed=seed, iseq=0)
    ow, _ = oracle.msc_init(L, R, seed, 0)
    E, M = st.msc_sweep(w, act, L, 3, beta, pa.RNG_NATIVE, seed=seed, iseq=0, step=step)
    T4, T8 = (int(x) for x in oracle.msc_thresholds(beta))
    ref = oracle.msc_sweep_native(ow, L, 3, T4, T8, seed, 1, oracle.NATIVE_TAG_MSC | step)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), ref)
    oE, oM = oracle.msc_energy(ref, L)
    assert np.array_equal(E.cpu().numpy(), oE) and np.array_equal(M.cpu().numpy(), oM)


@pytest.mark.parametrize("L,cs", [(8, 2), (48, 2), (96, 2), (96, 4), (120, 2), (128, 4), (160, 2), (160, 4),
                                  (232, 2), (256, 4)])
def test_cluster_sweep_at_the_table_limits(cuda, oracle, L, cs):
    """Clusters of 2 and 4 CTAs: both tables, the chains' alone, general and
    compile-time sizes."""
    from conftest import compare_rows
    threads = 256 if L <= 128 else {2: 1024, 4: 512}[cs]
    with pa.Engine(L=L, R=70, sweeps=2, dbeta=0.25, beta_final=0.5, seed=L, coding="msc", weights="fp64",
                   sweep_variant=cs) as e:
        e.run()
        got = e.rows(0)
    ref = oracle.anneal_msc_native(L, 70, 2, 0.25, 0.5, 1, L, L, oracle.NATIVE_TAG_MSC, threads, 1, cs)
    compare_rows(got, ref[0], rtol=2e-10)


@pytest.mark.parametrize("L", [80, 160, 192, 240])
def test_bit_plane_sweep_of_wide_rows(cuda, st, oracle, L):
    """SSC bit planes with several words per row, up to more than one batch of
    words per thread (L = 240: 1200 words per plane)."""
    R, seed, beta = 3, 90 + L, 0.4
    g = st.ssc_init(L, R, seed=seed, iseq=0)
    init = oracle.ssc_init(L, R, seed, 0)
    st.ssc_sweep_bits(g, L, 2, beta, seed=seed, step=1)
    T4, T8 = (int(x) for x in oracle.msc_thresholds(beta))
    ref = oracle.ssc_sweep_bits_native(init, L, 2, T4, T8, seed, 1, oracle.NATIVE_TAG_SSC | 1, oracle.bits_max_tile(L))
    assert np.array_equal(g.cpu().numpy(), ref)


@pytest.mark.parametrize("L,R,tile", [(8, 100, 8), (16, 70, 4), (16, 500, 64), (24, 40, 2), (32, 130, 16), (48, 33, 5),
                                      (96, 7, 1), (144, 5, 1)])
def test_bit_plane_tiles_of_at_most_a_word_per_thread(cuda, oracle, L, R, tile):
    """Small bit-plane tiles (one warp, several, all of them; rows of one and
    of several words; short last tiles) take the one-word form and still equal
    the oracle's anneal of that tile size."""
    from conftest import compare_rows
    with pa.Engine(L=L, R=R, sweeps=3, dbeta=0.25, beta_final=1.0, seed=L + tile, coding="ssc", weights="fp64",
                   tile_groups=tile) as e:
        assert e.sweep_form(0) == dict(spins_per_word=32, replicas_per_word=1, tile=tile, cluster_ctas=1)
        e.run()
        got = e.rows(0)
    ref = oracle.anneal_ssc_bits_native(L, R, 3, 0.25, 1.0, 1, L + tile, L + tile, oracle.NATIVE_TAG_SSC, tile)
    compare_rows(got, ref[0], rtol=2e-10)


@pytest.mark.parametrize("L", [8, 10, 14, 16, 20, 22, 24, 30, 32, 34, 40, 44, 46])
def test_one_batch_units_alone(cuda, st, oracle, L):
    """MSC units of one batch per thread (up to L = 44: one, two and up to four
    sites per thread, threads and slots without a site) and the first size
    beyond."""
    R, seed = 70, 300 + L
    w, act = st.msc_init(L, R, seed=seed, iseq=0)
    ow, _ = oracle.msc_init(L, R, seed, 0)
    st.msc_sweep(w, act, L, 4, 0.3, pa.RNG_NATIVE, seed=seed, iseq=0, step=3)
    T4, T8 = (int(x) for x in oracle.msc_thresholds(0.3))
    ref = oracle.msc_sweep_native(ow, L, 4, T4, T8, seed, 1, oracle.NATIVE_TAG_MSC | 3)
    assert np.array_equal(w.cpu().numpy().view(np.uint32), ref)


@pytest.mark.parametrize("L,tile,R", [(8, 2, 100), (8, 8, 300), (12, 2, 70), (16, 2, 90), (16, 4, 200), (16, 8, 520),
                                      (20, 2, 130), (20, 4, 97), (24, 4, 260), (32, 2, 170), (32, 4, 140)])
def test_one_batch_units_stacked(cuda, oracle, L, tile, R):
    """Stacked tiles of one batch per thread (rows wrapping inside their own
    group, short last tiles) and, at L = 32 with 4 groups, of two."""
    from conftest import compare_rows
    with pa.Engine(L=L, R=R, sweeps=3, dbeta=0.25, beta_final=1.0, seed=L + tile, coding="msc", weights="fp64",
                   sweep_variant=1, tile_groups=tile) as e:
        e.run()
        got = e.rows(0)
    ref = oracle.anneal_msc_native(L, R, 3, 0.25, 1.0, 1, L + tile, L + tile, oracle.NATIVE_TAG_MSC, 256, tile, 1)
    compare_rows(got, ref[0], rtol=2e-10)


@pytest.mark.parametrize("sizes", [(48, 72, 88), (64, 128), (16, 64), (32, 40), (32, 56), (96, 64, 16), (96, 80, 32)])
def test_batches_of_several_kinds_of_unit(cuda, oracle, sizes):
    """The MSC sweep kernel is chosen by the kinds of work unit in the batch:
    every population equals the oracle's anneal of it alone, whichever kernel
    its neighbours lead to."""
    from conftest import compare_rows
    pops = [dict(L=L, R=100 + 40 * k, sweeps=2, dbeta=0.2, beta_final=0.4, seed=500 + k) for k, L in enumerate(sizes)]
    with pa.Engine.batch(pops, coding="msc", weights="fp64", tile_groups=1, sweep_variant=1) as e:
        e.run()
        got = [e.rows(k) for k in range(len(pops))]
    for k, p in enumerate(pops):
        ref = oracle.anneal_msc_native(p["L"], p["R"], 2, 0.2, 0.4, 1, p["seed"], pops[0]["seed"],
                                       oracle.NATIVE_TAG_MSC | k, 256, 1, 1, iseq0=k << 40)
        compare_rows(got[k], ref[0], rtol=2e-10)
