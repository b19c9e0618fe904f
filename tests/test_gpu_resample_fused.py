"""The resampling plan as one launch (a cluster or one CTA per population, up
to 65536 slots with FP32 weights, 2048 with FP64) and as three beyond: exact
populations at the edges of its tiles, CTAs and ranges, and a batch of more
populations than one warp plans."""
import numpy as np
import pytest

import paising_gb300 as pa

pytestmark = pytest.mark.gpu



@pytest.mark.parametrize("weights", [pa.WEIGHTS_FP32, pa.WEIGHTS_FP64])
@pytest.mark.parametrize("coding,n,every", [
    ("ssc", 1, 1), ("ssc", 2, 1), ("ssc", 255, 3), ("ssc", 257, 1), ("msc", 33, 5), ("msc", 1000, 1), ("ssc", 2047, 7),
    ("ssc", 2048, 500), ("ssc", 2049, 1), ("msc", 2050, 11), ("ssc", 8193, 2000), ("msc", 20001, 6),
    ("ssc", 65535, 3), ("ssc", 65536, 30000), ("ssc", 65537, 9)])
def test_plan_of_exact_weights(cuda, st, oracle, coding, n, every, weights):
    """Every `every`-th replica has the lowest energy (weight exactly 1), the
    others weight exactly 0, so q is their number, every copy number is
    floor(mu) or one more by its own uniform with mu = R_init / q, and the
    offsets and the map follow: from one copy each to thousands of copies of
    a few replicas."""
    torch = cuda
    slots = n if coding == "ssc" else (n + 31) // 32 * 32
    E = np.full(slots, 400000, dtype=np.int32)
    live = np.zeros(slots, dtype=bool)
    live[np.arange(0, n, every)] = True
    E[live] = -800
    q = int(live.sum())
    Rinit, seed, iseq = max(1, n - n // 3), 17, 4000
    act = None if coding == "ssc" else torch.from_numpy((np.arange(slots) < n).astype(np.uint8)).cuda()
    # dbeta 0.01: exp(-0.01 * 400800) is 0 in both precisions
    roff, offs, src, lnq, gq, rn = st.resample_plan(torch.from_numpy(E).cuda(), act, pa.SSC if coding == "ssc" else pa.MSC,
                                                    n, Rinit, 2 * n + 8, 0.30, 0.31, -800.0, weights, seed, iseq)
    assert gq == q
    dB = 0.31 - 0.30
    assert lnq == pytest.approx(dB * 800.0 + np.log(q) - np.log(n), rel=1e-14, abs=1e-14)
    # FP64: mu = R_init/R_prev exp(-dB E - lnQ) rounds about R_init/q; the
    # uniforms are multiples of 2^-32, so ties within 1e-9 of the fraction are left out
    mu = float(np.float32(Rinit) / np.float32(q)) if weights == pa.WEIGHTS_FP32 else Rinit / q
    idx = np.flatnonzero(live)
    U = np.empty(len(idx))
    for k, j in enumerate(idx):
        U[k] = (oracle.H(seed, iseq + int(j), 0) + 1.0) / 2.0**32
    r = np.floor(mu) + (U < mu - np.floor(mu))
    got = roff.cpu().numpy().astype(np.int64)
    assert got[~live].sum() == 0
    sure = np.abs(U - (mu - np.floor(mu))) > (0.0 if weights == pa.WEIGHTS_FP32 else 1e-9)
    if mu == np.floor(mu) and weights == pa.WEIGHTS_FP64:
        assert (np.abs(got[idx] - mu) <= 1).all()  # mu may round to either side of the integer
    else:
        assert np.array_equal(got[idx][sure], r[sure].astype(np.int64))
    assert rn == got.sum()
    assert np.array_equal(offs.cpu().numpy().astype(np.int64), np.cumsum(got) - got)
    assert np.array_equal(src[:rn].cpu().numpy(), np.repeat(np.arange(slots), got))


@pytest.mark.parametrize("weights", ["fp32", "fp64"])
@pytest.mark.parametrize("coding", ["ssc", "msc"])
def test_batch_of_more_populations_than_a_warp(cuda, coding, weights):
    """40 populations of uneven sizes and schedules (several end early) in one
    batch, reference stream: each equals its own run to the last bit."""
    pops = [dict(L=8 * (1 + k % 3), R=40 + 61 * k, sweeps=1 + k % 2, dbeta=(0.05, 0.1, 0.25)[k % 3],
                 beta_final=0.3 + 0.01 * k, seed=500 + k) for k in range(40)]
    with pa.Engine.batch(pops, coding=coding, rng="reference", weights=weights, capacity=2.0) as e:
        e.run()
        got = [e.rows(k) for k in range(len(pops))]
    for k in (0, 1, 2, 17, 31, 32, 33, 39):
        with pa.Engine(coding=coding, rng="reference", weights=weights, capacity=2.0, **pops[k]) as e:
            e.run()
            one = e.rows(0)
        assert np.array_equal(got[k], one), k


@pytest.mark.parametrize("weights", ["fp32", "fp64"])
def test_one_launch_equals_three(cuda, weights):
    """A replica buffer beyond the one-launch range takes the three launches:
    the same anneal, bit for bit."""
    kw = dict(L=16, R=1200, sweeps=2, dbeta=0.05, seed=9, coding="msc", rng="reference", weights=weights)
    rows = []
    for cap in (1.4, 60.0):  # 1936 and 72256 slots
        with pa.Engine(capacity=cap, **kw) as e:
            e.run()
            rows.append(e.rows(0))
    assert np.array_equal(rows[0], rows[1])
