"""The native MSC gather's two routes -- rows through an asynchronous ring in
16-byte vectors, and bit by bit for groups spanning more than the window and
for buffers off 16-byte alignment -- against a numpy gather and each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(kind, R, rng):
    if kind == "identity":
        return np.arange(R)
    if kind == "near":  # copies 0, 1, 2
        return np.sort(rng.integers(0, R, R))
    if kind == "gaps":  # every group jumps beyond its window, some of them further inside
        return np.sort(np.concatenate([np.arange(0, R, 5), np.arange(0, R, 7), rng.integers(0, R, R // 3)]))[:R]
    if kind == "few":  # a few parents
        return np.sort(rng.choice([0, R // 3, R // 3 + 1, R - 1], R))
    raise ValueError(kind)


@pytest.mark.parametrize("kind", ["identity", "near", "gaps", "few"])
@pytest.mark.parametrize("L,R", [(4, 40), (10, 1000), (14, 33), (30, 2500), (64, 700), (100, 130)])
def test_native_gather_routes(cuda, st, L, R, kind):
    torch = cuda
    N, rng = L * L, np.random.default_rng(L + R)
    src = _map(kind, R, rng).astype(np.int32)
    Rn = len(src)
    old = rng.integers(0, 2**32, size=((R + 31) // 32, N), dtype=np.uint64).astype(np.uint32)
    bits = (old[src >> 5] >> (src & 31).astype(np.uint32)[:, None]) & 1  # [Rn, N]
    rgn = (Rn + 31) // 32
    ref = np.zeros((rgn, N), dtype=np.uint32)
    for s in range(Rn):
        ref[s >> 5] |= bits[s] << np.uint32(s & 31)
    srct = torch.from_numpy(src).cuda()
    for off in (0, 1):  # words off the allocation's alignment
        buf = torch.empty(old.size + off, dtype=torch.int32, device="cuda")
        t = buf[off:].view(old.shape)
        t.copy_(torch.from_numpy(old.view(np.int32)))
        new, act = st.msc_resample_native(t, L, R, srct, Rn)
        assert np.array_equal(new.cpu().numpy().view(np.uint32), ref), off
        assert np.array_equal(act.cpu().numpy(), (np.arange(rgn * 32) < Rn).astype(np.uint8))


@pytest.mark.parametrize("groups", [4076, 4100])
def test_native_gather_unit_sizes(cuda, st, groups):
    """Either side of the line between units of 4 and of 16 groups (L = 64: 32
    strips of 128 sites)."""
    torch = cuda
    L, R = 64, 32 * groups - 5
    g = torch.Generator(device="cuda").manual_seed(groups)
    old = torch.randint(-2**31, 2**31, (groups, L * L), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    src = torch.sort(torch.randint(0, R, (R,), generator=g, device="cuda", dtype=torch.int64))[0].to(torch.int32)
    new, _ = st.msc_resample_native(old, L, R, src, R)
    off = torch.empty(old.numel() + 1, dtype=torch.int32, device="cuda")[1:].view_as(old)
    off.copy_(old)
    ref, _ = st.msc_resample_native(off, L, R, src, R)
    assert torch.equal(new, ref)


def _many_groups(torch, chunks):
    L, R = 8, 131072 * chunks + 37
    g = torch.Generator(device="cuda").manual_seed(chunks)
    old = torch.randint(-2**31, 2**31, ((R + 31) // 32, L * L), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    src = torch.sort(torch.randint(0, R, (R,), generator=g, device="cuda", dtype=torch.int64))[0].to(torch.int32)
    return L, R, old, src


@pytest.mark.parametrize("chunks", [11, 12])  # chunk by chunk, and all at once
def test_native_gather_of_many_groups(cuda, st, chunks):
    """Pair lists of more groups than the library's scratch holds: the same as
    the gather of every 4096 groups by itself."""
    L, R, old, src = _many_groups(cuda, chunks)
    new, act = st.msc_resample_native(old, L, R, src, R)
    for s0 in range(0, R, 131072):
        part = src[s0:s0 + 131072]
        ref, ref_act = st.msc_resample_native(old, L, R, part, len(part))
        assert cuda.equal(new[s0 // 32:s0 // 32 + len(ref)], ref)
        assert cuda.equal(act[s0:s0 + len(ref_act)], ref_act)


def test_native_gather_of_very_many_groups_takes_no_longer_than_it_must(cuda, st):
    """Three launches for every 4096 groups made 4.7 million replicas of L = 8
    take 3.8 times as long as one million (0.68 ms; all at once 0.30)."""
    import time

    def best(chunks):
        L, R, old, src = _many_groups(cuda, chunks)
        times = []
        for _ in range(8):
            cuda.cuda.synchronize()
            t0 = time.perf_counter()
            st.msc_resample_native(old, L, R, src, R)
            times.append(time.perf_counter() - t0)
        return min(times)

    assert best(36) < 2.7 * best(8)
