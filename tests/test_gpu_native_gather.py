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
