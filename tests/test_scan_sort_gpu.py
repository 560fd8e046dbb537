"""GPU parity: exclusive scan (bit-exact, wrapping) and radix sort (keys
bit-exact and nondecreasing unsigned; payloads a multiset match per key, the
reference sort being unstable)."""
import hashlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_scan_golden(ctx, orc, golden):
    meta, _ = golden
    s = meta["cases"]["scan"]
    sin = orc.generate_rand_int(s["n"], s["n"], 0)
    got = ctx.scan_excl(dev(sin)).cpu().numpy()
    assert hashlib.sha256(got.tobytes()).hexdigest() == s["output_sha"]


@pytest.mark.parametrize("n", [0, 1, 2, 4095, 4096, 4097, 65536, 65537, 1000003])
def test_scan_sizes(ctx, orc, n):
    rng = np.random.default_rng(n)
    x = rng.integers(-(2 ** 31), 2 ** 31, n, dtype=np.int64).astype(np.int32)
    got = ctx.scan_excl(dev(x)).cpu().numpy() if n else np.zeros(0, np.int32)
    assert np.array_equal(got, orc.scan_excl(x))


def test_scan_in_place_and_unaligned(ctx, orc):
    x = np.random.default_rng(1).integers(-5, 5, 100001).astype(np.int32)
    t = dev(x)
    ctx.scan_excl(t, out=t)
    assert np.array_equal(t.cpu().numpy(), orc.scan_excl(x))
    # 4-byte aligned, not 16-byte aligned views
    big = dev(np.concatenate([[7], x]).astype(np.int32))
    out = torch.empty_like(big)
    got = ctx.scan_excl(big[1:], out=out[1:])
    assert np.array_equal(got.cpu().numpy(), orc.scan_excl(x))


def test_scan_full_size_property(ctx):
    # 2^28 ones: out[i] == i (size-independent check at full scale)
    n = 1 << 28
    x = torch.ones(n, dtype=torch.int32, device="cuda")
    y = ctx.scan_excl(x)
    assert torch.equal(y, torch.arange(n, dtype=torch.int32, device="cuda"))


def check_sorted_rec(got, rin):
    u = got[:, 1].view(np.uint32)
    assert (u[1:] >= u[:-1]).all()
    a = np.lexsort((rin[:, 0], rin[:, 1].view(np.uint32)))
    b = np.lexsort((got[:, 0], got[:, 1].view(np.uint32)))
    assert np.array_equal(rin[a], got[b])


@pytest.mark.parametrize("n", [2048, 1 << 15, 100003])
def test_sort_golden(ctx, orc, golden, n):
    meta, _ = golden
    c = meta["cases"][f"sort_{n}"]
    rin = orc.generate_rand(200, n, 0)
    got = ctx.sort_rec(dev(rin)).cpu().numpy()
    assert hashlib.sha256(np.ascontiguousarray(got[:, 1]).tobytes()).hexdigest() == c["keys_sorted_sha"]
    check_sorted_rec(got, rin)


@pytest.mark.parametrize("n,keyrange", [(0, 1), (1, 1), (2, 5), (4097, 3), (65536, 1 << 32),
                                        (1 << 20, 1 << 20), (3000001, 1 << 32)])
def test_sort_sizes(ctx, n, keyrange):
    rng = np.random.default_rng(n)
    rin = np.stack([np.arange(n, dtype=np.int64),
                    rng.integers(0, keyrange, n, dtype=np.int64)], 1).astype(np.uint32).view(np.int32)
    rin = np.ascontiguousarray(rin)
    if n == 0:
        return
    got = ctx.sort_rec(dev(rin)).cpu().numpy()
    check_sorted_rec(got, rin)


def test_sort_is_stable_lsd(ctx):
    # The passes are stable: equal keys keep input order (a property the
    # reference does not promise but the tests rely on for determinism).
    n = 200000
    rng = np.random.default_rng(9)
    rin = np.stack([np.arange(n), rng.integers(0, 1000, n)], 1).astype(np.int32)
    got = ctx.sort_rec(dev(rin)).cpu().numpy()
    order = np.argsort(rin[:, 1], kind="stable")
    assert np.array_equal(got, rin[order])


@pytest.mark.parametrize("mode", [0, 3, 4])
def test_sort_ranking_modes_stable(ctx, mode):
    # Every stable ranking form of the radix passes (eight ballots; a match on
    # the digit's high half and four ballots; a match on each half) gives the
    # same stable sort, over keys using every digit value and a ragged tail.
    assert ctx.lib.qg_sort_set_rank(mode) == 0
    try:
        n = 300001
        rng = np.random.default_rng(mode + 5)
        rin = np.stack([np.arange(n), rng.integers(0, 1 << 32, n, dtype=np.int64)], 1).astype(np.uint32).view(np.int32)
        rin = np.ascontiguousarray(rin)
        got = ctx.sort_rec(dev(rin)).cpu().numpy()
        order = np.argsort(rin[:, 1].view(np.uint32), kind="stable")
        assert np.array_equal(got, rin[order])
    finally:
        assert ctx.lib.qg_sort_set_rank(-1) == 0


# Tile edges (5120 records), and key masks whose digit positions give 0 to 4
# passes: in place (twice, so that both parities are remembered) and into
# another buffer.  Stable: equal keys keep their input order.
@pytest.mark.parametrize("n", [2, 5119, 5120, 5121, 3 * 5120 + 1, 100_003])
@pytest.mark.parametrize("mask", [0, 0xFF, 0xFF00FF, 0xFFFFFF, 0xFFFFFFFF])
def test_sort_rec_tiles_and_passes(ctx, n, mask):
    rng = np.random.default_rng(n ^ mask)
    for _ in range(2):
        y = (rng.integers(0, 2 ** 32, n, dtype=np.uint64) & np.uint64(mask)).astype(np.uint32)
        rec = np.stack([np.arange(n, dtype=np.uint32), y], 1).view(np.int32)
        exp = rec[np.argsort(y, kind="stable")]
        d = dev(rec)
        srt, start = ctx.groupby_rec(d)
        assert np.array_equal(srt.cpu().numpy(), exp) and np.array_equal(d.cpu().numpy(), rec)
        heads = np.flatnonzero(np.r_[True, exp[1:, 1] != exp[:-1, 1]])
        assert np.array_equal(start.cpu().numpy(), heads)
        assert np.array_equal(ctx.sort_rec(d).cpu().numpy(), exp)


def test_sort_rec_equal_keys_between_others(ctx):
    # many tiles of equal keys (no pass at all, twice), then keys that need passes, the
    # same buffer each time
    n = 10_500_000
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    buf = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    x = torch.arange(n, dtype=torch.int32, device="cuda")
    for key in (7, 7, None, 9, -1, None, None):
        y = torch.full((n,), key, dtype=torch.int32, device="cuda") if key is not None else \
            torch.randint(-(2 ** 31), 2 ** 31, (n,), generator=g, device="cuda").to(torch.int32)
        buf[:, 0], buf[:, 1] = x, y
        ctx.sort_rec(buf)
        order = torch.sort(y.to(torch.int64) & 0xFFFFFFFF, stable=True).indices
        assert torch.equal(buf[:, 0], x[order]) and torch.equal(buf[:, 1], y[order])


def test_sort_rec_timeout_reports_and_recovers(ctx):
    # Poll limit 0: look-backs give up, passes after the first read items other than the
    # counted ones.  The call reports it, writes nothing past the records, and the next
    # call is exact.
    from query_on_opencl_fpga_gb300 import QGError

    n = 4_000_001
    g = torch.Generator(device="cuda")
    g.manual_seed(6)
    rec = torch.randint(-(2 ** 31), 2 ** 31, (n + 300_000, 2), generator=g, device="cuda").to(torch.int32)
    rec[n:] = 77
    keep = rec[:n].clone()
    for _ in range(3):
        ctx.set_spin_limit(0)
        try:
            with pytest.raises(QGError) as e:
                ctx.sort_rec(rec[:n])
            assert e.value.status == 5
        finally:
            ctx.set_spin_limit(1 << 22)
        assert bool((rec[n:] == 77).all())
        rec[:n] = keep
        ctx.sort_rec(rec[:n])
        order = torch.sort(keep[:, 1].to(torch.int64) & 0xFFFFFFFF, stable=True).indices
        assert torch.equal(rec[:n], keep[order])
        rec[:n] = keep
