"""GPU parity: single-pass filter vs the oracle (bit-exact, positional:
filterImpl's scatter is stable, kernel/filter/filter_op.cl:220-238)."""
import numpy as np
import pytest
import torch

from query_on_opencl_fpga_gb300 import datagen

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_filter_rec_golden(ctx, orc, golden):
    meta, arrs = golden
    c = meta["cases"]["filter"]
    rin = orc.generate_rand(100, c["n"], 0)
    out = ctx.filter_range_rec(dev(rin), c["small"], c["large"]).cpu().numpy()
    assert np.array_equal(out, arrs["filter_out"])


@pytest.mark.parametrize("n", [0, 1, 2, 3, 5, 31, 4095, 4096, 4097, 8191, 100003, 1 << 20])
def test_filter_rec_sizes(ctx, orc, n):
    rin = orc.generate_rand(1000, n, n) if n else np.zeros((0, 2), np.int32)
    for lo, hi in [(0, 99), (-1000, 1000), (500, 400), (-(2 ** 31), 2 ** 31 - 1)]:
        exp = orc.filter_rec(rin, lo, hi)
        got = ctx.filter_range_rec(dev(rin) if n else torch.zeros((0, 2), dtype=torch.int32, device="cuda"),
                                   lo, hi).cpu().numpy()
        assert got.shape == exp.shape and np.array_equal(got, exp), (n, lo, hi)


def test_filter_rec_capacity(ctx, orc):
    from query_on_opencl_fpga_gb300 import QGError

    rin = orc.generate_rand(10, 10000, 1)
    with pytest.raises(QGError) as e:
        ctx.filter_range_rec(dev(rin), -100, 100, cap=5)
    assert e.value.status == 3
    # the context stays usable
    got = ctx.filter_range_rec(dev(rin), 0, 3).cpu().numpy()
    assert np.array_equal(got, orc.filter_rec(rin, 0, 3))


@pytest.mark.parametrize("n", [0, 1, 7, 4096, 65537, 1 << 21])
def test_filter_cols(ctx, orc, n):
    d = datagen.config0_filter(n, seed=n)
    key, pay = d["key"].numpy(), d["payload"].numpy()
    exp = orc.filter_cols(key, pay, d["lo"], d["hi"])
    got = ctx.filter_cols(dev(key), dev(pay), d["lo"], d["hi"]).cpu().numpy()
    assert np.array_equal(got, exp)


def test_filter_cols_config0_full_size(ctx, orc):
    # Full config-0 size: 16M rows, ~10 % selectivity, bit-exact.
    d = datagen.config0_filter(1 << 24, seed=0, device="cuda")
    got = ctx.filter_cols(d["key"], d["payload"], d["lo"], d["hi"])
    key, pay = d["key"].cpu().numpy(), d["payload"].cpu().numpy()
    exp = orc.filter_cols(key, pay, d["lo"], d["hi"], mt=True)
    assert got.shape[0] == exp.shape[0]
    assert np.array_equal(got.cpu().numpy(), exp)


def test_filter_cols_into_caller_buffer(ctx, orc):
    # out=: one caller-owned (cap, 2) buffer reused by calls of different selectivity
    d = datagen.config0_filter(1 << 20, seed=12)
    key, pay = d["key"].numpy(), d["payload"].numpy()
    out = torch.empty((1 << 20, 2), dtype=torch.int32, device="cuda")
    for lo, hi in ((d["lo"], d["hi"]), (0, 1 << 30), (5, 4)):
        got = ctx.filter_cols(dev(key), dev(pay), lo, hi, out=out)
        assert got.numel() == 0 or got.data_ptr() == out.data_ptr()  # an empty view reports 0
        assert np.array_equal(got.cpu().numpy(), orc.filter_cols(key, pay, lo, hi))
    with pytest.raises(ValueError):
        ctx.filter_cols(dev(key), dev(pay), 0, 1, out=out[:10])


def test_filter_repeat_is_deterministic(ctx):
    d = datagen.config0_filter(1 << 22, seed=5, device="cuda")
    a = ctx.filter_cols(d["key"], d["payload"], 0, 1 << 29).clone()
    for _ in range(3):
        b = ctx.filter_cols(d["key"], d["payload"], 0, 1 << 29)
        assert torch.equal(a, b)


def test_lookback_timeout_reports_and_recovers(ctx, orc):
    # A poll limit of 0 makes every look-back give up at once: the call must
    # report a timeout (no hang, no fault) and the context must stay usable.
    from query_on_opencl_fpga_gb300 import QGError

    rin = orc.generate_rand(100, 1 << 16, 0)
    ctx.set_spin_limit(0)
    try:
        with pytest.raises(QGError) as e:
            ctx.filter_range_rec(dev(rin), 0, 50)
        assert e.value.status == 5
    finally:
        ctx.set_spin_limit(1 << 22)
    got = ctx.filter_range_rec(dev(rin), 0, 50).cpu().numpy()
    assert np.array_equal(got, orc.filter_rec(rin, 0, 50))


@pytest.mark.parametrize("variant", [0, 1])
def test_filter_cols_timeout_reports_and_recovers(ctx, orc, variant):
    # Poll limit 0 on the single-pass column filters: every wait (look-back,
    # and for variant 1 the bulk-copy ring's barriers) gives up at once.  The
    # call reports a timeout, the ring stops refilling and drains its copies,
    # and the next call with the default limit is exact.
    from query_on_opencl_fpga_gb300 import QGError

    ctx.check(ctx.lib.qg_filter_set_variant(variant), "variant")
    d = datagen.config0_filter(1 << 22, seed=41)
    key, pay = d["key"].numpy(), d["payload"].numpy()
    try:
        ctx.set_spin_limit(0)
        try:
            with pytest.raises(QGError) as e:
                ctx.filter_cols(dev(key), dev(pay), d["lo"], d["hi"])
            assert e.value.status == 5
        finally:
            ctx.set_spin_limit(1 << 22)
        got = ctx.filter_cols(dev(key), dev(pay), d["lo"], d["hi"]).cpu().numpy()
        assert np.array_equal(got, orc.filter_cols(key, pay, d["lo"], d["hi"]))
    finally:
        ctx.lib.qg_filter_set_variant(2)


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 4095, 4099, 300007, 1 << 22, 1048576 + 4096 * 300 + 5])
def test_filter_cols_variants(ctx, orc, variant, n):
    ctx.check(ctx.lib.qg_filter_set_variant(variant), "variant")
    try:
        d = datagen.config0_filter(n, seed=n + variant)
        key, pay = d["key"].numpy(), d["payload"].numpy()
        got = ctx.filter_cols(dev(key), dev(pay), d["lo"], d["hi"]).cpu().numpy()
        assert np.array_equal(got, orc.filter_cols(key, pay, d["lo"], d["hi"]))
    finally:
        ctx.lib.qg_filter_set_variant(2)  # the default


# Edges of the two-phase kernel: a warp's unit (512 column rows, 256 records),
# a CTA of 8 warps, one unit per warp on every SM, and more units per warp than
# its shared memory keeps predicate bits for.
@pytest.mark.parametrize("rec", [False, True])
@pytest.mark.parametrize("units,extra", [(1, -1), (1, 0), (1, 1), (8, 0), (8, 1), (152 * 8, 3), (152 * 32, 0),
                                         (152 * 32, 1), (152 * 32 * 16, 1)])
def test_filter_two_phase_edges(ctx, orc, rec, units, extra):
    n = units * (256 if rec else 512) + extra
    d = datagen.config0_filter(n, seed=units, device="cuda")
    key, pay = d["key"], d["payload"]
    for lo, hi in [(d["lo"], d["hi"]), (1 << 29, 2 ** 31 - 1)]:
        if rec:
            r = datagen.records(key, pay)
            got = ctx.filter_range_rec(r, lo, hi).cpu().numpy()
            exp = orc.filter_rec(r.cpu().numpy(), lo, hi)
        else:
            got = ctx.filter_cols(key, pay, lo, hi).cpu().numpy()
            exp = orc.filter_cols(key.cpu().numpy(), pay.cpu().numpy(), lo, hi, mt=True)
        assert np.array_equal(got, exp)


def test_filter_rec_into_its_input(ctx, orc):
    import ctypes

    n = 300_007
    r = orc.generate_rand(1000, n, 9)
    buf = dev(r)
    cnt = ctypes.c_int64()
    st = ctx.lib.qg_filter_range_rec(ctx.handle, buf.data_ptr(), n, 0, 400, buf.data_ptr(), n, ctypes.byref(cnt))
    exp = orc.filter_rec(r, 0, 400)
    assert st == 0 and np.array_equal(buf[: cnt.value].cpu().numpy(), exp)


# Records kept in shared memory (512 a warp, units of 256): none and all selected,
# kept to the last one, run full in the middle of a warp's units or at once, and
# not kept at all (one unit, several, many per warp; a capacity among the kept).
@pytest.mark.parametrize("units", [1, 2, 5, 40])
@pytest.mark.parametrize("sel", [0.0, 0.004, 0.3, 0.45, 0.9, 1.0])
def test_filter_rec_kept_rows(ctx, orc, units, sel):
    from query_on_opencl_fpga_gb300 import QGError

    n = 152 * 32 * 256 * units - 77
    g = torch.Generator(device="cuda")
    g.manual_seed(units)
    key = torch.where(torch.rand(n, generator=g, device="cuda") < sel, 5, 900).to(torch.int32)
    key[: 256 * units] = 5  # the first warp's rows are all selected
    rec = torch.stack([torch.arange(n, dtype=torch.int32, device="cuda"), key], 1)
    got = ctx.filter_range_rec(rec, -3, 5)
    exp = rec[(key == 5).nonzero().flatten()]
    assert torch.equal(got, exp)
    with pytest.raises(QGError) as e:
        ctx.filter_range_rec(rec, -3, 5, cap=exp.shape[0] - 1)
    assert e.value.status == 3


# Two launches from 2^22 rows on: the line and beside it, sorted keys (the selected
# rows close together) and others, none, some and all selected, a capacity among them.
@pytest.mark.parametrize("n", [(1 << 22) - 1, 1 << 22, (1 << 22) + 513, 152 * 32 * 512 * 3 + 5])
@pytest.mark.parametrize("sorted_keys", [True, False])
def test_filter_cols_two_launches(ctx, n, sorted_keys):
    from query_on_opencl_fpga_gb300 import QGError

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    key = torch.randint(-(2 ** 31), 2 ** 31, (n,), generator=g, device="cuda")
    key = (key.sort().values if sorted_keys else key).to(torch.int32)
    pay = torch.randint(-(2 ** 31), 2 ** 31, (n,), generator=g, device="cuda").to(torch.int32)
    for lo, hi in [(0, 30_000_000), (-(2 ** 31), 2 ** 31 - 1), (5, 4), (-(2 ** 31), 0)]:
        at = ((key >= lo) & (key <= hi)).nonzero().flatten()
        exp = torch.stack([at.to(torch.int32), pay[at]], 1)
        assert torch.equal(ctx.filter_cols(key, pay, lo, hi), exp)
        m = exp.shape[0]
        if m > 1:
            out = torch.full((m + 64, 2), 7, dtype=torch.int32, device="cuda")
            with pytest.raises(QGError) as e:
                ctx.filter_cols(key, pay, lo, hi, cap=m - 1, out=out)
            assert e.value.status == 3
            assert torch.equal(out[: m - 1], exp[:-1]) and bool((out[m - 1:] == 7).all())


@pytest.mark.parametrize("n", [1, 5, 4097, 300_007, 5_000_003])
@pytest.mark.parametrize("sel", [0.1, 1.0])
def test_filter_cols_over_its_keys(ctx, n, sel):
    # the output lies over the key column: every key is read before a row is written
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    for _ in range(3):
        key = torch.randint(0, 1000, (n,), generator=g, device="cuda").to(torch.int32)
        pay = torch.randint(0, 1000, (n,), generator=g, device="cuda").to(torch.int32)
        hi = int(1000 * sel) - 1
        at = (key <= hi).nonzero().flatten()
        exp = torch.stack([at.to(torch.int32), pay[at]], 1)
        buf = torch.empty((n, 2), dtype=torch.int32, device="cuda")
        keys = buf.view(-1)[:n].copy_(key)
        assert torch.equal(ctx.filter_cols(keys, pay, 0, hi, out=buf), exp)


# The output over the input: at its start, before it (records that its rows have
# left behind) and inside it; one tile of 4096 records, its edges, many tiles.
@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 300_007, 5_000_001])
@pytest.mark.parametrize("shift", [0, -3000, 3000])
@pytest.mark.parametrize("sel", [0.02, 1.0])
def test_filter_rec_over_its_input(ctx, n, shift, sel):
    import ctypes

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    rec = torch.stack([torch.arange(n, device="cuda"), torch.randint(0, 1000, (n,), generator=g, device="cuda")], 1)
    rec = rec.to(torch.int32)
    hi = int(1000 * sel) - 1
    exp = rec[rec[:, 1] <= hi]
    buf = torch.full((n + 6000, 2), -9, dtype=torch.int32, device="cuda")
    buf[3000: 3000 + n] = rec
    cnt = ctypes.c_int64()
    out = buf[3000 + shift: 3000 + shift + n]
    st = ctx.lib.qg_filter_range_rec(ctx.handle, buf[3000:].data_ptr(), n, -5, hi, out.data_ptr(), n, ctypes.byref(cnt))
    assert st == 0 and cnt.value == exp.shape[0]
    assert torch.equal(out[: cnt.value], exp)


def test_filter_cols_without_scratch_takes_one_launch():
    # No room for the predicate bits: the one-launch form answers.
    from query_on_opencl_fpga_gb300.api import Context

    n = (1 << 22) + 513
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    key = torch.randint(0, 1000, (n,), generator=g, device="cuda").to(torch.int32)
    pay = torch.randint(0, 1000, (n,), generator=g, device="cuda").to(torch.int32)
    at = (key <= 99).nonzero().flatten()
    exp = torch.stack([at.to(torch.int32), pay[at]], 1)
    c = Context()
    try:
        for limit, kernels in [(200_000, {"k_filter_two"}), (0, {"k_filter_count", "k_filter_write"})]:
            c.check(c.lib.qg_ctx_set_arena_limit(c.handle, limit), "limit")
            c.enable_timing(True)
            got = c.filter_cols(key, pay, 0, 99)
            assert torch.equal(got, exp) and set(c.timing_report()) == kernels
            c.enable_timing(False)
    finally:
        c.close()
