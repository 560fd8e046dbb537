"""GPU parity of the join variants (radix / learned range partitions, hash +
sort) against the oracle, including the buckets that leave the shared-memory
bucket kernel (single-key cross products and recursive sub-joins), skewed
keys with heavy hitters, and the learned partition function itself."""
import numpy as np
import pytest
import torch

from query_on_opencl_fpga_gb300 import datagen

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def check_join(got, exp):
    gk, ga, gb = [t.cpu().numpy() for t in got]
    u = gk.view(np.uint32)
    assert (u[1:] >= u[:-1]).all(), "output not sorted by key"
    ek, ea, eb = [np.asarray(x) for x in exp]
    assert gk.size == ek.size
    g = np.lexsort((gb, ga, u))
    e = np.lexsort((eb, ea, ek.view(np.uint32)))
    assert np.array_equal(gk[g], ek[e])
    assert np.array_equal(ga[g], ea[e])
    assert np.array_equal(gb[g], eb[e])


@pytest.fixture
def knobs(ctx):
    yield ctx.join_set_knobs
    ctx.join_set_knobs(0, 0, 0, 0)


CASES = [
    # nR, nS, R keyspace, S keyspace (duplicates in R when nR > keyspace)
    (1, 1, 1, 1),
    (10, 1000, 20, 40),
    (4096, 100003, 8192, 16384),
    (1 << 16, 1 << 20, 1 << 17, 1 << 18),
    (100, 50000, 50, 100),
    (3000, 200000, 1 << 31, 1 << 31),  # sparse keys: wide buckets, bitonic path
]


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("nR,nS,kr,ks", CASES)
def test_join_variants(ctx, orc, knobs, variant, nR, nS, kr, ks):
    knobs(variant)
    rng = np.random.default_rng(nR * 7 + nS + variant)
    rkey = (rng.integers(0, kr, nR) - (kr // 2 if kr > 1 << 30 else 0)).astype(np.int64).astype(np.int32)
    rpay = rng.integers(0, 1000, nR).astype(np.int32)
    skey = (rng.integers(0, ks, nS) - (ks // 2 if ks > 1 << 30 else 0)).astype(np.int64).astype(np.int32)
    if ks > 1 << 30:  # make sparse keys hit R too
        pick = rng.random(nS) < 0.5
        skey[pick] = rkey[rng.integers(0, nR, int(pick.sum()))]
    spay = rng.integers(0, 1000, nS).astype(np.int32)
    got = ctx.join_filter_sort(dev(rkey), dev(rpay), dev(skey), dev(spay), -(2 ** 31), 299)
    exp = orc.join_filter_sort(rkey, rpay, skey, spay, -(2 ** 31), 299,
                               cap=nS * max(1, nR // max(1, min(kr, nR)) + 8), mt=True)
    check_join(got, exp)


@pytest.mark.parametrize("variant", [1, 2])
def test_join_outside_buckets(ctx, orc, knobs, variant):
    # Tiny bucket capacities and few buckets: most buckets leave the bucket
    # kernel -- heavy single keys become cross products, the rest take the
    # sort-merge path.
    knobs(variant, 4, 64, 32)
    rng = np.random.default_rng(5)
    base = rng.integers(0, 1 << 20, 3000)
    rkey = np.concatenate([base, np.full(5, 777), np.full(3, -5)]).astype(np.int32)
    rpay = rng.integers(0, 1000, rkey.size).astype(np.int32)
    skey = np.concatenate([rng.choice(base, 40000), np.full(3000, 777), np.full(500, -5),
                           rng.integers(0, 1 << 21, 5000)]).astype(np.int32)
    rng.shuffle(skey)
    spay = rng.integers(0, 1000, skey.size).astype(np.int32)
    got = ctx.join_filter_sort(dev(rkey), dev(rpay), dev(skey), dev(spay), -(2 ** 31), 499)
    st = ctx.join_stats()
    assert st["outside_buckets"] > 0
    exp = orc.join_filter_sort(rkey, rpay, skey, spay, -(2 ** 31), 499, cap=skey.size * 8, mt=True)
    check_join(got, exp)


@pytest.mark.parametrize("variant", [1, 2])
def test_join_sort_merge_with_duplicate_build_keys(ctx, orc, knobs, variant):
    # Every build key three times, tiny bucket capacities: the oversize buckets
    # hold several keys each (the sort-merge path) and every probe row that
    # hits matches three build rows.
    knobs(variant, 6, 256, 96)
    rng = np.random.default_rng(9)
    keys = rng.choice(1 << 22, 20000, replace=False).astype(np.int32)
    rkey = np.repeat(keys, 3)
    rng.shuffle(rkey)
    rpay = rng.integers(0, 1000, rkey.size).astype(np.int32)
    skey = np.concatenate([rng.choice(keys, 150000), rng.integers(0, 1 << 22, 20000)]).astype(np.int32)
    spay = rng.integers(0, 1000, skey.size).astype(np.int32)
    got = ctx.join_filter_sort(dev(rkey), dev(rpay), dev(skey), dev(spay), -(2 ** 31), 599, cap=skey.size * 4)
    st = ctx.join_stats()
    assert st["merge_buckets"] > 0
    exp = orc.join_filter_sort(rkey, rpay, skey, spay, -(2 ** 31), 599, cap=skey.size * 4, mt=True)
    check_join(got, exp)


@pytest.mark.parametrize("variant", [0, 1, 2])
def test_join_skewed_mixture(ctx, orc, knobs, variant):
    knobs(variant)
    d = datagen.config4_skewed(1 << 17, 1 << 21, seed=3)
    args = [d[k].numpy() for k in ("rkey", "rpay", "skey", "spay")]
    got = ctx.join_filter_sort(*[dev(a) for a in args], d["slo"], d["shi"])
    st = ctx.join_stats()
    assert st["path"] == {0: st["path"], 1: "radix", 2: "learned"}[variant]
    check_join(got, orc.join_filter_sort(*args, d["slo"], d["shi"], mt=True))


def test_learned_spreads_skew_better_than_radix(ctx, knobs):
    # On the skewed mixture, radix partitioning leaves most rows in buckets
    # too big for shared memory; the learned partition function does not.
    d = datagen.config4_skewed(1 << 18, 1 << 22, seed=4, device="cuda")
    rows = {}
    for v in (1, 2):
        knobs(v)
        ctx.join_filter_sort(d["rkey"], d["rpay"], d["skey"], d["spay"], d["slo"], d["shi"])
        rows[v] = ctx.join_stats()["outside_rows"]
    assert rows[2] * 4 < rows[1]


def test_part_model_monotone_and_heavy_keys_isolated(ctx):
    keys = datagen.skewed_keys(1 << 20, 9, device="cuda")
    nb = 4096
    model = ctx.part_learn(keys, nb)
    u = torch.unique(keys.to(torch.int64) & 0xFFFFFFFF)  # ascending unsigned
    probe = torch.cat([u, u + 1, u - 1]).clamp(0, 2 ** 32 - 1)
    probe = torch.unique(probe)
    probe32 = (probe - (probe >= 2 ** 31).to(torch.int64) * 2 ** 32).to(torch.int32)
    b = ctx.part_eval(probe32, model).to(torch.int64)
    assert int(b.min()) >= 0 and int(b.max()) < nb
    assert bool((b[1:] >= b[:-1]).all()), "bucket function not monotone in the unsigned key"
    # the most frequent key owns its bucket
    vals, cnt = torch.unique(keys, return_counts=True)
    top = vals[cnt.argmax()].reshape(1)
    tb = int(ctx.part_eval(top, model)[0])
    same = probe32[(b == tb)]
    assert same.numel() == 1 and int(same[0]) == int(top[0])
    # buckets are balanced within a few times the mean on the sample itself
    hb = torch.bincount(ctx.part_eval(keys, model).to(torch.int64), minlength=nb)
    heavy_mass = int(cnt.max())
    assert int(hb.max()) <= max(8 * keys.numel() // nb, heavy_mass)


def test_part_radix_eval(ctx):
    keys = torch.tensor([5, 6, 1029, -1], dtype=torch.int32, device="cuda")
    b = ctx.part_eval(keys, None, kmin=5, shift=10).cpu().tolist()
    assert b == [0, 0, 1, (2 ** 32 - 1 - 5) >> 10]


@pytest.mark.parametrize("variant", [1, 2])
def test_join_config4_full_size(ctx, knobs, variant):
    # The skewed config at the size the bench quotes (R 32M unique keys, S 256M
    # keys from 8 Gaussians + 5 % Zipf(1.2) heavy hitters, S.payload < 300),
    # radix (1) and learned (2) partitioning; both leave rows in oversize
    # buckets, so the sort-merge and cross-product paths run.  Size-independent
    # exact checks: the row count equals the filtered S rows whose key is in R,
    # keys ascend (unsigned), every R.payload is R's payload for that key, and
    # the multiset of (key, S.payload) equals the filtered, matching S rows'.
    knobs(variant)
    d = datagen.config4_skewed(1 << 25, 1 << 28, seed=0, device="cuda")
    ok, orp, osp = ctx.join_filter_sort(d["rkey"], d["rpay"], d["skey"], d["spay"], d["slo"], d["shi"],
                                        cap=120_000_000)
    st = ctx.join_stats()
    assert st["path"] == {1: "radix", 2: "learned"}[variant]
    assert st["outside_rows"] > 0, st
    ru = d["rkey"].long() & 0xFFFFFFFF
    ru_sorted, order = torch.sort(ru)
    rpay_sorted = d["rpay"][order]
    del ru, order
    m = d["spay"] <= 299
    sk = d["skey"][m].long() & 0xFFFFFFFF
    ss = d["spay"][m].long()
    del m
    pos = torch.searchsorted(ru_sorted, sk).clamp_(max=ru_sorted.numel() - 1)
    hit = ru_sorted[pos] == sk
    sk, ss = sk[hit], ss[hit]
    del pos, hit
    assert ok.numel() == sk.numel()
    gu = ok.long() & 0xFFFFFFFF
    assert bool((gu[1:] >= gu[:-1]).all())
    gpos = torch.searchsorted(ru_sorted, gu)
    assert torch.equal(orp, rpay_sorted[gpos])
    del gpos
    e = torch.sort(sk * 1024 + ss).values
    del sk, ss
    g = torch.sort(gu * 1024 + osp.long()).values
    assert torch.equal(e, g)


@pytest.fixture
def dense_knob(ctx):
    yield ctx.join_set_dense
    ctx.join_set_dense(True)


@pytest.mark.parametrize("wide_pay", [False, True])
@pytest.mark.parametrize("nR,nS,gap,base", [
    (1, 5, 1, 7),
    (1000, 50000, 1, 0),
    (1 << 16, 1 << 20, 1, 1000),
    (1 << 16, 1 << 20, 2, -(1 << 20)),      # every other key, all negative (one unsigned span)
    (50000, 3 << 20, 1, (1 << 31) - 25000),  # keys across 0x7fffffff / 0x80000000 (unsigned order)
])
def test_join_dense_build_side(ctx, orc, knobs, dense_knob, nR, nS, gap, base, wide_pay):
    # Unique R keys over a dense span: R becomes a payload table indexed by
    # key - min -- absent keys marked by a sentinel payload that no R row holds,
    # or, when R's payloads span every candidate (wide_pay), by a presence
    # bitmap -- and only S is partitioned.  Equal to the oracle, to the general
    # path (dense build side off) and to the learned partitioning (which takes
    # the general path).
    rng = np.random.default_rng(nR + nS + gap)
    rk = (rng.permutation(nR).astype(np.int64) * gap + base)
    rkey = ((rk + (1 << 31)) % (1 << 32) - (1 << 31)).astype(np.int32)
    rpay = rng.integers(-1000, 1000, nR).astype(np.int32)
    if wide_pay:
        rpay[0] = -(2 ** 31)
        rpay[-1] = 2 ** 31 - 1
    sk = rng.integers(base - 300, base + nR * gap + 300, nS)
    skey = ((sk + (1 << 31)) % (1 << 32) - (1 << 31)).astype(np.int32)
    spay = rng.integers(0, 1000, nS).astype(np.int32)
    skey[0], spay[0] = rkey[0], 0  # at least one S row passes the filters
    exp = orc.join_filter_sort(rkey, rpay, skey, spay, -(2 ** 31), 299, cap=nS + 16, mt=True)
    args = [dev(a) for a in (rkey, rpay, skey, spay)]
    check_join(ctx.join_filter_sort(*args, -(2 ** 31), 299), exp)
    assert ctx.join_stats()["path"] == "dense"
    knobs(0, 0, 1024, 0)  # groups of at most 1024 rows: the 512-thread form of the dense bucket kernel
    check_join(ctx.join_filter_sort(*args, -(2 ** 31), 299), exp)
    assert ctx.join_stats()["path"] == "dense"
    knobs(0)
    dense_knob(False)
    check_join(ctx.join_filter_sort(*args, -(2 ** 31), 299), exp)
    assert ctx.join_stats()["path"] == "radix"
    dense_knob(True)
    knobs(2)
    check_join(ctx.join_filter_sort(*args, -(2 ** 31), 299), exp)
    assert ctx.join_stats()["path"] == "learned"


def test_join_dense_span_duplicate_key_takes_general_path(ctx, orc):
    # A dense span with one key twice: the bitmap sees the duplicate, and the
    # general path (R records after all) joins both build rows.
    rng = np.random.default_rng(21)
    rkey = rng.permutation(20000).astype(np.int32)
    rkey[5] = rkey[6]
    rpay = rng.integers(0, 1000, rkey.size).astype(np.int32)
    skey = rng.integers(-10, 20010, 300000).astype(np.int32)
    spay = rng.integers(0, 1000, skey.size).astype(np.int32)
    got = ctx.join_filter_sort(dev(rkey), dev(rpay), dev(skey), dev(spay), -(2 ** 31), 299)
    assert ctx.join_stats()["path"] == "radix"
    check_join(got, orc.join_filter_sort(rkey, rpay, skey, spay, -(2 ** 31), 299, cap=skey.size * 2, mt=True))


def test_join_dense_oversize_bucket_falls_back(ctx, orc):
    # Unique R keys over a dense span, but one S key holds 200K rows: its
    # bucket exceeds the bucket kernel, so R's records are made after all and
    # the general path (with its outside buckets) finishes the join.
    rng = np.random.default_rng(22)
    nR = 1 << 16
    rkey = rng.permutation(nR).astype(np.int32)
    rpay = rng.integers(0, 1000, nR).astype(np.int32)
    skey = np.concatenate([rng.integers(0, nR, 1 << 20), np.full(200000, 4321)]).astype(np.int32)
    rng.shuffle(skey)
    spay = rng.integers(0, 1000, skey.size).astype(np.int32)
    got = ctx.join_filter_sort(dev(rkey), dev(rpay), dev(skey), dev(spay), -(2 ** 31), 299)
    st = ctx.join_stats()
    assert st["path"] == "radix" and st["outside_buckets"] > 0, st
    check_join(got, orc.join_filter_sort(rkey, rpay, skey, spay, -(2 ** 31), 299, cap=skey.size + 16, mt=True))


@pytest.mark.parametrize("full", [True, False])
def test_join_dense_capacity_error(ctx, orc, full):
    # The dense bucket kernel writes only below `cap` and the call reports the
    # size needed (QG_ERR_CAPACITY); the wrapper then retries with it.  With
    # and without every S' row matching (a permutation of the span, or gaps).
    from ctypes import byref, c_int64, c_void_p

    rng = np.random.default_rng(41)
    nR, nS = 1 << 14, 1 << 18
    rkey = (rng.permutation(nR) * (1 if full else 2)).astype(np.int32)
    rpay = rng.integers(0, 1000, nR).astype(np.int32)
    skey = rng.integers(0, nR * (1 if full else 2), nS).astype(np.int32)
    spay = rng.integers(0, 1000, nS).astype(np.int32)
    exp = orc.join_filter_sort(rkey, rpay, skey, spay, -(2 ** 31), 299, cap=nS + 16, mt=True)
    need = len(exp[0])
    r, rp, s, sp = (dev(a) for a in (rkey, rpay, skey, spay))
    small = need // 3
    out = [torch.full((small + 64,), 7, dtype=torch.int32, device="cuda") for _ in range(3)]
    m = c_int64()
    p = lambda t: c_void_p(t.data_ptr())  # noqa: E731
    st = ctx.lib.qg_join_filter_sort(ctx.handle, p(r), p(rp), nR, p(s), p(sp), nS, -(2 ** 31), 299,
                                     p(out[0]), p(out[1]), p(out[2]), small, byref(m))
    assert st == 3 and m.value == need
    assert ctx.join_stats()["path"] == "dense"
    assert all(int((o[small:] != 7).sum()) == 0 for o in out), "a row was written past cap"
    check_join(ctx.join_filter_sort(r, rp, s, sp, -(2 ** 31), 299), exp)


def _join_case(ctx, orc, rkey, rpay, skey, spay, path, hi=299, extra=16):
    exp = orc.join_filter_sort(rkey, rpay, skey, spay, -(2 ** 31), hi, cap=skey.size * extra, mt=True)
    args = [dev(a) for a in (rkey, rpay, skey, spay)]
    for _ in range(2):  # the second call knows what the first one found
        check_join(ctx.join_filter_sort(*args, -(2 ** 31), hi, cap=max(len(exp[0]), 1)), exp)
        assert ctx.join_stats()["path"] == path
    return len(exp[0])


# The counting path around its tiles (2 and 16 table entries per lane, 4096 probe
# rows, the most build rows that one CTA takes), spans of nR, 2 nR and 2 nR + 1 values, keys at the ends of the range,
# build payloads of every value, a key with the most rows it takes and one more.
@pytest.mark.parametrize("nR,nS,gap", [(1, 1, 1), (255, 4095, 1), (256, 4096, 2), (257, 4097, 1), (1025, 3000, 2),
                                       (2048, 70_000, 2), (2049, 70_000, 2), (1 << 18, 9000, 1),
                                       ((1 << 18) + 1, 50_001, 2), (5000, 300_003, 1)])
@pytest.mark.parametrize("base", [0, -(2 ** 31), 2 ** 31 - 600_000])
def test_join_counting_path_edges(ctx, orc, nR, nS, gap, base):
    rng = np.random.default_rng(nR + nS)
    off = rng.permutation(nR).astype(np.int64) * gap
    if gap == 2:
        off[np.argmax(off)] = 2 * nR - 1  # the widest dense span
    rkey = (base + off).astype(np.int64)
    rkey = ((rkey + 2 ** 31) % 2 ** 32 - 2 ** 31).astype(np.int32)
    rpay = rng.choice(np.array([-(2 ** 31), 2 ** 31 - 1, -1, 0, 7]), nR).astype(np.int32)
    skey = ((base + rng.integers(-3, nR * gap + 3, nS) + 2 ** 31) % 2 ** 32 - 2 ** 31).astype(np.int32)
    spay = rng.integers(0, 1000, nS).astype(np.int32)
    _join_case(ctx, orc, rkey, rpay, skey, spay, "dense")


def test_join_counting_path_limits(ctx, orc):
    rng = np.random.default_rng(3)
    n = 1000
    rpay = rng.integers(0, 1000, n).astype(np.int32)
    rkey = rng.permutation(n).astype(np.int32)
    skey = np.concatenate([rng.integers(0, n, 20_000), np.full(4000, n + 5)]).astype(np.int32)
    spay = np.full(skey.size, 5, np.int32)
    for rows, path in ((4096, "dense"), (4098, "radix")):  # rows of one key
        s = np.concatenate([skey[skey != 77], np.full(rows, 77, np.int32)])
        _join_case(ctx, orc, rkey, rpay, s, np.full(s.size, 5, np.int32), path)
    wide = rkey.astype(np.int64) * 2
    wide[np.argmax(wide)] = 2 * n  # one value too wide
    _join_case(ctx, orc, wide.astype(np.int32), rpay, skey, spay, "hash_sort")
    _join_case(ctx, orc, rkey, rpay, skey, spay, "dense")  # and back


# The hash join behind the default: 8192 and 8193 matches (one-CTA sort), key
# ranges of 1 to 4 digits, build keys twice, the key and payload that mark free
# slots, no match at all.
@pytest.mark.parametrize("bits", [14, 20, 27, 32])
@pytest.mark.parametrize("m", [0, 1, 8192, 8193, 60_000])
@pytest.mark.parametrize("twice", [False, True])
def test_join_sparse_keys_take_the_hash_join(ctx, orc, bits, m, twice):
    rng = np.random.default_rng(bits + m)
    nR = 3000
    keys = np.unique(np.concatenate([[0, 2 ** bits - 1], rng.integers(0, 2 ** bits, 2 * nR)]))[:nR].astype(np.int64)
    keys[-1] = 2 ** bits - 1
    gone = np.setdiff1d(rng.integers(0, 2 ** bits, 4000), keys)
    rkey = np.concatenate([keys, keys[:50]]) if twice else keys
    rpay = rng.integers(-5, 5, rkey.size).astype(np.int64)
    rpay[keys.size - 1] = -1
    hits = keys[rng.integers(50 if twice else 0, keys.size, m)]
    if twice:
        hits = np.concatenate([hits, keys[:50]])
    skey = np.concatenate([hits, gone])
    spay = np.zeros(skey.size, np.int64)
    p = rng.permutation(skey.size)
    as32 = lambda x: ((x + 2 ** 31) % 2 ** 32 - 2 ** 31).astype(np.int32)  # noqa: E731
    got = _join_case(ctx, orc, as32(rkey), as32(rpay), as32(skey[p]), as32(spay[p]), "hash_sort")
    assert got == m + (100 if twice else 0)


def test_join_sparse_crowded_key_takes_general_path(ctx, orc):
    # one build key 2000 times: more slots than a row may look at
    rng = np.random.default_rng(8)
    rkey = np.concatenate([rng.integers(-(2 ** 31), 2 ** 31, 5000), np.full(2000, 123)]).astype(np.int32)
    rpay = rng.integers(0, 9, rkey.size).astype(np.int32)
    skey = np.concatenate([rng.choice(rkey[:5000], 20_000), np.full(3, 123)]).astype(np.int32)
    spay = rng.integers(0, 400, skey.size).astype(np.int32)
    spay[-3:] = 1
    _join_case(ctx, orc, rkey, rpay, skey, spay, "radix")


def _hash32(x):
    x = x.astype(np.uint64)
    for mul, sh in ((0x85EBCA6B, 16), (0xC2B2AE35, 13)):
        x ^= x >> np.uint64(sh)
        x = x * np.uint64(mul) & np.uint64(0xFFFFFFFF)
    return x ^ (x >> np.uint64(16))


# Large probe inputs with a dense build side (one partition step): every value of
# R's span present, half of it (with a payload that leaves no sentinel), every row
# selected, few, none; a frequent key that the sample shows (another path), and
# rows off the sampled ones that overflow a bucket's room.
@pytest.mark.parametrize("kind", ["full", "half", "all", "few", "none", "hot", "missed"])
def test_join_large_dense(ctx, kind):
    nS = 20_000_003
    nR = 1_300_000
    step = 2 if kind == "half" else 1
    base = -(2 ** 31) + 5 if kind == "half" else 2 ** 31 - 1_000_000 if kind == "few" else 0
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    ints = lambda lo, hi, n: torch.randint(lo, hi, (n,), generator=g, device="cuda")  # noqa: E731
    roff = torch.randperm(nR, generator=g, device="cuda") * step
    rpay = ints(-(2 ** 31), 2 ** 31, nR) if kind != "half" else ints(0, 2, nR) * (2 ** 32 - 1) - 2 ** 31
    soff = ints(0, nR * step, nS) if kind in ("all", "missed") else ints(-nR, 3 * nR * step, nS)
    spay = ints(0, 1000, nS)
    row = np.arange(nS // 1024 * 1024)
    sampled = (row % 1024) // 16 == (_hash32(row // 1024) & np.uint64(63)).astype(np.int64)
    off = torch.from_numpy(np.flatnonzero(~sampled)).cuda()  # rows that the sample does not see
    hi = {"all": 999, "few": 3, "none": -1}.get(kind, 299)
    if kind == "hot":
        soff[::200] = 12_345
    elif kind == "missed":
        soff[off] = soff[off] % (nR // 3)
    i32 = lambda t: (((t + base + 2 ** 31) & 0xFFFFFFFF) - 2 ** 31).to(torch.int32)  # noqa: E731
    skey = i32(soff)
    for _ in range(2):  # the first call may follow one with sparse keys
        got = ctx.join_filter_sort(i32(roff), rpay.to(torch.int32), skey, spay.to(torch.int32), 0, hi, cap=nS)
    if kind not in ("hot", "missed"):
        assert ctx.join_stats()["path"] == "dense"
    table = torch.full((nR * step,), 2 ** 40, dtype=torch.int64, device="cuda")
    table[roff] = rpay
    sel = (spay <= hi) & (soff >= 0) & (soff < nR * step)
    so, sp = soff[sel], spay[sel]
    here = table[so] < 2 ** 40
    exp = (((so[here] + base) & 0xFFFFFFFF) * 1000 + sp[here]).sort().values
    uk = got[0].to(torch.int64) & 0xFFFFFFFF
    assert bool((uk[1:] >= uk[:-1]).all())
    assert torch.equal((uk * 1000 + got[2]).sort().values, exp)
    assert torch.equal(got[1].to(torch.int64), table[(uk - base) & 0xFFFFFFFF])


# Many probe rows on build keys three apart: partitioned, whichever path the last
# call took (keys three hundred apart are hashed).
def test_join_large_near_keys(ctx):
    nS, nR = 40_000_003, 700_000
    g = torch.Generator(device="cuda")
    g.manual_seed(12)
    ints = lambda lo, hi, n: torch.randint(lo, hi, (n,), generator=g, device="cuda")  # noqa: E731
    r = torch.randperm(nR, generator=g, device="cuda")
    rpay, soff, spay = ints(0, 1 << 20, nR), ints(0, 4 * nR, nS), ints(0, 1000, nS)
    hit = (soff % 3 == 0) & (soff < 3 * nR) & (spay <= 99)
    table = torch.empty(nR, dtype=torch.int64, device="cuda")
    table[r] = rpay
    exp = (soff[hit] // 3 * 1000 + spay[hit]).sort().values
    for stride in (3, 300, 3, 3):
        # rows that match no key lie between two of them
        key = torch.where(soff % 3 == 0, soff // 3 * stride, soff // 3 * stride + 1)
        got = ctx.join_filter_sort((r * stride).to(torch.int32), rpay.to(torch.int32), key.to(torch.int32),
                                   spay.to(torch.int32), 0, 99, cap=nS)
        k = got[0].to(torch.int64) // stride
        assert bool((k[1:] >= k[:-1]).all())
        assert torch.equal((k * 1000 + got[2]).sort().values, exp)
        assert torch.equal(got[1].to(torch.int64), table[k])
    assert ctx.join_stats()["path"] == "radix"


# Probe keys with far too many rows, met by some CTAs while others still start or
# wait for an SM that another stream's kernels hold: the attempt ends everywhere.
def test_join_counting_path_hot_keys_beside_other_work():
    from query_on_opencl_fpga_gb300.api import Context

    nR, nS = 30_000, 3_000_003
    g = torch.Generator(device="cuda")
    g.manual_seed(17)
    ints = lambda lo, hi, n: torch.randint(lo, hi, (n,), generator=g, device="cuda")  # noqa: E731
    roff, rpay = torch.randperm(nR, generator=g, device="cuda"), ints(0, 1000, nR)
    soff, spay = ints(0, 2 * nR, nS), ints(0, 1000, nS)
    soff[nS // 2:: 3] = 5 + ints(0, 3, soff[nS // 2:: 3].numel())
    sel = (spay <= 299) & (soff < nR)
    table = torch.empty(nR, dtype=torch.int64, device="cuda")
    table[roff] = rpay
    exp = (soff[sel] * 1000 + spay[sel]).sort().values
    args = [t.to(torch.int32) for t in (roff, rpay, soff, spay)]
    side, busy = torch.cuda.Stream(), torch.empty(1 << 26, dtype=torch.int32, device="cuda")
    for rep in range(6):
        c = Context()
        try:
            with torch.cuda.stream(side):
                for _ in range(rep * 3):
                    busy.add_(1)
            got = c.join_filter_sort(*args, 0, 299, cap=nS)
            assert c.join_stats()["path"] == "radix"
        finally:
            c.close()
        k = got[0].to(torch.int64)
        assert bool((k[1:] >= k[:-1]).all())
        assert torch.equal((k * 1000 + got[2]).sort().values, exp)
        assert torch.equal(got[1].to(torch.int64), table[k])
    torch.cuda.synchronize()


# Outputs over the probe columns: an attempt that is given up has written nothing
# when the next path reads them.
@pytest.mark.parametrize("kind", ["dup", "hot", "after_sparse"])
def test_join_outputs_over_inputs(orc, kind):
    import ctypes

    from query_on_opencl_fpga_gb300.api import Context

    rng = np.random.default_rng(31)
    nR, nS = 20_000, 300_000
    rkey = rng.permutation(nR).astype(np.int32)
    if kind == "dup":
        rkey[5] = rkey[6]
    rpay = rng.integers(0, 1000, nR).astype(np.int32)
    skey = rng.integers(-10, nR + 10, nS).astype(np.int32)
    if kind == "hot":
        skey[:6000] = 77
    spay = rng.integers(0, 1000, nS).astype(np.int32)
    c = Context()
    try:
        if kind == "after_sparse":  # the hash join is launched first, and meets a dense span
            c.join_filter_sort(dev(rkey * 100), dev(rpay), dev(skey), dev(spay))
            assert c.join_stats()["path"] == "hash_sort"
        exp = orc.join_filter_sort(rkey, rpay, skey, spay, -(2 ** 31), 299, cap=nS, mt=True)
        r, rp, s, sp = (dev(a) for a in (rkey, rpay, skey, spay))
        o = torch.empty_like(s)
        m = ctypes.c_int64()
        p = lambda t: t.data_ptr()  # noqa: E731
        st = c.lib.qg_join_filter_sort(c.handle, p(r), p(rp), nR, p(s), p(sp), nS, -(2 ** 31), 299, p(s), p(o), p(sp),
                                       nS, ctypes.byref(m))
        assert st == 0
        check_join([t[: m.value] for t in (s, o, sp)], exp)
    finally:
        c.close()


def launched(c, call):
    """Names of the kernels that a call launches."""
    c.timing_report()
    c.enable_timing(True)
    try:
        call()
        return set(c.timing_report())
    finally:
        c.enable_timing(False)


def _join_rows(rng, kind):
    nR, nS = 20_000, 300_000
    rkey = rng.permutation(nR).astype(np.int32)
    skey = rng.integers(-10, nR + 10, nS).astype(np.int32)
    if kind == "crowded":
        rkey = np.concatenate([rng.integers(-(2 ** 31), 2 ** 31, 5000), np.full(2000, 123)]).astype(np.int32)
        skey = np.concatenate([rng.choice(rkey[:5000], 20_000), np.full(3, 123)]).astype(np.int32)
    if kind == "marks":
        rkey = np.concatenate([rng.integers(-(2 ** 31), 2 ** 31, 5000), np.full(2000, -1)]).astype(np.int32)
        skey = np.concatenate([rng.choice(rkey[:5000], 20_000), np.full(3, -1)]).astype(np.int32)
    rpay = rng.integers(0, 1000, rkey.size).astype(np.int32)
    if kind == "marks":
        rpay[5000:] = -1
    return rkey, rpay, skey, rng.integers(0, 300, skey.size).astype(np.int32)


# Build keys that repeat (one of them, and the key and payload that mark free slots):
# given up by the hash join, and not tried again by the next calls; unique dense keys
# are counted all the same.
@pytest.mark.parametrize("kind,left_out", [("crowded", "k_join_build"), ("marks", "k_join_build")])
def test_join_failed_attempt_is_not_repeated(orc, kind, left_out):
    from query_on_opencl_fpga_gb300.api import Context

    rng = np.random.default_rng(33)
    a = _join_rows(rng, kind)
    exp = orc.join_filter_sort(*a, 0, 299, cap=a[2].size * 4 + 10_000, mt=True)
    c = Context()
    try:
        d = [dev(x) for x in a]
        for i in range(2):
            got = []
            names = launched(c, lambda: got.extend(c.join_filter_sort(*d, 0, 299, cap=len(exp[0]))))
            check_join(got, exp)
            assert c.join_stats()["path"] == "radix"
            if i:
                assert left_out not in names, names
        u = [dev(x) for x in _join_rows(rng, "unique")]
        for i in range(2):
            names = launched(c, lambda: c.join_filter_sort(*u, 0, 299))
            assert c.join_stats()["path"] == "dense"
        assert "k_jd_count" in names
    finally:
        c.close()


# Many build keys twice or more, in the sizes' three ranges, just below and far above
# what the hash join bears: the same rows whichever path answers.
@pytest.mark.parametrize("nR", [900, 40_000, 700_000])
@pytest.mark.parametrize("times,share", [(2, 0.1), (2, 1.0), (8, 0.02), (8, 1.0), (40, 1.0)])
def test_join_sparse_repeated_keys(ctx, nR, times, share):
    nS = 3 * nR
    g = torch.Generator(device="cuda")
    g.manual_seed(nR + times)
    rk = torch.randint(-(2 ** 31), 2 ** 31, (nR,), generator=g, device="cuda")
    many = int(nR * share) // times * times
    rk[:many] = rk[: many // times].repeat(times)
    rk = rk[torch.randperm(nR, generator=g, device="cuda")]
    sk = torch.where(torch.rand(nS, generator=g, device="cuda") < 0.3, rk[torch.randint(0, nR, (nS,), generator=g, device="cuda")],
                     torch.randint(-(2 ** 31), 2 ** 31, (nS,), generator=g, device="cuda"))
    rp, sp = torch.arange(nR, device="cuda"), torch.randint(0, 1000, (nS,), generator=g, device="cuda")
    order = torch.argsort(rk)
    rs = rk[order]
    sel = sp <= 299
    a, n = torch.searchsorted(rs, sk[sel]), torch.searchsorted(rs, sk[sel], right=True)
    n -= a
    row = torch.repeat_interleave(torch.arange(n.numel(), device="cuda"), n)
    at = a[row] + torch.arange(row.numel(), device="cuda") - (n.cumsum(0) - n)[row]
    exp = ((rp[order][at] << 10) | sp[sel][row]).sort().values  # a build row's payload tells its key
    for _ in range(2):
        got = ctx.join_filter_sort(rk.to(torch.int32), rp.to(torch.int32), sk.to(torch.int32), sp.to(torch.int32), 0, 299,
                                   cap=max(exp.numel(), 1))
        u = got[0].to(torch.int64) & 0xFFFFFFFF
        assert bool((u[1:] >= u[:-1]).all())
        assert torch.equal(((got[1].to(torch.int64) << 10) | got[2]).sort().values, exp)
        assert torch.equal(got[0].to(torch.int64), rk[got[1].to(torch.int64)])


# The line between hashing and partitioning close build keys: 24M probe rows and 2.5M
# build rows, a span of 5/8 of the probe rows' number, keys four apart.
@pytest.mark.parametrize("nS,nR,stride,path", [(24_000_001, 2_500_001, 5, "radix"), (24_000_001, 2_500_001, 7, "hash_sort"),
                                               (24_000_001, 2_500_000, 5, "hash_sort"), (24_000_000, 2_500_001, 5, "hash_sort"),
                                               (24_000_001, 5_000_000, 4, "radix")])
def test_join_near_line(nS, nR, stride, path):
    from query_on_opencl_fpga_gb300.api import Context

    g = torch.Generator(device="cuda")
    g.manual_seed(nR + stride)
    r = torch.randperm(nR, generator=g, device="cuda")
    soff, spay = (torch.randint(0, m, (nS,), generator=g, device="cuda") for m in (2 * nR, 1000))
    hit = (soff % 2 == 0) & (spay <= 99)
    key = torch.where(soff % 2 == 0, soff // 2 * stride, soff // 2 * stride + 1)
    exp = (soff[hit] // 2 * 1000 + spay[hit]).sort().values
    args = [t.to(torch.int32) for t in (r * stride, r, key, spay)]
    c = Context()
    try:
        for _ in range(2):
            got = c.join_filter_sort(*args, 0, 99, cap=nS)
            k = got[0].to(torch.int64) // stride
            assert torch.equal(got[1].to(torch.int64), k) and bool((k[1:] >= k[:-1]).all())
            assert torch.equal((k * 1000 + got[2]).sort().values, exp)
            assert c.join_stats()["path"] == path
    finally:
        c.close()


def _sparse_rows(g, nR, nS):
    ints = lambda lo, hi, n: torch.randint(lo, hi, (n,), generator=g, device="cuda")  # noqa: E731
    rk = torch.randperm(nR, generator=g, device="cuda") * (2 ** 32 // nR) - 2 ** 31
    s = ints(0, nR, nS)
    rp, sp = ints(0, 1000, nR), ints(0, 1000, nS)
    exp = (((rk[s] & 0xFFFFFFFF) * 1000 + rp[s]) * 1000 + sp)[sp <= 299].sort().values
    return [t.to(torch.int32) for t in (rk, rp, rk[s], sp)], exp


def _check_sparse(got, exp):
    u = got[0].to(torch.int64) & 0xFFFFFFFF
    assert bool((u[1:] >= u[:-1]).all())
    assert torch.equal(((u * 1000 + got[1]) * 1000 + got[2]).sort().values, exp)


def test_join_without_room_for_the_hash_join():
    # A generous capacity sizes the hash join's columns, not the partitioned path's
    # arrays: without memory for the former the latter answers.
    from query_on_opencl_fpga_gb300.api import Context

    g = torch.Generator(device="cuda")
    g.manual_seed(41)
    args, exp = _sparse_rows(g, 50_000, 200_000)
    c = Context()
    try:
        c.check(c.lib.qg_ctx_set_arena_limit(c.handle, 256 << 20), "limit")
        for _ in range(3):
            _check_sparse(c.join_filter_sort(*args, 0, 299, cap=40_000_000), exp)
            assert c.join_stats()["path"] == "radix"
        c.check(c.lib.qg_ctx_set_arena_limit(c.handle, 0), "limit")
    finally:
        c.close()


def test_join_hash_without_room_for_a_third_set_of_columns():
    # An even number of sort passes over more matches than the table's memory holds:
    # without the spare columns they end in the first set and are copied.
    from query_on_opencl_fpga_gb300.api import Context

    g = torch.Generator(device="cuda")
    g.manual_seed(42)
    small, small_exp = _sparse_rows(g, 3000, 9000)
    args, exp = _sparse_rows(g, 3000, 200_000)
    c = Context()
    try:
        for _ in range(2):  # the other arenas have their size then
            _check_sparse(c.join_filter_sort(*small, 0, 299, cap=2_000_000), small_exp)
        c.check(c.lib.qg_ctx_set_arena_limit(c.handle, 100_000), "limit")
        for _ in range(2):
            _check_sparse(c.join_filter_sort(*args, 0, 299, cap=200_000), exp)
            assert c.join_stats()["path"] == "hash_sort"
    finally:
        c.close()


def test_join_large_overflow_is_not_repeated():
    # Probe rows off the sampled ones crowd one bucket's range: the partition step runs
    # over, the next call leaves it out, and sparse build keys between are hashed.
    from query_on_opencl_fpga_gb300.api import Context

    nS, nR = 20_000_003, 1_300_000
    g = torch.Generator(device="cuda")
    g.manual_seed(13)
    ints = lambda lo, hi, n: torch.randint(lo, hi, (n,), generator=g, device="cuda")  # noqa: E731
    r, rpay, soff, spay = torch.randperm(nR, generator=g, device="cuda"), ints(0, 1000, nR), ints(0, nR, nS), ints(0, 1000, nS)
    row = np.arange(nS // 1024 * 1024)
    sampled = (row % 1024) // 16 == (_hash32(row // 1024) & np.uint64(63)).astype(np.int64)
    off = torch.from_numpy(np.flatnonzero(~sampled)).cuda()
    soff[off] = soff[off] % (nR // 3)
    sel = spay <= 299
    table = torch.empty(nR, dtype=torch.int64, device="cuda")
    table[r] = rpay
    exp = (soff[sel] * 1000 + spay[sel]).sort().values
    c = Context()
    try:
        for i, stride in enumerate((1, 1, 1000, 1)):
            args = [t.to(torch.int32) for t in (r * stride, rpay, soff * stride, spay)]
            got = []
            names = launched(c, lambda: got.extend(c.join_filter_sort(*args, 0, 299, cap=nS)))
            k = got[0].to(torch.int64) // stride
            assert bool((k[1:] >= k[:-1]).all())
            assert torch.equal((k * 1000 + got[2]).sort().values, exp) and torch.equal(got[1].to(torch.int64), table[k])
            assert c.join_stats()["path"] == ("hash_sort" if stride > 1 else c.join_stats()["path"])
            assert ("k_jp_part" in names) == (i == 0), (i, names)
    finally:
        c.close()


# Which form answers: each new one where it is meant to, and not where it hands over.
@pytest.mark.parametrize("nR,nS,kind,route", [(1000, 20_000, "unique", "counting"), (70_000, 1 << 20, "unique", "counting"),
                                              (1_000_000, 18_000_000, "unique", "counting"),
                                              (1_000_000, 18_000_001, "unique", "one_step"),
                                              (1_300_000, 20_000_003, "hot", "not one_step"),
                                              (20_000, 300_000, "twice", "radix"), (20_000, 300_000, "sparse", "hash"),
                                              (8_400_000, 1 << 20, "sparse", "radix"),
                                              (8_400_000, 1 << 20, "unique", "dense_buckets")])
def test_join_routes(nR, nS, kind, route):
    from query_on_opencl_fpga_gb300.api import Context

    g = torch.Generator(device="cuda")
    g.manual_seed(nR + nS)
    ints = lambda lo, hi, n: torch.randint(lo, hi, (n,), generator=g, device="cuda")  # noqa: E731
    stride = 200 if kind == "sparse" else 1
    r = torch.randperm(nR, generator=g, device="cuda") * stride
    rpay, s, spay = ints(0, 1000, nR), ints(-nR, 2 * nR, nS) * stride, ints(0, 1000, nS)
    if kind == "hot":
        s[::200] = 12_345
    if kind == "twice":
        r[5] = r[6]
    table = torch.zeros(nR * stride, dtype=torch.int64, device="cuda")
    table.index_add_(0, r, rpay + (1 << 20))  # rows of the key in the high bits, the sum of their payloads below
    hit = (spay <= 299) & (s >= 0) & (s < nR * stride)
    hit[hit.clone()] = table[s[hit]] > 0
    rows = table[s[hit]]
    c = Context()
    try:
        args = [t.to(torch.int32) for t in (r, rpay, s, spay)]
        for _ in range(2):
            k, a, b = c.join_filter_sort(*args, 0, 299, cap=2 * nS)
            assert k.numel() == int((rows >> 20).sum()) and bool((k[1:] >= k[:-1]).all())
            assert int(a.sum(dtype=torch.int64)) == int((rows & 0xFFFFF).sum())
            one = rows >> 20 == 1  # every row once: the pairs themselves
            if bool(one.all()):
                assert torch.equal((k.to(torch.int64) * 1000 + b).sort().values, (s[hit] * 1000 + spay[hit]).sort().values)
                assert torch.equal(a.to(torch.int64), table[k.to(torch.int64)] & 0xFFFFF)
            got = c.join_stats()["route"]
            assert got != "one_step" if route == "not one_step" else got == route
    finally:
        c.close()


def test_join_hot_probe_key_is_not_counted_again():
    # A key with too many rows ends the counting attempt; the next join of that size
    # leaves it out until one without such a key has been seen, smaller ones do not, and
    # sparse build keys find the hash join all the same.
    from query_on_opencl_fpga_gb300.api import Context

    g = torch.Generator(device="cuda")
    g.manual_seed(14)
    ints = lambda lo, hi, n: torch.randint(lo, hi, (n,), generator=g, device="cuda")  # noqa: E731
    nR = 20_000
    r, rpay = torch.randperm(nR, generator=g, device="cuda"), ints(0, 1000, nR)
    table = torch.empty(nR, dtype=torch.int64, device="cuda")
    table[r] = rpay
    c = Context()
    try:
        for nS, hot, stride, count, route in [(300_000, True, 1, True, "radix"), (300_000, True, 1, False, "radix"),
                                              (100_000, False, 1, True, "counting"), (300_000, True, 1, False, "radix"),
                                              (300_000, False, 1000, False, "hash"), (300_000, False, 1, False, "dense_buckets"),
                                              (300_000, False, 1, True, "counting")]:
            s, spay = ints(0, 2 * nR, nS), ints(0, 1000, nS)
            if hot:
                s[::20] = 77
            args = [t.to(torch.int32) for t in (r * stride, rpay, s * stride, spay)]
            got = []
            names = launched(c, lambda: got.extend(c.join_filter_sort(*args, 0, 299, cap=nS)))
            k = got[0].to(torch.int64) // stride
            hit = (spay <= 299) & (s < nR)
            assert bool((k[1:] >= k[:-1]).all()) and torch.equal(got[1].to(torch.int64), table[k])
            assert torch.equal((k * 1000 + got[2]).sort().values, (s[hit] * 1000 + spay[hit]).sort().values)
            assert ("k_jd_count" in names) == count and c.join_stats()["route"] == route, (nS, hot, stride, names)
    finally:
        c.close()
