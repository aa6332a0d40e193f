"""G1/G2 MSM, batch and sparse MSM parity on the GPU through the C-ABI.

Mirrors crates/gpu/tests/icicle_backend.rs:65-129 (sizes, identity points
every 7th index, zero scalars every 11th, [3]G, G + (-G), repeated bases)
and crates/gpu/tests/sparse_msm_backend.rs / batch_backend.rs.  The
expected values come from the CPU oracle and the golden vectors; results
must be byte-identical.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = bytes.fromhex


def _case_inputs(oracle, seed, n, g2=False):
    size = 128 if g2 else 64
    pts = bytearray((oracle.fixed_base_g2 if g2 else oracle.fixed_base_g1)(oracle.uniform_fr(seed, n)))
    scs = bytearray(oracle.uniform_fr(seed + 1, n))
    for i in range(0, n, 7):
        pts[i * size:(i + 1) * size] = bytes(size)
    for i in range(0, n, 11):
        scs[i * 32:(i + 1) * 32] = bytes(32)
    return bytes(pts), bytes(scs)


def test_golden_g1_msm(backend, golden):
    for case in golden["msm_g1"]:
        pts = b"".join(H(p) for p in case["points"])
        scs = b"".join(H(s) for s in case["scalars"])
        assert backend.msm(pts, scs).hex() == case["expected"], case["name"]


@pytest.mark.parametrize("seed", [7, 17, 2026])
def test_g1_msm_matches_oracle_across_sizes(backend, oracle, seed):
    for n in [0, 1, 2, 17, 511, 512, 1023, 1024, 2048, 6144, 8192]:
        pts, scs = _case_inputs(oracle, seed * 100 + n, n)
        expect = oracle.msm_g1(pts, scs)
        assert backend.msm(pts, scs) == expect, f"seed={seed} n={n}"
        assert backend.msm(pts, bytes(32 * n)) == bytes(64)
        assert backend.msm(pts, scs) == expect  # repeat: workspace reuse


def test_g1_msm_every_window_width(backend, oracle):
    pts, scs = _case_inputs(oracle, 555, 3000)
    expect = oracle.msm_g1(pts, scs)
    for c in range(4, 17):
        backend.set_window(c)
        try:
            assert backend.msm(pts, scs) == expect, f"c={c}"
        finally:
            backend.set_window(0)


def test_g1_msm_one_bucket_skew(backend, oracle):
    # every scalar equal: all entries of a window land in one bucket
    g = oracle.fixed_base_g1((1).to_bytes(32, "little"))
    for n in (1024, 8192):
        pts = g * n
        scs = (3).to_bytes(32, "little") * n
        expect = oracle.fixed_base_g1((3 * n).to_bytes(32, "little"))
        assert backend.msm(pts, scs) == expect


def test_g1_msm_2_16_matches_oracle(backend, oracle):
    n = 1 << 16
    pts, tau = oracle.srs_g1(2812, n)
    scs = oracle.uniform_fr(2813, n)
    assert backend.msm(pts, scs) == oracle.msm_g1(pts, scs)


def test_g1_msm_rejects_invalid_inputs_and_stays_healthy(backend, dv, oracle):
    pts, scs = _case_inputs(oracle, 9, 64)
    bad_point = bytearray(pts)
    bad_point[64 * 5:64 * 6] = (1).to_bytes(32, "little") + (1).to_bytes(32, "little")  # (1,1) off curve
    with pytest.raises(dv.DvgpuError) as e:
        backend.msm(bytes(bad_point), scs)
    assert e.value.status == -1
    bad_scalar = bytearray(scs)
    bad_scalar[32 * 3:32 * 4] = bytes([0xFF] * 32)
    with pytest.raises(dv.DvgpuError) as e:
        backend.msm(pts, bytes(bad_scalar))
    assert e.value.status == -1
    assert backend.msm(pts, scs) == oracle.msm_g1(pts, scs)


def test_golden_g2_msm(backend, golden):
    for case in golden["msm_g2"]:
        pts = b"".join(H(p) for p in case["points"])
        scs = b"".join(H(s) for s in case["scalars"])
        assert backend.msm_g2_host(pts, scs).hex() == case["expected"], case["name"]


def test_g2_msm_matches_oracle(backend, oracle):
    for n in [0, 1, 2, 17, 300, 1024, 4096]:
        pts, scs = _case_inputs(oracle, 4000 + n, n, g2=True)
        assert backend.msm_g2_host(pts, scs) == oracle.msm_g2(pts, scs), f"n={n}"


def test_padded_batch_matches_per_set_results(backend, oracle):
    length, count = 200, 5
    pts, scs = _case_inputs(oracle, 31, length * count)
    got = backend.msm_batch_padded(pts, scs, length, count)
    for k in range(count):
        sl = slice(k * length, (k + 1) * length)
        assert got[k] == oracle.msm_g1(pts[sl.start * 64:sl.stop * 64], scs[sl.start * 32:sl.stop * 32])


def test_uneven_batch_and_shared_scalars(backend, oracle):
    sizes = [0, 1, 5, 300, 17, 2048, 3]
    pts, scs = _case_inputs(oracle, 77, sum(sizes))
    offs = np.concatenate([[0], np.cumsum(sizes)]).tolist()
    got = backend.msm_batch_uneven(pts, scs, offs)
    for k in range(len(sizes)):
        a, b = offs[k], offs[k + 1]
        assert got[k] == oracle.msm_g1(pts[a * 64:b * 64], scs[a * 32:b * 32]), f"set {k}"
    # BatchMsmRequest form: point sets sharing one scalar vector
    sets = [pts[:64 * 10], pts[64 * 10:64 * 40]]
    got = backend.msm_batch(sets, scs, offsets=[0, 5], lengths=[10, 30])
    assert got[0] == oracle.msm_g1(pts[:640], scs[:320])
    assert got[1] == oracle.msm_g1(pts[640:64 * 40], scs[160:160 + 960])


def test_uneven_batch_with_long_reduction_segments(backend, oracle):
    """128 sets of 2^15 points: the batch's window model picks c = 11, so the
    launch holds 128 x 24 x 2^10 = 3.1 M buckets and the bucket reduction
    takes 16-bucket segments (2^21 buckets or more) instead of 8.  Every set
    is compared with the oracle."""
    from concurrent.futures import ThreadPoolExecutor
    count, n = 128, 1 << 15
    base, _ = oracle.srs_g1(7700, n)
    scs = oracle.uniform_fr(7701, count * n)
    offs = [k * n for k in range(count + 1)]
    got = backend.msm_batch_uneven(base * count, scs, offs)
    with ThreadPoolExecutor(8) as pool:
        want = list(pool.map(lambda k: oracle.msm_g1(base, scs[32 * k * n:32 * (k + 1) * n]), range(count)))
    for k in range(count):
        assert got[k] == want[k], f"set {k}"


def test_golden_sparse(backend, golden):
    reqs, expect = [], []
    for case in golden["sparse_g1"]:
        bases = b"".join(H(p) for p in case["bases"])
        entries = [(e[0], H(e[1])) for e in case["entries"]]
        reqs.append((bases, entries))
        expect.append(case["expected"])
    got = backend.msm_sparse_batch(reqs)
    assert [g.hex() for g in got] == expect
    # 70 copies of 17 x (5 G): splits nothing here, one launch sequence
    seventeen = reqs[0]
    got = backend.msm_sparse_batch([seventeen] * 70)
    assert all(g.hex() == expect[0] for g in got)


def test_sparse_resident_matches_oracle(backend, oracle):
    n = 1 << 14
    bases, _ = oracle.srs_g1(65536, n)
    h = backend.register_bases(bases)
    try:
        rng = np.random.default_rng(5)
        reqs = []
        for k in (16, 256, 1, 0, 1000):
            idx = rng.choice(n, size=k, replace=False).astype(np.uint64)
            vals = oracle.uniform_fr(900 + k, k)
            reqs.append((idx, vals))
        # repeated index and zero scalar
        reqs.append((np.array([7, 7, 3], dtype=np.uint64), (9).to_bytes(32, "little") + bytes(32) + (2).to_bytes(32, "little")))
        idx_all = np.concatenate([r[0] for r in reqs]) if reqs else np.zeros(0, np.uint64)
        vals_all = b"".join(r[1] for r in reqs)
        offs = np.concatenate([[0], np.cumsum([len(r[0]) for r in reqs])])
        expect = [oracle.sparse_msm_g1(bases, idx, vals) for idx, vals in reqs]
        got = backend.sparse_msm_resident(h, idx_all, vals_all, offs)
        assert got == expect
        with pytest.raises(Exception):
            backend.sparse_msm_resident(h, np.array([n], dtype=np.uint64), bytes(32), [0, 1])
        # with a table of precomputed window multiples the same requests take
        # the one-bucket-set path (host and device forms)
        import torch
        d_idx = torch.from_numpy(idx_all.view(np.int64)).cuda()
        d_vals = torch.frombuffer(bytearray(vals_all), dtype=torch.uint8).cuda()
        torch.cuda.synchronize()
        for c in (8, 11, 0):
            backend.precompute_bases(h, c)
            assert backend.sparse_msm_resident(h, idx_all, vals_all, offs) == expect, c
            assert backend.sparse_msm_device(h, d_idx.data_ptr(), d_vals.data_ptr(), offs) == expect, c
        bad = torch.tensor([n], dtype=torch.int64, device="cuda")
        with pytest.raises(Exception):
            backend.sparse_msm_device(h, bad.data_ptr(), d_vals.data_ptr(), [0, 1])
        assert backend.sparse_msm_resident(h, idx_all, vals_all, offs) == expect  # owner still healthy
    finally:
        backend.release_bases(h)


def test_sparse_direct_small_supports(backend, oracle, dv):
    """Small sparse requests over a table of window multiples take the direct
    path (one thread per entry and window, no bucket sort): results equal the
    oracle's for repeated indices, zero scalars, empty requests and many tiny
    requests, on both sides of the size limit, and bad inputs are rejected
    with the owner left healthy."""
    import torch
    n = 1 << 12
    bases, _ = oracle.srs_g1(4096, n)
    h = backend.register_bases(bases)
    try:
        rng = np.random.default_rng(11)
        sizes = [16, 1, 0, 3, 40] + [2] * 20
        reqs = []
        for j, k in enumerate(sizes):
            idx = rng.choice(n, size=k, replace=False).astype(np.uint64)
            reqs.append((idx, oracle.uniform_fr(1200 + j, k)))
        reqs.append((np.array([5, 5, 9], dtype=np.uint64), (3).to_bytes(32, "little") + bytes(32) + (7).to_bytes(32, "little")))
        idx_all = np.concatenate([r[0] for r in reqs])
        vals_all = b"".join(r[1] for r in reqs)
        offs = np.concatenate([[0], np.cumsum([len(r[0]) for r in reqs])])
        expect = [oracle.sparse_msm_g1(bases, idx, vals) for idx, vals in reqs]
        for c in (8, 11, 0):
            backend.precompute_bases(h, c)
            assert backend.sparse_msm_resident(h, idx_all, vals_all, offs) == expect, c
            d_idx = torch.from_numpy(idx_all.view(np.int64)).cuda()
            d_vals = torch.frombuffer(bytearray(vals_all), dtype=torch.uint8).cuda()
            assert backend.sparse_msm_device(h, d_idx.data_ptr(), d_vals.data_ptr(), offs) == expect, c
        # just below and above the direct path's limit (c = 8: 32 windows, 2^16 terms)
        backend.precompute_bases(h, 8)
        for k in (512, 2048, 2049):
            idx = rng.choice(n, size=k, replace=False).astype(np.uint64)
            vals = oracle.uniform_fr(1300 + k, k)
            assert backend.sparse_msm_resident(h, idx, vals, [0, k]) == [oracle.sparse_msm_g1(bases, idx, vals)]
        bad_idx = torch.tensor([1, n], dtype=torch.int64, device="cuda")
        two = torch.frombuffer(bytearray(oracle.uniform_fr(1400, 2)), dtype=torch.uint8).cuda()
        with pytest.raises(dv.DvgpuError) as e:
            backend.sparse_msm_device(h, bad_idx.data_ptr(), two.data_ptr(), [0, 2])
        assert e.value.status == -1 and "out of range" in e.value.message
        r_mod = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
        with pytest.raises(dv.DvgpuError) as e:
            backend.sparse_msm_resident(h, np.array([1, 2], dtype=np.uint64), bytes(32) + r_mod.to_bytes(32, "little"),
                                        [0, 2])
        assert e.value.status == -1 and "non-canonical scalar at index 1" in e.value.message
        assert backend.sparse_msm_resident(h, idx_all, vals_all, offs) == expect  # owner still healthy
    finally:
        backend.release_bases(h)


def test_autotune_picks_a_window_and_results_stay_exact(dv, oracle):
    with dv.DvgpuBackend() as b:
        c, log = b.autotune_msm(4096)
        assert 4 <= c <= 20 and log["best_c"] == c and len(log["candidates"]) >= 3
        assert b.window_for(4096) == c
        pts, scs = _case_inputs(oracle, 4242, 4000)
        assert b.msm(pts, scs) == oracle.msm_g1(pts, scs)
        c2, _ = b.autotune_msm(1000, g2=True)
        pts2, scs2 = _case_inputs(oracle, 4343, 1000, g2=True)
        assert b.msm_g2_host(pts2, scs2) == oracle.msm_g2(pts2, scs2)


def test_skewed_digits_long_bucket_chains(backend, oracle):
    """Buckets that span thousands of accumulation slices (every scalar equal)
    and tiny top windows (c = 14 and 18 leave 2 bits in the top window)."""
    n = 1 << 17
    pts, _ = oracle.srs_g1(1717, n)
    same = oracle.uniform_fr(1718, 1) * n
    assert backend.msm(pts, same) == oracle.msm_g1(pts, same)
    top = b"".join((((1 << 253) + (i % 3)) % (1 << 254)).to_bytes(32, "little") for i in range(n))
    expect = oracle.msm_g1(pts, top)
    rnd = oracle.uniform_fr(1719, n)
    expect_rnd = oracle.msm_g1(pts, rnd)
    for c in (14, 18):
        backend.set_window(c)
        try:
            assert backend.msm(pts, top) == expect, f"c={c}"
            assert backend.msm(pts, rnd) == expect_rnd, f"c={c}"
        finally:
            backend.set_window(0)


def test_precomputed_resident_msm_matches_oracle(backend, oracle):
    import torch
    n = 1 << 14
    pts, _ = oracle.srs_g1(777, n)
    scs = oracle.uniform_fr(778, n)
    expect = oracle.msm_g1(pts, scs)
    expect_prefix = oracle.msm_g1(pts[:1000 * 64], scs[:1000 * 32])
    d_sc = torch.frombuffer(bytearray(scs), dtype=torch.uint8).cuda()
    torch.cuda.synchronize()
    h = backend.register_bases(pts)
    try:
        assert backend.msm_resident(h, d_sc.data_ptr(), n) == expect
        for c in (0, 8, 13, 16):
            backend.precompute_bases(h, c)
            assert backend.msm_resident(h, d_sc.data_ptr(), n) == expect, f"c={c}"
            assert backend.msm_resident(h, d_sc.data_ptr(), 1000) == expect_prefix, f"c={c} prefix"
    finally:
        backend.release_bases(h)
    pts2, scs2 = _case_inputs(oracle, 779, 2000, g2=True)
    d_sc2 = torch.frombuffer(bytearray(scs2), dtype=torch.uint8).cuda()
    torch.cuda.synchronize()
    h2 = backend.register_bases(pts2, g2=True)
    try:
        backend.precompute_bases(h2, 0)
        assert backend.msm_resident(h2, d_sc2.data_ptr(), 2000, g2=True) == oracle.msm_g2(pts2, scs2)
    finally:
        backend.release_bases(h2)


def test_resident_host_msm(backend, oracle, dv):
    """Host-scalar MSMs over registered bases with a precomputed table
    (dvgpu_bn254_msm_resident_host, the e2e call of the headline bench): the
    same result as the oracle and the plain call; a bad scalar late in the
    call is reported with its index and leaves the result untouched."""
    n = (1 << 18) + 3
    pts, _ = oracle.srs_g1(6400, n, threads=16)
    sc = oracle.uniform_fr(6401, n)
    h = backend.register_bases(pts)
    try:
        backend.precompute_bases(h, 0)
        expect = oracle.msm_g1(pts, sc, threads=16)
        assert backend.msm_resident_host(h, sc) == expect == backend.msm(pts, sc)
        m = (1 << 18) - 5
        assert backend.msm_resident_host(h, sc[:32 * m]) == oracle.msm_g1(pts[:64 * m], sc[:32 * m], threads=16)
        bad = bytearray(sc)
        bad[32 * (n - 7):32 * (n - 6)] = b"\xff" * 32
        out = ctypes.create_string_buffer(b"\x5a" * 64, 64)
        err = ctypes.create_string_buffer(256)
        rc = dv.lib().dvgpu_bn254_msm_resident_host(backend.handle, h, bytes(bad), n, out, err, 256)
        assert rc == -1 and str(n - 7).encode() in err.value and out.raw == b"\x5a" * 64
        assert backend.msm_resident_host(h, sc) == expect  # owner still healthy
    finally:
        backend.release_bases(h)


@pytest.mark.parametrize("n", [230001, 420000])
@pytest.mark.parametrize("digits", ["uniform", "one value"])
def test_g1_msm_pairwise_levels(backend, oracle, n, digits):
    """Lists long enough for one and for two pairwise levels, over 64 distinct
    bases in turn (with infinity and opposite points), so that buckets are full
    of equal, opposite and absent points; with one scalar everywhere a bucket
    spans many lanes.  Expected: the 64-term sum of the collected scalars."""
    r = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
    q = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47
    half = oracle.fixed_base_g1(oracle.uniform_fr(6101, 32))
    bases = [half[64 * i:64 * i + 64] for i in range(32)]
    bases += [p[:32] + (q - int.from_bytes(p[32:], "little")).to_bytes(32, "little") for p in bases]
    bases[5] = bases[44] = bytes(64)
    if digits == "uniform":
        sc = bytearray(oracle.uniform_fr(6102, n))
        for i in range(0, n, 11):
            sc[32 * i:32 * i + 32] = bytes(32)
        sc = bytes(sc)
    else:
        sc = oracle.uniform_fr(6103, 1) * n
    pts = (b"".join(bases) * (n // 64 + 1))[:64 * n]
    limbs = np.frombuffer(sc, dtype="<u4").reshape(n, 8).astype(np.uint64)
    sums = [sum(int(x) << (32 * k) for k, x in enumerate(limbs[i::64].sum(axis=0))) % r for i in range(64)]
    expect = oracle.msm_g1(b"".join(bases), b"".join(x.to_bytes(32, "little") for x in sums))
    assert backend.msm(pts, sc) == expect


@pytest.mark.parametrize("g2", [False, True])
@pytest.mark.parametrize("n", [1, 9, 300, 2500, 20000])
def test_msm_repeated_scalars(backend, oracle, n, g2):
    """One scalar everywhere over four bases in turn: every window is one
    bucket over all slices, merged by a quad, a warp or a block as n grows, of
    equal and opposite partial sums; digits shared among up to W threads."""
    q = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47
    size, fixed = (128, oracle.fixed_base_g2) if g2 else (64, oracle.fixed_base_g1)
    p = fixed(oracle.uniform_fr(6201, 1))
    neg = p[:size // 2] + b"".join((-int.from_bytes(p[i:i + 32], "little") % q).to_bytes(32, "little")
                                   for i in range(size // 2, size, 32))
    bases = [p, p, neg, fixed(oracle.uniform_fr(6202, 1))]
    pts = (b"".join(bases) * (n // 4 + 1))[:size * n]
    run = backend.msm_g2_host if g2 else backend.msm
    ref = oracle.msm_g2 if g2 else oracle.msm_g1
    r = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
    for s in (1, r - 1, int.from_bytes(oracle.uniform_fr(6203, 1), "little")):
        counts = [(n + 3 - i) // 4 * s % r for i in range(4)]
        expect = ref(b"".join(bases), b"".join(c.to_bytes(32, "little") for c in counts))
        assert run(pts, s.to_bytes(32, "little") * n) == expect, s


def _collected_sum(oracle, bases, sc):
    """sum sc_i bases_(i mod len(bases)) from the sums of each base's scalars."""
    m = len(bases)
    r = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
    limbs = np.frombuffer(sc, dtype="<u4").reshape(-1, 8).astype(np.uint64)
    sums = [sum(int(x) << (32 * k) for k, x in enumerate(limbs[i::m].sum(axis=0))) % r for i in range(m)]
    return oracle.msm_g1(b"".join(bases), b"".join(x.to_bytes(32, "little") for x in sums))


@pytest.mark.parametrize("c", [8, 13, 16])
def test_msm_many_long_chains(backend, oracle, c):
    """Queues of long bucket chains over a window table: some hundred of block
    length (c = 8), thousands of warp length, more than one round of the queue
    (c = 13), and with one value everywhere one a window, among short ones
    with half the scalars equal."""
    n = 40000
    srs, _ = oracle.srs_g1(6301, 64)
    bases = [srs[64 * i:64 * i + 64] for i in range(64)]
    h = backend.register_bases((srs * (n // 64 + 1))[:64 * n])
    try:
        backend.precompute_bases(h, c)
        uniform, one = oracle.uniform_fr(6302, n), oracle.uniform_fr(6303, 1)
        half = b"".join(one if i % 2 else uniform[32 * i:32 * i + 32] for i in range(n))
        for sc in (uniform, one * n, half):
            assert backend.msm_resident_host(h, sc) == _collected_sum(oracle, bases, sc)
    finally:
        backend.release_bases(h)


@pytest.mark.parametrize("value", [0, 1, 255])
def test_msm_of_nearly_empty_lists(backend, oracle, value):
    """Plans with pairwise levels and next to nothing to sum: no digit at all,
    one entry, and the levels' least list of 4096 entries (value 1) from both
    sides; empty trees, and trees of one full bucket among empty ones."""
    n = 230001
    srs, _ = oracle.srs_g1(6401, 64)
    bases = [srs[64 * i:64 * i + 64] for i in range(64)]
    pts = (srs * (n // 64 + 1))[:64 * n]
    for k in (0, 1, 4095, 4096, 4097):
        sc = bytearray(32 * n)
        for i in range(k):
            sc[32 * (53 * i % n)] = value
        assert backend.msm(pts, bytes(sc)) == _collected_sum(oracle, bases, bytes(sc)), k


@pytest.mark.parametrize("n", [1700000, 3300000])
@pytest.mark.parametrize("skewed", ["half", "all"])
def test_msm_chunks_that_do_not_fit(backend, oracle, n, skewed):
    """Lists of two and of three chunks of pairwise levels, with half or all of
    the scalars equal and all their digits the same: the chunk of that digit's
    bucket is far over its room and summed from the sorted list, the middle one
    of three is empty, and with half of them the last one goes through the
    levels, its buckets behind the others'.  Over 64 bases in turn."""
    c, digit = 16, 1 << 14
    srs, _ = oracle.srs_g1(6601, 64)
    bases = [srs[64 * i:64 * i + 64] for i in range(64)]
    one = sum(digit << (c * w) for w in range(15)).to_bytes(32, "little")
    sc = np.frombuffer(one * n, dtype=np.uint8).reshape(n, 32).copy()
    if skewed == "half":
        sc[::2] = np.frombuffer(oracle.uniform_fr(6602, (n + 1) // 2), dtype=np.uint8).reshape(-1, 32)
    sc = sc.tobytes()
    h = backend.register_bases((srs * (n // 64 + 1))[:64 * n])
    try:
        assert backend.precompute_bases(h, c) == c
        assert backend.msm_resident_host(h, sc) == _collected_sum(oracle, bases, sc)
    finally:
        backend.release_bases(h)


def test_msm_with_little_device_memory_left(dv, backend):
    """A long G1 MSM takes 1.4 GB for its pairwise levels where they are to be
    had, runs without them where not, and gives them back to a call that finds
    no other memory; the sums are the same bytes, and the owner stays healthy."""
    import torch
    n = 1 << 20
    stream = torch.cuda.current_stream().cuda_stream
    scalars, powers, points = (torch.empty(k * n, dtype=torch.uint8, device="cuda") for k in (32, 32, 64))
    values = torch.empty(32 << 23, dtype=torch.uint8, device="cuda")
    backend.random_fr_device(6501, n, scalars.data_ptr(), stream)
    backend.random_fr_device(6502, 1 << 23, values.data_ptr(), stream)
    backend.fr_powers_device(values.data_ptr(), n, powers.data_ptr(), stream)
    backend.fixed_base_device(powers.data_ptr(), n, False, points.data_ptr(), stream)
    torch.cuda.synchronize()

    def leave(nbytes):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda")

    def msm(b):
        return b.msm_device(points.data_ptr(), scalars.data_ptr(), n, stream=stream)

    expect = msm(backend)
    with dv.DvgpuBackend() as b:
        held = leave(900 << 20)
        assert msm(b) == expect  # without levels
        del held
        torch.cuda.empty_cache()
        before = torch.cuda.mem_get_info()[0]
        assert msm(b) == expect  # with them
        assert before - torch.cuda.mem_get_info()[0] > 1 << 30
        out = torch.empty_like(values)
        held = leave(200 << 20)
        b.ntt_device(values.data_ptr(), 1 << 23, 0, out.data_ptr(), stream)  # 0.4 GB of its own
        assert msm(b) == expect
        del held
        ref = torch.empty_like(values)
        backend.ntt_device(values.data_ptr(), 1 << 23, 0, ref.data_ptr(), stream)
        assert torch.equal(out, ref)
    del out, ref, values, points, powers, scalars
    torch.cuda.empty_cache()


@pytest.mark.parametrize("c", [8, 13])
def test_sparse_direct_block_edges(backend, oracle, c):
    """One request around a block's 64 terms and around the direct path's
    16384 terms, with equal bases, for an even and an odd window width."""
    n = 1024
    bases, _ = oracle.srs_g1(4097, n)
    h = backend.register_bases(bases)
    try:
        backend.precompute_bases(h, c)
        rng = np.random.default_rng(12)
        windows = -(-255 // c)
        for k in (1, 2, 3, 64 // windows, 64 // windows + 1, 16384 // windows, 16384 // windows + 1):
            idx = rng.integers(0, n, size=k).astype(np.uint64)
            vals = oracle.uniform_fr(1500 + k, k)
            assert backend.sparse_msm_resident(h, idx, vals, [0, k]) == [oracle.sparse_msm_g1(bases, idx, vals)], k
    finally:
        backend.release_bases(h)


@pytest.mark.parametrize("c, requests, entries, direct",
                         [(8, 300, 4, True), (8, 70, 16, True), (8, 1100, 1, True), (8, 2, 900, False),
                          (8, 40, 75, False), (13, 300, 4, True), (13, 70, 16, True), (13, 1100, 1, True),
                          (13, 40, 75, True), (13, 2, 900, False)])
def test_sparse_many_requests(dv, backend, oracle, c, requests, entries, direct):
    """Calls of many requests between 16384 and 65536 terms stay one launch
    (blocks of quads for the shortest requests, of threads for the others), with
    empty requests, repeated indices and error words; few requests and
    more terms take the buckets."""
    n, r = 256, 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
    bases = oracle.fixed_base_g1(oracle.uniform_fr(8300, n))
    sizes = [0 if j % 17 == 5 else entries + j % 2 for j in range(requests)]
    offs = [0] + list(np.cumsum(sizes))
    k = int(offs[-1])
    idx = (np.arange(k, dtype=np.uint64) * 5 + 3) % n
    vals = bytearray(oracle.uniform_fr(8301, k))
    vals[64:96] = bytes(32)
    vals[96:128] = (r - 1).to_bytes(32, "little")
    vals = bytes(vals)
    expect = [oracle.sparse_msm_g1(bases, idx[a:b], vals[32 * a:32 * b]) if b > a else bytes(64)
              for a, b in zip(offs, offs[1:])]
    h = backend.register_bases(bases)
    try:
        backend.precompute_bases(h, c)
        before = backend.launch_count()
        assert backend.sparse_msm_resident(h, idx, vals, offs) == expect
        assert (backend.launch_count() - before == 1) == direct
        for bad in ([k - 1], [k // 2, k - 1], [0]):
            broken = bytearray(vals)
            for at in bad:
                broken[32 * at:32 * at + 32] = r.to_bytes(32, "little")
            with pytest.raises(dv.DvgpuError) as e:
                backend.sparse_msm_resident(h, idx, bytes(broken), offs)
            assert e.value.status == -1 and f"non-canonical scalar at index {min(bad)}" in e.value.message
        assert backend.sparse_msm_resident(h, idx, vals, offs) == expect
    finally:
        backend.release_bases(h)


@pytest.mark.parametrize("n", [1, 300, 5000])
@pytest.mark.parametrize("g2", [False, True])
def test_msm_error_words_reach_the_host(dv, backend, oracle, n, g2):
    """The last reduction kernel leaves the sums and both error words in host
    memory: a bad point, a bad scalar, both (the scalar is named), and good
    calls in between."""
    size = 128 if g2 else 64
    call = backend.msm_g2_host if g2 else backend.msm
    pts, scs = _case_inputs(oracle, 8100 + n, n, g2)
    expect = (oracle.msm_g2 if g2 else oracle.msm_g1)(pts, scs)
    r = (0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001).to_bytes(32, "little")
    assert call(pts, scs) == expect
    for at in sorted({0, n - 1}):
        bad_pts = pts[:at * size] + b"\x01" + bytes(size - 1) + pts[(at + 1) * size:]
        bad_scs = scs[:32 * at] + r + scs[32 * at + 32:]
        for p, s, message in ((bad_pts, scs, f"invalid point at index {at}"),
                              (pts, bad_scs, f"non-canonical scalar at index {at}"),
                              (bad_pts, bad_scs, f"non-canonical scalar at index {at}")):
            with pytest.raises(dv.DvgpuError) as e:
                call(p, s)
            assert e.value.status == -1 and message in e.value.message
            assert call(pts, scs) == expect


def test_sparse_direct_error_words_of_several_requests(dv, backend, oracle):
    """Each request's last block hands its error words to the host: the lowest
    bad scalar of all requests is named, empty requests give infinity, and the
    next call is good."""
    n, offs = 64, [0, 0, 3, 3, 12, 30, 30]
    bases = oracle.fixed_base_g1(oracle.uniform_fr(8200, n))
    idx = (np.arange(offs[-1], dtype=np.uint64) * 7) % n
    vals = oracle.uniform_fr(8201, offs[-1])
    r = (0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001).to_bytes(32, "little")
    expect = [oracle.sparse_msm_g1(bases, idx[a:b], vals[32 * a:32 * b]) if b > a else bytes(64)
              for a, b in zip(offs, offs[1:])]
    h = backend.register_bases(bases)
    try:
        backend.precompute_bases(h, 8)
        assert backend.sparse_msm_resident(h, idx, vals, offs) == expect
        for bad in ([29], [2, 29], [11, 12], [0]):
            broken = bytearray(vals)
            for at in bad:
                broken[32 * at:32 * at + 32] = r
            with pytest.raises(dv.DvgpuError) as e:
                backend.sparse_msm_resident(h, idx, bytes(broken), offs)
            assert e.value.status == -1 and f"non-canonical scalar at index {min(bad)}" in e.value.message
            assert backend.sparse_msm_resident(h, idx, vals, offs) == expect
    finally:
        backend.release_bases(h)
