"""Poly library on the GPU through the C ABI, bit-exact against the oracle / big integers."""
import numpy as np
import pytest

from conftest import lookup_case
import torch

pytestmark = pytest.mark.gpu

M = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
R = 1 << 256


def dev(zk, a):
    return zk.ScalarArray.from_numpy(a)


def scal(zk, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.uint64).view(np.int32).reshape(1, 8).copy()).cuda()


def ints(orc, a):
    """canonical integers of Montgomery-form limbs"""
    return [orc.limbs_to_int(x) * pow(R, -1, M) % M for x in a]


@pytest.mark.parametrize("la,lb", [(1000, 1000), (1000, 300), (300, 1000)])
def test_binary_ops_unequal_lengths(zk, orc, la, lb):
    a, b = orc.gen_fr(1, la), orc.gen_fr(2, lb)
    up, lo = max(la, lb), min(la, lb)
    for name, fn in (("add", zk.poly.poly_add), ("sub", zk.poly.poly_sub), ("mul", zk.poly.poly_mul)):
        r = zk.ScalarArray.zeros(up)
        fn(r, dev(zk, a), dev(zk, b))
        got = r.numpy_u64()
        head = {"add": orc.vec_add, "sub": orc.vec_sub, "mul": orc.vec_mul}[name](a[:lo], b[:lo])
        assert np.array_equal(got[:lo], head), name
        longer = a if la >= lb else b
        tail = longer[lo:]
        if name == "sub" and la < lb:
            tail = np.stack([orc.neg(x) for x in tail])
        assert np.array_equal(got[lo:], tail), name


def test_binary_ops_rotated(zk, orc):
    n = 512
    a, b = orc.gen_fr(3, n), orc.gen_fr(4, n)
    xa, xb = dev(zk, a), dev(zk, b)
    xa.rotate(5)
    xb.rotate(n - 7)
    r = zk.ScalarArray.zeros(n)
    r.rotate(11)
    zk.poly.poly_mul(r, xa, xb)
    va = orc.poly_ptr_view(a, n, rotate=5)
    vb = orc.poly_ptr_view(b, n, rotate=n - 7)
    assert np.array_equal(r.numpy_u64(), orc.vec_mul(va, vb))


def test_fills(zk, orc):
    t = dev(zk, orc.gen_fr(5, 100))
    zk.poly.poly_one_lagrange(t)
    assert np.array_equal(t.numpy_u64(), np.repeat(orc.one()[None], 100, 0))
    zk.poly.poly_one_coef(t)
    got = t.numpy_u64()
    assert np.array_equal(got[0], orc.one()) and not got[1:].any()
    zk.poly.poly_zero(t)
    assert not t.numpy_u64().any()


@pytest.mark.parametrize("n", [1, 5, 64, 65, 512, 513, 4097, 32769, 1 << 20])
def test_poly_eval(zk, orc, n):
    a = orc.gen_fr(6, n)
    x = orc.gen_fr(7, 1)[0]
    res = torch.zeros((1, 8), dtype=torch.int32, device="cuda")
    zk.poly.poly_eval(dev(zk, a), scal(zk, x), res)
    assert np.array_equal(res.cpu().numpy().view(np.uint64)[0], orc.eval_poly(a, x))


@pytest.mark.parametrize("n", [1, 63, 64, 65, 512, 513, 5000, 32769, 1 << 20])
def test_batched_invert(zk, orc, n):
    a = orc.gen_fr(8, n)
    if n > 10:
        a[3] = 0
        a[n - 1] = 0
        a[64:128 if n > 128 else n] = 0  # a whole zero chunk
    t = dev(zk, a)
    zk.poly.batched_invert(t)
    assert np.array_equal(t.numpy_u64(), orc.batch_invert(a))


@pytest.mark.parametrize("n", [1, 64, 65, 512, 513, 4100, 32769, 70000])
def test_scan_mul(zk, orc, n):
    a = orc.gen_fr(9, n)
    t = dev(zk, a)
    zk.poly.scan_mul(t)
    got = ints(orc, t.numpy_u64())
    acc, expect = 1, []
    for v in ints(orc, a):
        acc = acc * v % M
        expect.append(acc)
    assert got == expect


@pytest.mark.parametrize("log_n", [0, 1, 4, 6, 7, 9, 10, 12, 15, 16])
def test_kate_division(zk, orc, log_n):
    n = 1 << log_n
    p = orc.gen_fr(10, n)
    b = orc.gen_fr(11, 1)[0]
    q = zk.ScalarArray.zeros(n)
    xp = dev(zk, p)
    xp.rotate(2 % n if n > 1 else 0)
    zk.poly.kate_division(xp, scal(zk, b), q)
    pv = ints(orc, orc.poly_ptr_view(p, n, rotate=2 % n if n > 1 else 0))
    bi = ints(orc, [b])[0]
    expect = [0] * n
    for i in range(n - 2, -1, -1):
        expect[i] = (pv[i + 1] + bi * expect[i + 1]) % M
    assert ints(orc, q.numpy_u64()) == expect


def test_scalar_inv_and_pow(zk, orc):
    x = orc.gen_fr(12, 1)[0]
    t = scal(zk, x)
    zk.poly.inv_scalar(t)
    assert np.array_equal(t.cpu().numpy().view(np.uint64)[0], orc.inv(x))
    t = scal(zk, x)
    zk.poly.scalar_pow(t, 12345678901)
    assert np.array_equal(t.cpu().numpy().view(np.uint64)[0], orc.pow_(x, 12345678901))
    z = scal(zk, np.zeros(4, dtype=np.uint64))
    zk.poly.inv_scalar(z)
    assert not z.cpu().numpy().any()


def test_scalar_inv_edge_words(zk, orc):
    """The inversion (batched binary-GCD steps, fixed 17 x 30 iterations) on the stored words
    it inverts: small values, values next to m and to powers of two, R mod m, R^2 mod m, and
    seeded values; each equals the oracle's Montgomery inverse."""
    words = [1, 2, 3, 5, M - 1, M - 2, (M - 1) // 2, (M + 1) // 2, 1 << 253, (1 << 254) % M, (1 << 128) + 1,
             (1 << 32) - 1, R % M, R * R % M, M - (1 << 200)]
    vals = [orc.int_to_limbs(w) for w in words] + list(orc.gen_fr(13, 48))
    for x in vals:
        t = scal(zk, x)
        zk.poly.inv_scalar(t)
        assert np.array_equal(t.cpu().numpy().view(np.uint64)[0], orc.inv(x)), orc.limbs_to_int(x)


def test_square_matches_mul(zk, orc):
    """The dedicated Montgomery squaring equals a * a bit for bit (edge values included)."""
    n = 20000
    a = orc.gen_fr(13, n)
    M_limbs = orc.int_to_limbs(M - 1)
    a[0] = 0
    a[1] = M_limbs                      # m - 1
    a[2] = orc.int_to_limbs(1)
    a[3] = orc.int_to_limbs((1 << 253) + 12345)
    r = zk.ScalarArray.zeros(n)
    zk.poly.poly_square(r, dev(zk, a))
    assert np.array_equal(r.numpy_u64(), orc.vec_mul(a, a))


@pytest.mark.parametrize("log_n", [6, 10, 14])
def test_permute_matches_oracle(zk, orc, log_n):
    n = 1 << log_n
    usable = n - min(25, n // 4)
    inp, table = lookup_case(zk, n, usable, 70 + log_n)
    ri, rt = zk.ScalarArray.alloc(usable), zk.ScalarArray.alloc(usable)
    zk.poly.permute(inp, table, usable, ri, rt)
    ei, et = orc.permute(inp.numpy_u64(), table.numpy_u64(), usable)
    assert np.array_equal(ri.numpy_u64(), ei)
    assert np.array_equal(rt.numpy_u64(), et)


@pytest.mark.parametrize("n", [2, 255, 511, 512, 1023, 1025, 75776, 75777, 606209])
def test_sweeps_at_chunk_edges(zk, orc, n):
    """Lengths around one CTA of two-element chunks, and where the chunk length changes."""
    a = orc.gen_fr(15, n)
    x = orc.gen_fr(16, 1)[0]
    res = torch.zeros((1, 8), dtype=torch.int32, device="cuda")
    zk.poly.poly_eval(dev(zk, a), scal(zk, x), res)
    assert np.array_equal(res.cpu().numpy().view(np.uint64)[0], orc.eval_poly(a, x))
    z = a.copy()
    z[::7] = 0
    t = dev(zk, z)
    zk.poly.batched_invert(t)
    assert np.array_equal(t.numpy_u64(), orc.batch_invert(z))
    t = dev(zk, a)
    zk.poly.scan_mul(t)
    acc, expect = 1, []
    for v in ints(orc, a):
        acc = acc * v % M
        expect.append(acc)
    assert ints(orc, t.numpy_u64()) == expect


@pytest.mark.parametrize("log_n", [8, 11, 13, 17, 20])
def test_kate_division_chunk_edges(zk, orc, log_n):
    """q (X - b) + p(b) = p: checked as q[i - 1] - b q[i] = p[i] for every i, with q[n - 1] = 0."""
    n = 1 << log_n
    p, b = orc.gen_fr(17, n), orc.gen_fr(18, 1)[0]
    q = zk.ScalarArray.zeros(n)
    zk.poly.kate_division(dev(zk, p), scal(zk, b), q)
    got = q.numpy_u64()
    assert not got[n - 1].any()
    bq = orc.vec_mul(got, np.repeat(b[None], n, axis=0))
    assert np.array_equal(orc.vec_sub(got[:-1], bq[1:]), p[1:])


@pytest.mark.parametrize("n", [1, 2, 31, 2047, 2048, 2049, 9000])
@pytest.mark.parametrize("kind", ["random", "small", "signed", "clash"])
def test_permute_key_shapes(zk, orc, n, kind):
    """Sort keys of every shape the word choice meets: random field elements, a small range, small
    values and their negatives (one word cannot tell them apart), and values that agree in their
    top bits in runs longer than the insertion step takes."""
    rng = np.random.default_rng(n)
    if kind == "random":
        vals = [int.from_bytes(rng.bytes(32), "little") % M for _ in range(n)]
    elif kind == "small":
        vals = [int(v) for v in rng.integers(0, max(2, n // 3), n)]
    elif kind == "signed":
        vals = [int(v) if s else (M - 1 - int(v)) for v, s in zip(rng.integers(0, n + 1, n), rng.integers(0, 2, n))]
    else:
        tops = [int.from_bytes(rng.bytes(3), "little") << 220 for _ in range(3)]
        vals = [tops[int(t)] | (int(m) << 100) | int(v)
                for t, m, v in zip(rng.integers(0, 3, n), rng.integers(0, 4, n), rng.integers(0, 50, n))]
    table = np.stack([orc.to_mont(orc.int_to_limbs(v % M)) for v in vals])
    usable = max(1, n - 3)
    inp = table[rng.integers(0, usable, n)]
    ri, rt = zk.ScalarArray.alloc(usable), zk.ScalarArray.alloc(usable)
    zk.poly.permute(dev(zk, inp), dev(zk, table), usable, ri, rt)
    ei, et = orc.permute(inp, table, usable)
    assert np.array_equal(ri.numpy_u64(), ei)
    assert np.array_equal(rt.numpy_u64(), et)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 16, 17, 63, 64, 65, 66, 127, 129, 513])
def test_sweeps_of_few_chunks(zk, orc, n):
    """One CTA whose scans stop at the chunks there are: one chunk, part of a warp, one more than a
    warp's, several warps; zeros at both ends for the inversion."""
    a = orc.gen_fr(19, n)
    x = orc.gen_fr(20, 1)[0]
    res = torch.zeros((1, 8), dtype=torch.int32, device="cuda")
    zk.poly.poly_eval(dev(zk, a), scal(zk, x), res)
    assert np.array_equal(res.cpu().numpy().view(np.uint64)[0], orc.eval_poly(a, x))
    for zeros in ([], [0], [n - 1], list(range(n))):
        z = a.copy()
        z[zeros] = 0
        t = dev(zk, z)
        zk.poly.batched_invert(t)
        assert np.array_equal(t.numpy_u64(), orc.batch_invert(z)), zeros
    t = dev(zk, a)
    zk.poly.scan_mul(t)
    acc, expect = 1, []
    for v in ints(orc, a):
        acc = acc * v % M
        expect.append(acc)
    assert ints(orc, t.numpy_u64()) == expect
    if n & (n - 1) == 0:
        q = zk.ScalarArray.zeros(n)
        zk.poly.kate_division(dev(zk, a), scal(zk, x), q)
        b, p, acc, expect = ints(orc, x[None])[0], ints(orc, a), 0, []
        for i in reversed(range(n)):
            acc = (acc * b + (p[i + 1] if i + 1 < n else 0)) % M
            expect.append(acc)
        assert ints(orc, q.numpy_u64()) == expect[::-1]


def test_empty_polynomial_through_the_size_query(zk):
    """Length 0 with buffers of exactly the queried sizes: the query asks for some bytes (a buffer of
    none is a null pointer, which would be a query again), and the evaluation writes zero."""
    import ctypes
    lib = zk.poly._lib()
    stream = torch.cuda.current_stream().cuda_stream
    empty = zk.native.PolyPtr(None, 0, 0, 0, 0)
    x = torch.ones(8, dtype=torch.int32, device="cuda")
    res = torch.full((8,), 7, dtype=torch.int32, device="cuda")
    for fn, args in ((lib.poly_eval, (res.data_ptr(), x.data_ptr())), (lib.batched_invert, ()), (lib.scan_mul, ())):
        size = ctypes.c_ulong(0)
        assert fn(None, ctypes.byref(size), empty, *args, stream) == 0
        temp = torch.empty(size.value, dtype=torch.uint8, device="cuda")
        assert size.value > 0 and fn(temp.data_ptr(), ctypes.byref(size), empty, *args, stream) == 0
    assert not res.any()


def permute_expected(vals, table):
    """canonical integers: the input sorted; the table's arrangement (see oracle.permute)"""
    a, left = sorted(vals), {}
    for v in table:
        left[v] = left.get(v, 0) + 1
    out = list(a)
    repeated = []
    for i, v in enumerate(a):
        if i == 0 or v != a[i - 1]:
            left[v] -= 1
        else:
            repeated.append(i)
    for i, v in zip(repeated, sorted(v for v, c in left.items() for _ in range(c))):
        out[i] = v
    return a, out


def mont_words(vals):
    return np.frombuffer(b"".join((v * R % M).to_bytes(32, "little") for v in vals), dtype=np.uint64).reshape(-1, 4)


def permute_table(kind, n, rng):
    if kind == "random":
        return [int.from_bytes(rng.bytes(32), "little") % M for _ in range(n)]
    if kind == "signed":  # a range around zero
        return [(int(v) - n // 2) % M for v in rng.permutation(n)]
    if kind == "wide":  # 62-bit magnitudes of either sign
        return [int(v) * int(s) % M for v, s in zip(rng.integers(0, 1 << 62, n), rng.choice([-1, 1], n))]
    if kind == "clash":  # three top words, a few middle ones, values below
        tops = [int.from_bytes(rng.bytes(3), "little") << 220 for _ in range(3)]
        return [tops[int(t)] | (int(m) << 100) | int(v)
                for t, m, v in zip(rng.integers(0, 3, n), rng.integers(0, 4, n), rng.integers(0, 1 << 20, n))]
    vals = permute_table("random", n, rng)
    if kind == "some":  # small values among random ones
        vals[: n // 8] = range(n // 8)
    if kind == "nested":  # long runs under one top word, under two, under three, ...
        for w in range(7):
            part = range(w * n // 16, (w + 1) * n // 16)
            for i in part:
                vals[i] = (0x1234567 << 228 | vals[i] >> (26 + 32 * w)) % M
    if kind == "repeated":  # few values, many rows of each
        vals = [vals[int(i)] for i in rng.integers(0, max(1, n // 40), n)]
    return [vals[int(i)] for i in rng.permutation(n)]


@pytest.mark.parametrize("kind", ["random", "signed", "wide", "clash", "some", "nested", "repeated"])
@pytest.mark.parametrize("n", [40, 1024, 2048, 2049, 65536, 65537, 152000])
def test_permute_sort_rounds(zk, n, kind):
    """Every way the sort settles ties (none, insertion, one or more further words, all words), on one CTA
    an array, several, and all of them, with the 24-bit and the 32-bit word."""
    rng = np.random.default_rng(n)
    table = permute_table(kind, n, rng)
    vals = [table[int(i)] for i in rng.integers(0, n, n)]
    ri, rt = zk.ScalarArray.alloc(n), zk.ScalarArray.alloc(n)
    zk.poly.permute(dev(zk, mont_words(vals)), dev(zk, mont_words(table)), n, ri, rt)
    ei, et = permute_expected(vals, table)
    assert np.array_equal(ri.numpy_u64(), mont_words(ei))
    assert np.array_equal(rt.numpy_u64(), mont_words(et))


@pytest.mark.parametrize("kind", ["random", "signed", "some"])
def test_permute_2_20_rows(zk, kind):
    test_permute_sort_rounds(zk, 1 << 20, kind)


def permute_case(zk, n, kind="some"):
    rng = np.random.default_rng(n)
    table = permute_table(kind, n, rng)
    vals = [table[int(i)] for i in rng.integers(0, n, n)]
    ei, et = permute_expected(vals, table)
    return (dev(zk, mont_words(vals)), dev(zk, mont_words(table)), zk.ScalarArray.alloc(n), zk.ScalarArray.alloc(n),
            mont_words(ei), mont_words(et))


def test_permute_captured_and_beside_other_work(zk):
    """The cooperative launch in a stream capture, replayed on other values, and while another stream
    keeps the GPU busy with transforms."""
    n = 30000
    inp, table, ri, rt, ei, et = permute_case(zk, n)
    other = permute_case(zk, n, "signed")
    stream, busy = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        zk.poly.permute(inp, table, n, ri, rt)
    graph.replay()
    assert np.array_equal(ri.numpy_u64(), ei) and np.array_equal(rt.numpy_u64(), et)
    inp.values.copy_(other[0].values)
    table.values.copy_(other[1].values)
    graph.replay()
    assert np.array_equal(ri.numpy_u64(), other[4]) and np.array_equal(rt.numpy_u64(), other[5])
    x = zk.ScalarArray(zk.gen.fr(3, 1 << 20))
    zk.ntt.ntt(x)
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        for _ in range(20):
            zk.ntt.ntt(x)
    with torch.cuda.stream(stream):
        zk.poly.permute(other[0], other[1], n, other[2], other[3])
    torch.cuda.synchronize()
    assert np.array_equal(other[2].numpy_u64(), other[4]) and np.array_equal(other[3].numpy_u64(), other[5])


def test_permute_on_a_partition(zk):
    """A stream of a green context with a few SMs: the grid is cut to what is resident there at once."""
    driver = pytest.importorskip("cuda.bindings.driver")
    import ctypes

    def ok(r):
        if int(r[0]) != 0:
            pytest.skip(f"green contexts: {r[0]}")
        return r[1] if len(r) == 2 else r[1:]
    torch.zeros(1, device="cuda")
    device = ok(driver.cuDeviceGet(0))
    sms = ok(driver.cuDeviceGetDevResource(device, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups = ok(driver.cuDevSmResourceSplitByCount(1, sms, 0, 8))[0]
    desc = ok(driver.cuDevResourceGenerateDesc([groups[0]], 1))
    green = ok(driver.cuGreenCtxCreate(desc, device, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(driver.cuGreenCtxStreamCreate(green, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    try:
        n = 65536
        ctas = ctypes.c_uint(0)
        assert zk.poly._lib().zkp_permute_ctas(n, None, ctypes.byref(ctas)) == 0 and ctas.value == 64
        assert zk.poly._lib().zkp_permute_ctas(n, int(stream), ctypes.byref(ctas)) == 0
        assert 2 <= ctas.value <= groups[0].sm.smCount < 64  # no launch unless all its CTAs fit
        inp, table, ri, rt, ei, et = permute_case(zk, n)
        torch.cuda.synchronize()
        zk.poly.permute(inp, table, n, ri, rt, stream=torch.cuda.ExternalStream(int(stream)))
        ok(driver.cuStreamSynchronize(stream) + (None,))
        assert np.array_equal(ri.numpy_u64(), ei) and np.array_equal(rt.numpy_u64(), et)
    finally:
        driver.cuStreamDestroy(stream)
        driver.cuGreenCtxDestroy(green)
