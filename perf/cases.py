"""Workloads of the framework's main path, through its public entry points.

Each case is one thing a prover built on this framework does over and over: a transform, a coset
extension, a multi-scalar multiplication over resident bases, a round of polynomial kernels, or a
handful of prover requests put through the serving loop.  All results are exact integers (canonical
Montgomery-form field elements and affine points), so outputs are compared bit for bit.
"""
import importlib
import math

import numpy as np
import torch

zk = importlib.import_module("zkpoly-compiler_b200")

FR = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
FQ = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47
R = 1 << 256
SHIFT = 7  # the coset shift of the extended domain (the multiplicative generator of Fr)
PRODUCT = 256.0  # operations of one Montgomery product: 64 + 64 multiply-adds of 32-bit words


def listed():
    return [
        # one small vector: what a call costs when there is hardly any work in it
        {"name": "ntt_1k", "kind": "ntt", "log_n": 10, "inverse": False, "abi": False},
        # a column of an ordinary circuit back to coefficients
        {"name": "intt_64k", "kind": "ntt", "log_n": 16, "inverse": True, "abi": False},
        # the drop-in symbol with the Montgomery root table alone, as the original host code calls it
        {"name": "ssip_ntt_1m", "kind": "ntt", "log_n": 20, "inverse": False, "abi": True},
        # the largest transform of the benchmark
        {"name": "ntt_16m", "kind": "ntt", "log_n": 24, "inverse": False, "abi": False},
        # coefficients to evaluations on the four times larger coset, before a quotient
        {"name": "lde_256k_to_1m", "kind": "lde", "log_n": 18, "ext": 2},
        # a commitment of a small circuit: almost all latency
        {"name": "msm_4k", "kind": "msm", "n": 4096, "batch": 1, "tables": True},
        # the four commitments of one prover request in one batch
        {"name": "msm_4x64k", "kind": "msm", "n": 65536, "batch": 4, "tables": True},
        # the largest commitment of the benchmark, over precomputed tables
        {"name": "msm_4m", "kind": "msm", "n": 1 << 22, "batch": 1, "tables": True},
        # bases without precomputed tables, and a length that is no power of two
        {"name": "msm_plain_1000003", "kind": "msm", "n": 1000003, "batch": 1, "tables": False},
        # lookup permutation, grand product, division and evaluation over a short ragged column
        {"name": "poly_4095", "kind": "poly", "n": 4095},
        # the same round over a large column
        {"name": "poly_1m", "kind": "poly", "n": 1 << 20},
        # eight requests of uneven sizes that arrive together at the serving loop
        {"name": "serve_8", "kind": "serve", "requests": 8, "k_lo": 14, "k_hi": 17, "mix": 5},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ntt", "ntt", "lde", "msm", "msm", "poly", "serve"])
    if kind == "ntt":
        return {"kind": kind, "log_n": rng.randint(10, 24), "inverse": rng.random() < 0.5, "abi": rng.random() < 0.3}
    if kind == "lde":
        ext = rng.randint(1, 3)
        return {"kind": kind, "log_n": rng.randint(10, 23 - ext), "ext": ext}
    if kind == "msm":
        batch = rng.choice([1, 1, 2, 3, 4])
        tables = rng.random() < 0.7
        top = (1 << 22) // batch if tables else (1 << 21) // batch
        return {"kind": kind, "n": _log_uniform(rng, 4096, top), "batch": batch, "tables": tables}
    if kind == "poly":
        return {"kind": kind, "n": _log_uniform(rng, 4000, 1 << 20)}
    lo = rng.randint(14, 16)
    return {"kind": kind, "requests": rng.randint(2, 10), "k_lo": lo, "k_hi": min(lo + rng.randint(0, 3), 17),
            "mix": rng.randint(0, 1000)}


# ------------------------------------------------------------------ inputs
def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    return g


def _fr(seed, salt, n):
    """(n, 8) int32: uniform below the modulus but for its last sliver (the top word is drawn below
    the modulus's top word)."""
    g = _generator(seed, salt)
    w = torch.randint(-(1 << 31), 1 << 31, (n, 8), generator=g, device="cuda", dtype=torch.int64)
    w[:, 7] = torch.randint(0, FR >> 224, (n,), generator=g, device="cuda", dtype=torch.int64)
    return w.to(torch.int32)


def _table_column(seed, n):
    """A lookup table of n distinct random values and a column of n values out of its first n - 5
    rows (the last rows of a column are blinding rows and are not permuted)."""
    table = _fr(seed, 21, n)
    pick = torch.randint(0, max(1, n - 5), (n,), generator=_generator(seed, 22), device="cuda")
    return table[pick].contiguous(), table


def _request_sizes(case):
    rng = np.random.default_rng(case["mix"])
    return [int(k) for k in rng.integers(case["k_lo"], case["k_hi"] + 1, case["requests"])]


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "ntt":
        log_n, inverse = case["log_n"], case["inverse"]
        s["x"] = zk.ScalarArray(_fr(seed, 1, 1 << log_n))
        s["twiddle"] = zk.ntt.twiddle_table(log_n, inverse)
        s["n_inv"] = zk.ntt.n_inv(log_n)
        if not case["abi"]:
            zk.ntt.shoup_table(log_n, inverse)  # the table that ntt() and intt() keep for a size
    elif kind == "lde":
        log_out = case["log_n"] + case["ext"]
        s["coef"] = zk.ScalarArray(_fr(seed, 1, 1 << case["log_n"]))
        s["out"] = zk.ScalarArray.alloc(1 << log_out)
        zk.ntt.twiddle_table(log_out)
        zk.ntt.shoup_table(log_out)
    elif kind == "msm":
        n, batch = case["n"], case["batch"]
        s["points"] = zk.gen.points(seed, n)
        s["scalars"] = [_fr(seed, 1 + i, n) for i in range(batch)]
        s["results"] = [torch.zeros(16, dtype=torch.int32, device="cuda") for _ in range(batch)]
        if case["tables"]:
            window, n_tables = zk.tuner.msm_resident_config(n)
        else:
            window, n_tables = zk.tuner.msm_window(n), 1
        s["bases"] = zk.msm.ResidentBases(s["points"], window=window, n_tables=n_tables)
        if batch == 1:
            s["workspace"] = s["bases"].workspace()
        else:
            s["batch"] = zk.msm.MsmBatch([
                {"points": s["bases"].tables, "n_tables": n_tables, "scalars": sc, "n": n,
                 "window": s["bases"].window, "result": r} for sc, r in zip(s["scalars"], s["results"])])
    elif kind == "poly":
        n = case["n"]
        k = n.bit_length() - 1
        s["p"] = zk.ScalarArray(_fr(seed, 1, n))
        s["divisor"], s["point"] = _fr(seed, 2, 1), _fr(seed, 3, 1)
        s["value"] = torch.zeros((1, 8), dtype=torch.int32, device="cuda")
        s["dividend"] = zk.ScalarArray(_fr(seed, 4, 1 << k))
        s["quotient"] = zk.ScalarArray.alloc(1 << k)
        s["inverted"] = zk.ScalarArray(_fr(seed, 5, n))
        s["scanned"] = zk.ScalarArray(_fr(seed, 6, n))
        column, table = _table_column(seed, n)
        s["column"], s["table"] = zk.ScalarArray(column), zk.ScalarArray(table)
        s["perm"] = [zk.ScalarArray.zeros(n - 5), zk.ScalarArray.zeros(n - 5)]
    else:
        sizes = _request_sizes(case)
        s["requests"] = [(k, seed * 4096 + i) for i, k in enumerate(sizes)]
        s["points"] = zk.gen.points(2, 1 << case["k_hi"])
        s["sets"] = zk.serving.resident_sets(s["points"], case["k_lo"], case["k_hi"])
        s["server"] = zk.serving.Server(s["sets"], 8 << 30, max_inflight=8, min_k=case["k_lo"], max_k=case["k_hi"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "ntt":
        case, x = s["case"], s["x"]
        if case["abi"] and case["inverse"]:
            zk.ntt.ntt_ex(x, s["twiddle"], None, s["n_inv"])
        elif case["abi"]:
            zk.ntt.ssip_ntt(x, s["twiddle"])
        elif case["inverse"]:
            zk.ntt.intt(x)
        else:
            zk.ntt.ntt(x)
        return x.values
    if kind == "lde":
        zk.ntt.coset_ntt(s["out"], s["coef"], SHIFT)
        return s["out"].values
    if kind == "msm":
        if "batch" in s:
            s["batch"].run()
        else:
            s["bases"].msm(s["scalars"][0], s["results"][0], s["workspace"])
        return s["results"]
    if kind == "poly":
        n = s["case"]["n"]
        zk.poly.permute(s["column"], s["table"], n - 5, s["perm"][0], s["perm"][1])
        zk.poly.batched_invert(s["inverted"])
        zk.poly.scan_mul(s["scanned"])
        zk.poly.kate_division(s["dividend"], s["divisor"], s["quotient"])
        zk.poly.poly_eval(s["p"], s["point"], s["value"])
        return {"perm_input": s["perm"][0].values, "perm_table": s["perm"][1].values, "inverted": s["inverted"].values,
                "scanned": s["scanned"].values, "quotient": s["quotient"].values, "value": s["value"]}
    server = s["server"]
    tickets = [server.submit(k, seed) for k, seed in s["requests"]]
    results = [server.wait(t) for t in tickets]
    assert all(r.status == 0 for r in results)
    return [zk.serving.result_words(r).view(np.int32) for r in results]


# ------------------------------------------------------------------ what a pass cannot do without
def _msm_work(n, batch):
    # each scalar and base once; 254 bits in windows of 16, six products to add a point
    return 32.0 * n * batch + 64.0 * n, PRODUCT * 16 * 6 * n * batch


def work(case):
    kind = case["kind"]
    if kind == "ntt":
        n = 1 << case["log_n"]
        return {"bytes": 64.0 * n, "flops": PRODUCT * n / 2 * case["log_n"]}
    if kind == "lde":
        n, N = 1 << case["log_n"], 1 << (case["log_n"] + case["ext"])
        return {"bytes": 32.0 * (n + N), "flops": PRODUCT * (n + N / 2 * (case["log_n"] + case["ext"]))}
    if kind == "msm":
        b, f = _msm_work(case["n"], case["batch"])
        return {"bytes": b, "flops": f}
    if kind == "poly":
        # permute 4 columns, invert / scan / divide 2 each, evaluate 1; 3 + 1 + 1 + 1 products
        return {"bytes": 32.0 * 11 * case["n"], "flops": PRODUCT * 6 * case["n"]}
    total = {"bytes": 0.0, "flops": 0.0}
    for k in _request_sizes(case):
        n, N = 1 << k, 4 << k
        b, f = _msm_work(n, 4)
        # 3 INTTs, one coset transform at 4x, the quotient (3 products a value), two evaluations
        total["bytes"] += b + 3 * 64.0 * n + 32.0 * (n + N) + 160.0 * N + 64.0 * n
        total["flops"] += f + PRODUCT * (3 * n / 2 * k + n + N / 2 * (k + 2) + 3 * N + 2 * n)
    return total


def tolerance(case):
    return "exact"  # whole numbers: canonical field elements and affine points


# ------------------------------------------------------------------ the same results in Python integers
def _ints(t, words=8):
    a = np.ascontiguousarray(t.cpu().numpy()).view(np.uint8).reshape(-1, 4 * words)
    return [int.from_bytes(row.tobytes(), "little") for row in a]


def _words(values, shape=None):
    raw = b"".join(v.to_bytes(32, "little") for v in values)
    a = np.frombuffer(raw, dtype=np.int32)
    return a.reshape(shape if shape is not None else (-1, 8)).copy()


def _root(log_n):
    return pow(pow(SHIFT, (FR - 1) >> 28, FR), 1 << (28 - log_n), FR)


def _dft(a, w):
    """sum_j a_j w^(ij), natural order in and out."""
    n = len(a)
    if n == 1:
        return a
    bits = n.bit_length() - 1
    a = [a[int(format(i, "0%db" % bits)[::-1], 2)] for i in range(n)]
    half = 1
    while half < n:
        step, tw = pow(w, n // (2 * half), FR), [1] * half
        for i in range(1, half):
            tw[i] = tw[i - 1] * step % FR
        for base in range(0, n, 2 * half):
            for i in range(half):
                u, v = a[base + i], a[base + half + i] * tw[i] % FR
                a[base + i], a[base + half + i] = (u + v) % FR, (u - v) % FR
        half *= 2
    return a


def _jac_add(p, q):
    """Jacobian p plus Jacobian q over Fq (y^2 = x^3 + 3); None is the identity."""
    if p is None:
        return q
    if q is None:
        return p
    x1, y1, z1 = p
    x2, y2, z2 = q
    z1z1, z2z2 = z1 * z1 % FQ, z2 * z2 % FQ
    u1, u2 = x1 * z2z2 % FQ, x2 * z1z1 % FQ
    s1, s2 = y1 * z2 * z2z2 % FQ, y2 * z1 * z1z1 % FQ
    if u1 == u2:
        if s1 != s2:
            return None
        a, b = x1 * x1 % FQ, y1 * y1 % FQ
        s, m = 4 * x1 * b % FQ, 3 * a % FQ
        x3 = (m * m - 2 * s) % FQ
        return x3, (m * (s - x3) - 8 * b * b) % FQ, 2 * y1 * z1 % FQ
    h, r = (u2 - u1) % FQ, (s2 - s1) % FQ
    hh = h * h % FQ
    hhh, v = h * hh % FQ, u1 * hh % FQ
    x3 = (r * r - hhh - 2 * v) % FQ
    return x3, (r * (v - x3) - s1 * hhh) % FQ, z1 * z2 * h % FQ


def _multiexp(scalars, points):
    c, total = 9, None
    for w in reversed(range(-(-254 // c))):
        for _ in range(c):
            total = _jac_add(total, total) if total is not None else None
        buckets = [None] * (1 << c)
        for k, p in zip(scalars, points):
            d = (k >> (w * c)) & ((1 << c) - 1)
            if d and p is not None:
                buckets[d] = _jac_add(buckets[d], p)
        run = acc = None
        for b in reversed(buckets[1:]):
            run = _jac_add(run, b)
            acc = _jac_add(acc, run)
        total = _jac_add(total, acc)
    if total is None:
        return [0, 0]
    x, y, z = total
    zi = pow(z, -1, FQ)
    return [x * zi * zi % FQ * R % FQ, y * zi * zi * zi % FQ * R % FQ]


def exact(case, seed):
    """The outputs of the small cases in Python integers, from the inputs that prepare() makes."""
    kind = case["kind"]
    r_inv = pow(R, -1, FR)
    if kind == "ntt" and case["log_n"] <= 17:
        a = _ints(prepare(case, seed)["x"].values)
        n = len(a)
        w = _root(case["log_n"])
        if not case["inverse"]:
            return _words(_dft(a, w))
        n_inv = pow(n, -1, FR)
        return _words([v * n_inv % FR for v in _dft(a, pow(w, -1, FR))])
    if kind == "lde" and case["log_n"] + case["ext"] <= 17:
        a = _ints(prepare(case, seed)["coef"].values)
        g, power = SHIFT, 1
        for i in range(len(a)):
            a[i] = a[i] * power % FR
            power = power * g % FR
        N = len(a) << case["ext"]
        return _words(_dft(a + [0] * (N - len(a)), _root(case["log_n"] + case["ext"])))
    if kind == "msm" and case["n"] * case["batch"] <= 5000:
        s = prepare(case, seed)
        q_inv = pow(R, -1, FQ)
        xy = [v * q_inv % FQ for v in _ints(s["points"])]
        pts = [(x, y, 1) if y else None for x, y in zip(xy[::2], xy[1::2])]
        return [_words(_multiexp([v * r_inv % FR for v in _ints(sc)], pts), (16,)) for sc in s["scalars"]]
    if kind == "poly" and case["n"] <= 70000:
        s = prepare(case, seed)
        n, usable = case["n"], case["n"] - 5
        plain = lambda v: v * r_inv % FR  # noqa: E731
        column, table = _ints(s["column"].values)[:usable], _ints(s["table"].values)[:usable]
        order = sorted(column, key=plain)
        left = {}
        for v in table:
            left[v] = left.get(v, 0) + 1
        first = [i == 0 or order[i] != order[i - 1] for i in range(usable)]
        for i, v in enumerate(order):
            if first[i]:
                left[v] -= 1
        rest = iter(sorted((v for v, m in left.items() for _ in range(m)), key=plain))
        perm_table = [v if first[i] else next(rest) for i, v in enumerate(order)]
        inverted = [pow(v, -1, FR) * R * R % FR if v else 0 for v in _ints(s["inverted"].values)]
        scanned, acc = [], R % FR
        for v in _ints(s["scanned"].values):
            acc = acc * v * r_inv % FR
            scanned.append(acc)
        b = plain(_ints(s["divisor"])[0])
        p = _ints(s["dividend"].values)
        quotient, acc = [0] * len(p), 0
        for i in range(len(p) - 2, -1, -1):
            acc = (p[i + 1] + b * acc) % FR
            quotient[i] = acc
        x, value = plain(_ints(s["point"])[0]), 0
        for v in reversed(_ints(s["p"].values)):
            value = (value * x + v) % FR
        return {"perm_input": _words(order), "perm_table": _words(perm_table), "inverted": _words(inverted),
                "scanned": _words(scanned), "quotient": _words(quotient), "value": _words([value])}
    return None
