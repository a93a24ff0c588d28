"""The device integer library evaluated ON THE DEVICE against the CPU oracle: a million seeded
operand tuples per primitive. The host build of the same header (tests/test_device_int_host.py)
cannot execute the device-only halves -- the rcp.approx / rsqrt.approx estimates behind the exact
divisions and roots, and the attention kernels' 32-bit softmax element -- so they are swept here.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import harness as H

pytestmark = pytest.mark.gpu

N = 1 << 20
I64 = np.int64


def device_sweep(lib, which, a, b, c, e):
    f = lib.dll.sslm_b200_int_sweep
    f.argtypes = [C.c_int32] + [C.c_void_p] * 4 + [C.c_int64] + [C.c_void_p] * 3
    outs = [np.zeros(a.size, dtype=I64) for _ in range(3)]
    assert f(which, a.ctypes.data, b.ctypes.data, c.ctypes.data, e.ctypes.data, a.size, *[o.ctypes.data for o in outs]) == 0
    return outs


def oracle_sweep(which, a, b, c, e):
    outs = [np.zeros(a.size, dtype=I64) for _ in range(3)]
    H.port().osc_sweep(which, a.ctypes.data, b.ctypes.data, c.ctypes.data, e.ctypes.data, a.size, *[o.ctypes.data for o in outs])
    return outs


def pack(hi, lo):
    return ((hi.astype(I64) << 32) | (lo.astype(I64) & 0xFFFFFFFF)).astype(I64)


def canonical(rng, n):
    return rng.integers(1 << 30, 1 << 31, n, dtype=I64)


def zeros():
    return np.zeros(N, dtype=I64)


def test_reciprocal_on_the_device(gpu_lib):
    rng = np.random.default_rng(1)
    a = canonical(rng, N)
    a[::9] = rng.integers(-(1 << 40), 1 << 40, a[::9].size, dtype=I64)     # non-canonical mantissas take the reference's sequence
    a[::11] = rng.integers(1, 1 << 20, a[::11].size, dtype=I64)
    a[:4] = [1 << 30, (1 << 31) - 1, (1 << 30) + 1, 1090717716]
    got, want = device_sweep(gpu_lib, 0, a, zeros(), zeros(), zeros()), oracle_sweep(0, a, zeros(), zeros(), zeros())
    assert (got[0] == want[0]).all()


def test_square_root_and_floor_divisions_on_the_device(gpu_lib):
    rng = np.random.default_rng(2)
    bits = rng.integers(0, 62, N)
    a = (rng.integers(0, 1 << 62, N, dtype=I64) >> (61 - bits)).astype(I64)
    a[:6] = [0, 1, 2, 3, (1 << 62) - 1, (1 << 32)]
    sq = rng.integers(1, 1 << 31, N // 4, dtype=I64)
    a[1000:1000 + sq.size] = sq * sq - rng.integers(0, 2, sq.size)          # perfect squares and their predecessors
    got, want = device_sweep(gpu_lib, 1, a, zeros(), zeros(), zeros()), oracle_sweep(1, a, zeros(), zeros(), zeros())
    assert (got[0] == want[0]).all()
    h = rng.integers(-127, 128, N, dtype=I64)
    root = (rng.integers(1, 1 << 39, N, dtype=I64) >> rng.integers(0, 38, N)).astype(I64)
    root[root < 1] = 1
    got, want = device_sweep(gpu_lib, 2, h, root, zeros(), zeros()), oracle_sweep(2, h, root, zeros(), zeros())
    assert (got[0] == want[0]).all()
    den = (rng.integers(1, 1 << 40, N, dtype=I64) >> rng.integers(0, 39, N)).astype(I64)
    den[den < 1] = 1
    q = rng.integers(0, 1 << 20, N, dtype=I64)
    num = q * den + (rng.integers(0, 1 << 40, N, dtype=I64) % den)
    got, want = device_sweep(gpu_lib, 5, num, den, zeros(), zeros()), oracle_sweep(5, num, den, zeros(), zeros())
    assert (got[0] == want[0]).all()


def test_requant_codes_and_funnel_scalars_on_the_device(gpu_lib):
    rng = np.random.default_rng(3)
    dn = canonical(rng, N)
    dn[::13] = 1 << 30                                                      # R = 2^32: the coders' edge
    r = oracle_sweep(0, dn, zeros(), zeros(), zeros())[0]
    s = rng.integers(-1, 31, N, dtype=I64)
    x = rng.integers(-(1 << 31), (1 << 31) + 1, N, dtype=I64)
    x[::7] = rng.integers(-(1 << 33), 1 << 33, x[::7].size, dtype=I64)
    x[:4] = [1 << 31, -(1 << 31), (1 << 31) + 1, 0]
    got, want = device_sweep(gpu_lib, 3, x, r, s, zeros()), oracle_sweep(3, x, r, s, zeros())
    for k in range(3):                   # the general composite and both per-row coders
        assert (got[k] == want[0]).all(), k
    mx = rng.integers(0, (1 << 31) + 3, N, dtype=I64)
    mx[::5] = (rng.integers(1, 1 << 31, mx[::5].size, dtype=I64) >> rng.integers(0, 30, mx[::5].size)).astype(I64)
    inc_m, inc_e = canonical(rng, N), rng.integers(-60, -20, N, dtype=I64)
    site = pack(canonical(rng, N), rng.integers(-60, -30, N, dtype=I64))
    got, want = device_sweep(gpu_lib, 6, mx, inc_m, inc_e, site), oracle_sweep(6, mx, inc_m, inc_e, site)
    assert (got[2] == want[2]).all()
    ok = want[2] == 0
    assert ok.sum() > N // 2
    assert (got[0][ok] == want[0][ok]).all() and (got[1][ok] == want[1][ok]).all()


def test_landing_rescale_on_the_device(gpu_lib):
    rng = np.random.default_rng(4)
    code = rng.integers(-(1 << 31), 1 << 31, N, dtype=I64)
    code[::3] = rng.integers(-127, 128, code[::3].size, dtype=I64)
    m_a = canonical(rng, N) * rng.choice(np.array([1, 1, 1, -1], dtype=I64), N)
    r_t = rng.integers((1 << 31) + 1, (1 << 32) + 1, N, dtype=I64)
    e = pack(rng.integers(-90, 40, N, dtype=I64), rng.integers(-70, 20, N, dtype=I64))
    got, want = device_sweep(gpu_lib, 4, code, m_a, r_t, e), oracle_sweep(4, code, m_a, r_t, e)
    exceeded = (want[1] & 2) != 0
    assert (got[1] == want[1]).all()
    assert (got[0][~exceeded] == want[0][~exceeded]).all()


def test_softmax_element_and_probability_on_the_device(gpu_lib):
    rng = np.random.default_rng(5)
    port = H.port()
    # constant triples of scales inside the softmax window, as k_qkv_post derives them
    sets = []
    for i in range(64):
        m, e = int(rng.integers(1 << 30, 1 << 31)), int(rng.integers(-51, -33))
        ln2, qb, qc = C.c_int64(0), C.c_int64(0), C.c_int64(0)
        if port.osc_iexp_scale_constants(m, e, C.byref(ln2), C.byref(qb), C.byref(qc)) == 0 and ln2.value >= 1 and \
           qb.value * qb.value + qc.value <= (1 << 47):
            sets.append((ln2.value, qb.value, qc.value))
    assert len(sets) >= 16
    pick = rng.integers(0, len(sets), N)
    ln2 = np.array([sets[i][0] for i in pick], dtype=I64)
    qb = np.array([sets[i][1] for i in pick], dtype=I64)
    qc = np.array([sets[i][2] for i in pick], dtype=I64)
    peak16 = ((qb * qb + qc) >> 16) + 1                                     # peak rounded up to a multiple of 2^16
    dq = (rng.integers(0, 34, N) * ln2 + rng.integers(-3, 4, N)).clip(0, (1 << 32) - 1).astype(I64)
    dq[::17] = rng.integers(0, 1 << 32, dq[::17].size, dtype=I64)
    e = pack(qc, peak16)
    got, want = device_sweep(gpu_lib, 7, dq, ln2, qb, e), oracle_sweep(7, dq, ln2, qb, e)
    assert (want[1] == 0).all()
    assert (got[0] == want[0]).all() and (got[2] == want[0]).all()
    bound = peak16 << 16
    assert (got[1] == ((want[0] < 0) | (want[0] > bound)).astype(I64)).all()
    tot = (rng.integers(1, 1 << 62, N, dtype=I64) >> rng.integers(0, 61, N)).astype(I64)
    tot[tot < 1] = 1
    ev = (rng.integers(0, 1 << 47, N, dtype=I64) % (np.minimum(tot, (1 << 47) - 1) + 1)).astype(I64)
    got = device_sweep(gpu_lib, 8, ev, tot, zeros(), zeros())
    want = ((ev.astype(np.uint64) << np.uint64(15)) // tot.astype(np.uint64)).astype(I64)
    assert (got[0] == want).all()


def funnel_scalars(d):
    """(R, s) of a row of maximum d, as NormalizeScale and DynamicScaleReciprocal give them."""
    s = 30 - np.floor(np.log2(d.astype(np.float64))).astype(I64)
    dn = np.where(s >= 0, d << np.maximum(s, 0), d >> 1)
    assert ((dn >= 1 << 30) & (dn < 1 << 31)).all()
    return oracle_sweep(0, dn, np.zeros_like(dn), np.zeros_like(dn), np.zeros_like(dn))[0], s


def near_ties(rng, d, low, spread):
    """elements of rows of maximum d: near (2 c + 1) d / 254, the ties, for |c| from `low` up, and anywhere."""
    n = d.size
    c = rng.integers(low, 127, n, dtype=I64)
    x = ((2 * c + 1) * d) // 254 + rng.integers(-spread, spread + 1, n, dtype=I64)
    x[::3] = rng.integers(0, 1 << 62, x[::3].size, dtype=I64) % (d[::3] + 1)
    return np.minimum(np.abs(x), d) * rng.choice(np.array([1, -1], dtype=I64), n)


def test_row_codes_on_the_device(gpu_lib):
    rng = np.random.default_rng(6)
    for lo, hi, low, spread in [(24, 31, 118, 40), (24, 31, 0, 3), (30, 31, 120, 400), (16, 24, 0, 2), (1, 16, 0, 1)]:
        d = np.exp2(rng.uniform(lo, hi, N)).astype(I64)
        d[::11] = (1 << rng.integers(lo, hi + 1, d[::11].size, dtype=I64)) + rng.integers(-3, 4, d[::11].size, dtype=I64)
        d[::13] = 1 << hi
        d = np.clip(d, 1, (1 << 31) - 1)
        if hi == 31:
            d[5] = 1 << 31      # (the maximum of a row may be 2^31; an element that is no int32 may not be given here)
        x = np.clip(near_ties(rng, d, low, spread), -(1 << 31) + 1, (1 << 31) - 1)
        r, s = funnel_scalars(d)
        want = oracle_sweep(3, x, r, s, zeros())[0]
        got = device_sweep(gpu_lib, 9, x, d, zeros(), zeros())
        assert (got[0] == want).all() and (got[1] == want).all() and not got[2].any(), (lo, hi)
    d = rng.integers(1, 1 << 16, N, dtype=I64)
    d[::2] = rng.integers(1, 600, d[::2].size, dtype=I64)
    x = near_ties(rng, d, 0, 1)
    r, s = funnel_scalars(d)
    want = oracle_sweep(3, x, r, s, zeros())[0], oracle_sweep(3, -x, r, s, zeros())[0]
    got = device_sweep(gpu_lib, 10, x, d, zeros(), zeros())
    assert (got[0] == want[0]).all() and (got[1] == want[1]).all()


def test_landings_of_the_row_kernels_on_the_device(gpu_lib):
    rng = np.random.default_rng(7)
    code = rng.integers(-127, 128, N, dtype=I64)
    bs_m, ss_m = canonical(rng, N), canonical(rng, N)
    bs_m[::4] = np.clip(ss_m[::4] + rng.integers(-300, 301, bs_m[::4].size, dtype=I64), 1 << 30, (1 << 31) - 1)   # ratios near powers of two: true ties
    bs_m[::17] *= -1
    bs_e, ss_e = rng.integers(-60, -20, N, dtype=I64), rng.integers(-60, -20, N, dtype=I64)
    ss_e[::2] = bs_e[::2] + rng.integers(-9, 8, ss_e[::2].size, dtype=I64)
    e = pack(bs_e, ss_e)
    want = oracle_sweep(4, code, bs_m, oracle_sweep(0, ss_m, zeros(), zeros(), zeros())[0], e)
    got = device_sweep(gpu_lib, 11, code, bs_m, ss_m, e)
    covered = got[1] != 0
    assert covered.sum() > N // 3 and (np.abs(want[0][covered]) < 1 << 15).all()
    assert (got[0][covered] == want[0][covered]).all()
    acc = rng.integers(-(1 << 31), (1 << 31) + 1, N, dtype=I64)
    acc[::3] = rng.integers(-127, 128, acc[::3].size, dtype=I64)
    r_t = rng.integers((1 << 31) + 1, (1 << 32) + 1, N, dtype=I64)
    e = pack(rng.integers(-90, 40, N, dtype=I64), rng.integers(-70, 20, N, dtype=I64))
    want = oracle_sweep(4, acc, bs_m, r_t, e)
    got = device_sweep(gpu_lib, 15, acc, bs_m, r_t, e)
    covered = got[1] != 0
    assert covered.sum() > N // 4
    assert (got[0][covered] == want[0][covered]).all()


def test_norm_quotients_of_the_row_kernels_on_the_device(gpu_lib):
    rng = np.random.default_rng(8)
    n = rng.choice(np.array([128, 256, 896, 1536, 2048, 3584, 8192, 16384], dtype=I64), N)
    rms = np.exp2(rng.uniform(-1, 6.98, N))
    ss = np.clip((n * rms * rms).astype(I64), 1, n * 127 * 127)
    ss[::5] = n[::5] * rng.integers(1, 128, ss[::5].size, dtype=I64) ** 2          # the root a whole code, and its neighbours
    ss[::5] += rng.integers(-1, 2, ss[::5].size, dtype=I64)
    h = rng.integers(-127, 128, N, dtype=I64)
    root = np.maximum(oracle_sweep(1, (ss << 32) // n, zeros(), zeros(), zeros())[0], 1)
    got = device_sweep(gpu_lib, 12, h, ss, n, zeros())
    covered = got[1] != 0
    assert (covered == (root >= 1 << 16)).all() and covered.sum() > N // 2
    assert (got[2][covered] == root[covered]).all()
    assert (got[0][covered] == ((h << 32) // root)[covered]).all()


def test_prefill_softmax_on_the_device(gpu_lib):
    rng = np.random.default_rng(9)
    port = H.port()
    sets = []
    for i in range(64):
        m, e = int(rng.integers(1 << 30, 1 << 31)), int(rng.integers(-51, -33))
        ln2, qb, qc = C.c_int64(0), C.c_int64(0), C.c_int64(0)
        if port.osc_iexp_scale_constants(m, e, C.byref(ln2), C.byref(qb), C.byref(qc)) == 0 and ln2.value >= 1 and \
           qb.value * qb.value + qc.value <= (1 << 47):
            sets.append((ln2.value, qb.value, qc.value))
    assert len(sets) >= 16
    pick = rng.integers(0, len(sets), N)
    ln2, qb, qc = (np.array([sets[i][k] for i in pick], dtype=I64) for k in range(3))
    dq = (rng.integers(0, 34, N) * ln2 + rng.integers(-3, 4, N)).clip(0, (1 << 32) - 1).astype(I64)
    dq[::17] = rng.integers(0, 1 << 32, dq[::17].size, dtype=I64)
    x = np.minimum(dq, 30 * ln2)
    value = ((qb - x % ln2) ** 2 + qc) >> (x // ln2)
    got = device_sweep(gpu_lib, 13, dq, ln2, qb, qc)
    assert (got[0] == value).all()
    words = got[1]
    z, base = words >> 24, words & 0xFFFFFF
    assert ((base * base + qc) >> z == value).all()
    # totals from the element alone to rows of 32,768 of the largest; some for quotients beside a whole number
    tot = np.maximum(value, 1) + (rng.integers(0, 1 << 62, N, dtype=I64) >> rng.integers(0, 61, N)) % ((qb * qb + qc) * 32767)
    k = rng.integers(1, 1 << 15, N, dtype=I64)
    near = (value << 15) // k + rng.integers(-2, 3, N, dtype=I64)
    use = (rng.integers(0, 2, N) == 0) & (near >= value) & (near > 0)
    tot[use] = near[use]
    words[::41] = 63 << 24                                                          # elements that count for nothing
    value[::41] = 0
    got = device_sweep(gpu_lib, 14, words, tot, qc, zeros())
    want = ((value.astype(np.uint64) << np.uint64(15)) // tot.astype(np.uint64)).astype(I64)
    assert (got[0] == want).all()


def test_softmax_at_the_width_gate_on_the_device(gpu_lib):
    """the smallest scale that the gate admits: q_b and the peak at their largest"""
    rng = np.random.default_rng(10)
    port = H.port()
    ln2, qb, qc = C.c_int64(0), C.c_int64(0), C.c_int64(0)
    lo, hi, limit = (1 << 30), (1 << 31) - 1, None
    while lo <= hi:
        m = (lo + hi) // 2
        ok = port.osc_iexp_scale_constants(m, -53, C.byref(ln2), C.byref(qb), C.byref(qc)) == 0 and qb.value ** 2 + qc.value <= 1 << 47
        if ok:
            limit, hi = (ln2.value, qb.value, qc.value), m - 1
        else:
            lo = m + 1
    ln2, qb, qc = limit
    peak = qb ** 2 + qc
    assert peak > 0.9999 * (1 << 47)
    dq = (rng.integers(0, 34, N) * ln2 + rng.integers(-3, 4, N)).clip(0, (1 << 32) - 1).astype(I64)
    dq[::17] = rng.integers(0, 1 << 32, dq[::17].size, dtype=I64)
    x = np.minimum(dq, 30 * ln2)
    value = ((qb - x % ln2) ** 2 + qc) >> (x // ln2)
    got = device_sweep(gpu_lib, 13, dq, zeros() + ln2, zeros() + qb, zeros() + qc)
    assert (got[0] == value).all()
    words = got[1]
    z, base = words >> 24, words & 0xFFFFFF
    assert ((base * base + qc) >> z == value).all()
    tot = np.maximum(value, 1) + (rng.integers(0, 1 << 62, N, dtype=I64) >> rng.integers(0, 61, N)) % (peak * 32767)
    k = rng.integers(1, 1 << 15, N, dtype=I64)
    near = (value << 15) // k + rng.integers(-2, 3, N, dtype=I64)
    use = (rng.integers(0, 2, N) == 0) & (near >= value) & (near > 0)
    tot[use] = near[use]
    got = device_sweep(gpu_lib, 14, words, tot, zeros() + qc, zeros())
    want = ((value.astype(np.uint64) << np.uint64(15)) // tot.astype(np.uint64)).astype(I64)
    assert (got[0] == want).all()
