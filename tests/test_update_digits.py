"""The digit scheme of the int8-emulated FP64 update restated in numpy: 48-bit rows of six balanced 8-bit
digits below scales of six bits, products of levels s + t <= 7, K = 256 columns at a time -- against the six
7-bit digits with levels <= 8 and K = 128 of test_digit_schemes.py."""
import numpy as np
import pytest

from test_digit_schemes import _blocked_forms, _system


def _product8(a, b):
    """a @ b.T: exact level sums of the digits that k_slice_panel64 cuts."""
    def digits(m):
        frac, e = np.frexp(np.abs(m).max(axis=1))
        scale = np.where(frac > 0, np.ldexp(np.ceil(frac * (64.0 / 0.996)) / 32.0, e), 1.0)
        u = np.rint(m / scale[:, None] * 2.0**48).astype(np.int64) + 0x808080808080
        assert u.min() >= 0 and u.max() < 1 << 48
        return [((u >> 8 * (5 - s)) & 255) - 128 for s in range(6)], scale

    (da, sa), (db, sb) = digits(a), digits(b)
    g = np.zeros((len(a), len(b)), dtype=np.longdouble)
    for level in range(5, -1, -1):
        total = sum(da[s] @ db[level - s].T for s in range(level + 1))
        assert np.abs(total).max() < 1 << 31
        g += total.astype(np.longdouble) * np.longdouble(2.0) ** (-8 * (level + 2))
    return (g * sa[:, None].astype(np.longdouble) * sb[None, :]).astype(np.float64)


def _forms8(tall, n):
    """_blocked_forms with the blocks in pairs: the first updates the second's columns, both the rest."""
    a = tall.copy()
    for k0 in range(0, n, 128):
        k1 = min(k0 + 128, n)
        a[k0:k1, k0:k1] = np.linalg.cholesky(a[k0:k1, k0:k1])
        a[k1:, k0:k1] = np.linalg.solve(a[k0:k1, k0:k1], a[k1:, k0:k1].T).T
        second = k0 % 256 == 128
        kb, c1 = (k0 - 128, n) if second else (k0, min(k1 + 128, n))
        if k1 < c1:
            a[k1:, k1:c1] -= _product8(a[k1:, kb:k1], a[k1:c1, kb:k1])
    return -np.sum(a[n:, :n] ** 2, axis=1)


@pytest.mark.parametrize("omega", [0.05, 1.0, 30.0])
def test_no_further_off_than_seven_bit_digits(omega):
    inp, de, v = _system(40, 12, seed=117)
    n = v.shape[0]
    eri = inp.eri_mo.reshape(40, 40, 40, 40)
    io, av = np.repeat(np.arange(12), 28), np.tile(np.arange(12, 40), 12)
    x = np.concatenate([eri[s, :, io, av].T for s in (10, 11, 12, 13)])
    dh = np.sqrt(4 * de / (de * de + omega**2))
    tall = np.concatenate([np.eye(n) + dh[:, None] * v * dh[None, :], x * dh[None, :]])
    ref = _blocked_forms(tall, n, None)
    old = np.abs(_blocked_forms(tall, n, (6, 8, True)) - ref).max()
    new = np.abs(_forms8(tall, n) - ref).max()
    assert new <= old + 1e-15 * np.abs(ref).max()  # 1e-15: the FP64 sums themselves
