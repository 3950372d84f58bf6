"""CPU model of the back-projection tables' entries (bp_line and bp_taps_on of
csrc/update.cuh): a detector position A + q B held in two floats each gives the bin
and the fraction of the position in 64 bits, the fraction rounded once (2^-25), next to
bin boundaries too."""
import numpy as np

f = np.float32


def _fma(a, b, c):  # exact product and a sum to 64 bits or more, then one rounding
    return (np.asarray(a, np.longdouble) * np.asarray(b, np.longdouble) + c).astype(f)


def taps_on(A, B, q):
    ah, bh = f(A), f(B)
    al, bl = f(A - np.float64(ah)), f(B - np.float64(bh))
    p = q * bh
    pe = _fma(q, bh, -p)
    s = ah + p
    t = s - ah
    se = (ah - (s - t)) + (p - t)
    lo = se + (pe + _fma(q, bl, al))
    fl = np.floor(s)
    r = (s - fl) + lo
    off = (r >= 1) | (r < 0)
    fl = np.where(off, fl + np.where(r < 0, f(-1), f(1)), fl)
    r = np.where(off, np.maximum((s - fl) + lo, f(0)), r)
    assert all(v.dtype == f for v in (p, pe, s, se, lo, fl, r))
    return fl, r


def test_bin_and_fraction():
    rng = np.random.default_rng(0)
    q = np.arange(0, 2048, 7).astype(f)
    for k in range(300):
        B = rng.uniform(0.05, 3.0)
        A = rng.uniform(-4000.0, 4000.0)
        if k % 3 == 0:   # position q[k] within a few 2^-40 of a bin boundary
            A = np.round(A) - q[k % q.size] * B + rng.integers(-4, 5) * 2.0 ** -40
        fl, r = taps_on(A, B, q)
        assert (r >= 0).all() and (r <= 1).all()
        x = np.longdouble(A) + q.astype(np.longdouble) * np.longdouble(B)
        assert np.abs(fl.astype(np.longdouble) + r - x).max() <= 2.0 ** -25 + 2.0 ** -33
