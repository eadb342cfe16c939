"""FP32 arithmetic with every rounding named, on NumPy arrays: what a kernel that
names its roundings gives, bit for bit."""
import numpy as np

f32, f64 = np.float32, np.float64


def fma(x, y, z):
    """x y + z with one rounding (the FP64 sum's own rounding shows in about one of 2^29 values)."""
    return (np.asarray(x, f32).astype(f64) * np.asarray(y, f32) + np.asarray(z, f32)).astype(f32)


def tables(profile, delta):
    """ik, ad, b, ikh, adh, bh of one axis, as the solvers hold them."""
    K, A, B, Kh, Ah, Bh = profile.packed()
    return [t.astype(f32) for t in (1.0 / (delta * K), A / delta, B, 1.0 / (delta * Kh), Ah / delta, Bh)]


def strip(n, w):
    i = np.arange(n)
    return (i < w) | (i >= n - w)


def ahead(f, axis):
    """f at the next cell of an axis (wrapping: the last cells lie outside every loop that looks ahead)."""
    return np.roll(f, -1, axis)


def behind(f, axis):
    return np.roll(f, 1, axis)
