"""CPU test of which grid sides have a transform of the library's own (the others
take cuFFT): compile-time lengths for powers of two from 32 to 8192 pixels, run-time
ones for the other multiples of four from 16 to 4,800 whose G / 3 has no prime factor
above the limit."""
import ctypes

import fastimagingpipe_b200 as fip


class Plan(ctypes.Structure):
    _fields_ = [(k, ctypes.c_int) for k in ("g", "m", "any", "passes")] + [
        ("radix", ctypes.c_int * 12), ("rest", ctypes.c_int * 32)]


def plan(n):
    """The plan of an n x n image's grid, or None."""
    f = fip.lib()._Z12fip_fft_planiRN6fipfft4PlanEi
    f.restype = ctypes.c_bool
    p = Plan()
    return p if f(ctypes.c_int(3 * n // 2), ctypes.byref(p), ctypes.c_int(0)) else None


def largest_prime(m):
    f, big = 2, 1
    while m > 1:
        while m % f == 0:
            m //= f
            big = f
        f += 1
    return big


def test_sides_up_to_the_limit():
    for n in range(16, 4801, 4):
        m = n // 2
        limit = 509 if m >= 1500 else 251 if m >= 500 else 199
        p = plan(n)
        if m & (m - 1) == 0 and m >= 16:
            assert p and not p.any
        elif largest_prime(m) > limit:
            assert p is None
        else:
            assert p and p.any == 1 and p.m == m
            product = 1
            for r in p.radix[:p.passes]:
                product *= r
            assert product == m


def test_sides_beyond_it_take_cufft():
    for n in list(range(4804, 9470, 4)) + [10000, 12288, 16384]:
        assert (plan(n) is not None) == (n == 8192), n
