"""Where a blind-rotation kernel adds an FP64 product sum in another order than the others, the bits agree only if
every sum rounds to its exact integer.  A numpy model of the FP64 arithmetic (folded negacyclic transforms,
multiply-accumulate over the (k+1)l rows, inverse transform) measures the error of the sums against the exact
products, with the widest digits that those kernels are given: l Bgbit <= 22 at l = 2, any accepted width at l = 3.
1/2 must stay at least 12 sigma away (a wrong rounding is then below 1e-30 per coefficient)."""
import numpy as np
import pytest


def sigma(N, l, Bgbit, seed=1):
    rng = np.random.default_rng(seed)
    M = N // 2
    tw = np.exp(-1j * np.pi * np.arange(M) / N)

    def fwd(a):
        return np.fft.fft((a[:M] - 1j * a[M:]) * tw)

    acc, exact = np.zeros(M, complex), np.zeros(N, np.int64)  # |sums| below 2^53 here
    for _ in range(2 * l):
        d = rng.integers(-(1 << (Bgbit - 1)), 1 << (Bgbit - 1), N)
        k = rng.integers(-2**31, 2**31, N)
        acc += fwd(d.astype(float)) * fwd(k.astype(float))
        full = np.convolve(d, k)
        full[:N - 1] -= full[N:]
        exact += full[:N]
    z = np.fft.ifft(acc) / tw
    v = np.concatenate([z.real, -z.imag])
    nearest = np.rint(v)
    return float(np.sqrt(np.mean(((nearest.astype(np.int64) - exact) + (v - nearest)) ** 2)))


@pytest.mark.parametrize("N,l,Bgbit", [(1024, 2, 11), (1024, 3, 10), (2048, 3, 10)])
def test_reordered_sums_round_to_the_exact_integer(N, l, Bgbit):
    s = sigma(N, l, Bgbit)
    assert 0.5 / s >= 12, s


def test_wider_digits_do_not():
    assert 0.5 / sigma(1024, 2, 14) < 6
