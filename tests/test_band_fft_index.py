"""Index arithmetic of the band-pruned transforms (cg_fft_band.cu), restated in
numpy and checked against numpy.fft: decimation-in-frequency passes in place,
inputs taken from the window's start on (a rotation that the first pass's factors
undo), a half-filled line as two transforms of half the length, outputs in
digit-reversed position."""
import numpy as np
import pytest


def factor(n):
    a = b = c = 0
    while n % 2 == 0:
        n, a = n // 2, a + 1
    while n % 3 == 0:
        n, b = n // 3, b + 1
    while n % 5 == 0:
        n, c = n // 5, c + 1
    assert n == 1
    r = []
    while a >= 4 and a != 5:
        r, a = r + [16], a - 4
    if a == 5:
        r, a = r + [8], 2
    while c and b:
        r, c, b = r + [15], c - 1, b - 1
    while c and a:
        r, c, a = r + [10], c - 1, a - 1
    r, c = r + [5] * c, 0
    while b >= 2 and a == 0:
        r, b = r + [9], b - 2
    while b and a >= 2:
        r, b, a = r + [12], b - 1, a - 2
    while b and a:
        r, b, a = r + [6], b - 1, a - 1
    while b >= 2:
        r, b = r + [9], b - 2
    r = r + [3] * b
    return r + ([1 << a] if a else [])


def transform(x, L, i0, ni, o0, no):
    """Outputs {k: X[k]} of the window [o0, o0 + no) for inputs in [i0, i0 + ni)."""
    H = 2 if ni <= L // 2 else 1
    n = L // H
    radix = factor(n)
    sub0 = n // radix[0]
    m0, delta = divmod(i0 % n, sub0)
    out = {}
    for s in range(H):
        sm = np.zeros(n, complex)
        blk = n
        for i, R in enumerate(radix):
            sub = blk // R
            dft = np.exp(2j * np.pi * np.outer(np.arange(R), np.arange(R)) / R)
            for bf in range(n // R):
                q, j = divmod(bf, sub)
                pos = q * blk + j + np.arange(R) * sub
                if i == 0:
                    v = np.zeros(R, complex)
                    for m in range(R):
                        o = bf - delta + m * sub
                        if m == 0 and o < 0:
                            o += n
                        if o < ni:
                            k = (i0 + o) % L
                            v[m] = x[k] * np.exp(2j * np.pi * k * s / L)
                    j = j + m0 * sub
                else:
                    v = sm[pos]
                sm[pos] = dft @ v
                if i < len(radix) - 1:
                    sm[pos] *= np.exp(2j * np.pi * np.arange(R) * j / blk)
                elif i == 0:
                    sm[pos] *= np.exp(2j * np.pi * np.arange(R) * j / blk)
            blk = sub
        last = radix[-1]
        for k0 in range(n // last):
            b, k = 0, k0
            for R in radix[:-1]:
                k, r = divmod(k, R)
                b = b * R + r
            for m in range(last):
                k = H * (k0 + m * (n // last)) + s
                if (k - o0) % L < no:
                    out[k] = sm[b * last + m]
    return out


@pytest.mark.parametrize("L", [36, 72, 100, 128, 216, 300, 512, 540, 750, 1152])
@pytest.mark.parametrize("seed", range(4))
def test_windows_and_passes(L, seed):
    rng = np.random.default_rng(1000 * seed + L)
    i0 = int(rng.integers(0, L))
    ni = [L // 2, int(rng.integers(1, L // 2)), int(rng.integers(L // 2 + 1, L)), L][seed]
    o0, no = int(rng.integers(0, L)), int(rng.integers(1, L + 1))
    x = np.zeros(L, complex)
    idx = (i0 + np.arange(ni)) % L
    x[idx] = rng.standard_normal(ni) + 1j * rng.standard_normal(ni)
    ref = np.fft.ifft(x) * L
    got = transform(x, L, i0, ni, o0, no)
    assert sorted(got) == sorted((o0 + np.arange(no)) % L)
    assert max(abs(got[k] - ref[k]) for k in got) < 1e-11 * np.sqrt(L)
