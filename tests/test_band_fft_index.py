"""Shapes and index arithmetic of the band-pruned transforms (cg_band_shape.cuh): the
library's radices, halves and window offsets drive the passes restated in numpy,
checked against numpy.fft (decimation in frequency in place, inputs taken from the
window's start on, a half-filled line as two transforms of half the length, outputs
in digit-reversed position); its shared-memory indices are checked pass by pass."""
import ctypes

import numpy as np
import pytest


@pytest.fixture(scope="module")
def shape(host_index):
    """The library's own shape of a transform (cg_band_shape.cuh)."""

    def get(L, i0, ni, o0, no, rows, esz):
        v = (ctypes.c_int * 64)()
        if not host_index.t_band_shape(L, i0, ni, o0, no, int(rows), esz, v):
            return None
        keys = ("H", "n", "NB", "apart", "threads", "smem", "m0", "delta", "npass")
        s = dict(zip(keys, v))
        s["radix"] = [v[9 + 2 * i] for i in range(s["npass"])]
        return s

    return get


def transform(x, L, i0, ni, o0, no, sh):
    """Outputs {k: X[k]} of the window [o0, o0 + no) for inputs in [i0, i0 + ni)."""
    H, n, radix, m0, delta = (sh[k] for k in ("H", "n", "radix", "m0", "delta"))
    assert H * n == L and np.prod(radix) == n
    assert (i0 % n) == m0 * (n // radix[0]) + delta and 0 <= delta < n // radix[0]
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
@pytest.mark.parametrize("rows", [False, True])
def test_windows_and_passes(shape, L, seed, rows):
    rng = np.random.default_rng(1000 * seed + L)
    i0 = int(rng.integers(0, L))
    ni = [L // 2, int(rng.integers(1, L // 2)), int(rng.integers(L // 2 + 1, L)), L][seed]
    o0, no = int(rng.integers(0, L)), int(rng.integers(1, L + 1))
    x = np.zeros(L, complex)
    idx = (i0 + np.arange(ni)) % L
    x[idx] = rng.standard_normal(ni) + 1j * rng.standard_normal(ni)
    ref = np.fft.ifft(x) * L
    sh = shape(L, i0, ni, o0, no, rows, 16)
    if sh is None:  # a line of one pass
        assert L // 2 <= 50
        return
    got = transform(x, L, i0, ni, o0, no, sh)
    assert sorted(got) == sorted((o0 + np.arange(no)) % L)
    assert max(abs(got[k] - ref[k]) for k in got) < 1e-11 * np.sqrt(L)


def test_shared_memory_indices(host_index, shape):
    """Every supported length up to the largest, narrow windows apart from and meeting the
    outputs, and whole lines: padding, strides, reciprocals, output blocks, stash and
    table of the launch that the library makes."""
    seen = set()
    for L in range(32, 16385, 2):
        m = L
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m != 1:
            continue
        for i0, ni, o0, no in ((L // 2 - L // 8, L // 4, L - L // 4, L // 2), (L // 3, L // 2, 0, L // 2),
                               (L - L // 4, L // 2, L // 2 - L // 4, L // 2), (0, L, L - L // 4, L // 2), (5, L - 7, 3, L)):
            for rows in (0, 1):
                for esz in (8, 16):
                    assert host_index.t_band_check(L, i0, ni, o0, no, rows, esz) in (0, -1), (L, i0, ni, rows, esz)
                    sh = shape(L, i0, ni, o0, no, rows, esz)
                    if sh is None:
                        continue
                    assert sh["smem"] <= 227 * 1024 and sh["threads"] <= (1024 if esz == 8 else 512), (L, rows, esz)
                    seen.add((rows, esz, sh["H"], sh["apart"]))
    # columns and long rows as two half transforms, apart and (columns) through the stash
    for esz in (8, 16):
        assert {(0, esz, 1, 0), (0, esz, 2, 0), (0, esz, 2, 1), (1, esz, 1, 0), (1, esz, 2, 1)} <= seen
