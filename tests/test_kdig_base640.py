"""The digits of the exact K rho product (k_kdig) at their limits, in numpy:
K - (L + 1) / 2 as three balanced base-64 digits (L < 2^18), |rho_q| <= 2^27
(and the few units the own-state entry may exceed it by) as three balanced
base-640 digits, sums over segments of 1536 sequences.  The largest product
times a segment must stay below 2^24, and the combination 64^k 640^p plus the
middle times the column sums must give K rho exactly."""
import numpy as np
import pytest

SEG = 1536
MOST = 2 ** 27 + 64


def split_k(v):
    d0 = ((v + 32) & 63) - 32
    v = (v - d0) >> 6
    d1 = ((v + 32) & 63) - 32
    return [d0, d1, (v - d1) >> 6]


def split_rho(v):
    out = []
    up = 2 ** 28 // 640
    for _ in range(2):
        t = v + 320 + up * 640
        assert np.all(t >= 0) and np.all(t < 2 ** 32)
        out.append(t % 640 - 320)
        v = t // 640 - up
    return out + [v]


def test_digit_bounds():
    k = np.arange(-2 ** 17, 2 ** 17 + 1, dtype=np.int64)
    ds = split_k(k)
    assert all(np.abs(d).max() <= 32 for d in ds)
    np.testing.assert_array_equal(ds[0] + 64 * ds[1] + 4096 * ds[2], k)
    rng = np.random.default_rng(3)
    v = np.concatenate([rng.integers(-MOST, MOST + 1, 200000), np.arange(-2000, 2001), MOST - np.arange(2000),
                        np.arange(2000) - MOST]).astype(np.int64)
    ds = split_rho(v)
    assert all(np.abs(d).max() <= 320 for d in ds[:2]) and np.abs(ds[2]).max() <= 328
    np.testing.assert_array_equal(ds[0] + 640 * ds[1] + 640 ** 2 * ds[2], v)
    assert 32 * 328 * SEG < 2 ** 24


@pytest.mark.parametrize("N,L", [(1536, 2 ** 18 - 1), (1537, 94000), (4000, 2 ** 18 - 1)])
def test_combination_gives_k_rho(N, L):
    rng = np.random.default_rng(N)
    c = (L + 1) // 2
    K = rng.integers(0, L + 1, size=(16, N), dtype=np.int64)
    K[0], K[1], K[2] = 0, L, rng.choice([0, L], N)
    rho = rng.integers(-MOST, MOST + 1, size=(N, 3), dtype=np.int64)
    rho[:, 0] = MOST
    got = np.zeros((16, 3), dtype=np.int64)
    for j in range(0, N, SEG):
        for k, kd in enumerate(split_k(K[:, j:j + SEG] - c)):
            for p, rd in enumerate(split_rho(rho[j:j + SEG])):
                s = kd @ rd
                assert np.abs(s).max() < 2 ** 24
                got += s * 64 ** k * 640 ** p
    np.testing.assert_array_equal(got + c * rho.sum(0), K @ rho)
