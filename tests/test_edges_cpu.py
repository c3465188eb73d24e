"""CPU model of the specialised edges of fft_edges.cuh (no GPU): the four-step
line transform with idle owners, every line position inside the padded line,
the radix-9 and prime-factor index maps, and the register mirror images the x
passes exchange by warp shuffles (fft_fast.cuh: separate_lines, join_lines)."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "fft_method_test_gb300", "csrc")


def _edges():
    out = {}
    src = open(os.path.join(CSRC, "fft_edges.cuh")).read()
    for n, r1, r2, tpl in re.findall(r"\bE\((\d+), (\d+), (\d+), (\d+)\)", src):
        out[int(n)] = (int(r1), int(r2), int(tpl))
    src = open(os.path.join(CSRC, "fft_fast.cuh")).read()
    for n, r1, r2, tpl in re.findall(
            r"struct Split<(\d+)>\s*{\s*static constexpr int R1 = (\d+), R2 = (\d+), TPL = (\d+);", src):
        out[int(n)] = (int(r1), int(r2), int(tpl))
    return out


EDGES = _edges()


def _dft(v, sign):
    k = np.arange(len(v))
    return np.exp(sign * 2j * np.pi * np.outer(k, k) / len(v)) @ v


def test_every_smooth_edge_is_listed_once():
    smooth = {2 ** a * 3 ** b * 5 ** c for a in range(9) for b in range(6) for c in range(4)}
    want = {n for n in smooth if 20 <= n <= 256} - {125, 128, 243, 250, 256} | {128, 256}
    assert set(EDGES) == want
    for n, (r1, r2, tpl) in EDGES.items():
        assert r1 * r2 == n and 32 % tpl == 0
        assert max(r1, r2) <= 20
        # values per thread and stage
        assert max(-(-r2 // tpl) * r1, -(-r1 // tpl) * r2) <= 40


@pytest.mark.parametrize("sign", [-1, 1])
def test_radix_9(sign):
    v = np.random.default_rng(9).standard_normal(9) + 0.25j
    a = v.astype(complex).copy()
    for n2 in range(3):
        a[[n2, 3 + n2, 6 + n2]] = _dft(a[[n2, 3 + n2, 6 + n2]], sign)
    w = np.exp(sign * 2j * np.pi * np.arange(9) / 9)
    for k1 in (1, 2):
        for n2 in (1, 2):
            a[3 * k1 + n2] *= w[k1 * n2]
    for k1 in range(3):
        a[3 * k1:3 * k1 + 3] = _dft(a[3 * k1:3 * k1 + 3], sign)
    out = a[[0, 3, 6, 1, 4, 7, 2, 5, 8]]
    np.testing.assert_allclose(out, _dft(v, sign), atol=1e-12)


@pytest.mark.parametrize("p,q", [(2, 3), (2, 5), (3, 5), (2, 9)])
def test_prime_factor_maps(p, q):
    r = p * q
    v = np.random.default_rng(r).standard_normal(r) + 0.5j
    a = np.array([[v[(q * i + p * j) % r] for j in range(q)] for i in range(p)])
    a = np.array([_dft(row, -1) for row in a])
    a = np.array([_dft(a[:, j], -1) for j in range(q)]).T
    np.testing.assert_allclose([a[k % p, k % q] for k in range(r)], np.fft.fft(v), atol=1e-12)


def _line(x, ra, rb, tpl, sign, span):
    n = ra * rb
    tw = np.exp(sign * 2j * np.pi * np.arange(n) / n)
    line = np.full(span, np.nan + 0j)
    for t in range(tpl):
        for j in range(-(-rb // tpl)):
            a = t + tpl * j
            if a < rb:  # owned
                v = _dft(np.array([x[rb * i + a] for i in range(ra)]), sign)
                for k in range(ra):
                    line[k * (rb + 1) + a] = v[k] * tw[a * k]
    out = np.full(n, np.nan + 0j)
    for t in range(tpl):
        for j in range(-(-ra // tpl)):
            k = t + tpl * j
            if k < ra:
                y = _dft(np.array([line[k * (rb + 1) + a] for a in range(rb)]), sign)
                for m in range(rb):
                    out[k + ra * m] = y[m]
    return out


@pytest.mark.parametrize("n", sorted(EDGES))
def test_line_matches_numpy(n):
    r1, r2, tpl = EDGES[n]
    span = n + max(r1, r2)
    x = np.random.default_rng(n).standard_normal(n) + 1j * np.random.default_rng(n + 1).standard_normal(n)
    np.testing.assert_allclose(_line(x, r1, r2, tpl, -1, span), np.fft.fft(x), atol=1e-9)
    np.testing.assert_allclose(_line(x, r2, r1, tpl, +1, span), n * np.fft.ifft(x), atol=1e-9)


@pytest.mark.parametrize("n", [n for n, (r1, r2, t) in sorted(EDGES.items()) if r1 % t == 0 and r2 % 2 == 0])
def test_mirror_registers(n):
    """Z[N - k] of z[t][j][m] = Z[t + TPL j + R1 m] in thread (TPL - t) % TPL."""
    r1, r2, tpl = EDGES[n]
    J = r1 // tpl
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n), rng.standard_normal(n)
    Z, A, B = np.fft.fft(a + 1j * b), np.fft.fft(a), np.fft.fft(b)
    z = [[[Z[t + tpl * j + r1 * m] for m in range(r2)] for j in range(J)] for t in range(tpl)]
    w = [[[None] * (r2 // 2) for _ in range(J)] for _ in range(tpl)]  # Z[N - k] as join_lines forms it
    for t in range(tpl):
        for m in range(r2 // 2):
            for j in range(J):
                k = t + tpl * j + r1 * m
                if t == 0:
                    zn = z[0][J - j][r2 - 1 - m] if j else z[0][0][(r2 - m) % r2]
                else:
                    zn = z[(tpl - t) % tpl][J - 1 - j][r2 - 1 - m]
                assert zn == Z[(n - k) % n]
                np.testing.assert_allclose((z[t][j][m] + np.conj(zn)) / 2, A[k], atol=1e-10)
                np.testing.assert_allclose((z[t][j][m] - np.conj(zn)) / 2j, B[k], atol=1e-10)
                w[t][j][m] = np.conj(A[k]) + 1j * np.conj(B[k])
    for t in range(tpl):  # the upper half of the inverse's inputs
        for m in range(r2 // 2):
            for j in range(J):
                if t == 0:
                    own = w[0][j + 1][m] if j + 1 < J else (w[0][0][m + 1] if m + 1 < r2 // 2 else Z[n // 2])
                else:
                    own = w[(tpl - t) % tpl][j][m]
                np.testing.assert_allclose(own, z[t][J - 1 - j][r2 - 1 - m], atol=1e-10)
