"""The error budget of the double-float reciprocal kernels' FP32 vectors, restated
on the CPU: wave vectors whose force weight |G| c(n) is below 1e-8 of the largest
(RECIP_DF_SPLIT, read from the source) summed in float32, the others in FP64, next
to all of them in FP64.  The kernels rest on the float32 ones leaving below 1e-14 of
the reciprocal forces' norm.
"""
import math
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "md-lab_gb300", "csrc", "xmd_kernels.cuh")


def _line():
    return float(re.search(r"RECIP_DF_SPLIT = ([0-9.e+-]+);", open(SRC).read()).group(1))


def _vectors(nsum, alphaL):
    r = np.arange(-nsum, nsum + 1)
    n = np.stack(np.meshgrid(r[nsum:], r, r, indexing="ij"), -1).reshape(-1, 3)
    half = (n[:, 0] > 0) | ((n[:, 0] == 0) & ((n[:, 1] > 0) | ((n[:, 1] == 0) & (n[:, 2] > 0))))
    n = n[half]
    g2 = (n ** 2).sum(1).astype(np.float64)
    c = np.exp(-math.pi ** 2 * g2 / alphaL ** 2) / g2
    return n, c, np.sqrt(g2) * c


def _phases(x, n, cdtype):
    """e_xy and e_z of every vector and particle, harmonics rounded from FP64"""
    h = [np.exp(2j * np.pi * np.arange(np.abs(n).max() + 1)[:, None] * x[:, d]).astype(cdtype) for d in range(3)]
    row = [np.where(n[:, d, None] < 0, np.conj(h[d][np.abs(n[:, d])]), h[d][np.abs(n[:, d])]) for d in range(3)]
    return (row[0] * row[1]).astype(cdtype), row[2].astype(cdtype)


def _forces(x, n, c, dtype, cdtype):
    """sum over n of c n Im(e conj(S)), as the kernels add it: S from products of e_xy and e_z, eight particles
    at a time in dtype and those sums exactly; the forces' terms of a column (n_x, n_y) in dtype, the columns' exactly"""
    exy, ez = _phases(x, n, cdtype)
    e = (exy * ez).astype(cdtype)
    S = sum(e[:, i:i + 8].sum(1, dtype=cdtype).astype(np.complex128) for i in range(0, len(x), 8))
    W = (c * np.conj(S)).astype(cdtype)
    F = np.zeros((len(x), 3))
    columns = {}
    for i, (a, b, _) in enumerate(n):
        columns.setdefault((a, b), []).append(i)
    for (a, b), at in columns.items():
        U = np.zeros(len(x), dtype=cdtype)
        V = np.zeros(len(x), dtype=cdtype)
        for i in at:
            U = (U + (ez[i] * W[i]).astype(cdtype)).astype(cdtype)
            V = (V + dtype(n[i, 2]) * (ez[i] * W[i]).astype(cdtype)).astype(cdtype)
        T, Z = (exy[at[0]] * U).astype(cdtype).imag, (exy[at[0]] * V).astype(cdtype).imag
        F += np.stack([dtype(a) * T, dtype(b) * T, Z], 1).astype(np.float64)
    return F


@pytest.mark.parametrize("N,nsum,alphaL", [(20, 6, 5.6), (64, 8, 5.6), (128, 10, 5.6), (40, 10, 7.0), (40, 9, 4.0)])
def test_vectors_below_the_line_fit_float32(N, nsum, alphaL):
    x = np.random.default_rng(N).uniform(0, 1, (N, 3))
    n, c, w = _vectors(nsum, alphaL)
    kept = w >= 1e-17 * w.max()
    small = kept & (w < _line() * w.max())
    assert small.any() and (kept & ~small).any()
    whole = _forces(x, n[kept], c[kept], np.float64, np.complex128)
    part = _forces(x, n[small], c[small], np.float64, np.complex128)
    part32 = _forces(x, n[small], c[small], np.float32, np.complex64).astype(np.float64)
    off = np.linalg.norm(part32 - part) / np.linalg.norm(whole)
    print("%d of %d vectors in float32: %.1e of the norm" % (small.sum(), kept.sum(), off))
    assert off <= 1e-14
