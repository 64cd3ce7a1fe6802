"""FP64 products on the int8 tensor cores (csrc/gemm_rns.cu) against extended-precision sums:
tile edges, K remainders, every op, split and unsplit A, several products in one launch, badly
scaled, graded and non-finite input.

Bound of an entry: a row is scaled by a power of two to a 2-norm of 2^57.3 .. 2^58.3 and
every real part rounded to an integer, so each of its K complex values is off by at most
2^-1/2 and, by Cauchy-Schwarz, the sum of K products by sqrt(K / 2) (1 / |a| + 1 / |b|) of the
norms' product in scaled units: sqrt(2 K) 2^-57.3 |a| |b|.  The result is rounded to FP64
twice more (2^-51 |c| covers that and the final addition).  A B with A split in the launch
takes the norms of A D and D^-1 B, D_k the power of two below max_j |B_kj| / |b_j| (real and
imaginary parts apart, norms up to a factor of two): 4 |a D'| |b / D'| with D' that ratio itself.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from baandi_b200 import _lib as L

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (64, 16, 3), (127, 15, 64), (128, 16, 65), (129, 17, 63), (255, 128, 130), (257, 129, 1000),
         (300, 256, 1144), (256, 257, 1146), (513, 40, 1152), (40, 300, 4099)]


def product(mode, a, b, c, op, presplit):
    """a, b, c: CUDA complex128 rows = columns of the column-major matrices."""
    lib = L.load()
    m = a.shape[0] if mode == 0 else a.shape[1]
    k, n = b.shape[1], b.shape[0]
    rc = lib.bg_test_residue_product(ctypes.c_int32(mode), ctypes.c_int64(m), ctypes.c_int64(n), ctypes.c_int64(k),
                                     ctypes.c_void_p(a.data_ptr()), ctypes.c_int64(a.shape[1]),
                                     ctypes.c_void_p(b.data_ptr()), ctypes.c_int64(k),
                                     ctypes.c_void_p(c.data_ptr()), ctypes.c_int64(m), ctypes.c_int32(op),
                                     ctypes.c_int32(presplit))
    assert rc == 0, rc


def matrices(mode, m, n, k, seed):
    rng = np.random.default_rng(seed)
    z = lambda r, c: rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))
    a = z(m, k) if mode == 0 else z(k, m)
    return a, z(n, k), z(n, m)


def exact(mode, a, b, balanced=False, skip=()):
    """(n, m) product in 80-bit arithmetic and the bound's norm products.  skip: columns of B that
    the balance does not see (non-finite ones)."""
    left = (a.conj() if mode == 0 else a.T).astype(np.clongdouble)
    la, lb = np.abs(left).astype(np.float64), np.abs(b)
    factor = 1.0
    if balanced and mode == 1:
        parts, size = np.maximum(np.abs(b.real), np.abs(b.imag)), np.linalg.norm(b, axis=1)
        rel = parts / np.where(size > 0.0, size, 1.0)[:, None]
        d = np.maximum(np.max(np.delete(rel, list(skip), axis=0), axis=0), 2.0 ** -58)
        la, lb, factor = la * d, lb / d, 4.0
    norms = factor * np.linalg.norm(lb, axis=1)[:, None] * np.linalg.norm(la, axis=1)[None, :]
    return b.astype(np.clongdouble) @ left.T, norms


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("m,n,k", SIZES)
def test_tile_edges(mode, m, n, k):
    torch = pytest.importorskip("torch")
    op, presplit = (m + n + k) % 3, (m + k) % 2
    a, b, c0 = matrices(mode, m, n, k, m + 7 * n + 31 * k)
    a[..., 0] *= 1e-3  # a graded row or column
    c = torch.from_numpy(c0.copy()).cuda()
    product(mode, torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), c, op, presplit)
    want, norms = exact(mode, a, b, not presplit)
    if op == 1:
        want = c0 + want
    if op == 2:
        want = c0 - want
    diff = np.abs((c.cpu().numpy() - want).astype(np.complex128))
    bound = np.sqrt(2 * k) * 2.0 ** -57.3 * norms + 2.0 ** -51 * (np.abs(want).astype(np.float64) + (np.abs(c0) if op else 0.0))
    assert np.all(diff <= bound), float(np.max(diff / bound))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("power", [660, 940])   # 940: one scale alone overflows the intermediate
def test_scales_and_nonfinite(mode, power):
    torch = pytest.importorskip("torch")
    m, n, k = 130, 33, 200
    a, b, c0 = matrices(mode, m, n, k, 5)
    rows = a if mode == 0 else a.T          # row i of the left factor
    rows[2] = 0.0
    b[1] = 0.0
    want, norms = exact(mode, a, b, True, skip=[3])
    ea, eb = np.zeros(m, np.int64), np.zeros(n, np.int64)
    ea[0], ea[1], eb[0] = power, -power, -power   # squares overflow and underflow; one product vanishes
    rows *= np.ldexp(1.0, ea)[:, None]
    b *= np.ldexp(1.0, eb)[:, None]
    rows[5, 11] = np.inf
    b[3, 7] = np.nan
    c = torch.from_numpy(c0.copy()).cuda()
    product(mode, torch.from_numpy(np.ascontiguousarray(a)).cuda(), torch.from_numpy(b).cuda(), c, 0, 0)
    got = c.cpu().numpy()
    assert np.all(np.isnan(got[3].real)) and np.all(np.isnan(got[:, 5].real))
    fine = np.ix_(np.arange(n) != 3, np.arange(m) != 5)
    e = (eb[:, None] + ea[None, :])[fine]
    w = want[fine].astype(np.complex128)
    w = np.ldexp(w.real, e) + 1j * np.ldexp(w.imag, e)
    bound = np.ldexp(np.sqrt(2 * k) * 2.0 ** -57.3 * norms[fine], e) + 2.0 ** -51 * np.abs(w) + 4 * np.finfo(np.float64).smallest_subnormal
    assert np.all(np.abs(got[fine] - w) <= bound)


@pytest.mark.parametrize("steep", [0.35, 1.0])
def test_graded_rotation(steep):
    """Ritz vectors with steep tails and corrections with slow ones, rotated with coefficients of
    order one and 1e-8: every entry within the FP64 sum's own bound, K 2^-53 (|A| |B|)."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(0)
    m, n = 1500, 100
    z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    q2 = np.linspace(0.01, 30.0, m)
    a = np.concatenate([z(n, m) * np.exp(-steep * q2), z(n, m) / (1.0 + q2) ** 2])
    a /= np.linalg.norm(a, axis=1)[:, None]
    b = np.concatenate([np.linalg.qr(z(n, n))[0], 1e-8 * z(n, n)], axis=1)
    c = torch.zeros((n, m), dtype=torch.complex128, device="cuda")
    product(1, torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), c, 0, 0)
    want, _ = exact(1, a, b)
    bound = 2 * n * 2.0 ** -53 * (np.abs(b) @ np.abs(a))
    diff = np.abs((c.cpu().numpy() - want).astype(np.complex128))
    assert np.all(diff <= bound), float(np.max(diff / bound))


@pytest.mark.parametrize("presplit", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_several_products(mode, presplit):
    """Ragged products of one launch, empty slots among them, in a workspace made for larger ones
    (fewer K splits than the products alone would take), as the Davidson's slots and k points."""
    import torch
    lib = L.load()
    shapes = [(300, 96, 2100), (0, 0, 0), (129, 17, 4099), (513, 257, 70), (40, 1, 1300), (0, 5, 9), (256, 128, 64)]
    rng = np.random.default_rng(11)
    hosts, devs = [], []
    for i, (m, n, k) in enumerate(shapes):
        a, b, c = matrices(mode, max(m, 1), max(n, 1), max(k, 1), 40 + i)
        a = a * np.exp(rng.uniform(-8, 8, a.shape[1]))[None, :] if i % 2 else a
        hosts.append((a, b, c))
        devs.append([torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (a, b, c)])
    count = len(shapes)
    ptrs = lambda j: (ctypes.c_void_p * count)(*[d[j].data_ptr() for d in devs])
    lds = lambda j: (ctypes.c_int64 * count)(*[d[j].shape[1] for d in devs])
    flat = (ctypes.c_int64 * (3 * count))(*[v for s in shapes for v in s])
    for bounds in (None, (600, 300, 5000), (513, 257, 4100)):
        bp = (ctypes.c_int64 * 3)(*bounds) if bounds else None
        for d, h in zip(devs, hosts):
            d[2].copy_(torch.from_numpy(h[2]))
        rc = lib.bg_test_residue_products(mode, count, flat, ptrs(0), lds(0), ptrs(1), lds(1), ptrs(2), lds(2), 1,
                                          presplit, bp, -1)
        assert rc == 0
        for (m, n, k), h, d in zip(shapes, hosts, devs):
            got = d[2].cpu().numpy()
            if m == 0 or n == 0 or k == 0:
                assert np.array_equal(got, h[2])   # an empty slot's output is not touched
                continue
            want, norms = exact(mode, h[0], h[1], not presplit)
            want = h[2] + want
            diff = np.abs((got - want).astype(np.complex128))
            bound = np.sqrt(2 * k) * 2.0 ** -57.3 * norms + 2.0 ** -51 * (np.abs(want).astype(np.float64) + np.abs(h[2]))
            assert np.all(diff <= bound), ((m, n, k), float(np.max(diff / bound)))
