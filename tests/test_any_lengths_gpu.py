"""Apply and band density on boxes of every line length (csrc/fft_any.cuh, planes_any.cu) and of
lengths outside it, against numpy's FFT: each length once along every axis, one and two plane
blocks per SM, odd unit counts; densities in one group of units and in several.  Bound: FP64 transforms of up to 128^3
points, errors of a few eps times log2 N of the column's norm (the suite's 1e-12 parity bound
holds them with room; 1e-13 here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [15, 16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108, 120, 128]
BOXES = [(n, LENGTHS[(i + 5) % 15], LENGTHS[(i + 11) % len(LENGTHS)]) for i, n in enumerate(LENGTHS)]
BOXES += [(LENGTHS[(i + 3) % 14], n, LENGTHS[(i + 8) % 20]) for i, n in enumerate(LENGTHS)]
BOXES += [(108, 100, 16), (96, 96, 20), (128, 108, 15), (8, 125, 30), (60, 9, 12), (1, 25, 24), (45, 45, 60)]


def basis(dims, rng, count):
    """Distinct grid points, G = 0 first, filling a ball of the box's lowest frequencies."""
    m = np.stack(np.meshgrid(*[np.arange(-((d - 1) // 2), d // 2 + 1) for d in dims], indexing="ij"), -1).reshape(-1, 3)
    m = m[np.all((m >= -(np.asarray(dims) // 2)) & (m <= (np.asarray(dims) - 1) // 2), axis=1)]
    r2 = np.sum((m / np.maximum(np.asarray(dims) / 4.0, 1.0)) ** 2, axis=1)
    order = np.argsort(r2, kind="stable")[: max(4 * count, 1)]
    pick = np.sort(rng.choice(len(order), size=min(count, len(order)), replace=False))
    pick[0] = 0
    return m[order[np.unique(pick)]].astype(np.int32)


@pytest.mark.parametrize("dims", BOXES, ids=lambda d: "x".join(map(str, d)))
def test_box(ctx, dims):
    import torch
    from baandi_b200.hamiltonian import ComplexHamiltonian, KPointSet
    from baandi_b200.operands import PlaneWaves
    rng = np.random.default_rng(sum(dims))
    miller = basis(dims, rng, 700)
    n, cols = len(miller), 5
    q = miller.astype(np.float64) * 0.1
    pw = PlaneWaves(miller, q, np.sum(q * q, axis=1), (0.1, 0.0, 0.0))
    op = ComplexHamiltonian.new_owned(pw, dims, None, cols, ctx)
    v = rng.standard_normal(dims)
    op.set_owned_potential(v, 1)
    x = np.asfortranarray(rng.standard_normal((n, cols)) + 1j * rng.standard_normal((n, cols)))
    idx = tuple(np.mod(miller, np.asarray(dims)).T)
    box = np.zeros((cols,) + tuple(dims), np.complex128)
    box[(slice(None),) + idx] = x.T
    psi = np.fft.ifftn(box, axes=(1, 2, 3)) * np.prod(dims)
    want = np.fft.fftn(psi * v, axes=(1, 2, 3))[(slice(None),) + idx].T / np.prod(dims) + (0.5 * pw.kpg2)[:, None] * x
    got = op.apply_block(x)
    assert np.linalg.norm(got - want) <= 1e-13 * np.linalg.norm(want)
    w = rng.uniform(0.1, 2.0, cols)
    rho_want = np.einsum("b,bxyz->xyz", w, np.abs(psi) ** 2) / 7.0
    rho = op.band_density_sum(x, w, 7.0)
    assert np.linalg.norm(rho - rho_want) <= 1e-13 * np.linalg.norm(rho_want)
    # groups of two units and a last one of one: the same sums in the same order
    assert op._lib.bg_test_density_budget(op.handle, None, 2 * 8 * int(np.prod(dims))) == 0
    assert np.array_equal(op.band_density_sum(x, w, 7.0), rho)
    ks = KPointSet([op], ctx)
    ks.set_stream(torch.cuda.current_stream().cuda_stream)
    rho = ks.band_density_sum([torch.from_numpy(np.ascontiguousarray(x.T)).cuda()], w[None, :], 7.0)
    assert np.linalg.norm(rho.cpu().numpy() - rho_want) <= 1e-13 * np.linalg.norm(rho_want)
    ks.close()
    op.close()
