"""Band densities whose units pass in groups (a set's slices beyond the budget): any group gives
the sums of a single group, bit for bit, since the units are added in order; the single group is
pinned to the FP64 transforms elsewhere (test_kset_fields_gpu.py, test_any_lengths_gpu.py).
Groups of one, two and five of seven units, the last one ragged, complex and Gamma, overwriting
and accumulating, for the tuned, the any-length and the run-time plane kernels; and the buffer's
growth call by call."""
import numpy as np
import pytest

from baandi_b200 import _lib as L
from baandi_b200.hamiltonian import ComplexHamiltonian, KPointSet, RealGammaHamiltonian
from baandi_b200.operands import PlaneWaves

pytestmark = pytest.mark.gpu

DIMS = [(25, 25, 25), (45, 45, 45), (24, 30, 18), (8, 125, 30)]


def operators(ctx, dims, gamma, nk, units):
    import torch
    half = np.asarray([(x, y, z) for x in range(0, 3) for y in range(-2, 3) for z in range(-2, 3)
                       if (x, y, z) > (0, 0, 0)], np.int32)
    miller = np.concatenate([np.zeros((1, 3), np.int32), half, -half])
    miller = miller[np.lexsort((miller[:, 2], miller[:, 1], miller[:, 0], np.sum(miller * miller, axis=1)))]
    q = miller * 0.1
    ops = []
    for _ in range(nk):
        pw = PlaneWaves(miller, q, np.sum(q * q, axis=1), (0.0, 0.0, 0.0))
        cls = RealGammaHamiltonian if gamma else ComplexHamiltonian
        ops.append(cls.new_owned(pw, dims, None, 2 * units if gamma else units, ctx))
        ops[-1].set_stream(torch.cuda.current_stream().cuda_stream)
    return ops, len(miller)


@pytest.mark.parametrize("gamma", [False, True])
@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_groups(ctx, dims, gamma):
    import torch
    lib = L.load()
    nk, units = 3, 7
    cols = 2 * units - 1 if gamma else units   # Gamma: an odd column count, the last unit half empty
    ops, n = operators(ctx, dims, gamma, nk, units)
    ks = KPointSet(ops, ctx)
    ks.set_stream(torch.cuda.current_stream().cuda_stream)
    gen = torch.Generator(device="cuda").manual_seed(3)
    xs = [torch.randn((cols, n), dtype=torch.float64 if gamma else torch.complex128, device="cuda", generator=gen)
          for _ in range(nk)]
    w = np.random.default_rng(1).uniform(0.1, 1.0, (nk, cols))
    add = torch.rand(dims, dtype=torch.float64, device="cuda", generator=gen)
    slice_bytes = 8 * int(np.prod(dims))
    want = ks.band_density_sum(xs, w, 3.0)
    want_add = ks.band_density_sum(xs, w, 3.0, out=add.clone(), accumulate=True)
    one = ops[1].band_density_sum(xs[1], w[1], 3.0)
    for group in (1, 2, 5):
        assert lib.bg_test_density_budget(ops[1].handle, ks.handle, group * nk * slice_bytes) == 0
        assert torch.equal(ks.band_density_sum(xs, w, 3.0), want)
        assert torch.equal(ks.band_density_sum(xs, w, 3.0, out=add.clone(), accumulate=True), want_add)
        assert lib.bg_test_density_budget(ops[1].handle, None, group * slice_bytes) == 0
        assert torch.equal(ops[1].band_density_sum(xs[1], w[1], 3.0), one)
    total = sum(ops[k].band_density_sum(xs[k], w[k], 3.0) for k in range(nk))
    assert torch.linalg.vector_norm(total - want) <= 1e-15 * nk * torch.linalg.vector_norm(want)
    ks.close()


def test_growing_calls(ctx):
    import torch
    dims, units = (24, 30, 18), 12
    ops, n = operators(ctx, dims, False, 1, units)
    ks = KPointSet(ops, ctx)
    ks.set_stream(torch.cuda.current_stream().cuda_stream)
    x = torch.randn((units, n), dtype=torch.complex128, device="cuda")
    w = np.linspace(0.5, 1.0, units)
    for cols in (1, 3, 2, 12, 5):   # each width on the buffer that the calls before it left
        fresh, _ = operators(ctx, dims, False, 1, cols)
        want = fresh[0].band_density_sum(x[:cols].contiguous(), w[:cols], 2.0)
        assert torch.equal(ops[0].band_density_sum(x[:cols].contiguous(), w[:cols], 2.0), want)
        assert torch.equal(ks.band_density_sum([x[:cols].contiguous()], w[None, :cols], 2.0), want)
    ks.close()
