"""Davidson solves whose Grams and rotations run as residue products (csrc/kset_davidson.cu,
k_dv_rns_descs): a k-point set just above the size where they pay, against the same solves on the
FP64 tiles, which the small solves pin to the reference (test_kset_davidson_gpu.py).  The tiles are
reached through short memory, which must also leave the results and every later call alone.

Bound: both sides form each product to a few eps of its operands' norms, and the iterations'
rotations carry that to the Ritz values; a start block changed in its last bit moves them by
5e-15 and 3e-14 of their size on the timed cells, so 1e-12 holds with room."""
import ctypes

import numpy as np
import pytest

from baandi_b200 import _lib as L
from baandi_b200 import davidson as DV
from baandi_b200 import systems as W
from baandi_b200.hamiltonian import ComplexHamiltonian, Context, KPointSet

pytestmark = pytest.mark.gpu

BANDS, RTOL = 200, 1e-12   # capacity 400: 400 x 200 x 23,847 is 1.9e9, the products pay from 1.5e9


def state(op, ks):
    p, r = ctypes.c_int32(), ctypes.c_int32()
    assert L.load().bg_test_residue_state(op.handle, ks.handle, ctypes.byref(p), ctypes.byref(r)) == 0
    return p.value, r.value


class Problem:
    """Si64 at Gamma and at one more k point (other row counts), potential set."""

    def __init__(self, free=-1):
        import torch
        self.ctx = Context(0)
        self.lib = L.load()
        assert self.lib.bg_test_memory(self.ctx.handle, free, 0) == 0
        self.w = W.si64_gamma()
        self.ops = []
        for k in ((0.0, 0.0, 0.0), (0.25, 0.25, 0.0)):
            pw = self.w.plane_waves(k)
            self.ops.append(ComplexHamiltonian.new_owned(pw, self.w.dims(), self.w.nonlocal_table(pw), BANDS, self.ctx))
            self.ops[-1].set_stream(torch.cuda.current_stream().cuda_stream)
        self.ks = KPointSet(self.ops, self.ctx)
        self.ks.set_stream(torch.cuda.current_stream().cuda_stream)
        v = torch.from_numpy(self.w.ionic_potential()).cuda()
        self.ks.set_potential_device(v, 1)
        mean = float(v.mean())
        self.starts = [torch.from_numpy(np.ascontiguousarray(self.w.random_block(op.npw, BANDS, seed_offset=9 + i).T)).cuda()
                       for i, op in enumerate(self.ops)]
        self.diags = [torch.from_numpy(op.diagonal_static() + mean).cuda() for op in self.ops]

    def solve(self, tensor=False, iterations=4):
        o = DV.Options(BANDS, 1e-10, 128, max_iterations=iterations,
                       apply_precision="tensor" if tensor else "fp64")
        sols = DV.solve_kset(self.ks, self.starts, self.diags, o)
        return sols, np.stack([s.eigenvalues for s in sols])

    def close(self):
        self.ks.close()
        for op in self.ops:
            op.close()


def test_residue_solve_matches_the_tiles():
    import torch
    a, b = Problem(), Problem(free=0)
    sa, ea = a.solve()
    sb, eb = b.solve()
    assert state(a.ops[0], a.ks) == (1, 1) and state(b.ops[0], b.ks) == (0, 0)
    assert sum(s.contractions for s in sa) > 0   # contractions exchange the basis buffers
    assert [s.contractions for s in sa] == [s.contractions for s in sb]
    assert np.max(np.abs(ea - eb)) <= RTOL * np.max(np.abs(eb))
    # the density of all bands, which no phase or rotation among them enters: rounding times the
    # spectrum's width over the level spacing at the last band, 1e4 to 1e5
    wts = np.ones((2, BANDS))
    rho = [p.ks.band_density_sum([s.eigenvectors for s in ss], wts, 1.0) for p, ss in ((a, sa), (b, sb))]
    assert torch.linalg.vector_norm(rho[0] - rho[1]) <= 1e-10 * torch.linalg.vector_norm(rho[1])
    # the same solve again (captured iterations replayed)
    assert np.array_equal(a.solve()[1], ea)
    a.close()
    b.close()


def test_short_memory_gives_the_buffers_back():
    """A tensor-form solve that finds no memory for its own buffers takes the residue buffers'
    (and the captured iterations that hold their addresses) and runs."""
    a, b = Problem(), Problem()
    first = a.solve()[1]
    b.solve()
    want = b.solve(tensor=True)[1]
    assert a.lib.bg_test_memory(a.ctx.handle, -1, 1) == 0
    got = a.solve(tensor=True)[1]
    assert state(a.ops[0], a.ks) == (1, 0) and state(b.ops[0], b.ks) == (1, 1)
    assert np.max(np.abs(got - want)) <= 1e-6 * np.max(np.abs(want))   # the tensor phase's own precision
    again = a.solve()[1]                                               # FP64, captured anew on the tiles
    assert np.max(np.abs(again - first)) <= RTOL * np.max(np.abs(first))
    a.close()
    b.close()


def test_applies_without_memory_for_workspaces():
    """Panels made, then no spare memory at the first apply: the tiles serve, also later."""
    import torch
    a, b = Problem(), Problem(free=0)
    assert a.lib.bg_test_memory(a.ctx.handle, 0, 0) == 0
    ya, yb = a.ks.apply_blocks(a.starts), b.ks.apply_blocks(b.starts)
    assert all(torch.equal(x, y) for x, y in zip(ya, yb))
    y = a.ops[0].apply_block(a.starts[0])
    assert torch.linalg.vector_norm(y - ya[0]) <= 1e-14 * torch.linalg.vector_norm(y)
    a.close()
    b.close()
