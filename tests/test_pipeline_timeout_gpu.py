"""A pipeline wait of the residue products that gives up: the kernel ends by itself and says so,
the library reports BG_ETIMEOUT before whatever the wrong values led to, and the next call is
clean.  The wait runs out on its try limit; the library's side sees the error bit set on the
operator as the kernel sets it."""
import ctypes

import numpy as np
import pytest

from baandi_b200 import _lib as L
from baandi_b200 import davidson as DV
from baandi_b200 import systems as W
from baandi_b200.hamiltonian import ComplexHamiltonian, DenseOperator, KPointSet, SolverError
from oracle import davidson_ref as D

pytestmark = pytest.mark.gpu

GAVE_UP = 4   # rns::kErrBit


def code_of(call):
    with pytest.raises(SolverError) as e:
        call()
    return e.value.code


@pytest.mark.parametrize("mode", [0, 1])
def test_wait_limit(mode):
    import torch
    m, n, k = 300, 70, 900   # several K tiles: the copies in flight at the give-up are waited for
    a = torch.randn((m, k) if mode == 0 else (k, m), dtype=torch.complex128, device="cuda")
    b = torch.randn((n, k), dtype=torch.complex128, device="cuda")
    c = torch.zeros((n, m), dtype=torch.complex128, device="cuda")
    lib = L.load()
    shape = (ctypes.c_int64 * 3)(m, n, k)
    one = lambda v: (ctypes.c_int64 * 1)(v)
    ptr = lambda t: (ctypes.c_void_p * 1)(t.data_ptr())

    def product(limit):
        return lib.bg_test_residue_products(mode, 1, shape, ptr(a), one(a.shape[1]), ptr(b), one(k), ptr(c), one(m), 0,
                                            0, None, limit)
    assert product(0) == L.BG_ETIMEOUT
    assert product(-1) == L.BG_OK
    want = b @ (a.conj().T if mode == 0 else a)
    assert torch.linalg.vector_norm(c - want) <= 1e-13 * torch.linalg.vector_norm(want)


def test_solve_reports_the_wait_before_its_consequences(ctx):
    lib = L.load()
    dim, bands = 32, 6
    hs = [D.dct_fixture(dim, False).astype(np.complex128), D.dct_fixture(dim, True).astype(np.complex128)]
    ops = [DenseOperator(h, dim, ctx) for h in hs]
    ks = KPointSet(ops, ctx)
    good = [D.dct_start(dim, bands).astype(np.complex128) for _ in hs]
    bad = [good[0], good[1].copy()]
    bad[1][:, 1] = bad[1][:, 0]
    diags = [np.diag(h).real.copy() for h in hs]
    opts = DV.Options(bands, 1e-10, bands, max_iterations=100)
    solve = lambda starts: DV.solve_kset(ks, starts, diags, opts)
    want = solve(good)
    for starts, then in ((bad, L.BG_EINVAL), (good, None)):
        for k in (0, 1):
            assert lib.bg_test_raise_error(ops[k].handle, GAVE_UP) == 0
            assert code_of(lambda: solve(starts)) == L.BG_ETIMEOUT
            ks.sync()   # reported once
            if then is not None:
                assert code_of(lambda: solve(starts)) == then
                ks.sync()
    for x, y in zip(want, solve(good)):
        assert np.array_equal(x.eigenvalues, y.eigenvalues)
    ks.close()


def test_potential_install_and_sync_name_the_wait(ctx):
    import torch
    lib = L.load()
    w = W.si8_k444()
    ops = []
    for i in (0, 5):
        pw = w.plane_waves(w.kpoints[i][0])
        ops.append(ComplexHamiltonian.new_owned(pw, w.dims(), w.nonlocal_table(pw), 4, ctx))
        ops[-1].set_stream(torch.cuda.current_stream().cuda_stream)
    ks = KPointSet(ops, ctx)
    ks.set_stream(torch.cuda.current_stream().cuda_stream)
    v = torch.from_numpy(w.ionic_potential()).cuda()
    ks.set_potential_device(v, 1)
    assert lib.bg_test_raise_error(ops[0].handle, GAVE_UP) == 0
    assert code_of(lambda: ks.set_potential_device(v, 2)) == L.BG_ETIMEOUT
    ks.set_potential_device(v, 3)
    for k, bits in ((0, 1), (1, GAVE_UP)):   # the wait outranks another operator's non-finite block
        assert lib.bg_test_raise_error(ops[k].handle, bits) == 0
    assert code_of(ks.sync) == L.BG_ETIMEOUT
    ks.sync()
    ks.close()
