"""The one-launch Arnoldi step (csrc/arnoldi.cu) at the widths of its kernels: a basis of one, the widest that are held in
registers, the ones that are read twice and the widest, against the oracle's solver, and two lockstep instances against
single solves.  Tolerances are those of the solver tests with restarts: the same iterations, misfits within 1e-5,
solutions within 1e-8.
"""
import numpy as np
import pytest

from giem2g_b200.synthetic import csiga_from_sigma
from tests.helpers import random_sigma, rel, tiny_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("outer,inner", [(31, 1), (31, 2), (3, 7), (4, 15), (4, 16), (3, 31), (1, 1)])
def test_basis_widths(g2lib, orc, outer, inner):
    m = tiny_model(8, 8, 4, freq=10.0)
    sig = random_sigma(m, seed=4, lo=-2.5, hi=0.5)
    symm, asym = orc.green_tensor(m)
    op = g2lib.IEOperator.from_model(m)
    op.set_background(m.csigma, m.thick, m.omega)
    op.set_ie_kernel_spatial(symm, asym)
    op.calc_fft_of_ie_kernel()
    csiga = csiga_from_sigma(sig, m.freq)
    op.set_anomaly_conductivity(csiga)
    sh, ah = orc.tensor_spectrum(m.Nx, m.Ny, m.Nz, symm, asym)
    csigb, sqsigb = orc.background_cells(m)
    E0 = [orc.plane_wave(m, p) for p in (1, 0)]
    ref = [orc.solve(m.Nx, m.Ny, m.Nz, sh, ah, csiga, csigb, sqsigb, m.dz, e, None, outer, inner, 60, 1e-9) for e in E0]
    got, info = op.solve_equation(E0[0], tol=1e-9, max_restart=60, outer_buf=outer, inner_buf=inner)
    Eo, io, ho = ref[0]
    assert info.iterations == io.iterations and info.stat == io.stat
    assert np.allclose(info.misfits, ho, rtol=1e-5, atol=0)
    assert rel(got, Eo) < 1e-8
    batch = g2lib.Batch([op, op], outer_buf=outer, inner_buf=inner, precision=0, max_restart=60)
    sols, infos = batch.solve(E0, tol=1e-9)
    batch.delete()
    for s, i, (Er, ir, _) in zip(sols, infos, ref):
        assert i.iterations == ir.iterations and rel(s, Er) < 1e-8
    op.delete()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", [(2, 2, 1), (2, 4, 3), (16, 8, 9), (32, 16, 7)])
def test_cycle_start(g2lib, orc, shape, precision):
    """The two launches that start an inner cycle, from one block to many, for one, two and three lockstep instances of
    which one has a vanishing right side; mixed precision: converged, within 1e-5 of the oracle's FP64 solution."""
    m = tiny_model(*shape, freq=10.0)
    sig = random_sigma(m, seed=6, lo=-2.5, hi=0.5)
    symm, asym = orc.green_tensor(m)
    op = g2lib.IEOperator.from_model(m)
    op.set_background(m.csigma, m.thick, m.omega)
    op.set_ie_kernel_spatial(symm, asym)
    op.calc_fft_of_ie_kernel()
    csiga = csiga_from_sigma(sig, m.freq)
    op.set_anomaly_conductivity(csiga)
    sh, ah = orc.tensor_spectrum(m.Nx, m.Ny, m.Nz, symm, asym)
    csigb, sqsigb = orc.background_cells(m)
    E0 = [orc.plane_wave(m, p) for p in (1, 0)]
    tol = 1e-6 if precision else 1e-9
    ref = [orc.solve(m.Nx, m.Ny, m.Nz, sh, ah, csiga, csigb, sqsigb, m.dz, e, None, 10, 10, 60, tol) for e in E0]
    got, info = op.solve_equation(E0[0], tol=tol, max_restart=60, outer_buf=10, inner_buf=10, precision=precision)
    batch = g2lib.Batch([op, op, op], outer_buf=10, inner_buf=10, precision=precision, max_restart=60)
    sols, infos = batch.solve([E0[0], np.zeros_like(E0[0]), E0[1]], tol=tol)
    batch.delete()
    assert infos[1].stat == 1 and not np.any(sols[1])
    for s, i, (Er, ir, _) in ((got, info, ref[0]), (sols[0], infos[0], ref[0]), (sols[2], infos[2], ref[1])):
        assert i.stat == ir.stat and (precision or i.iterations == ir.iterations)
        assert rel(s, Er) < (1e-5 if precision else 1e-8)
    op.delete()
