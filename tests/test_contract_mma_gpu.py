"""The tensor-core contraction (csrc/contract_mma.cu), the default of every operator, against the oracle apply.

Nz at the edges of its tiles: one z, whole and part tiles of 8 and of 4 z, the largest of each tile count, single-stage
rings, the largest Nz an operator takes (57); one unit per CTA and (the last rows) rings that wrap many times.
Tolerances are the apply's: 1e-12 for complex128, 2e-5 for complex64 and for pairs.
"""
import numpy as np
import pytest

from giem2g_b200.synthetic import csiga_from_sigma
from tests.helpers import random_sigma, random_spatial_tensor, random_vec, rel, tiny_model

pytestmark = pytest.mark.gpu

EDGES = [1, 4, 5, 8, 9, 12, 13, 17, 20, 21, 24, 25, 28, 29, 32, 33, 37, 40, 41, 45, 48, 49, 53, 57]


def _op(g2, orc, m):
    symm, asym = random_spatial_tensor(m, seed=13)
    op = g2.IEOperator.from_model(m)
    op.set_background(m.csigma, m.thick, m.omega)
    op.set_ie_kernel_spatial(symm, asym)
    op.calc_fft_of_ie_kernel()
    csiga = csiga_from_sigma(random_sigma(m, 4), m.freq)
    op.set_anomaly_conductivity(csiga)
    csigb, sqsigb = orc.background_cells(m)
    sh, ah = orc.tensor_spectrum(m.Nx, m.Ny, m.Nz, symm, asym)
    vs = [random_vec(m, s) for s in (31, 32)]
    return op, vs, [orc.apply(m.Nx, m.Ny, m.Nz, sh, ah, csiga, csigb, sqsigb, m.dz, v) for v in vs]


def _run(g2, op, vs, form):
    import torch
    dt = torch.complex128 if form == 0 else torch.complex64
    xs = [torch.from_numpy(v.ravel()).to("cuda", dt) for v in vs]
    ys = [torch.full_like(x, complex(np.nan, np.nan)) for x in xs]
    if form == 2:
        g2.apply_device_batch(op, [x.data_ptr() for x in xs], [y.data_ptr() for y in ys], 1)
    else:
        op.apply_device(xs[0].data_ptr(), ys[0].data_ptr(), form)
    op.check_device_error()
    return [y.cpu().numpy() for y in ys[: (2 if form == 2 else 1)]]


@pytest.mark.parametrize("shape", [(4, 4, n) for n in EDGES] + [(64, 32, 3), (32, 64, 11), (32, 32, 27), (64, 16, 44)])
def test_every_tile_edge(g2lib, orc, shape):
    m = tiny_model(*shape)
    op, vs, refs = _op(g2lib, orc, m)
    for form, tol in ((0, 1e-12), (1, 2e-5), (2, 2e-5)):
        for got, ref in zip(_run(g2lib, op, vs, form), refs):
            assert rel(got.astype(np.complex128).reshape(ref.shape), ref) < tol, form
    op.delete()


def test_switching_to_the_other_kernels_and_back(g2lib, orc):
    """Selecting a shape of the other kernels makes their copy of the tensor, the default selection frees it; a new
    tensor replaces the copy; the default's result is the same bits before and after."""
    m = tiny_model(16, 8, 16)
    op, vs, refs = _op(g2lib, orc, m)
    before = [_run(g2lib, op, vs, f) for f in (0, 1, 2)]
    for form in (0, 1, 2):
        n = op.contract_variants(form)
        op.set_contract_variant(form, 0)
        assert rel(_run(g2lib, op, vs, form)[0].astype(np.complex128).reshape(refs[0].shape), refs[0]) < 2e-5
        symm, asym = random_spatial_tensor(m, seed=13)
        op.set_ie_kernel_spatial(symm, asym)
        op.calc_fft_of_ie_kernel()
        assert rel(_run(g2lib, op, vs, form)[0].astype(np.complex128).reshape(refs[0].shape), refs[0]) < 2e-5
        op.set_contract_variant(form, n - 1)
    for form in (0, 1, 2):
        for a, b in zip(_run(g2lib, op, vs, form), before[form]):
            assert np.array_equal(a, b)
    op.delete()
