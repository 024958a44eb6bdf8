"""Rounding of the tensor-core contraction (csrc/contract_mma.cu) against the apply in 80-bit numbers.

On a 2x2 grid the transforms have four points, whose twiddles are 1 and +-i: they only add, so nearly all of an apply's
rounding is the contraction's.  The tensor is scaled so that the contraction outweighs the a x term of the apply.
"""
import numpy as np
import pytest

from giem2g_b200.synthetic import csiga_from_sigma
from tests.helpers import random_sigma, random_spatial_tensor, random_vec, tiny_model

pytestmark = pytest.mark.gpu

# (row component, column component): sign of the transposed block, parity in x and in y
PARITY = {(0, 0): (1, 1), (1, 1): (1, 1), (2, 2): (1, 1), (0, 1): (-1, -1), (0, 2): (-1, 1), (1, 2): (1, -1)}


def _blocks(m, symm, asym):
    """{(a, b): [Nx, Ny, Nz, Nz]} for a <= b, rows z and columns z'."""
    Nz = m.Nz
    hi, lo = np.maximum.outer(np.arange(Nz), np.arange(Nz)), np.minimum.outer(np.arange(Nz), np.arange(Nz))
    packed = lo + hi * (hi + 1) // 2
    out = {ab: symm[:, :, i][:, :, packed] for i, ab in enumerate([(0, 0), (0, 1), (1, 1), (2, 2)])}
    for i, ab in enumerate([(0, 2), (1, 2)]):
        out[ab] = asym[:, :, i].reshape(m.Nx, m.Ny, Nz, Nz).transpose(0, 1, 3, 2)  # column-major
    return out


def exact_apply(m, symm, asym, csiga, csigb, v, single=False):
    """s (a v - (G * (g v)) / dz), the convolution lag by lag, in 80-bit numbers; single: with the coefficients s, a, g
    and 1 / (4 Nx Ny dz) as the complex64 apply holds them, in FP32 (s and dz are few, so their rounding would not
    average out)."""
    L = np.clongdouble
    sb = csigb.astype(L)[:, None, None]
    a = 2 * np.sqrt(sb.real) / (csiga.astype(L) + np.conj(sb))
    g, s, d = (csiga.astype(L) - sb) * a, np.sqrt(sb.real), 1 / (4 * m.Nx * m.Ny * m.dz.astype(np.longdouble))
    if single:
        a, g = (t.astype(np.complex64).astype(L) for t in (a, g))
        s, d = (t.astype(np.float32).astype(np.longdouble) for t in (s, d))
    u = v.astype(L) * g
    w = np.zeros(v.shape, L)
    for (p, q), blk in _blocks(m, symm, asym).items():
        blk = blk.astype(L)
        for lx in range(-(m.Nx - 1), m.Nx):
            for ly in range(-(m.Ny - 1), m.Ny):
                sign = (PARITY[p, q][0] if lx < 0 else 1) * (PARITY[p, q][1] if ly < 0 else 1)
                B = sign * blk[abs(lx), abs(ly)]
                dst = (slice(max(ly, 0), m.Ny + min(ly, 0)), slice(max(lx, 0), m.Nx + min(lx, 0)))
                src = (slice(max(-ly, 0), m.Ny + min(-ly, 0)), slice(max(-lx, 0), m.Nx + min(-lx, 0)))
                w[p][(slice(None), *dst)] += np.tensordot(B, u[q][(slice(None), *src)], 1)
                if p != q:  # the transposed block: out_y takes xy as it is, out_z takes -xz^T and -yz^T
                    Bt = -B.T if q == 2 else B
                    w[q][(slice(None), *dst)] += np.tensordot(Bt, u[p][(slice(None), *src)], 1)
    return s * (a * v.astype(L) - w * (4 * m.Nx * m.Ny * d)[:, None, None])


def _case(g2, orc, Nz, seed, components=(0, 1, 2)):
    m = tiny_model(2, 2, Nz)
    symm, asym = random_spatial_tensor(m, seed=seed, scale=1e4)
    op = g2.IEOperator.from_model(m)
    op.set_background(m.csigma, m.thick, m.omega)
    op.set_ie_kernel_spatial(symm, asym)
    op.calc_fft_of_ie_kernel()
    csiga = csiga_from_sigma(random_sigma(m, seed), m.freq)
    op.set_anomaly_conductivity(csiga)
    v = random_vec(m, seed + 1)
    for c in range(3):
        if c not in components:
            v[c] = 0
    return m, op, symm, asym, csiga, orc.background_cells(m)[0], v


def _run(g2, op, vs, form):
    import torch
    dt = torch.complex128 if form == 0 else torch.complex64
    xs = [torch.from_numpy(v.ravel()).to("cuda", dt) for v in vs]
    ys = [torch.empty_like(x) for x in xs]
    if form == 2:
        g2.apply_device_batch(op, [x.data_ptr() for x in xs], [y.data_ptr() for y in ys], 1)
    else:
        op.apply_device(xs[0].data_ptr(), ys[0].data_ptr(), form)
    op.check_device_error()
    return [y.cpu().numpy().reshape(v.shape) for y, v in zip(ys, vs)][: 2 if form == 2 else 1]


def test_statement_in_80_bits_is_the_oracles(orc):
    m = tiny_model(4, 2, 5)
    symm, asym = random_spatial_tensor(m, seed=3)
    csiga = csiga_from_sigma(random_sigma(m, 3), m.freq)
    csigb, sqsigb = orc.background_cells(m)
    v = random_vec(m, 4)
    sh, ah = orc.tensor_spectrum(m.Nx, m.Ny, m.Nz, symm, asym)
    ref = orc.apply(m.Nx, m.Ny, m.Nz, sh, ah, csiga, csigb, sqsigb, m.dz, v)
    e = exact_apply(m, symm, asym, csiga, csigb, v)
    assert np.linalg.norm((e - ref).ravel()) < 1e-13 * np.linalg.norm(ref.ravel())


@pytest.mark.parametrize("components", [(0,), (2,), (0, 1, 2)])
@pytest.mark.parametrize("Nz", [9, 13, 32, 48])
def test_complex64_sums_keep_their_size(g2lib, orc, Nz, components):
    """<exact, result - exact> / <exact, exact>: roundings average out, a truncation or a gain that does not belong to the
    sums stays.  Truncating sums lose half a unit, 4.3e-8; what is left has to be under half of that, whichever components
    of the vector are there."""
    for form in (1, 2):
        num, den = 0.0, 0.0
        for seed in range(12):
            m, op, symm, asym, csiga, csigb, v = _case(g2lib, orc, Nz, 10 * seed + 5, components)
            v = v.astype(np.complex64).astype(np.complex128)
            vs = [v, v[:, ::-1].copy()]
            for got, x in zip(_run(g2lib, op, vs, form), vs):
                e = exact_apply(m, symm, asym, csiga, csigb, x, single=True)
                num += float(np.sum(np.conj(e) * (got.astype(np.clongdouble) - e)).real)
                den += float(np.sum(np.abs(e) ** 2))
            op.delete()
        assert abs(num / den) < 2.1e-8, (form, num / den)


def test_complex128_sums_are_split(g2lib, orc):
    """57 layers: one chain of FMAs per output has an error of 4.4e-16, two chains 3.2e-16; the apply's other roundings add
    about 1e-16 in quadrature, so 4.5e-16 and 3.4e-16 for the whole."""
    num, den = 0.0, 0.0
    for seed in range(6):
        m, op, symm, asym, csiga, csigb, v = _case(g2lib, orc, 57, 10 * seed + 5)
        e = exact_apply(m, symm, asym, csiga, csigb, v)
        got = _run(g2lib, op, [v], 0)[0].astype(np.clongdouble)
        num += float(np.sum(np.abs(got - e) ** 2))
        den += float(np.sum(np.abs(e) ** 2))
        op.delete()
    assert np.sqrt(num / den) < 3.9e-16, np.sqrt(num / den)
