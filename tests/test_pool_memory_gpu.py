"""Device memory that the set-up keeps (csrc/mem_pool.cu): what a call used is given back when it returns, operators share one
pool, and nothing is left after the last one."""
import pytest

from giem2g_b200.synthetic import csiga_from_sigma
from tests.helpers import random_sigma, tiny_model

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def test_call_gives_back_what_it_used(g2lib):
    """The receivers' weights at 128x128 take 1.6 GB: after the call at most the 512 MB that the pool keeps are missing."""
    import torch
    m = tiny_model(128, 128, 4)
    rc = g2lib.RCOperator.from_model(m, [0.0])
    torch.cuda.synchronize()
    before = _free()
    rc.calc_rc_kernel(m.csigma, m.thick, m.omega)
    assert before - _free() < 576 * MB
    op = g2lib.IEOperator.from_model(tiny_model(128, 128, 16))
    torch.cuda.synchronize()
    before = _free()
    op.calc_ie_kernel(m.csigma, m.thick, m.omega)  # weights 394 MB; the spatial tensor, 277 MB, stays
    assert before - _free() < (277 + 576) * MB
    op.delete()
    rc.delete()


def test_operators_share_one_pool(g2lib):
    """64x64x16: an operator holds 104 MB of tensors and about 35 MB of vectors and scratch; its set-up uses 250 MB more."""
    import torch
    m = tiny_model(64, 64, 16)
    csiga = csiga_from_sigma(random_sigma(m, 4), m.freq)
    torch.cuda.synchronize()
    start, ops, used = _free(), [], []
    for _ in range(4):
        before = _free()
        op = g2lib.IEOperator.from_model(m)
        op.calc_ie_kernel(m.csigma, m.thick, m.omega)
        op.calc_fft_of_ie_kernel()
        op.set_anomaly_conductivity(csiga)
        ops.append(op)
        used.append(before - _free())
    assert used[3] < 200 * MB, used
    for op in ops:
        op.delete()
    torch.cuda.synchronize()
    assert start - _free() < 64 * MB
