"""The layouts of the spectral tensor: one per precision where one will do, what a failed or a captured selection leaves."""
import numpy as np
import pytest

from giem2g_b200.autotune import _one_layout, _second_tensor_fits
from giem2g_b200.synthetic import csiga_from_sigma
from tests.helpers import random_sigma, random_spatial_tensor, random_vec, tiny_model


def test_tuner_weighs_the_second_tensor():
    class Op:
        Nx, Ny, Nz = 256, 256, 48

    need = 8 * 256 * 256 * 96 * 97
    assert not _second_tensor_fits(Op, 31 * need) and _second_tensor_fits(Op, 32 * need)
    # the paired apply decides, the single one follows in its layout
    assert _one_layout([0.20, 0.25, 0.17], [0.28, 0.40, 0.30]) == (0, 0)
    assert _one_layout([0.10, 0.25, 0.17], [0.28, 0.40, 0.27]) == (2, 2)
    assert _one_layout([0.10, 0.25, None], [0.28, 0.27, None]) == (1, 1)
    assert _one_layout([0.10, None, None], [0.28, 0.27, None]) == (0, 0)


def _op(g2, m, seed=13):
    op = g2.IEOperator.from_model(m)
    op.set_background(m.csigma, m.thick, m.omega)
    op.set_ie_kernel_spatial(*random_spatial_tensor(m, seed=seed))
    op.calc_fft_of_ie_kernel()
    op.set_anomaly_conductivity(csiga_from_sigma(random_sigma(m, 4), m.freq))
    return op


def _vectors(m):
    import torch
    x = {dt: torch.from_numpy(random_vec(m, 7).ravel()).to("cuda", dt) for dt in (torch.complex128, torch.complex64)}
    return x, {dt: torch.empty_like(t) for dt, t in x.items()}


def _applies(g2, op, x, y):
    """The bits of an FP64, a complex64 and a paired apply."""
    import torch
    out = []
    for prec, dt in ((0, torch.complex128), (1, torch.complex64)):
        op.apply_device(x[dt].data_ptr(), y[dt].data_ptr(), prec)
        out.append(y[dt].cpu().numpy())
    a, b = x[torch.complex64], y[torch.complex64]
    b2 = torch.empty_like(b)
    g2.apply_device_batch(op, [a.data_ptr(), a.data_ptr()], [b.data_ptr(), b2.data_ptr()], 1)
    op.check_device_error()
    return out + [b.cpu().numpy(), b2.cpu().numpy()]


@pytest.mark.gpu
def test_one_tensor_per_precision(g2lib):
    """64x64x32: 273 MB in FP64, 136 MB in complex64.  Selections that one layout serves hold no second tensor, and the
    spectral tensor that a host reads back is the same in either."""
    import torch
    m = tiny_model(64, 64, 32)
    op = _op(g2lib, m)
    x, y = _vectors(m)
    before = _applies(g2lib, op, x, y)
    tensor = op.get_ie_kernel_spectral()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for form, v in ((0, 5), (1, 21), (2, 14)):
        op.set_contract_variant(form, v)
    other = _applies(g2lib, op, x, y)
    assert torch.cuda.mem_get_info()[0] > free - (64 << 20)
    for a, b in zip(op.get_ie_kernel_spectral(), tensor):
        assert np.array_equal(a, b)
    # a new tensor while the other layout is held
    symm, asym = random_spatial_tensor(m, seed=13)
    op.set_ie_kernel_spatial(symm, asym)
    op.calc_fft_of_ie_kernel()
    for a, b in zip(_applies(g2lib, op, x, y), other):
        assert np.array_equal(a, b)
    for form in (0, 1, 2):
        op.set_contract_variant(form, 0)
    for a, b in zip(_applies(g2lib, op, x, y), before):
        assert np.array_equal(a, b)
    op.delete()


@pytest.mark.gpu
def test_failed_selection_leaves_the_old_one(g2lib):
    """No memory for a second complex64 tensor (136 MB): the selection is refused and the applies go on as they were."""
    import torch
    m = tiny_model(64, 64, 32)
    op = _op(g2lib, m)
    x, y = _vectors(m)
    before = _applies(g2lib, op, x, y)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filler = [torch.empty(torch.cuda.mem_get_info()[0] - (96 << 20), dtype=torch.uint8, device="cuda")]
    try:
        with pytest.raises(torch.OutOfMemoryError):  # what memory pools give back on demand
            for _ in range(64):
                filler.append(torch.empty(64 << 20, dtype=torch.uint8, device="cuda"))
        with pytest.raises(g2lib.Giem2gError):
            op.set_contract_variant(1, 21)
        after = _applies(g2lib, op, x, y)
    finally:
        del filler
        torch.cuda.empty_cache()
    for a, b in zip(after, before):
        assert np.array_equal(a, b)
    op.set_contract_variant(1, 21)  # there is memory again
    assert not np.array_equal(_applies(g2lib, op, x, y)[1], before[1])
    op.delete()


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [0, 1])
def test_captured_apply_outlives_selections_and_new_tensors(g2lib, variant):
    """A graph that the host captured reads the operator's tensor as it was selected then: replays stay right after another
    selection, and after a new tensor."""
    import torch
    m = tiny_model(16, 16, 16)
    op = _op(g2lib, m)
    op.set_contract_variant(0, variant)
    x, y = _vectors(m)
    xd, yd = x[torch.complex128], y[torch.complex128]
    op.apply_device(xd.data_ptr(), yd.data_ptr(), 0)
    first = yd.cpu().numpy()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op.apply_device(xd.data_ptr(), yd.data_ptr(), 0)

    def replay():
        yd.zero_()
        graph.replay()
        torch.cuda.synchronize()
        return yd.cpu().numpy()

    assert np.array_equal(replay(), first)
    op.set_contract_variant(0, 1 - variant)
    assert np.array_equal(replay(), first)
    op.set_ie_kernel_spatial(*random_spatial_tensor(m, seed=99))
    op.calc_fft_of_ie_kernel()
    second = replay()
    op.set_contract_variant(0, variant)
    op.apply_device(xd.data_ptr(), yd.data_ptr(), 0)
    torch.cuda.synchronize()
    assert np.array_equal(yd.cpu().numpy(), second) and not np.array_equal(second, first)
    del graph
    op.delete()


@pytest.mark.gpu
@pytest.mark.parametrize("fits", [True, False])
def test_tuner_keeps_one_layout_when_memory_is_short(g2lib, monkeypatch, fits):
    """A grid without the fused pass: its last number is the default again and is not picked; without room for a second
    tensor the complex64 and the paired apply get kernels of one layout."""
    import giem2g_b200.autotune as at
    monkeypatch.setattr(at, "_second_tensor_fits", lambda op, free: fits)
    m = tiny_model(32, 32, 16)
    op = _op(g2lib, m)
    picks = at.autotune_contraction(op, reps=2, rounds=1)
    for form in (0, 1, 2):
        assert 0 <= picks[str(form)]["variant"] < op.contract_variants(form) - 1
    if not fits:
        assert (picks["1"]["variant"] == 0) == (picks["2"]["variant"] == 0)
    op.delete()
