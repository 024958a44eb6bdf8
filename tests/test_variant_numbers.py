"""What the contraction's variant numbers mean stays what it is: hosts keep them, and the tuner's file does."""
import numpy as np
import pytest

from giem2g_b200.autotune import _cached
from giem2g_b200.synthetic import csiga_from_sigma
from tests.helpers import random_sigma, random_spatial_tensor, random_vec, tiny_model


def test_cached_pick_of_another_set_of_variants_is_not_used():
    pick = {"variant": 27, "ms": 0.3, "all_ms": [0.4] * 28}
    assert _cached({"k": pick}, "k", 28) is pick
    assert _cached({"k": pick}, "k", 27) is None  # one fewer: 27 would not even be a variant
    assert _cached({"k": pick}, "k", 29) is None
    assert _cached({"k": {"variant": 3, "ms": 0.3}}, "k", 4) is None and _cached({}, "k", 4) is None


@pytest.mark.gpu
@pytest.mark.parametrize("shape,counts", [((4, 32, 32), (14, 27, 23)), ((16, 8, 32), (13, 26, 22)), ((16, 8, 16), (3, 5, 5)),
                                          ((8, 8, 48), (3, 5, 7)), ((8, 8, 20), (0, 0, 0))])
def test_numbers(g2lib, shape, counts):
    """0 is the default.  Where the fused pass exists (4x32x32) it has the two numbers after the 12, 25 and 21 of the
    separate passes and nothing follows; elsewhere the number after the shapes is the default too."""
    import torch
    m = tiny_model(*shape)
    op = g2lib.IEOperator.from_model(m)
    op.set_background(m.csigma, m.thick, m.omega)
    op.set_ie_kernel_spatial(*random_spatial_tensor(m, seed=13))
    op.calc_fft_of_ie_kernel()
    op.set_anomaly_conductivity(csiga_from_sigma(random_sigma(m, 4), m.freq))
    assert tuple(op.contract_variants(f) for f in (0, 1, 2)) == counts
    x = [torch.from_numpy(random_vec(m, 7).ravel()).to("cuda", dt) for dt in (torch.complex128, torch.complex64)]
    y = [torch.empty_like(t) for t in x]

    def apply(prec):
        n0 = g2lib.kernel_launch_count()
        op.apply_device(x[prec].data_ptr(), y[prec].data_ptr(), prec)
        op.check_device_error()
        return y[prec].cpu().numpy(), g2lib.kernel_launch_count() - n0

    for prec in (0, 1):
        n, fused = counts[prec], shape == (4, 32, 32)
        default = apply(prec)[0]
        for v in range(n):
            op.set_contract_variant(prec, v)
            out, launches = apply(prec)
            assert launches == (3 if fused and v >= n - 2 else 5), v
            same = v == 0 or (not fused and v == n - 1)
            assert np.array_equal(out, default) == same, v
        op.set_contract_variant(prec, 0)
        assert np.array_equal(apply(prec)[0], default)
        with pytest.raises(g2lib.Giem2gError):
            op.set_contract_variant(prec, max(n, 1))
    op.delete()
