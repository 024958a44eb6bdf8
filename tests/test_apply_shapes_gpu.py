"""Applies at shapes where a kernel's loops run in full, against the oracle, at tolerances near the kernels' errors: 1e-14 for
complex128 (both sides are within 1e-15 of the exact result), 1e-6 for complex64 and pairs (within 3.2e-7)."""
import numpy as np
import pytest

from tests.helpers import rel, tiny_model
from tests.test_contract_mma_gpu import _op, _run

pytestmark = pytest.mark.gpu


def _check(g2, orc, shape):
    m = tiny_model(*shape)
    op, vs, refs = _op(g2, orc, m)
    for form, tol in ((0, 1e-14), (1, 1e-6), (2, 1e-6)):
        for got, ref in zip(_run(g2, op, vs, form), refs):
            assert rel(got.astype(np.complex128).reshape(ref.shape), ref) < tol, form
    op.delete()


def _stages(Nz, points, size):
    """Stages of the tensor-core contraction's ring: what fits 227 KB, at most 16."""
    pitch = 3 * Nz + (4 - 3 * Nz) % 8
    stage = -(-(2 * Nz * (2 * Nz + 1) + points * pitch + 1) * size // 128) * 128
    return min(16, (232448 - 512) // (stage + 16))


@pytest.mark.parametrize("shape", [(128, 64, 4), (128, 64, 11), (128, 64, 13), (128, 64, 20), (64, 64, 27), (64, 64, 32),
                                   (64, 64, 37), (64, 32, 44), (32, 32, 53), (32, 32, 58)])
def test_rings_wrap(g2lib, orc, shape):
    """Every stage of the ring is filled three times or more, in all three forms and at every tile count; 58 layers are the
    most that an operator takes."""
    import torch
    ctas = torch.cuda.get_device_properties(0).multi_processor_count
    for points, size in ((4, 16), (4, 8), (8, 8)):
        assert shape[0] * shape[1] >= 3 * ctas * _stages(shape[2], points, size)
    _check(g2lib, orc, shape)


@pytest.mark.parametrize("shape", [(256, 4, 3), (4, 256, 3), (256, 2, 9), (256, 256, 2)])
def test_512_point_lines(g2lib, orc, shape):
    """The three-step transform, along x (k_fx, k_bx) and along y (k_fy, k_by)."""
    _check(g2lib, orc, shape)
