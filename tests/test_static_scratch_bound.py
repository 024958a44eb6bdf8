"""The static scratch array holds the padded intermediates of every grid that its limit on the unpadded ones lets in."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "giem2g_b200", "csrc", "static_scratch.cu")


def _mib(name):
    return int(re.search(rf"{name} = size_t\((\d+)\) << 20", open(SRC).read()).group(1)) << 20


@pytest.mark.parametrize("es", [16, 8])
def test_every_accepted_grid_fits(es):
    limit, array = _mib("kStaticScratchBytes"), _mib("kStaticArrayBytes")
    state = 64 << 10  # the fused pass's counters and the alignment between the two parts
    worst = 0
    for nx in (2 ** k for k in range(1, 10)):
        for ny in (2 ** k for k in range(1, 10)):
            for nz in range(1, 59):
                pitch = 3 * nz + (4 - 3 * nz) % 8
                assert pitch % 8 == 4
                u1, rows = 6 * nx * ny * nz, 4 * nx * ny
                if (u1 + rows * 3 * nz) * es <= limit:
                    worst = max(worst, (u1 + rows * pitch) * es + state)
    assert worst <= array, worst / 2 ** 20
