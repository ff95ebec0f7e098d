"""The four-launch factorised gam_4 build (csrc/k_gam4f.cu) on both sides of the
lines where its CTAs change their width and their tiles: n = 22 | 23 and 32 | 33,
five and six nuclear functions, and at large n."""
from __future__ import annotations

import pytest

import test_gpu_gam4_factored as factored

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,np_", [(22, 5), (23, 5), (23, 6), (25, 1), (26, 4), (32, 6), (33, 5), (33, 6), (48, 2), (49, 2), (52, 6)])
def test_widths(nx, ne, np_):
    factored.test_factored_build(nx, ne, np_)
