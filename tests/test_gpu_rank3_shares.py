"""The open-shell rank-3 contraction (csrc/k_rank3.cu) where its CTAs take shares
of the walk over i3 (few proton pairs): even and uneven shares, weights formed in
the CTAs (up to eight functions) and tabulated, one class with all of its flags
and one with few."""
from __future__ import annotations

import pytest

import test_gpu_rank3 as rank3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,np_,na,nb", [(2, 1, 3, 2), (4, 3, 2, 1), (6, 2, 4, 3), (7, 2, 2, 2), (8, 1, 1, 3), (8, 3, 3, 3),
                                          (9, 1, 4, 1), (12, 1, 2, 3), (14, 1, 3, 2), (17, 1, 2, 2)])
def test_shares(nx, ne, np_, na, nb):
    rank3.test_xcuhf_omg3(nx, ne, np_, na, nb)
