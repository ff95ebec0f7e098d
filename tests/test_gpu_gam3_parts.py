"""The gam_3 passes with a block's bras cut into parts (csrc/k_gam3.cu,
fb_parts): one to eight parts of contracted functions, blocks with fewer parts
than the cluster has CTAs, remainders of a part, against the oracle; and the
persistent launch of many systems, which takes the parts one after the other."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import OracleTensors, assert_close_scaled

pytestmark = pytest.mark.gpu
RTOL = 1e-10   # the oracle tolerance of the parity tests

# mean bras of a block and parts: 441 (8), 81 (8), 44 (4), 21 (2), 4 (1), 44 (4)
CASES = [dict(seed=201, nat=2, nebf=2, nprim=3, npbf=1, ngtg=3, lmax_e=0, lmax_p=0),
         dict(seed=202, nat=2, nebf=2, nprim=2, npbf=2, ngtg=3, lmax_e=0, lmax_p=1),
         dict(seed=203, nat=2, nebf=2, nprim=2, npbf=1, ngtg=2, lmax_e=0, lmax_p=2),
         dict(seed=204, nat=2, nebf=3, nprim=(1, 2), npbf=1, ngtg=3, lmax_e=1, lmax_p=0),
         dict(seed=205, nat=2, nebf=3, nprim=1, npbf=2, ngtg=2, lmax_e=1, lmax_p=1)]


@pytest.mark.parametrize("kw", CASES)
def test_parts_against_oracle(nx, orc, kw):
    from neoxc import basis
    s = basis.synthetic(**kw)
    ref = OracleTensors(orc, s).get("g3")
    got = nx.gam3_ic1(s)
    assert_close_scaled(got, ref, RTOL, "GM3ICR")
    assert np.array_equal(got, nx.gam3_ic1(s))   # the parts are added in their order


@pytest.mark.parametrize("mixed", [False, True])
def test_parts_of_many_systems(nx, mixed):
    from neoxc import basis
    systems = [basis.synthetic(**kw) for kw in CASES]
    outs, _ = nx.gam3_ic1_batch(systems, mixed=mixed)
    for s, x in zip(systems, outs):
        ref = nx.gam3_ic1(s, mixed=mixed)
        assert np.abs(x - ref).max() <= 1e-14 * np.abs(ref).max(), s.name
