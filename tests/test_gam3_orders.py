"""The FP64 (bra, ket) integral of the gam_2 and gam_3 builders
(csrc/g3_fatbra.cuh) at the Hermite orders that only electronic d together with
nuclear p or d functions reach (13 to 16 in one direction): on the host under
the address and bounds checkers, and the gam_3 tensor against the oracle."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, OracleTensors, assert_close_scaled


def test_every_order_of_a_direction(tmp_path):
    exe = str(tmp_path / "g3_orders_check")
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-ffp-contract=off", "-fsanitize=address,undefined",
                    "-fno-sanitize-recover=all",
                    os.path.join(ROOT, "tests", "hostcheck", "g3_orders_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    a = np.array([[float(x) for x in line.split()] for line in r.stdout.splitlines()])
    assert set(a[:, 0].astype(int)) == set(range(8, 17))
    # T carries a few roundings, which F_m's dependence on T (as T^-(m+1/2), m <= 16, or over T <= 20)
    # multiplies by at most 20, and a term some hundred operations: 1024 units of 2^-53
    assert (np.abs(a[:, 1] - a[:, 2]) <= 1024 * 2.0 ** -53 * a[:, 3]).all()


def _d_along_x(npbf_l):
    """Electrons d_xx, s and p_x with one primitive each, proton functions of
    the given l along x: Hermite orders up to 12 + 2 l in the x direction."""
    from neoxc import basis
    s = basis.synthetic(seed=31, nat=2, nebf=3, nprim=1, npbf=2, ngtg=1, lmax_e=1, lmax_p=1)
    s.ELCAM[:] = [[2, 0, 0], [0, 0, 0], [1, 0, 0]]
    s.NUCAM[:] = [[0, 0, 0], [npbf_l, 0, 0]]
    s.AGEBFCC[:] = basis.elcnorm3(s.AMPEB2C, np.ones(3), s.ELCEX, s.ELCAM, s.ELCBFC)
    s.AGNBFCC[:] = basis.nucnorm(np.ones(2), s.NUCEX, s.NUCAM)
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("l", [1, 2])
def test_gam3_of_d_electrons_and_excited_protons(nx, orc, l):
    s = _d_along_x(l)
    ref = OracleTensors(orc, s).get("g3")
    assert_close_scaled(nx.gam3_ic1(s), ref, 1e-10, "GM3ICR")   # the tolerance of the parity tests
    (got,), _ = nx.gam3_ic1_batch([s])
    assert_close_scaled(got, ref, 1e-10, "GM3ICR, batch")
