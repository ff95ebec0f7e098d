"""Pairs of primitives so far apart that their Gaussian product factor is
subnormal: every integral of the gam_2 and gam_3 builders has to be the
negligible number that it is, on the host and in the tensors."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, OracleTensors, assert_close_scaled


def test_subnormal_product_factor(tmp_path):
    exe = str(tmp_path / "g3_far_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off",
                    os.path.join(ROOT, "tests", "hostcheck", "g3_far_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    a = np.array([[float(x) for x in line.split()] for line in r.stdout.splitlines()])
    assert np.isfinite(a).all(), a[~np.isfinite(a[:, 3])][:4]
    # nothing above 1e-250 is dropped, and what is kept agrees as far as fb_eval's own numbers are normal
    assert (np.abs(a[:, 3] - a[:, 4]) <= 1e-250 + 1e-10 * np.abs(a[:, 4])).all()
    assert r.returncode == 0


@pytest.mark.gpu
@pytest.mark.parametrize("am,dist", [((1, 0, 0), 8.45), ((2, 0, 0), 8.45), ((1, 0, 0), 8.40), ((0, 1, 0), 8.55)])
def test_tensors_of_distant_centres(nx, orc, am, dist):
    """p (or d) functions of exponent 20 on two centres: q Q^2 = 706 to 731."""
    from neoxc import basis
    s = basis.synthetic(seed=41, nat=2, nebf=2, nprim=1, npbf=1, ngtg=2, lmax_e=1, lmax_p=0)
    s.cat[:] = [[0.0, dist], [0.0, 0.0], [0.0, 0.0]]
    s.ELCAM[:] = am
    s.ELCEX[:] = 20.0
    s.ELCBFC[:] = s.cat.T
    s.NUCBFC[:] = 0.0
    s.AGEBFCC[:] = basis.elcnorm3(s.AMPEB2C, np.ones(2), s.ELCEX, s.ELCAM, s.ELCBFC)
    T = OracleTensors(orc, s)
    got = dict(zip(("g2", "g2s"), nx.gam2_ic1(s)))
    got.update(zip(("rx2", "rx2ex"), nx.rxchfne_gam2_ic1(s)))
    got["g3"], got["gee"] = nx.gam3_ic1(s), nx.calc_gam_ee(s)
    for k, v in got.items():
        assert np.isfinite(v).all(), k
        assert_close_scaled(v, T.get(k), 1e-10, k)   # the tolerance of the parity tests
