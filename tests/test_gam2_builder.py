"""The gam_2 builder (csrc/k_gam2.cu, csrc/g2_threebody.cuh): its pair-density
integrals compiled for the host against the element-wise MD integrals, and the
tensors on the GPU against the oracle at the edges of its work decomposition
(32 primitive pairs a warp, splits over primitives, chunks of proton pairs)."""
from __future__ import annotations

import ctypes as C
import dataclasses
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, OracleTensors, assert_close_scaled

RTOL = 1e-10   # the FP64 integral tolerance of the parity tests


class _HP(C.Structure):
    _fields_ = [("l", C.c_int * 3), ("a", C.c_double), ("c", C.c_double * 3)]


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("g2") / "g2_host_check.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    os.path.join(ROOT, "tests", "hostcheck", "g2_host_check.cpp"), "-o", so], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("le,ln", [(0, 0), (0, 2), (1, 2), (2, 2)])
def test_pair_density_integrals_match_element_integrals(host, le, ln):
    rng = np.random.Generator(np.random.PCG64(100 * le + ln))

    def prim(lmax, lo, hi, centre=None):
        p = _HP()
        p.a = float(np.exp(rng.uniform(np.log(lo), np.log(hi))))
        for _ in range(int(rng.integers(0, lmax + 1))):
            p.l[int(rng.integers(0, 3))] += 1
        for d in range(3):
            p.c[d] = float(rng.uniform(-1.2, 1.2)) if centre is None else centre[d]
        return p

    V = C.c_void_p
    for _ in range(60):
        cp = rng.uniform(-1, 1, 3)
        A = (_HP * 3)(prim(le, 0.1, 20), prim(le, 0.1, 20), prim(ln, 4, 32, cp))
        B = (_HP * 3)(prim(le, 0.1, 20), prim(le, 0.1, 20), prim(ln, 4, 32, cp))
        gm, cat, zan = rng.uniform(0.2, 10, 2), rng.uniform(-1.5, 1.5, 9), np.array([1.0, 2.0, 3.0])
        ref, got, pair, ov = np.zeros(4), np.zeros(3), np.zeros(4), np.zeros(2)
        host.hc_gam2(A, B, 2, gm.ctypes.data_as(V), 3, cat.ctypes.data_as(V), zan.ctypes.data_as(V),
                     C.c_double(1836.0), *[x.ctypes.data_as(V) for x in (ref, got, pair, ov)])
        # sums of terms of both signs: against the sum of magnitudes
        assert np.abs(got - ref[:3]).max() <= 1e-11 * ref[3]
        for x, y in ((pair[0], pair[2]), (pair[1], pair[3]), (ov[0], ov[1])):
            assert abs(x - y) <= 1e-10 * abs(y) + 1e-14 * max(abs(pair).max(), abs(ov).max())


@pytest.mark.parametrize("le,ln", [(0, 0), (1, 2), (2, 2)])
def test_two_particle_integrals_match_element_integrals(host, le, ln):
    """GAM_1's kinetic, multiplicative and overlap integrals and the plain
    Coulomb integral of two pair densities (csrc/k_pair.cu)."""
    rng = np.random.Generator(np.random.PCG64(7 + 10 * le + ln))
    V, D = C.c_void_p, C.c_double

    def prim(lmax, lo, hi, centre):
        p = _HP()
        p.a = float(np.exp(rng.uniform(np.log(lo), np.log(hi))))
        for _ in range(int(rng.integers(0, lmax + 1))):
            p.l[int(rng.integers(0, 3))] += 1
        for d in range(3):
            p.c[d] = float(centre[d])
        return p
    for _ in range(80):
        cp = rng.uniform(-1, 1, 3)
        A = (_HP * 2)(prim(le, 0.1, 20, rng.uniform(-1, 1, 3)), prim(ln, 4, 32, cp))
        B = (_HP * 2)(prim(le, 0.1, 20, rng.uniform(-1, 1, 3)), prim(ln, 4, 32, cp))
        gk, gl = rng.uniform(0.1, 10, 2)
        cat, zan = rng.uniform(-1.5, 1.5, 6), np.array([1.0, 3.0])
        got, ref, mag = np.zeros(4), np.zeros(4), np.zeros(1)
        host.hc_gam1(A, B, D(gk), D(gl), 2, cat.ctypes.data_as(V), zan.ctypes.data_as(V), D(1836.0),
                     *[x.ctypes.data_as(V) for x in (got, ref, mag)])
        err = np.abs(got - ref)
        assert err[0] <= 1e-11 * abs(ref[0]) + 1e-16
        assert err[1] <= 1e-11 * mag[0]
        assert (err[2:] <= 1e-10 * np.abs(ref[2:]) + 1e-16).all()


@pytest.mark.parametrize("L", [0, 1, 2, 7, 12, 16])
def test_boys_dot_is_the_boys_function(host, L):
    """One recursion for both ranges of T: the table's grid points and their
    midpoints, the branch at T = 20, tiny, large and enormous T (positive
    weights, so the sum has the relative accuracy of its terms)."""
    host.hc_boys_dot.restype = host.hc_boys_ref.restype = C.c_double
    rng = np.random.Generator(np.random.PCG64(L))
    T = [0.0, 1e-300, 1e-12, 1 / 32, 1 / 16, 19.96875, np.nextafter(20, 0), 20.0, np.nextafter(20, 21), 35.0, 1e4,
         1e14, 1e16, 1e60] + list(rng.uniform(0, 40, 200))
    for t in T:
        B = rng.uniform(0.1, 1.0, L + 1)
        if t > 1e14:
            B[:] = 0.0
            B[0] = 1.0
        x, y = (f(L, C.c_double(t), B.ctypes.data_as(C.c_void_p)) for f in (host.hc_boys_dot, host.hc_boys_ref))
        assert abs(x - y) <= 2e-14 * abs(y), (t, x, y)
    assert np.isnan(host.hc_boys_dot(L, C.c_double(float("nan")), B.ctypes.data_as(C.c_void_p)))


def _system(**kw):
    from neoxc import basis
    return basis.synthetic(**kw)


# one function; 31 / 32 / 33 primitive pairs around a warp; uneven contraction
# lengths; d shells; s-only classes; one geminal term
EDGE = [dict(seed=1, nat=1, nebf=1, nprim=1, npbf=1, ngtg=1, lmax_e=0, lmax_p=0),
        dict(seed=2, nat=2, nebf=2, nprim=(3, 5), npbf=2, ngtg=2, lmax_e=0, lmax_p=2),
        dict(seed=3, nat=3, nebf=3, nprim=(1, 3), npbf=3, ngtg=2, lmax_e=1, lmax_p=0),
        dict(seed=4, nat=2, nebf=7, nprim=1, npbf=1, ngtg=1, lmax_e=2, lmax_p=1),
        dict(seed=5, nat=1, nebf=8, nprim=1, npbf=2, ngtg=1, lmax_e=1, lmax_p=2)]


@pytest.mark.gpu
@pytest.mark.parametrize("kw", EDGE)
def test_tensors_at_the_edges(nx, orc, kw):
    s = _system(**kw)
    T = OracleTensors(orc, s)
    g2, g2s = nx.gam2_ic1(s)
    assert_close_scaled(g2, T.get("g2"), RTOL, "GM2ICR")
    assert_close_scaled(g2s, T.get("g2s"), RTOL, "GM2sICR")
    g, gx = nx.rxchfne_gam2_ic1(s)
    assert_close_scaled(g, T.get("rx2"), RTOL, "GM2ICR (RXCHF-ne)")
    assert_close_scaled(gx, T.get("rx2ex"), RTOL, "GM2exICR")


@pytest.mark.gpu
def test_long_contractions(nx):
    """A contracted function of 34 primitives (1156 primitive pairs, beyond a
    tile of the pair tables) of which two have a coefficient: the tensor of
    the two-primitive function, to the rounding of the same sums."""
    s = _system(seed=6, nat=2, nebf=1, nprim=34, npbf=1, ngtg=1, lmax_e=0, lmax_p=0)
    c = np.zeros(34)
    c[[3, 30]] = s.AGEBFCC[[3, 30]]
    long = dataclasses.replace(s, AGEBFCC=c)
    two = dataclasses.replace(s, npebf=2, ELCAM=s.ELCAM[[3, 30]], ELCEX=s.ELCEX[[3, 30]],
                              ELCBFC=s.ELCBFC[[3, 30]], AMPEB2C=s.AMPEB2C[:2], AGEBFCC=c[[3, 30]],
                              KPESTR=np.array([1]), KPEEND=np.array([2]))
    for f in (nx.gam2_ic1, nx.rxchfne_gam2_ic1):
        for x, y in zip(f(long), f(two)):
            assert_close_scaled(x, y, 1e-12, f.__name__)


@pytest.mark.gpu
def test_chunks_of_proton_pairs_match_single_slices(nx):
    """nebf = 20, npbf = 16: the scratch of one chunk does not hold all 136
    proton pairs.  The in-core energies equal those of the direct build, which
    takes one proton pair at a time, to the rounding of 4e7-term sums."""
    from neoxc import basis
    s = _system(seed=7, nat=2, nebf=20, nprim=1, npbf=16, ngtg=1, lmax_e=1, lmax_p=2)
    DE, DP = basis.random_density(20, 2, 3), basis.random_density(16, 1, 4, 1.0)
    g2, g2s = nx.gam2_ic1(s)
    a = nx.eg2ic1(20, 16, DE, DP, g2, g2s)
    b = nx.gam2_dscf(s, DE, DP)
    for x, y in ((a[0], b[0]), (a[2], b[1]), (a[1], b[2]), (a[3], b[3])):
        assert np.abs(x - y).max() <= 1e-11 * np.abs(y).max()
    assert abs(a[4] - b[4]) <= 1e-11 * np.abs(a[0]).max() * 20 and abs(a[5] - b[5]) <= 1e-11 * np.abs(a[1]).max() * 20
