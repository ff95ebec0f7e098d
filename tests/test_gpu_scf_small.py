"""The one-CTA kernels of an SCF iteration at odd and even orders (Jacobi pairs
with and without a dummy index, one to two warps of elements): the core guess
and its energies against LAPACK, and the solved density's idempotency.

Tolerances: the eigenvectors' rounding, 100 n eps, is scaled by the condition
of the overlap matrix through X = S^(-1/2); both sides then carry it."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,np_", [(1, 1), (2, 2), (3, 1), (5, 3), (6, 4), (8, 2), (9, 5)])
def test_core_guess_and_density(nx, ne, np_):
    from scipy.linalg import eigh
    from neoxc import basis
    s = basis.synthetic(seed=400 + ne, nat=3, nebf=ne, nprim=2, npbf=np_, ngtg=2, lmax_e=1, lmax_p=1, nelec=2)
    r = nx.xchf_scf(s, None, maxit=1)
    t = nx.onebody_integrals(s)
    m = {k: t[k].reshape(n, n) for k, n in (("Se", ne), ("GAM_ecore", ne), ("Sp", np_), ("GAM_pcore", np_))}
    D = {}
    for S, H, nn, pre in (("Se", "GAM_ecore", ne, 2.0), ("Sp", "GAM_pcore", np_, 1.0)):
        k = 0 if S == "Se" else s.nucst - 1
        c = eigh(m[H], m[S])[1][:, k]
        D[S] = pre * np.outer(c, c)
    gep = t["GAM_ep"].reshape(np_, np_, ne, ne)
    cond = max(np.linalg.cond(m["Se"]), np.linalg.cond(m["Sp"]))
    tol = 100 * max(ne, np_) * 2.2e-16 * cond
    ini = r["initial"]
    for got, want in ((ini["E_ecore"], (D["Se"] * m["GAM_ecore"]).sum()), (ini["E_pcore"], (D["Sp"] * m["GAM_pcore"]).sum()),
                      (ini["E_ep"], np.einsum("pqij,pq,ij->", gep, D["Sp"], D["Se"]))):
        assert abs(got - want) <= tol * abs(want), (got, want)
    for S, d, pre in (("Se", r["DE"], 2.0), ("Sp", r["DP"], 1.0)):
        assert np.abs(d @ m[S] @ d - pre * d).max() <= tol * np.abs(d).max()
        assert abs(np.trace(d @ m[S]) - pre) <= tol * pre
