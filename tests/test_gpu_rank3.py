"""Stored rank-3 contractions (csrc/k_rank3.cu): EG3IC1 and the open-shell
FAE / UFP_OMG3 against the ket-permutation formulas in plain torch FP64, on
unsymmetric tensors, at the edges of the kernel's range (one function, fewer
ket pairs than threads, odd sizes, the largest nebf of each routine)."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

# every output is a sum of at most 28^4 * 4 products of FP64 numbers; its
# rounding error stays below 1e-12 of the sum of their magnitudes
TOL = 1e-12


def _perm(t, o):
    import torch
    return torch.einsum("a%sb%sc%s->axbycz" % tuple("xyz"[k - 1] for k in o), t)


def _rows(t, terms, flip=False):
    """sum over kets of coef * G(ket permutation) * d2 * d3 -> [i1, j1]."""
    import torch
    out = 0
    for coef, order, d2, d3 in terms:
        g = _perm(t, order) if order != (1, 2, 3) else t
        out = out + (abs(coef) if flip else coef) * torch.einsum("axbycz,by,cz->ax", g, d2, d3)
    return out


def _tensors(ne, np_, seed):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def r(*n):
        return torch.rand(*n, generator=gen, dtype=torch.float64, device="cuda") - 0.3
    return r(np_ * np_, ne ** 6), r(ne, ne), r(ne, ne), r(np_, np_)


def _check(got, ref, scale):
    assert (got - ref).abs().max().item() <= TOL * scale


def _col(d):
    return d.T.contiguous().view(-1)


@pytest.mark.parametrize("ne,np_", [(1, 1), (2, 3), (3, 2), (7, 2), (16, 1), (20, 1)])
def test_eg3ic1(nx, ne, np_):
    import torch
    G, D, _, DP = _tensors(ne, np_, 10 * ne + np_)
    fe, fp = torch.ones(ne * ne, dtype=torch.float64, device="cuda"), torch.ones(np_ * np_, dtype=torch.float64, device="cuda")
    E = torch.zeros(1, dtype=torch.float64, device="cuda")
    nx.dev_eg3ic1(torch.cuda.current_stream().cuda_stream, ne, np_, _col(D), _col(DP), G.view(-1), fe, fp, E)
    terms = [(1.0, (1, 2, 3), D, D), (-0.5, (2, 1, 3), D, D), (0.25, (3, 1, 2), D, D),
             (-0.5, (1, 3, 2), D, D), (0.25, (2, 3, 1), D, D), (-0.5, (3, 2, 1), D, D)]
    dp = DP.reshape(-1)
    A = [_rows(G[p].view((ne,) * 6), terms) for p in range(np_ * np_)]
    S = [_rows(G[p].abs().view((ne,) * 6), [(c, o, D.abs(), D.abs()) for c, o, _, _ in terms], True)
         for p in range(np_ * np_)]
    f = sum(3.0 * w * a for w, a in zip(dp, A))
    p = torch.stack([(D * a).sum() for a in A])
    sf = 1 + max(3.0 * s.max().item() for s in S) * np_ * np_
    sp = 1 + max((D.abs() * s).sum().item() for s in S)
    _check(fe, 1 + _col(f), sf)
    _check(fp, 1 + _col(p.view(np_, np_)), sp)
    _check(E, (p * dp).sum().view(1), sp * np_ * np_)


@pytest.mark.parametrize("ne,np_,na,nb", [(1, 1, 2, 2), (3, 2, 1, 3), (5, 1, 4, 2), (11, 2, 3, 1), (28, 1, 2, 2)])
def test_xcuhf_omg3(nx, ne, np_, na, nb):
    import torch
    G, A, B, DP = _tensors(ne, np_, 100 + ne)
    z = lambda n: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
    FA, FB, FP, E = z(ne * ne), z(ne * ne), z(np_ * np_), z(6)
    nx.dev_xcuhf_omg(torch.cuda.current_stream().cuda_stream, 3, ne, np_, na, nb, G.view(-1), None, _col(A),
                     _col(B), _col(DP), d_FAE=FA, d_FBE=FB, d_FP=FP, d_E=E)

    def terms(na, nb, a, b):
        t = []
        if na >= 3:
            t += [(1.0, (1, 2, 3), a, a), (-1.0, (2, 1, 3), a, a), (1.0, (3, 1, 2), a, a),
                  (-1.0, (1, 3, 2), a, a), (1.0, (2, 3, 1), a, a), (-1.0, (3, 2, 1), a, a)]
        if na >= 2 and nb >= 1:
            t += [(1.0, (1, 2, 3), a, b), (-1.0, (2, 1, 3), a, b), (1.0, (1, 2, 3), b, a), (-1.0, (3, 2, 1), b, a)]
        if nb >= 2:
            t += [(1.0, (1, 2, 3), b, b), (-1.0, (1, 3, 2), b, b)]
        return t
    ta, tb = terms(na, nb, A, B), terms(nb, na, B, A)
    dp = DP.reshape(-1)
    ra, rb = z(ne * ne).view(ne, ne), z(ne * ne).view(ne, ne)
    fp, s = [], 1.0
    for p in range(np_ * np_):
        t = G[p].view((ne,) * 6)
        a, b = ra + _rows(t, ta), rb + _rows(t, tb)
        s = max(s, (_rows(t.abs(), [(c, o, x.abs(), y.abs()) for c, o, x, y in ta + tb], True)).max().item())
        fp.append((A * a).sum() + (B * b).sum())
        FA -= 3.0 * dp[p] * _col(a)
        FB -= 3.0 * dp[p] * _col(b)
    s *= 3.0 * np_ * np_
    _check(FA, z(ne * ne), s)
    _check(FB, z(ne * ne), s)
    fp = torch.stack(fp).view(np_, np_)
    _check(FP, _col(fp), s * ne * ne)
    _check(E[2:3], (fp * DP).sum().view(1), s * ne * ne * np_ * np_)
