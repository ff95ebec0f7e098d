"""Edges of the tensor-core factorised gam_4 build: tables whose rows can or
cannot be read two at a time, sizes beside the 8-wide load tiles, the 64-wide
K steps and the batches of the fockp dots, and accumulators that hold zeros
(which the integer FP32 -> FP64 widening leaves to the general conversion).

Compared with the FP64 factorised build.  Tolerance 2e-5 of the sum of the
magnitudes of an output's terms (the 24 permutations with every sign taken as
plus and |D|; four electrons in one orbital, as here for nebf < 6, cancel to
exactly zero): 3xTF32 products are good to about 2^-21, and K of them
accumulated in FP32 over at most 256 terms between FP64 folds stay below
2^-21 + 256 2^-24, 1.6e-5, even if every rounding had the same sign.
"""
from __future__ import annotations

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 2e-5


def _magnitudes(ne, np_, gee, g2s, DE, DP):
    import torch
    d = DE.abs().requires_grad_(True)
    D = d.view(ne, ne).T
    g = g2s.view(np_ * np_, -1)
    G = torch.mv(g.T, DP.abs().view(np_, np_).T.reshape(-1)).requires_grad_(True)

    def ket(t):
        return torch.einsum("abcy,xb->axcy", torch.einsum("abcd,yd->abcy", t.view((ne,) * 4), D), D)
    Gt, Et = ket(G), ket(gee)
    E = 0.0
    for s in itertools.permutations(range(4)):
        cycles, seen = 0, set()
        for i in range(4):
            if i not in seen:
                cycles += 1
                while i not in seen:
                    seen.add(i)
                    i = s[i]
        L = "abcd"
        E = E + 16.0 * 0.5 ** (4 - cycles) / 32.0 * torch.einsum(
            L[0] + L[s[0]] + L[1] + L[s[1]] + "," + L[2] + L[s[2]] + L[3] + L[s[3]] + "->", Gt, Et)
    E.backward()
    return [v.abs().max().item() for v in (d.grad, torch.mv(g, G.grad), E.detach())]


@pytest.mark.parametrize("ne,np_,zero,scale", [
    (1, 1, 0, 1.0), (2, 3, 0, 1.0), (5, 7, 0, 1.0), (8, 1, 0, 1.0), (9, 2, 0, 1.0), (16, 5, 0, 1.0),
    (23, 3, 0, 1.0), (24, 4, 0, 1.0), (31, 2, 0, 1.0), (40, 3, 0, 1.0), (12, 3, 7, 1.0), (10, 2, 0, 1e-20)])
def test_tc_factored_edges(nx, ne, np_, zero, scale):
    torch = pytest.importorskip("torch")
    from neoxc import basis
    dev = torch.device("cuda:0")
    f64 = torch.float64
    rng = np.random.default_rng(77 + 31 * ne + np_)
    ee = rng.uniform(0.0, scale, (ne,) * 4)
    ee[zero and ne - zero:zero and ne] = 0.0
    gs = rng.uniform(0.0, 1.0, (np_, np_) + (ne,) * 4)
    t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=f64, device=dev)  # noqa: E731
    gee = t(0.5 * (ee + ee.transpose(2, 3, 0, 1))).ravel()
    g2s = t(0.5 * (gs + gs.transpose(0, 1, 4, 5, 2, 3))).ravel()
    DE = t(basis.random_density(ne, max(1, ne // 3), ne, 2.0).ravel(order="F"))
    DP = t(basis.random_density(np_, 1, ne + 1, 1.0).ravel(order="F"))
    s = torch.cuda.current_stream(dev).cuda_stream
    out = []
    for fn in (nx.dev_gam4_fock_factored, nx.dev_gam4_fock_factored_tc):
        fe = torch.zeros(ne * ne, dtype=f64, device=dev)
        fp = torch.zeros(np_ * np_, dtype=f64, device=dev)
        E = torch.zeros(1, dtype=f64, device=dev)
        fn(s, ne, np_, gee, g2s, DE, DP, fe, fp, E)
        torch.cuda.synchronize(dev)
        out.append([x.cpu().numpy() for x in (fe, fp, E)])
    for x, y, m, w in zip(out[1], out[0], _magnitudes(ne, np_, gee, g2s, DE, DP), ("focke", "fockp", "E")):
        assert np.isfinite(x).all(), w
        assert np.abs(x - y).max() <= TOL * m, w
