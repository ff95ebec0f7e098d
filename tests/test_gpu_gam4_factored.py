"""The four-launch factorised gam_4 build (csrc/k_gam4f.cu) against E as a sum
over the 24 permutations in plain torch FP64 and its gradients, at the edges
of its tiles: one function, tiles smaller than a CTA with idle and shared
proton-pair groups, just below and above 32 and 1024 elements, the largest
nebf, proton-pair counts that are no multiple of four or 32."""
from __future__ import annotations

import itertools

import pytest

pytestmark = pytest.mark.gpu
RTOL = 1e-10   # the contraction tolerance of the parity tests, of the output's scale


def _reference(ne, np_, gee, g2s, DE, DP):
    import torch
    d = DE.clone().requires_grad_(True)
    D = d.view(ne, ne).T
    dp = DP.view(np_, np_).T.reshape(-1)
    g = g2s.view(np_ * np_, -1)
    G = torch.mv(g.T, dp).requires_grad_(True)

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
        E = E + 16.0 * (-0.5) ** (4 - cycles) / 32.0 * torch.einsum(
            L[0] + L[s[0]] + L[1] + L[s[1]] + "," + L[2] + L[s[2]] + L[3] + L[s[3]] + "->", Gt, Et)
    E.backward()
    return d.grad, torch.mv(g, G.grad).view(np_, np_).T.reshape(-1), E.detach()


@pytest.mark.parametrize("ne,np_", [(1, 1), (2, 7), (5, 3), (6, 1), (16, 2), (17, 3), (31, 1), (32, 2), (33, 1), (64, 1)])
def test_factored_build(nx, ne, np_):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(ne * 100 + np_)

    def table(p):
        t = torch.rand(p, ne * ne, ne * ne, generator=gen, dtype=torch.float64, device="cuda") - 0.2
        return (0.5 * (t + t.transpose(1, 2))).reshape(-1)
    gee, g2s = table(1), table(np_ * np_)
    DE = torch.rand(ne * ne, generator=gen, dtype=torch.float64, device="cuda") / ne
    DP = torch.rand(np_ * np_, generator=gen, dtype=torch.float64, device="cuda")
    z = lambda n: torch.full((n,), 0.5, dtype=torch.float64, device="cuda")  # noqa: E731
    fe, fp, E = z(ne * ne), z(np_ * np_), z(1)
    for _ in range(2):   # outputs accumulate, E is overwritten, the scratch is reused
        nx.dev_gam4_fock_factored(torch.cuda.current_stream().cuda_stream, ne, np_, gee, g2s, DE, DP, fe, fp, E)
    rfe, rfp, rE = _reference(ne, np_, gee, g2s, DE, DP)
    assert (fe - 0.5 - 2 * rfe).abs().max() <= RTOL * max(1.0, rfe.abs().max().item())
    assert (fp - 0.5 - 2 * rfp).abs().max() <= RTOL * max(1.0, rfp.abs().max().item())
    assert (E - rE).abs().max() <= RTOL * max(1.0, (DP * rfp).abs().sum().item())
