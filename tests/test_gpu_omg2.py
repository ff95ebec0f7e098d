"""The fused RXCHF-ne OMG2 contraction (csrc/k_contract.cu omg2_kernel) against
torch at the edges of its panels and row blocks: one column, a lane's worth,
one column below and above a panel, several panels, row counts that are no
multiple of eight, the largest nebf."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,np_", [(1, 1), (3, 2), (5, 3), (6, 1), (17, 2), (18, 3), (25, 1), (40, 2), (57, 1), (128, 1)])
def test_omg2(nx, ne, np_):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(ne)
    r = lambda *n: torch.rand(*n, generator=gen, dtype=torch.float64, device="cuda") - 0.3  # noqa: E731
    n2, p2 = ne * ne, np_ * np_
    M, DP = r(p2 * n2, n2), r(np_, np_)
    DA, DB = r(ne, ne), r(ne, ne)
    DA = DA + DA.T   # densities are symmetric
    col = lambda x: x.T.contiguous().view(-1)  # noqa: E731
    fa, fp, fb, E = (torch.full((n,), 2.0, dtype=torch.float64, device="cuda") for n in (n2, p2, n2, 1))
    nx.dev_rxchfne_omg2(torch.cuda.current_stream().cuda_stream, ne, np_, col(DA), col(DB), col(DP), M.view(-1),
                        fa, fp, fb, E)
    u = torch.outer(DP.reshape(-1), DB.reshape(-1)).view(-1)
    v = M @ DA.reshape(-1)
    va = M.abs() @ DA.abs().reshape(-1)
    FA, FAs = u @ M, u.abs() @ M.abs()
    FB, FP = DP.reshape(-1) @ v.view(p2, n2), v.view(p2, n2) @ DB.reshape(-1)
    FBs, FPs = DP.abs().reshape(-1) @ va.view(p2, n2), va.view(p2, n2) @ DB.abs().reshape(-1)
    # sums of at most 2.7e8 FP64 products: their rounding stays below 1e-12 of
    # the sum of magnitudes
    for got, ref, s, n in ((fa, FA, FAs, ne), (fb, FB, FBs, ne), (fp, FP, FPs, np_)):
        assert ((got.view(n, n).T.reshape(-1) - 2.0 - ref).abs() <= 1e-12 * (s + 2.0)).all()
    assert (E - (FP * DP.reshape(-1)).sum()).abs().item() <= 1e-12 * (FPs * DP.abs().reshape(-1)).sum().item()
