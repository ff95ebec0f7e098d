"""Device entry points under stream capture: their scratch becomes nodes of the
graph (never the library's own pool), and a replay gives what a call gives."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["factored", "eg3", "omg2", "omg3"])
def test_captured_call_replays(nx, which):
    import torch
    ne, np_ = 6, 3
    f64 = dict(dtype=torch.float64, device="cuda")
    r, z = (lambda n: torch.rand(n, **f64)), (lambda n: torch.zeros(n, **f64))
    g2, g3, gee, DE, DP = r(ne ** 4 * np_ ** 2), r(ne ** 6 * np_ ** 2), r(ne ** 4), r(ne * ne), r(np_ * np_)
    o = [z(ne * ne), z(np_ * np_), z(1)]
    call = {"factored": lambda s: nx.dev_gam4_fock_factored(s, ne, np_, gee, g2, DE, DP, *o),
            "eg3": lambda s: nx.dev_eg3ic1(s, ne, np_, DE, DP, g3, *o)}
    if which == "omg2":
        o = [z(ne * ne), z(np_ * np_), z(ne * ne), z(1)]
        call[which] = lambda s: nx.dev_rxchfne_omg2(s, ne, np_, DE, DE, DP, g2, *o)
    if which == "omg3":
        o = [z(ne * ne), z(ne * ne), z(np_ * np_), z(6)]
        call[which] = lambda s: nx.dev_xcuhf_omg(s, 3, ne, np_, 2, 2, g3, None, DE, DE, DP, d_FAE=o[0], d_FBE=o[1],
                                                 d_FP=o[2], d_E=o[3])
    st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    call[which](st.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=st):
        call[which](torch.cuda.current_stream().cuda_stream)
    for x in o:
        x.zero_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    got = [x.clone() for x in o]
    for x in o:
        x.zero_()
    torch.cuda.synchronize()
    call[which](st.cuda_stream)
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(got, o))
