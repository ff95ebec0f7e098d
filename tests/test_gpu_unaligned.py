"""Device entry points on arrays that start at an odd multiple of eight bytes:
the results of the same values on an aligned start, bit for bit."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fn", ["dev_gam4_fock_factored_tc", "dev_gam4_fock_factored"])
@pytest.mark.parametrize("ne,np_", [(10, 2), (24, 3), (7, 2)])
def test_factored_gam4(nx, fn, ne, np_):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(ne)

    def r(*n):
        return torch.rand(*n, generator=gen, dtype=torch.float64, device="cuda") - 0.3

    def table(p):
        t = r(p, ne * ne, ne * ne)
        return (0.5 * (t + t.transpose(1, 2))).reshape(-1)
    ins = [table(1), table(np_ * np_), r(ne * ne), r(np_ * np_)]
    got = []
    for off in (0, 1):
        def at(x):
            buf = torch.empty(x.numel() + 2, dtype=torch.float64, device="cuda")
            v = buf[off:off + x.numel()]
            v.copy_(x)
            assert v.data_ptr() % 16 == 8 * off
            return v
        out = [at(torch.zeros(n, dtype=torch.float64, device="cuda")) for n in (ne * ne, np_ * np_, 1)]
        getattr(nx, fn)(torch.cuda.current_stream().cuda_stream, ne, np_, *[at(x) for x in ins], *out)
        got.append(out)
    for x, y in zip(*got):
        assert torch.isfinite(x).all() and torch.equal(x, y)
