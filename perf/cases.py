"""What a user of this framework has it do, as cases that can be timed and compared.

Families (the public entry point each one calls):

  scf        neoxc.xchf_scf          one whole XCHF solve from host arrays, integrals included
  batch      neoxc.xchf_scf_batch    a proton-position scan of the same molecule, 8 worker streams
  gam2       neoxc.gam2_ic1          the contracted XCHF gam_2 tensors
  gam2_rx    neoxc.rxchfne_gam2_ic1  the contracted RXCHF-ne gam_2 tensors
  gam3       neoxc.gam3_ic1          the contracted gam_3 tensor (FP64, or FP32 tables)
  gam4f      neoxc.dev_gam4_fock_factored      the factorised gam_4 Fock build, FP64
  gam4f_tc   neoxc.dev_gam4_fock_factored_tc   the same with its GEMMs on the tensor cores
  gam4_dscf  neoxc.dev_gam4_dscf     the element-wise direct-SCF gam_4 Fock build
  eg3        neoxc.dev_eg3ic1        the stored gam_3 tensor into the Fock matrices
  omg2       neoxc.dev_rxchfne_omg2  the stored RXCHF-ne gam_2 tensor into FAE, FP, FBE
  spin3      neoxc.dev_xcuhf_omg     the stored gam_3 tensor into the open-shell Fock matrices

The tensors of the contraction families are device-resident torch tensors (an SCF keeps them there
between iterations); the builders and solves take and return host arrays, as their callers hold them.
"""
import itertools
import json
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "neo-rxchf_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import neoxc  # noqa: E402
from neoxc import basis  # noqa: E402

F64 = torch.float64


def listed():
    return [
        # The molecule of the reference's xchf example with its proton displaced: one point of a scan,
        # solved from host arrays. The smallest whole call: latency of builders and iterations.
        {"name": "scf_example", "kind": "scf", "points": 1, "diis": True, "mixed": "none"},
        # A scan of 16 such points as one job list, gam_3 with FP32 tables: throughput of small solves.
        {"name": "scf_batch16", "kind": "batch", "points": 16, "diis": True, "mixed": "gam3"},
        # The gam_2 build of an ordinary small molecule (s/p electrons, s/p/d proton): one of the two
        # integral builds that a first solve waits for.
        {"name": "gam2_8x3", "kind": "gam2", "nat": 3, "nebf": 8, "nprim": 2, "npbf": 3, "ngtg": 3, "lmax_e": 1, "lmax_p": 2},
        # The RXCHF-ne gam_2 build with electronic d functions and five nuclei.
        {"name": "gam2_rx_9x4_d", "kind": "gam2_rx", "nat": 5, "nebf": 9, "nprim": 2, "npbf": 4, "ngtg": 4, "lmax_e": 2, "lmax_p": 2},
        # The gam_3 build, the largest cost of a solve with more than two electrons.
        {"name": "gam3_6x4", "kind": "gam3", "nat": 3, "nebf": 6, "nprim": 3, "npbf": 4, "ngtg": 3, "lmax_e": 1, "lmax_p": 2, "mixed": False},
        # The same at the smallest end with the FP32-table option.
        {"name": "gam3_4x2_mixed", "kind": "gam3", "nat": 3, "nebf": 4, "nprim": 2, "npbf": 2, "ngtg": 3, "lmax_e": 1, "lmax_p": 2, "mixed": True},
        # The gam_4 Fock build of every iteration, at a first solve's shape: short kernels.
        {"name": "gam4f_12x8", "kind": "gam4f", "ne": 12, "np": 8, "nocc": 2},
        # The same build at a large basis, on the tensor cores.
        {"name": "gam4f_tc_48x12", "kind": "gam4f_tc", "ne": 48, "np": 12, "nocc": 4},
        # The element-wise gam_4 build, for callers that want the reference's own evaluation.
        {"name": "gam4_dscf_8x4", "kind": "gam4_dscf", "ne": 8, "np": 4, "nocc": 2},
        # The in-core gam_3 contraction of every iteration: a 1.5 GB tensor.
        {"name": "eg3_12x8", "kind": "eg3", "ne": 12, "np": 8, "nocc": 2},
        # The RXCHF-ne contraction of every iteration at the largest in-core shape: an 8 GB tensor.
        {"name": "omg2_40x20", "kind": "omg2", "ne": 40, "np": 20, "nocc": 5},
        # The open-shell gam_3 contraction (alpha, beta and proton matrices in one call).
        {"name": "spin3_12x4", "kind": "spin3", "ne": 12, "np": 4, "nae": 2, "nbe": 2},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("scf", "batch", "gam2", "gam2_rx", "gam3", "gam4f", "gam4f", "gam4f_tc",
                       "gam4_dscf", "eg3", "omg2", "spin3"))
    if kind in ("scf", "batch"):
        return {"kind": kind, "points": 1 if kind == "scf" else rng.randint(2, 16), "diis": rng.random() < 0.75,
                "mixed": "none" if kind == "scf" else rng.choice(("none", "gam3")), "shift": rng.randint(1, 10 ** 6)}
    if kind in ("gam2", "gam2_rx", "gam3"):
        while True:
            c = {"kind": kind, "nat": rng.randint(2, 5), "nebf": rng.randint(3, 9 if kind != "gam3" else 6),
                 "nprim": rng.randint(1, 3), "npbf": rng.randint(1, 4), "ngtg": rng.randint(2, 4),
                 "lmax_e": rng.choice((0, 1, 1, 2) if kind == "gam2_rx" else (0, 1, 1)), "lmax_p": rng.choice((0, 1, 2))}
            if kind == "gam3":
                c["mixed"] = rng.random() < 0.4
            top = {"gam2": 5.5e6, "gam2_rx": 1.7e7, "gam3": 1.2e9}[kind]
            if _items(c) <= top:
                return c
    if kind == "gam4f":
        return {"kind": kind, "ne": _log(rng, 4, 40), "np": _log(rng, 1, 10), "nocc": rng.randint(2, 3)}
    if kind == "gam4f_tc":
        return {"kind": kind, "ne": rng.randint(10, 48), "np": _log(rng, 2, 12), "nocc": rng.randint(2, 6)}
    # (with one doubly occupied orbital the three- and four-electron terms vanish)
    if kind == "gam4_dscf":
        return {"kind": kind, "ne": rng.randint(3, 8), "np": _log(rng, 1, 4), "nocc": 2}
    if kind == "eg3":
        return {"kind": kind, "ne": rng.randint(3, 12), "np": _log(rng, 1, 8), "nocc": rng.randint(2, 3)}
    if kind == "omg2":
        return {"kind": kind, "ne": _log(rng, 6, 40), "np": _log(rng, 2, 20), "nocc": rng.randint(1, 5)}
    return {"kind": kind, "ne": rng.randint(3, 12), "np": _log(rng, 1, 4), "nae": rng.randint(2, 4), "nbe": rng.randint(1, 3)}


def _items(c):
    """Primitive integral evaluations of a builder case, the pair symmetry of the tensor not used
    (gam_2: primitive quartet and geminal term) or used (gam_3: composite bra and pair ket)."""
    n, m, g = c["nebf"] * c["nprim"], c["npbf"], c["ngtg"]
    if c["kind"] == "gam2":
        return n ** 4 * m ** 2 * (g + g * g)
    if c["kind"] == "gam2_rx":
        return n ** 4 * m ** 2 * g * g
    pairs = c["nebf"] * (c["nebf"] + 1) // 2 * c["nprim"] ** 2
    return m * (m + 1) * pairs ** 3 * g * g


# ---- inputs -------------------------------------------------------------------------------------
def _example():
    with open(os.path.join(_ROOT, "tests", "golden", "xchf_example.json")) as f:
        g = json.load(f)
    s = basis.parse_inp(g["inp"], name="examples/xchf")
    vec = basis.read_mo_file(g["guessCE"], s.nebf)
    return s, basis.density(vec, s.nelec // 2, 2.0)


def _rand(gen, n):
    """Signed values over several orders of magnitude, as geminal integrals have them."""
    u = torch.rand(n, generator=gen, dtype=F64, device="cuda")
    v = torch.rand(n, generator=gen, dtype=F64, device="cuda")
    return v.mul_(-6.0).exp_().mul_(u.sub_(0.25))


def _table(gen, ne, p2):
    """A pair-symmetric table t(p; ab; cd) = t(p; cd; ab), the layout of GAM_ee and GAM_2s."""
    t = _rand(gen, p2 * ne ** 4).view(p2, ne * ne, ne * ne)
    for p in range(p2):
        t[p] = 0.5 * (t[p] + t[p].T)
    return t.view(-1)


def _density(n, nocc, seed, prefac):
    d = basis.random_density(n, min(nocc, n), seed, prefac)
    return torch.from_numpy(np.ascontiguousarray(d.ravel(order="F"))).cuda()


def prepare(case, seed):
    c, k = dict(case), case["kind"]
    if k in ("scf", "batch"):
        s, DE = _example()
        pts = basis.proton_scan(s, c["points"], amplitude=0.3, seed=seed * 7919 + c.get("shift", 0))
        return {"c": c, "systems": pts, "DE": DE}
    if k in ("gam2", "gam2_rx", "gam3"):
        s = basis.synthetic(seed=seed, nat=c["nat"], nebf=c["nebf"], nprim=c["nprim"], npbf=c["npbf"],
                            ngtg=c["ngtg"], lmax_e=c["lmax_e"], lmax_p=c["lmax_p"])
        return {"c": c, "system": s}
    ne, np_ = c["ne"], c["np"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    st = {"c": c, "stream": torch.cuda.current_stream().cuda_stream, "DP": _density(np_, 1, seed + 2, 1.0)}
    n2, p2 = ne * ne, np_ * np_
    if k in ("gam4f", "gam4f_tc", "gam4_dscf"):
        st.update(gee=_table(gen, ne, 1), g2s=_table(gen, ne, p2), DE=_density(ne, c["nocc"], seed + 1, 2.0))
        sizes = (n2, p2, 1)
    elif k == "eg3":
        st.update(g=_rand(gen, ne ** 6 * p2), DE=_density(ne, c["nocc"], seed + 1, 2.0))
        sizes = (n2, p2, 1)
    elif k == "omg2":
        st.update(g=_rand(gen, ne ** 4 * p2), DA=_density(ne, c["nocc"], seed + 1, 2.0), DB=_density(ne, 1, seed + 3, 1.0))
        sizes = (n2, p2, n2, 1)
    else:
        st.update(g=_rand(gen, ne ** 6 * p2), DA=_density(ne, c["nae"], seed + 1, 1.0), DB=_density(ne, c["nbe"], seed + 3, 1.0))
        sizes = (n2, n2, p2, 6)
    # the output matrices in one buffer, so that a pass clears them (the calls add to them) with one fill
    st["out"] = torch.zeros(sum(sizes), dtype=F64, device="cuda")
    st["parts"] = list(st["out"].split(sizes))
    return st


# ---- one pass -----------------------------------------------------------------------------------
def _solve_out(r):
    return [np.array(list(r["initial"].values())), np.array(list(r["final"].values())), r["DE"], r["DP"],
            int(r["niter"]), bool(r["converged"])]


def run(st):
    c = st["c"]
    k = c["kind"]
    if k == "scf":
        r = neoxc.xchf_scf(st["systems"][0], st["DE"], diis=c["diis"], mixed=False if c["mixed"] == "none" else c["mixed"])
        return _solve_out(r)
    if k == "batch":
        r = neoxc.xchf_scf_batch(st["systems"], [st["DE"]] * len(st["systems"]), nworkers=8, diis=c["diis"],
                                 mixed=False if c["mixed"] == "none" else c["mixed"])
        o = [_solve_out(x) for x in r]
        return [np.stack([x[i] for x in o]) for i in range(4)] + [np.array([x[4] for x in o]), np.array([x[5] for x in o])]
    if k == "gam2":
        return list(neoxc.gam2_ic1(st["system"]))
    if k == "gam2_rx":
        return list(neoxc.rxchfne_gam2_ic1(st["system"]))
    if k == "gam3":
        return [neoxc.gam3_ic1(st["system"], mixed=c["mixed"])]
    o = st["parts"]
    st["out"].zero_()
    sp, ne, np_ = st["stream"], c["ne"], c["np"]
    if k == "gam4f":
        neoxc.dev_gam4_fock_factored(sp, ne, np_, st["gee"], st["g2s"], st["DE"], st["DP"], *o)
    elif k == "gam4f_tc":
        neoxc.dev_gam4_fock_factored_tc(sp, ne, np_, st["gee"], st["g2s"], st["DE"], st["DP"], *o)
    elif k == "gam4_dscf":
        neoxc.dev_gam4_dscf(sp, ne, np_, st["gee"], st["g2s"], st["DE"], st["DP"], *o)
    elif k == "eg3":
        neoxc.dev_eg3ic1(sp, ne, np_, st["DE"], st["DP"], st["g"], *o)
    elif k == "omg2":
        neoxc.dev_rxchfne_omg2(sp, ne, np_, st["DA"], st["DB"], st["DP"], st["g"], *o)
    else:
        neoxc.dev_xcuhf_omg(sp, 3, ne, np_, c["nae"], c["nbe"], st["g"], None, st["DA"], st["DB"], st["DP"],
                            d_FAE=o[0], d_FBE=o[1], d_FP=o[2], d_E=o[3])
    return o


# ---- the least work of one pass -----------------------------------------------------------------
#: Operations that one Coulomb evaluation over primitives cannot do without, whatever its angular
#: momenta: its exponent, distance, Boys function and one product.
_EVAL = 40


def work(case):
    c, k = case, case["kind"]
    if k in ("scf", "batch"):
        # the builders of the example's 6 contracted functions of 1 or 3 primitives (27 primitive pairs
        # of canonical contracted pairs times about 2), 3 geminal terms; the tensors are written once
        # and read twice (two Fock builds) in each of about 8 iterations
        pairs, ng3 = 63, 6 ** 6
        one = 2 * pairs ** 3 * 9 + 12 * pairs ** 2 * 12
        return {"bytes": c["points"] * 8.0 * (ng3 + 2 * 6 ** 4) * 17, "flops": float(c["points"]) * one * _EVAL}
    if k in ("gam2", "gam2_rx", "gam3"):
        n, m, g = c["nebf"], c["npbf"], c["ngtg"]
        pairs = n * (n + 1) // 2 * c["nprim"] ** 2
        mp = m * (m + 1) // 2
        if k == "gam3":
            return {"bytes": 8.0 * n ** 6 * m * m, "flops": 2.0 * mp * pairs ** 3 * g * g * _EVAL}
        terms = 3 * g * g if k == "gam2_rx" else 2 * g + g * g * (7 + 2 * c["nat"])
        return {"bytes": 16.0 * n ** 4 * m * m, "flops": 1.0 * mp * pairs ** 2 * terms * _EVAL}
    ne, p2 = c["ne"], c["np"] ** 2
    if k == "gam4_dscf":
        return {"bytes": 8.0 * ne ** 4 * (1 + p2), "flops": 2.0 * 42 * ne ** 8 * p2}
    if k in ("gam4f", "gam4f_tc"):
        # GAM_2s into G and, once W is known, into fockp: read once if it stays on the chip, else twice
        return {"bytes": 8.0 * ne ** 4 * (1 + p2), "flops": 2.0 * (2 * ne ** 4 * p2 + 8 * ne ** 5)}
    if k == "omg2":
        return {"bytes": 8.0 * ne ** 4 * p2, "flops": 4.0 * ne ** 4 * p2}
    return {"bytes": 8.0 * ne ** 6 * p2, "flops": 6.0 * ne ** 6 * p2}


# ---- the same in plain torch, 64 bits -----------------------------------------------------------
def _exact_gam4(st, ne, np_):
    """E = 1/32 sum over the 24 permutations s of c_s <G'(i1,i_s1,i2,i_s2), E'(i3,i_s3,i4,i_s4)>,
    c_s = 16 (-1/2)^(4 - cycles), T'(a,x,c,y) = sum_bd T(a,b,c,d) DE(x,b) DE(y,d), G = sum_p DP(p)
    GAM_2s(p); focke = dE/dDE, fockp(p) = dE/dDP(p) (both tables pair-symmetric)."""
    n = (ne,) * 4
    DE = st["DE"].clone().requires_grad_(True)
    d = DE.view(ne, ne).T   # DE(i,j) from the column-major buffer
    # DP(ip,jp) column-major against GAM_2s blocks with jp fastest
    dp = st["DP"].view(np_, np_).T.reshape(-1)
    g2s = st["g2s"].view(np_ * np_, -1)
    G = torch.mv(g2s.T, dp).requires_grad_(True)

    def ket(t):
        return torch.einsum("abcy,xb->axcy", torch.einsum("abcd,yd->abcy", t.view(n), d), d)
    Gt, Et = ket(G), ket(st["gee"])
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
        left, right = L[0] + L[s[0]] + L[1] + L[s[1]], L[2] + L[s[2]] + L[3] + L[s[3]]
        E = E + 16.0 * (-0.5) ** (4 - cycles) / 32.0 * torch.einsum(left + "," + right + "->", Gt, Et)
    E.backward()
    fp = torch.mv(g2s, G.grad).view(np_, np_).T.reshape(-1)
    return [DE.grad, fp.contiguous(), E.detach().view(1)]


def _exact_rank3(st, ne, np_, rows):
    """rows(t): the electron Fock rows [i1,j1] (one per class) of the proton-contracted tensor t =
    sum_p DP(p) G(p); each class's density weights its row into the energy, whose derivative by t
    gives the proton matrix."""
    dp = st["DP"].view(np_, np_).T.reshape(-1)
    g = st["g"].view(np_ * np_, -1)
    t = torch.mv(g.T, dp).requires_grad_(True)
    mats, dens = rows(t.view((ne,) * 6))
    E = sum((m * w).sum() for m, w in zip(mats, dens))
    grad = torch.autograd.grad(E, t)[0]
    fp = torch.mv(g, grad).view(np_, np_).T.reshape(-1).contiguous()
    return [m.detach() for m in mats], fp, E.detach()


def _perm(t, order):
    """t(i1,j,i2,j',i3,j'') with the kets taken in the given order of (j1,j2,j3)."""
    return torch.einsum("a%sb%sc%s->axbycz" % tuple("xyz"[o - 1] for o in order), t)


def exact(case, seed):
    k = case["kind"]
    if k not in ("gam4f", "gam4f_tc", "gam4_dscf", "eg3", "omg2", "spin3"):
        # a whole solve, or a builder: the primitive loops of the reference's integral formulas, which
        # take plain torch or numpy far over 20 seconds
        return None
    st = prepare(case, seed)
    ne, np_ = case["ne"], case["np"]
    if k in ("gam4f", "gam4f_tc", "gam4_dscf"):
        return _exact_gam4(st, ne, np_)
    if k == "omg2":
        m = st["g"].view(np_ * np_, ne * ne, ne * ne)          # [jp + np ip][j1 + ne i1][j2 + ne i2]
        flat = lambda v, n: v.view(n, n).T.reshape(-1)         # noqa: E731  column-major -> i*n + j
        da, db, dp = flat(st["DA"], ne), flat(st["DB"], ne), flat(st["DP"], np_)
        v = torch.matmul(m, da)                                # [p][i1 j1]
        fae = torch.mv(m.view(-1, ne * ne).T, torch.outer(dp, db).view(-1))
        fp, fbe = torch.mv(v, db), torch.mv(v.T, dp)
        return [flat(fae, ne).contiguous(), flat(fp, np_).contiguous(), flat(fbe, ne).contiguous(), (fp * dp).sum().view(1)]
    col = lambda x: x.T.reshape(-1).contiguous()               # noqa: E731  [i][j] -> column-major
    if k == "eg3":
        d = st["DE"].view(ne, ne).T

        def rows(t):
            g = (8.0 * t - 4.0 * _perm(t, (2, 1, 3)) + 2.0 * _perm(t, (3, 1, 2)) - 4.0 * _perm(t, (1, 3, 2))
                 + 2.0 * _perm(t, (2, 3, 1)) - 4.0 * _perm(t, (3, 2, 1))) / 8.0
            return [torch.einsum("axbycz,by,cz->ax", g, d, d)], [d]
        (f,), fp, E = _exact_rank3(st, ne, np_, rows)
        return [3.0 * col(f), fp, E.view(1)]
    a, b = st["DA"].view(ne, ne).T, st["DB"].view(ne, ne).T
    na, nb = case["nae"], case["nbe"]

    def classes(t, na, nb, a, b, proton):
        o213, o132, o321 = _perm(t, (2, 1, 3)), _perm(t, (1, 3, 2)), _perm(t, (3, 2, 1))
        r = torch.zeros((ne, ne), dtype=F64, device="cuda")
        con = lambda g, p, q: torch.einsum("axbycz,by,cz->ax", g, p, q)  # noqa: E731
        if na >= 3:
            r = r + con(t - o213 + _perm(t, (3, 1, 2)) - o132 + _perm(t, (2, 3, 1)) - o321, a, a)
        if na >= 2 and nb >= 1:
            r = r + con(t - o213, a, b) + con(t - o321, b, a)
        if nb >= 2 and (na >= 1 or not proton):
            r = r + con(t - o132, b, b)
        return r
    (fa, fb), fp, E = _exact_rank3(st, ne, np_, lambda t: (
        [classes(t, na, nb, a, b, False), classes(t, nb, na, b, a, False)], [a, b]))
    zero = torch.zeros((), dtype=F64, device="cuda")
    return [3.0 * col(fa), 3.0 * col(fb), fp, torch.stack([(fa * a).sum(), (fb * b).sum(), E, zero, zero, zero])]
