"""Jobs of a batch or a server whose sizes no solve accepts: each gets its own
error, and the jobs beside them their results."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _jobs(nx, s, DE):
    """The molecule, and the same with nebf = 0, npbf = 0, nebf = -3, ngtg1 = 0,
    nebf beyond the limit (one electron: its tensors are not counted)."""
    bad = [("nebf", 0), ("npbf", 0), ("nebf", -3), ("ngtg1", 0), ("nebf", 65)]
    jobs = (nx.XchfJob * (len(bad) + 1))()
    bufs = [nx._fill_job(j, s, DE, None, 40) for j in jobs]
    for j, (name, v) in zip(jobs[1:], bad):
        setattr(j, name, v)
    jobs[len(bad)].nelec = 1
    return jobs, bufs


def test_batch(nx, xchf):
    jobs, bufs = _jobs(nx, xchf["sys"], xchf["DE0"])
    opts = nx._scf_options(True, True, False, False)
    rc = nx.lib().neoxc_xchf_scf_batch(C.cast(jobs, C.c_void_p), len(jobs), 2, opts, 40)
    st = [int(j.status) for j in jobs]
    assert rc != 0 and st[0] == 0 and all(x != 0 for x in st[1:]), st
    ref = nx.xchf_scf(xchf["sys"], xchf["DE0"], maxit=40, diis=True)
    got = nx._job_result(jobs[0], bufs[0])
    assert np.array_equal(got["DE"], ref["DE"]) and got["final"] == ref["final"]
