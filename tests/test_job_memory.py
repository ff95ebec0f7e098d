"""The scratch of an XCHF solve's builders stays within what the batch and the
server admit its job for (neoxc_xchf_job_bytes counts the gam_2 build's scratch:
gam2_scratch_bound)."""
from __future__ import annotations

import ctypes as C
import random


def _functions():
    import neoxc
    L = neoxc.lib(build_if_missing=True)
    bound, factors = L["_ZN5neoxc18gam2_scratch_boundEiiiii"], L["_ZN5neoxc20gam3_factors_scratchEiiiiib"]
    bound.restype = factors.restype = C.c_size_t
    bound.argtypes, factors.argtypes = [C.c_int] * 5, [C.c_int] * 5 + [C.c_bool]
    return bound, factors


def test_gam3_factors_of_a_solve_take_no_more_than_its_gam2_build():
    bound, factors = _functions()
    rng = random.Random(3)
    sizes = [(34, 2, 3, 3)] + [(rng.randint(1, 64), rng.randint(1, 20), rng.randint(1, 6), rng.randint(1, 8))
                               for _ in range(300)]
    for ne, np_, prim, ng in sizes:
        nket, most = ne * (ne + 1) // 2 * prim * prim, prim * prim
        have = bound(ne, np_, nket, most, ng)
        assert factors(ne, np_, nket, most, ng, True) <= have, (ne, np_, prim, ng)
    # without W3 at hand its own chunks can take more: only a plain gam_3 build does that
    assert factors(34, 2, 34 * 35 // 2 * 9, 9, 3, False) > bound(34, 2, 34 * 35 // 2 * 9, 9, 3)
