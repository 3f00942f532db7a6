"""K+ on the device over the cluster sizes it picks (1, 2, 4 and 8 CTAs per subdomain), ragged last blocks and
unequal subdomains: K+ x of every subdomain against the host factor, and the whole solve (K+ at the
touched DOFs for b, the primal recovery) against the global direct solve."""
import numpy as np
import pytest

from espreso_b200 import feti4i as F
from espreso_b200 import problems
from tests.helpers import direct_u

pytestmark = pytest.mark.gpu

# blocks of 32 DOFs per subdomain: 1, 4, 24, 48 and 94 (cluster sizes 1, 1, 2, 4, 8), and unequal ones
CASES = {
    "heat_1": lambda: problems.heat_cube(domains=(3, 2, 1), elements=(2, 2, 2), seed=3),
    "heat_4": lambda: problems.heat_cube(domains=(2, 2, 2), elements=(4, 4, 4), seed=1),
    "elast_24": lambda: problems.elasticity_cube(domains=(2, 1, 1), elements=(5, 5, 6)),
    "elast_48": lambda: problems.elasticity_cube(domains=(2, 1, 1), elements=(7, 7, 7)),
    "elast_94": lambda: problems.elasticity_cube(domains=(2, 1, 1), elements=(9, 9, 9)),
    "uneven": lambda: problems.uneven_cube("elasticity", side=(16, 12, 12), levels=4, lo=3, hi=9, seed=2),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_kplus_and_solve(name):
    P = CASES[name]()
    opts = dict(iopts={F.PRECONDITIONER: F.PREC_LUMPED, F.VERBOSE_LEVEL: 0, F.MAX_ITERATIONS: 2000},
                ropts={F.PRECISION: 1e-11})
    inst = problems.make_instance(P, **opts)
    host = problems.make_instance(P, ext={F.EXT_HOST_ONLY: 1}, **opts)
    try:
        rng = np.random.default_rng(0)
        for d in range(int(inst.stats()["subdomains"])):
            x = rng.standard_normal(inst.subdomain_info(d)["ndofs"])
            a, b = inst.kplus(d, x), host.kplus(d, x)
            # two FP64 factorisations of one matrix, summed in different orders (the bound of the
            # device preprocessing's own K+ test)
            assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)
        u, ref = inst.solve().reshape(-1, P.dpn), direct_u(P)
        assert np.linalg.norm(u - ref) <= 1e-8 * np.linalg.norm(ref)
    finally:
        inst.destroy()
        host.destroy()


@pytest.mark.parametrize("name", ["heat_4", "elast_48", "elast_94", "uneven"])
@pytest.mark.parametrize("nrhs", [2, 9, 17])
def test_kplus_columns(name, nrhs):
    """The multi-column K+ (padded groups of 8 and 16, a last single column; 94 blocks keep 8 columns in
    shared memory) through whole solves: every column equals its own solve.  Both stop at 1e-11."""
    P = CASES[name]()
    inst = problems.make_instance(P, iopts={F.PRECONDITIONER: F.PREC_LUMPED, F.VERBOSE_LEVEL: 0, F.MAX_ITERATIONS: 2000},
                                  ropts={F.PRECISION: 1e-11})
    try:
        R = problems.traction_loads(P, nrhs, seed=nrhs)
        U = inst.solve_multi(R)
        for j in (0, nrhs // 2, nrhs - 1):
            inst.update_rhs(R[j])
            u = inst.solve()
            assert np.linalg.norm(U[j] - u) <= 1e-8 * np.linalg.norm(u)
    finally:
        inst.destroy()
