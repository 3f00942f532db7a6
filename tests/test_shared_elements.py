"""A matrix and the instances made from it share their element data until one of them changes: later changes
of the matrix do not reach an instance, scaled updates do not reach the matrix (CPU, host preprocessing)."""
import numpy as np

from espreso_b200 import feti4i as F
from espreso_b200 import problems

OPTS = dict(iopts={F.PRECONDITIONER: F.PREC_LUMPED, F.VERBOSE_LEVEL: 0})


def _matrix(P):
    M = F.Matrix(0)
    M.add_elements(P.elem_nodes, P.elem_dofs(), P.Ke)
    M.set_partition(P.elem_domain)
    return M


def _instance(M, P):
    F.set_extended(F.EXT_HOST_ONLY, 1)
    try:
        dd, dv = P.dirichlet_dofs()
        return F.Instance(M, P.rhs(), dd, dv, **OPTS)
    finally:
        F.set_extended(F.EXT_HOST_ONLY, 0)


def test_matrix_changes_after_the_instance():
    P = problems.heat_cube(domains=(2, 2, 1), elements=(3, 3, 3), seed=2)
    M = _matrix(P)
    inst = _instance(M, P)
    S = [inst.schur(d) for d in range(4)]
    M.add_element(P.elem_nodes[0], P.elem_dofs()[0], 5.0 * P.Ke[0])   # the matrix takes its own copy
    assert inst.stats()["elements"] == P.elem_nodes.shape[0]
    inst.set_extended(F.EXT_SCALING, 0)                               # rebuilds from the instance's elements
    for d in range(4):
        assert np.allclose(inst.schur(d), S[d], rtol=1e-12, atol=1e-12 * np.abs(S[d]).max())
    M.destroy()
    inst.destroy()


def test_scaled_updates_leave_the_matrix():
    P = problems.elasticity_cube(domains=(2, 1, 1), elements=(2, 2, 3))
    M = _matrix(P)
    inst, other = _instance(M, P), _instance(M, P)
    S = inst.schur(0)
    ne = P.elem_nodes.shape[0]
    inst.update_matrix_scaled(M, 4.0 * np.ones(ne))
    tol = dict(rtol=0, atol=1e-9 * np.abs(S).max())   # S scales with 1/K up to the regularisation's rounding
    assert np.allclose(4.0 * inst.schur(0), S, **tol)
    assert np.allclose(other.schur(0), S, rtol=0, atol=0)
    inst.update_matrix_scaled(M, np.ones(ne))
    assert np.allclose(inst.schur(0), S, **tol)
    other.update_matrix(M)
    assert np.allclose(other.schur(0), S, **tol)
    M.destroy()
    inst.destroy()
    other.destroy()


def test_blocks_with_skipped_elements():
    """A block of elements with a zero one falls back to the element-by-element rule (it is skipped)."""
    P = problems.heat_cube(domains=(2, 1, 1), elements=(2, 2, 2), seed=1)
    K = P.Ke.copy()
    K[3] = 0.0
    M = F.Matrix(0)
    M.add_elements(P.elem_nodes, P.elem_dofs(), K)
    M.set_partition(np.delete(P.elem_domain, 3))
    inst = _instance(M, P)
    assert inst.stats()["elements"] == P.elem_nodes.shape[0] - 1
    M.destroy()
    inst.destroy()
