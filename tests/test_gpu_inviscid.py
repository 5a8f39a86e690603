"""The inviscid kernel at the edges of its chunks: lines of one chunk, one point
more than a chunk (32 points, 64 along i), several uneven chunks, and flagged
ends (walls, far field, freestream, extrapolation) at both ends of short and
long lines.  Chunked lines give what the parts of a split case give: a case and
its one-kernel halves are compared in the other tests; here the mixed path's
RHS is held to the plain one's, which the reference fixtures pin."""
import numpy as np
import pytest

from orion_b200 import _lib, cases, solver

pytestmark = pytest.mark.gpu

OPEN = {"imin": cases.BC_FREESTREAM, "imax": cases.BC_EXTRAPOLATION, "kmax": cases.BC_EXTRAPOLATION}
SHAPES = [((12, 12, 12), None), ((64, 32, 32), None), ((65, 33, 33), None), ((129, 65, 34), OPEN), ((70, 97, 13), OPEN)]


def _rhs(case, precision):
    fs = solver.FlowFieldSet(case, precision=precision)
    solver.apply_physical_bc(None, fs)
    solver.StateUpdater.update_flow_states(fs)
    solver.InviscidFluxComputer.compute_inviscid_rhs(fs)
    dq = fs.download(0, "dq")
    fs.close()
    return dq[:, 3:-3, 3:-3, 3:-3]


@pytest.mark.parametrize("dims,physical", SHAPES, ids=["x".join(map(str, s[0])) for s in SHAPES])
def test_mixed_rhs_follows_the_plain_one(dims, physical):
    case = cases.small_case("inv", dims=dims, noise_seed=6, nvis=0, physical=physical)
    a, b = _rhs(case, _lib.PREC_FP64), _rhs(case, _lib.PREC_MIXED)
    # FP32 fluxes of size p |k| differenced with weights of at most 27/24 x 4 per direction: each rounds
    # within a few eps32 (6e-8) of the largest flux, about 3 |k|; the noise makes dq about 1e-2 of it
    assert np.isfinite(a).all() and np.isfinite(b).all()
    err = np.sqrt(((a - b) ** 2).sum() / (a ** 2).sum())
    assert err <= 1e-3, err


@pytest.mark.parametrize("component", [1, 2, 3])
def test_overflowing_smoothness_drops_its_stencils(component):
    """A velocity of 1e80 at one point overflows the squared smoothness measure
    of every stencil that holds it.  Those weights are c / inf = 0, so a state
    one or two points away comes from the stencils without it and is finite:
    only the two faces at the point are not, and dq only up to three points
    from it along its three lines."""
    n, s = 40, 20
    case = cases.small_case("inf", dims=(n, n, n), noise_seed=6, nvis=0)
    fs = solver.FlowFieldSet(case, precision=_lib.PREC_FP64)
    solver.apply_physical_bc(None, fs)
    prim = fs.download(0, "prim")
    prim[component, 3 + s, 3 + s, 3 + s] = 1e80
    fs.upload(0, "prim", prim)
    solver.StateUpdater.update_flow_states(fs)
    solver.InviscidFluxComputer.compute_inviscid_rhs(fs)
    dq = fs.download(0, "dq")[:, 3:-3, 3:-3, 3:-3]
    fs.close()
    near = np.zeros((n, n, n), bool)
    near[s - 3:s + 4, s, s] = near[s, s - 3:s + 4, s] = near[s, s, s - 3:s + 4] = True
    assert np.isfinite(dq[:, ~near]).all()
