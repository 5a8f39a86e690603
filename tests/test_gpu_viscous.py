"""The viscous kernel at the edges of its chunks (32 points, 64 along i): one
chunk, one point more, several uneven chunks, walls and open faces.  The mixed
path's viscous RHS follows the plain one's, which the reference fixtures pin."""
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
    solver.FluxComputer.compute_viscous_rhs(fs)
    dq = fs.download(0, "dq")
    fs.close()
    return dq[:, 3:-3, 3:-3, 3:-3]


@pytest.mark.parametrize("dims,physical", SHAPES, ids=["x".join(map(str, s[0])) for s in SHAPES])
def test_mixed_rhs_follows_the_plain_one(dims, physical):
    case = cases.small_case("visc", dims=dims, noise_seed=6, physical=physical)
    a, b = _rhs(case, _lib.PREC_FP64), _rhs(case, _lib.PREC_MIXED)
    assert np.isfinite(a).all() and np.isfinite(b).all() and (a[0] == 0).all()
    # gradients of 1e-2 noise on velocities of 1 lose two digits of FP32's seven, the second difference another two
    err = np.sqrt(((a - b) ** 2).sum() / (a ** 2).sum())
    assert err <= 1e-3, err
