"""The tile wavefront sweeps at the edges of their tiling: one tile, ragged
last tiles, thin blocks, several tiles a direction, several blocks.  The plain
path is bit-identical to one launch per hyperplane (the same operations in the
same order); the mixed path's neighbour term is the same sum simplified, held
to the mixed tolerance (1e-6 relative L2)."""
import numpy as np
import pytest

from orion_b200 import _lib, cases, solver

pytestmark = pytest.mark.gpu

SHAPES = [((12, 12, 12), (1, 1, 1), 1), ((13, 47, 12), (1, 1, 1), 1), ((12, 12, 61), (1, 1, 1), 1),
          ((97, 33, 29), (1, 1, 1), 0), ((45, 26, 41), (2, 2, 3), 1), ((61, 75, 37), (3, 1, 2), 1)]


def _run(case, precision, sweep):
    fs = solver.FlowFieldSet(case, precision=precision)
    fs.set_schedule(sweep, 0, 16)
    h = fs.step(3)
    st = [fs.download(b, "prim") for b in range(len(case.blocks))]
    fs.close()
    return h, st


@pytest.mark.parametrize("dims,split,nvis", SHAPES, ids=["x".join(map(str, s[0])) for s in SHAPES])
def test_tiles_match_the_hyperplane_launches(dims, split, nvis):
    case = cases.small_case("tiles", dims=dims, split=split, noise_seed=3, moo=0.7, nvis=nvis)
    a, b = (_run(case, _lib.PREC_FP64, s) for s in ("planes", "tiles"))
    assert np.array_equal(a[0], b[0])
    assert all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))
    a, b = (_run(case, _lib.PREC_MIXED, s)[1] for s in ("planes", "tiles"))
    cut = (slice(0, 5),) + (slice(3, -3),) * 3
    num = sum(float(np.sum((x[cut] - y[cut]) ** 2)) for x, y in zip(a, b))
    assert (num / sum(float(np.sum(x[cut] ** 2)) for x in a)) ** 0.5 <= 1e-6


def test_switching_forms_keeps_the_arrays_apart():
    """The tile form and the hyperplane forms share their memory: going back
    and forth steps exactly as one form does."""
    case = cases.small_case("switch", dims=(33, 25, 23), split=(2, 1, 1), noise_seed=8)
    ref, _ = _run(case, _lib.PREC_FP64, "planes")
    fs = solver.FlowFieldSet(case, precision=_lib.PREC_FP64)
    got = []
    for sweep in ("tiles", "planes", "tiles"):
        fs.set_schedule(sweep, 0, 16)
        got.append(fs.step(1))
    fs.close()
    assert np.array_equal(np.vstack(got), ref)


# More than 9,472 lines, the least that FP64 cases take tiles of up to 96 lines for
LARGE = [((25, 131, 97), (1, 1, 1), 1), ((17, 140, 143), (1, 2, 3), 0), ((13, 12, 797), (1, 1, 1), 1)]


@pytest.mark.parametrize("dims,split,nvis", LARGE, ids=["x".join(map(str, s[0])) for s in LARGE])
def test_large_tiles_match_the_hyperplane_launches(dims, split, nvis):
    case = cases.small_case("tiles_large", dims=dims, split=split, uneven_seed=3 if max(split) > 1 else None,
                            noise_seed=3, moo=0.7, nvis=nvis)
    assert sum(b.jdim * b.kdim for b in case.blocks) > 9472
    a, b = (_run(case, _lib.PREC_FP64, s) for s in ("planes", "tiles"))
    assert np.array_equal(a[0], b[0])
    assert all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))


@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED], ids=["plain", "mixed"])
def test_a_group_of_small_and_large_tiles_steps_as_its_members_alone(precision):
    """Plain: members of 64-line tiles run in the launch of the 96-line ones."""
    specs = [dict(name="tl", dims=(25, 131, 97), noise_seed=3), dict(name="ts", dims=(33, 25, 23), split=(2, 1, 1), noise_seed=4),
             dict(name="to", dims=(13, 47, 12), noise_seed=5, moo=0.7)]
    sets = [solver.FlowFieldSet(cases.small_case(**sp), precision=precision) for sp in specs]
    alone = []
    for sp in specs:
        fs = solver.FlowFieldSet(cases.small_case(**sp), precision=precision)
        alone.append((fs.step(3), [fs.download(b, "prim") for b in range(len(fs.case.blocks))]))
        fs.close()
    g = solver.CaseGroup(sets)
    hists = g.step(3)
    g.close()
    for (h, st), hg, fs in zip(alone, hists, sets):
        assert np.array_equal(h, hg)
        assert all(np.array_equal(x, fs.download(b, "prim")) for b, x in enumerate(st))
        fs.close()
