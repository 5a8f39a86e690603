"""The packed output's staging buffer: sized for the case's largest block
whichever is packed first, one call at a time over it, and never taken from a
capturing stream.  Packed values are compared with numpy's on the same state
(FP64, then rounded to FP32)."""
import concurrent.futures as cf

import numpy as np
import pytest

from orion_b200 import _lib, cases, output, solver
from test_output_cpu import _fields_from_prim

pytestmark = pytest.mark.gpu


def test_blocks_of_different_sizes_from_several_threads():
    case = cases.small_case("pack", dims=(59, 17, 13), split=(3, 1, 1), uneven_seed=4, noise_seed=5)
    fs = solver.FlowFieldSet(case)
    want = [_fields_from_prim(fs.download(b, "prim"), case.params.gamma) for b in range(len(case.blocks))]
    order = sorted(range(len(case.blocks)), key=lambda b: int(np.prod(case.blocks[b].dims))) * 4
    with cf.ThreadPoolExecutor(4) as pool:
        got = list(pool.map(lambda b: output.pack_block(fs, b), order))
    for b, g in zip(order, got):
        # the temperature and Mach number are one division or square root away: an ulp of FP32
        np.testing.assert_allclose(g, want[b], rtol=2.4e-7, atol=0)
    fs.close()


def test_a_capturing_stream_is_refused():
    import torch

    fs = solver.FlowFieldSet(cases.small_case("pack_cap", dims=(17, 13, 13), noise_seed=3))
    fs.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.ExternalStream(fs.stream_ptr())):
        g.capture_begin()
        try:
            with pytest.raises(_lib.OrionError, match="capturing"):
                output.pack_block(fs, 0)
        finally:
            g.capture_end()
    del g
    assert np.isfinite(output.pack_block(fs, 0)).all()
    fs.close()


@pytest.mark.parametrize("split", [(1, 1, 1), (2, 1, 1)])
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED], ids=["plain", "mixed"])
def test_the_footprint_counts_the_staging_buffer(precision, split):
    case = cases.small_case("pack_fp", dims=(49, 45, 41), split=split, noise_seed=3)
    fs = solver.FlowFieldSet(case, precision=precision)
    before = fs.footprint()
    for b in range(len(case.blocks)):
        output.pack_block(fs, b)
    assert fs.footprint() == before + 28 * max(int(np.prod(b.dims)) for b in case.blocks)
    # the work lists too: 1/64 of the arena
    assert solver.footprint_estimate(case, precision) >= fs.footprint() + before // 64
    fs.close()
