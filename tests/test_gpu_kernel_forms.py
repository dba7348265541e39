"""Launch variants at level sizes where they are different kernels: each form
of a sweep against another one that does not share its launch."""
import numpy as np
import pytest
import torch

from ucfd_sparse_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def checkerboard(m):
    c = np.arange(m ** 3)
    return ((c % m + c // m % m + c // (m * m)) & 1).astype(np.int32)


@pytest.mark.parametrize("threads", [64, 256])
def test_chained_float_block_sweeps_equal_the_face_loop(threads, port, ucfd):
    """FP32 levels above and below 16384 cells (greedy colours of 40^3 cells):
    the kernels whose launches are chained (variant 0: unrolled, and blocks in
    registers for small levels) against the face loop launched level after
    level (variant 1), bit for bit, and within 1e-4 of the FP64 mode's change."""
    from tests.test_gpu_blusgs import make, run_sweeps
    from ucfd_sparse_gb300 import coloredlusgs as cl
    b = mg.blusgs_case(40, seed=6)
    _, rg, lc = cl.greedy_coloring_csr(b["rowptr"], b["colidx"])
    sizes = np.diff([0] + rg)
    assert sizes.max() > 16384 and sizes.min() < 16384
    outs = []
    for prec, var in ((2, 0), (2, 1), (0, 0)):
        S, e = make(b, prec=prec, on_device=True, colored=lc)
        S.set_launch_config(threads_per_block=threads, sweep_variant=var)
        run_sweeps(S, 3)
        outs.append(e["upts"].cpu().numpy())
    np.testing.assert_array_equal(outs[1], outs[0])
    d, r = outs[0] - b["upts"], outs[2] - b["upts"]
    assert np.abs(d - r).max() <= 1e-4 * np.abs(r).max()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("threads", [64, 256])
def test_block_variants_of_large_fp64_levels(prec, threads, ucfd):
    """Colours of 8788 cells, more than the lane-per-row kernel takes: the
    unrolled kernel and the face loop in FP64, with kept terms or sums."""
    from tests.test_gpu_blusgs import make, run_sweeps
    b = mg.blusgs_case(26, permute=False, seed=9)
    outs = []
    for var in (0, 1):
        S, e = make(b, prec=prec, on_device=True, colored=checkerboard(26))
        S.set_launch_config(threads_per_block=threads, sweep_variant=var)
        run_sweeps(S, 3)
        outs.append(e["upts"].cpu().numpy())
    np.testing.assert_array_equal(outs[1], outs[0])


@pytest.mark.parametrize("nvars", [5, 6])
@pytest.mark.parametrize("prec", [0, 1])
def test_scalar_register_caps_of_fp64_levels(nvars, prec, port, ucfd):
    """Colours of 13500 cells, between the levels of the lanes kernel and those
    with a thread per active face: the three register budgets (variants 0-2),
    two threads per cell (3, 4) and the face lists (5)."""
    from tests.test_gpu_lusgs import make_flowsys
    fs = mg.lusgs_flowsys_case(30, nvars=nvars, permute=False)
    fs["dsrc"] = 0.1 * np.abs(fs["rhs"])
    color = checkerboard(30)
    outs = []
    for var in range(6):
        S, e = make_flowsys(fs, fs, prec=prec, on_device=True, colored=color)
        S.set_launch_config(threads_per_block=64, sweep_variant=var)
        S.lusgs_pack(0, 1.5, 0.3)
        S.lusgs_ns_prepare(1.01)
        S.lusgs_ns_lower(1.01)
        S.lusgs_ns_upper(1.01)
        if nvars > 5:
            S.lusgs_rans_prepare(1.01)
            S.lusgs_rans_lower(1.01)
            S.lusgs_rans_upper(1.01)
        S.lusgs_update(0)
        outs.append(e["upts"].cpu().numpy())
    for o in outs[1:]:
        np.testing.assert_array_equal(o, outs[0])
    if prec == 0:
        new = np.empty(fs["nlocal"], dtype=np.int64)
        new[np.argsort(color, kind="stable")] = np.arange(fs["nlocal"])
        ref = port.flowsys_lusgs_step(mg.renumber_flowsys(fs, new), fs["upts"], fs["rhs"], fs["dt"], fs["dsrc"],
                                      fs["fspr"], fs["tfspr"], kappa=1.01, a0=0.3, turb_factor=1.5,
                                      rans=nvars > 5)[0]
        np.testing.assert_array_equal(outs[0], ref)


# colours of 8064 / 8065 (two lanes per face) and 8320 / 8321 quadrilaterals
# (one thread per cell): either side of the line for rows of four faces
@pytest.mark.parametrize("m", [127, 129])
@pytest.mark.parametrize("nvars", [4, 6])
@pytest.mark.parametrize("prec", [0, 1])
def test_plane_levels_either_side_of_the_lane_kernel(m, nvars, prec, ucfd):
    from tests.test_gpu_level_shapes import test_plane_levels as same_as_two_threads_per_cell
    same_as_two_threads_per_cell(m, nvars, prec, ucfd)
