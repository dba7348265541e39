"""Sweeps of levels at the sizes where the launch changes its shape."""
import numpy as np
import pytest
import torch

from ucfd_sparse_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


# checkerboard colours of 13/14, 6083/6084 (two lanes per face) and 6912 cells
# (one thread per cell): either side of the FP64 kernels' boundary at 6144
@pytest.mark.parametrize("m", [3, 23, 24])
def test_scalar_levels_either_side_of_the_lane_kernel(m, port, ucfd):
    from ucfd_sparse_gb300 import coloredlusgs as cl
    c = mg.lusgs_case(m)
    icolor = cl.make_coloring(m, m, m)
    ranges = [(m ** 3 + 1) // 2, m ** 3]
    c["lcolor"] = mg.colors_from_icolor(icolor, ranges)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    d = dict(c, **{k: dev(c[k]) for k in ("nei_ele", "fnorm_vol", "vec_fnorm", "fspr", "dt", "upts", "rhs", "lcolor")})
    diag = torch.zeros(c["neles"], dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    cl.colored_step(d, dev(icolor), ranges, diag, torch.zeros_like(d["rhs"]))
    ref = port.legacy_step(c, icolor, ranges, c["lcolor"])[0]
    np.testing.assert_array_equal(d["upts"].cpu().numpy(), ref)
