"""Pack through records, and without them where their memory is not to be had."""
import numpy as np
import pytest
import torch

from ucfd_sparse_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvars", [5, 6])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_pack_without_room_for_records(nvars, prec, ucfd):
    """51^3 = 132651 cells, from 131072 on through records: the schedule built
    and the steps made with and without room for them."""
    from tests.test_gpu_lusgs import make_flowsys
    from ucfd_sparse_gb300 import lib
    fs = mg.lusgs_flowsys_case(51, nvars=nvars)
    fs["dsrc"] = 0.1 * np.abs(fs["rhs"])
    c = np.arange(51 ** 3)
    color = np.empty(51 ** 3, dtype=np.int32)
    color[fs["cell_ids"]] = (c % 51 + c // 51 % 51 + c // 51 ** 2) & 1
    got = []
    for limit in (0, 8):
        lib.call("UCFDSelfTestScratchLimit", limit)
        try:
            S, e = make_flowsys(fs, fs, prec=prec, on_device=True, colored=color)
            for k in range(2):
                S.lusgs_pack(0, 1.5, 0.3)
                S.lusgs_run(2, rans=nvars > 5)
                S.lusgs_update(0)
                S.lusgs_pack(0, 1.0, 0.0)
                S.lusgs_ns_prepare(1.0)
                S.lusgs_ns_lower(1.0)
                S.lusgs_ns_upper(1.0)
                S.lusgs_update(0)
                e["rhs"].mul_(-0.5)
                torch.cuda.synchronize()
        finally:
            lib.call("UCFDSelfTestScratchLimit", 0)
        got.append(e["upts"].cpu().numpy())
    assert np.isfinite(got[0]).all() and not np.array_equal(got[0], fs["upts"])
    np.testing.assert_array_equal(got[0], got[1])
