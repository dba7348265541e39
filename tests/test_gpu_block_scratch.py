"""What the block sweeps keep between calls: allocated before the first sweep,
and not needed for one."""
import numpy as np
import pytest
import torch

from ucfd_sparse_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def checkerboard(m):
    c = np.arange(m ** 3)
    return ((c % m + c // m % m + c // (m * m)) & 1).astype(np.int32)


@pytest.mark.parametrize("m", [4, 26])
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("reset", [False, True])
def test_first_sweeps_of_a_handle_are_captured(reset, prec, m, ucfd):
    """In the default capture mode, which refuses allocations."""
    from tests.test_gpu_blusgs import make
    b = mg.blusgs_case(m, permute=False, seed=m)
    got = []
    for graph in (False, True):
        S, e = make(b, prec=prec, on_device=True, colored=checkerboard(m))
        st = torch.cuda.Stream()
        S.set_stream(st.cuda_stream, True)
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            S.blusgs_pack(0, 0.0)
            S.blusgs_reset()
            S.blusgs_ns_prepare()
            if reset:
                S.blusgs_reset()
            torch.cuda.synchronize()
            if graph:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=st):
                    S.blusgs_ns_lower()
                    S.blusgs_ns_upper()
                g.replay()
            else:
                S.blusgs_ns_lower()
                S.blusgs_ns_upper()
            S.blusgs_update(0)
        torch.cuda.synchronize()
        got.append(e["upts"].cpu().numpy())
    assert not np.array_equal(got[0], b["upts"])
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("m", [4, 26])
@pytest.mark.parametrize("graph", [False, True])
def test_exact_sweeps_without_room_for_terms(graph, m, ucfd):
    """Where the terms' memory is not to be had every sweep forms every face;
    the values are the same."""
    from tests.test_gpu_blusgs import make
    from ucfd_sparse_gb300 import lib
    b = mg.blusgs_case(m, permute=False, seed=m)
    got = []
    for limit in (0, 8):
        lib.call("UCFDSelfTestScratchLimit", limit)
        try:
            S, e = make(b, on_device=True, colored=checkerboard(m))
            st = torch.cuda.Stream()
            S.set_stream(st.cuda_stream, True)
            torch.cuda.synchronize()
            with torch.cuda.stream(st):
                S.blusgs_pack(0, 0.0)
                S.blusgs_ns_prepare()
                for step in "RluulRlu":
                    {"R": S.blusgs_reset, "l": S.blusgs_ns_lower, "u": S.blusgs_ns_upper}[step]()
                if graph:
                    g = torch.cuda.CUDAGraph()
                    torch.cuda.synchronize()
                    with torch.cuda.graph(g, stream=st):
                        S.blusgs_ns_lower()
                        S.blusgs_ns_upper()
                    g.replay()
                    g.replay()
                    S.blusgs_ns_lower()
                S.blusgs_solve(1e-30, 3, 2)
                S.blusgs_update(0)
            torch.cuda.synchronize()
            got.append(e["upts"].cpu().numpy())
        finally:
            lib.call("UCFDSelfTestScratchLimit", 0)
    np.testing.assert_array_equal(got[0], got[1])
