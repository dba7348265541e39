"""Scalar LU-SGS calls captured into a caller's graph and launched between
eager calls: the values of the calls in the order in which the work runs."""
import numpy as np
import pytest
import torch

from ucfd_sparse_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu

# P Pack, n / r / b Prepare of the mean-flow system, of the turbulence system
# and of both, L / U sweeps of both, F spectral radii scaled by 1.5 in place,
# D Update; "(...)" is captured there, "g" launches the graph
ORDERS = {
    "sweeps_of_a_graph_after_separate_prepares": "Pb(LU)FPnrgD",
    "separate_prepares_in_the_graph": "Pnr(nr)FPbFPgLUD",
    "step_in_a_graph": "PbLU(PbLUD)gFgPbLUD",
    "captured_but_not_launched": "Pb(Fnr)LUD",
}


def run(fs, prec, color, order, graph):
    from tests.test_gpu_lusgs import make_flowsys
    S, e = make_flowsys(fs, fs, prec=prec, on_device=True, colored=color)
    lam = [torch.from_numpy(np.ascontiguousarray(fs[k])).cuda() for k in ("fspr", "tfspr")]
    S.set_lusgs(*lam)
    st = torch.cuda.Stream()
    S.set_stream(st.cuda_stream, True)
    torch.cuda.synchronize()

    def call(step):
        if step == "F":
            for t in lam:
                t.mul_(1.5)
        else:
            {"P": lambda: S.lusgs_pack(0, 1.5, 0.3), "n": S.lusgs_ns_prepare, "r": S.lusgs_rans_prepare,
             "b": S.lusgs_nsrans_prepare, "L": S.lusgs_nsrans_lower, "U": S.lusgs_nsrans_upper,
             "D": S.lusgs_update}[step]()

    with torch.cuda.stream(st):
        for step in "PbLU":  # every buffer a call needs is there before a capture
            call(step)
        inner, k = "", 0
        while k < len(order):
            if order[k] == "(":
                end = order.index(")", k)
                inner, k = order[k + 1:end], end + 1
                if graph:
                    g = torch.cuda.CUDAGraph()
                    torch.cuda.synchronize()
                    with torch.cuda.graph(g, stream=st):
                        for step in inner:
                            call(step)
                continue
            if order[k] == "g" and graph:
                g.replay()
            else:
                for step in inner if order[k] == "g" else order[k]:
                    call(step)
            k += 1
    torch.cuda.synchronize()
    return e["upts"].cpu().numpy()


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("order", sorted(ORDERS))
def test_launched_graph_equals_the_calls(order, prec, ucfd):
    m = 12
    fs = mg.lusgs_flowsys_case(m, nvars=6, permute=False)
    fs["dsrc"] = 0.1 * np.abs(fs["rhs"])
    c = np.arange(m ** 3)
    color = ((c % m + c // m % m + c // (m * m)) & 1).astype(np.int32)
    ref = run(fs, prec, color, ORDERS[order], False)
    got = run(fs, prec, color, ORDERS[order], True)
    assert np.isfinite(ref).all() and not np.array_equal(ref, fs["upts"])
    np.testing.assert_array_equal(got, ref)
