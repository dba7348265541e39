"""Block LU-SGS calls captured into a caller's graph and launched between
eager calls: the same values as the eager calls in the order in which the work
runs, bit for bit, whatever the host knew when the graph was captured."""
import ctypes

import numpy as np
import pytest
import torch

from ucfd_sparse_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


# One letter a call: l / u lower / upper sweep, R Reset, P Pack of a right-hand
# side scaled by -0.75, J Prepare of Jacobians scaled by 1.25, S a Solve of a
# few sweeps.  "(...)" is captured there, not run; "g" launches the graph (the
# eager twin runs its calls instead).
ORDERS = {
    "one_direction_launched_twice": "R(l)gg",
    "upper_alone_launched_twice": "Rl(u)gg",
    "captured_but_not_launched": "lu(l)uu",
    "pair": "R(lu)gggl",
    "pair_after_eager_pair": "Rlu(lu)gglug",
    "solve_between_launches": "R(lu)gSgl",
    "solve_before_update": "R(lu)gS",
    "solve_then_launch": "R(lu)gSg",
    "prepare_between_launches": "R(lu)gJgl",
    "pack_between_launches": "Rlu(lu)PgPgu",
    "pack_and_prepare_in_the_graph": "Rl(PJlu)gguPl",
    "reset_in_the_graph": "lu(Rllu)gulg",
    "reset_before_launch": "lu(lu)Rg",
    "uneven": "R(luulul)gug",
}


def run(b, prec, color, order, graph):
    from tests.test_gpu_blusgs import make
    from ucfd_sparse_gb300 import lib
    S, e = make(b, prec=prec, on_device=True, colored=color)
    jmat = torch.from_numpy(np.ascontiguousarray(b["jmat"])).cuda()
    S.set_blusgs(jmat)
    st = torch.cuda.Stream()
    S.set_stream(st.cuda_stream, True)
    torch.cuda.synchronize()

    def call(step):
        if step == "P":
            e["rhs"].mul_(-0.75)
            S.blusgs_pack(0, 0.0)
        elif step == "J":
            jmat.mul_(1.25)
            S.blusgs_ns_prepare()
        elif step == "S":
            S.blusgs_solve(1e-30, 3, 2)
        else:
            {"l": S.blusgs_ns_lower, "u": S.blusgs_ns_upper, "R": S.blusgs_reset}[step]()

    with torch.cuda.stream(st):
        S.blusgs_pack(0, 0.0)
        S.blusgs_ns_prepare()
        S.blusgs_reset()
        S.blusgs_ns_lower()  # every buffer a call needs is there before a capture
        S.blusgs_ns_upper()
        inner, k = "", 0
        while k < len(order):
            if order[k] == "(":
                end = order.index(")", k)
                inner, k = order[k + 1:end], end + 1
                if graph:
                    g = torch.cuda.CUDAGraph()
                    torch.cuda.synchronize()
                    with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
                        for step in inner:
                            call(step)
                continue
            if order[k] == "g" and graph:
                g.replay()
            else:
                for step in inner if order[k] == "g" else order[k]:
                    call(step)
            k += 1
        S.blusgs_update(0)
        S.blusgs_sub_residual(0)
    torch.cuda.synchronize()
    rel = S.blusgs_residual()
    h = ctypes.c_double(-1.0)
    lib.call("UCFDBLUSGS_ResidualNoAlloc", S._h, ctypes.addressof(h))
    assert abs(h.value - rel) <= 1e-12 * rel
    return e["upts"].cpu().numpy(), e["res"].cpu().numpy(), rel


# colours of 32 (levels of the small-level kernels) and of 8788 cells
@pytest.mark.parametrize("m", [4, 26])
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("order", sorted(ORDERS))
def test_launched_graph_equals_the_calls(order, prec, m, ucfd):
    b = mg.blusgs_case(m, permute=False, seed=m)
    c = np.arange(m ** 3)
    color = ((c % m + c // m % m + c // (m * m)) & 1).astype(np.int32)
    ref = run(b, prec, color, ORDERS[order], False)
    got = run(b, prec, color, ORDERS[order], True)
    for r, g in zip(ref, got):
        assert np.isfinite(r).all()
        np.testing.assert_array_equal(g, r)
