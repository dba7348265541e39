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


# checkerboard colours of 32, 7812/7813 (a lane per block row) and 8788 cells
# (one thread per cell): either side of the FP64 kernels' boundary at 8192
@pytest.mark.parametrize("m", [4, 25, 26])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_block_levels_and_kept_terms(m, prec, ucfd):
    """A sweep that reads the other side's terms or sums from the sweep before
    equals one that forms every face itself (Prepare before each sweep makes
    the kept ones stale), bit for bit, in any order of sweeps and with a
    Reset in between."""
    from tests.test_gpu_blusgs import make
    b = mg.blusgs_case(m, permute=False, seed=m)
    c = np.arange(m ** 3)
    color = ((c % m + c // m % m + c // (m * m)) & 1).astype(np.int32)
    got = []
    for stale in (False, True):
        S, e = make(b, prec=prec, on_device=True, colored=color)
        S.blusgs_pack(0, 0.0)
        S.blusgs_ns_prepare()
        S.blusgs_reset()
        for step in "luluullRluul":
            if step == "R":
                S.blusgs_reset()
                continue
            if stale:
                S.blusgs_ns_prepare()
            (S.blusgs_ns_lower if step == "l" else S.blusgs_ns_upper)()
        S.blusgs_update(0)
        got.append(e["upts"].cpu().numpy())
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("m", [25, 26])
def test_block_levels_match_the_oracle(m, port, ucfd):
    from tests.test_gpu_blusgs import host, make, run_sweeps
    b = mg.blusgs_case(m, seed=m)
    from ucfd_sparse_gb300 import coloredlusgs as cl
    ic, rg, lc = cl.greedy_coloring_csr(b["rowptr"], b["colidx"])
    S, e = make(b, colored=lc)
    run_sweeps(S, 2)
    new = np.empty(b["nlocal"], dtype=np.int64)
    new[ic] = np.arange(b["nlocal"])
    br = mg.renumber_flowsys(b, new)
    up, _, res, _ = port.flowsys_blusgs(br, b["rhs"], b["dt"], b["jmat"], b["vol"], b["upts"], nsweeps=2)
    np.testing.assert_array_equal(host(e["upts"]), up)
    np.testing.assert_array_equal(host(e["res"]), res)


# either side of the size from which Pack goes through records (131072 cells);
# 51^3 is no multiple of a warp's 32 cells
@pytest.mark.parametrize("m", [50, 51])
@pytest.mark.parametrize("nvars", [5, 7])
@pytest.mark.parametrize("prec", [0, 2])
def test_pack_of_large_systems(m, nvars, prec, ucfd):
    """Two Packs with new inputs, a step after each: elements in an order of
    their own and in the order of the sweeps give the same cells the same
    values."""
    from ucfd_sparse_gb300.flowsys import FlowSys
    fs = mg.lusgs_flowsys_case(m, nvars=nvars, permute=False)
    N = fs["nlocal"]
    c = np.arange(N)
    color = ((c % m + c // m % m + c // (m * m)) & 1).astype(np.int32)
    rng = np.random.default_rng(m)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    got = []
    for order in (np.arange(N), rng.permutation(N)):
        # element e is cell order[e]; its inputs move with it
        t = {k: dev(fs[k]) for k in ("rowptr", "colidx", "slots", "sides", "face_area", "face_normal", "rcp_vol")}
        S = FlowSys(N, nvars, 5, 3, fs["nfaces"], 1, *t.values())
        S.set_coloring(color)
        S.set_precision(prec)
        e = dict(upts=dev(fs["upts"][:, order]), rhs=dev(fs["rhs"][:, order]), dt=dev(fs["dt"][order]),
                 dsrc=dev(0.1 * np.abs(fs["rhs"][:, order])), vol=dev(fs["vol"][order]))
        ids = dev(order.astype(np.int32))
        S.set_element(0, N, 6, ids, e["upts"], e["rhs"], e["dt"], e["dsrc"], e["vol"], torch.zeros_like(e["rhs"]))
        S.set_lusgs(dev(fs["fspr"]), dev(fs["tfspr"]))
        for k in range(2):
            S.lusgs_pack(0, 1.5, 0.3)
            S.lusgs_run(2, rans=nvars > 5)
            S.lusgs_update(0)
            e["rhs"].mul_(-0.5)
            torch.cuda.synchronize()
        back = np.empty(N, dtype=np.int64)
        back[order] = np.arange(N)
        got.append(e["upts"].cpu().numpy()[:, back])
    assert np.abs(got[0] - fs["upts"]).max() > 0
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("m", [4, 25])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_block_sweeps_follow_a_new_right_hand_side(m, prec, ucfd):
    """A sweep whose first level would only repeat the sweep before is not
    launched for that level; after a Pack with a new right-hand side, in any
    direction, it is.  Against the same calls with a Prepare before each sweep
    (every level and face formed), bit for bit."""
    from tests.test_gpu_blusgs import make
    b = mg.blusgs_case(m, permute=False, seed=m + 1)
    c = np.arange(m ** 3)
    color = ((c % m + c // m % m + c // (m * m)) & 1).astype(np.int32)
    got = []
    for stale in (False, True):
        S, e = make(b, prec=prec, on_device=True, colored=color)
        S.blusgs_pack(0, 0.0)
        S.blusgs_ns_prepare()
        S.blusgs_reset()
        for step in "luluPluPulPuluPllu":
            if step == "P":
                e["rhs"].mul_(-0.75)
                torch.cuda.synchronize()
                S.blusgs_pack(0, 0.0)
                continue
            if stale:
                S.blusgs_ns_prepare()
            (S.blusgs_ns_lower if step == "l" else S.blusgs_ns_upper)()
        S.blusgs_update(0)
        got.append(e["upts"].cpu().numpy())
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("m", [4, 26])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_captured_sweeps(m, prec, ucfd):
    """A lower + upper pair captured once gives, launched between calls, what
    the calls themselves give; in the exact mode also with another right-hand
    side packed before the launch (the other modes form D^-1 rhs in the first
    sweep call after a Pack, which a graph captured earlier does not hold)."""
    from tests.test_gpu_blusgs import make
    b = mg.blusgs_case(m, permute=False, seed=m)
    c = np.arange(m ** 3)
    color = ((c % m + c // m % m + c // (m * m)) & 1).astype(np.int32)
    got = []
    for graph in (False, True):
        S, e = make(b, prec=prec, on_device=True, colored=color)
        st = torch.cuda.Stream()
        S.set_stream(st.cuda_stream, True)

        def pair():
            S.blusgs_ns_lower()
            S.blusgs_ns_upper()

        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            S.blusgs_pack(0, 0.0)
            S.blusgs_ns_prepare()
            S.blusgs_reset()
            pair()
            if graph:
                g = torch.cuda.CUDAGraph()
                torch.cuda.synchronize()
                with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
                    pair()
            for scale in (1.0, -0.5, 3.0):
                if prec == 0:
                    e["rhs"].mul_(scale)
                    S.blusgs_pack(0, 0.0)
                if graph:
                    g.replay()
                    pair()
                else:
                    pair()
                    pair()
            S.blusgs_update(0)
        torch.cuda.synchronize()
        got.append(e["upts"].cpu().numpy())
    np.testing.assert_array_equal(got[0], got[1])


# a square of m x m cells in two colours: levels of 32, 12168 (lanes), 12800
# (one thread per cell) and 17298 cells (one thread per active face) in FP64
@pytest.mark.parametrize("m", [8, 156, 160, 186])
@pytest.mark.parametrize("nvars", [4, 5, 6])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_plane_levels(m, nvars, prec, ucfd):
    """Two-dimensional cells: the kernels chosen by the level's size and two
    threads per cell (variant 3) agree bit for bit."""
    from ucfd_sparse_gb300.flowsys import FlowSys
    rng = np.random.default_rng(m)
    N = m * m
    c = np.arange(N)
    x, y = c % m, c // m
    right, up = c[x < m - 1], c[y < m - 1]
    a, b = np.concatenate([right, up]), np.concatenate([right + 1, up + m])
    nF = a.size
    row, col = np.concatenate([a, b]), np.concatenate([b, a])
    slot, side = np.tile(np.arange(nF), 2), np.repeat([1, -1], nF)
    k = np.lexsort((rng.random(2 * nF), row))
    rowptr = np.searchsorted(row[k], np.arange(N + 1)).astype(np.int32)
    ang = rng.uniform(0, 2 * np.pi, nF)
    upts = np.empty((nvars, N))
    upts[:4] = np.array([1.0, 0.4, -0.2, 2.5])[:, None] * rng.uniform(0.95, 1.05, (4, N))
    upts[4:] = rng.uniform(0.1, 1.0, (nvars - 4, N))
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()  # noqa: E731
    rhs, dt = rng.standard_normal((nvars, N)) * 1e-2, rng.uniform(1e-3, 1e-2, N)
    got = []
    for variant in (0, 3):
        t = [dev(v) for v in (rowptr, col[k].astype(np.int32), slot[k].astype(np.int32), side[k].astype(np.int8),
                              1.25 + 0.5 * np.sin(ang), np.stack([np.cos(ang), np.sin(ang)], 1),
                              1.0 / (1.0 + 0.1 * x / m))]
        S = FlowSys(N, nvars, 4, 2, nF, 1, *t)
        S.set_coloring(((x + y) & 1).astype(np.int32))
        S.set_precision(prec)
        S.set_launch_config(sweep_variant=variant)
        e = [dev(v) for v in (upts, rhs, dt, np.zeros((nvars, N)), np.ones(N), np.zeros((nvars, N)))]
        ids = dev(c.astype(np.int32))
        S.set_element(0, N, 4, ids, *e)
        f = dev(1.0 + 0.5 * np.sin(np.arange(nF))), dev(1.0 + 0.5 * np.cos(np.arange(nF)))
        S.set_lusgs(*f)
        S.lusgs_pack(0, 1.5, 0.3)
        S.lusgs_run(2, rans=nvars > 4)
        S.lusgs_update(0)
        torch.cuda.synchronize()
        got.append(e[0].cpu().numpy())
    assert np.isfinite(got[0]).all() and not np.array_equal(got[0], upts)
    np.testing.assert_array_equal(got[0], got[1])
