"""Cells with 5 to 9 neighbours, two dimensions and the pressure floor: forms
that a box of hexahedra does not reach (the scalar kernels with eight face
slots, the loops over wider rows, the block sweeps' face loop with kept terms,
the transposed sweeps six faces at a time)."""
import numpy as np
import pytest
import torch

from ucfd_sparse_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def pairs(m, width, rng):
    """Neighbour pairs of the m^3 cells of a box and further ones, even to odd
    cells of the checkerboard, up to width neighbours a cell (width 5: some of
    the box's are left out)."""
    c = np.arange(m ** 3)
    x, y, z = c % m, c // m % m, c // (m * m)
    box = [np.stack([c[t < m - 1], c[t < m - 1] + s], 1) for t, s in ((x, 1), (y, m), (z, m * m))]
    even, odd = c[(x + y + z) % 2 == 0], c[(x + y + z) % 2 == 1]
    more = np.stack([rng.choice(even, 4 * c.size), rng.choice(odd, 4 * c.size)], 1)
    deg, out, seen = np.zeros(c.size, dtype=int), [], set()
    for a, b in np.concatenate([rng.permutation(np.concatenate(box)), more]).tolist():
        key = (min(a, b), max(a, b))
        if deg[a] < width and deg[b] < width and key not in seen:
            seen.add(key)
            deg[a] += 1
            deg[b] += 1
            out.append((a, b))
    assert deg.max() == width and deg.min() < width
    return np.array(out), ((x + y + z) & 1).astype(np.int32)


def ragged(m, width, nvars, seed):
    """FlowSys arrays of such a mesh, rows in random face order, and inputs of
    both systems and of the block system."""
    rng = np.random.default_rng(seed)
    e, color = pairs(m, width, rng)
    N, nF = m ** 3, e.shape[0]
    row, col = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    k = np.lexsort((rng.random(2 * nF), row))
    n = rng.standard_normal((3, nF))
    b = dict(nlocal=N, nfaces=nF, nvars=nvars, nfvars=5, ndims=3, neles=N,
             rowptr=np.searchsorted(row[k], np.arange(N + 1)).astype(np.int32), colidx=col[k].astype(np.int32),
             slots=np.tile(np.arange(nF), 2)[k].astype(np.int32), sides=np.repeat([1, -1], nF)[k].astype(np.int8),
             face_area=rng.uniform(0.5, 1.5, nF), face_normal=n / np.linalg.norm(n, axis=0),
             rcp_vol=rng.uniform(0.8, 1.2, N), cell_ids=rng.permutation(N).astype(np.int32),
             dt=rng.uniform(1e-3, 1e-2, N), rhs=rng.standard_normal((nvars, N)) * 1e-2, vol=rng.uniform(0.8, 1.2, N),
             dsrc=rng.uniform(0, 1, (nvars, N)), fspr=rng.uniform(0.5, 2, nF), tfspr=rng.uniform(0.5, 2, nF))
    b["upts"] = mg.free_stream(nvars, N) * rng.uniform(0.95, 1.05, (nvars, N))
    if nvars > 5:
        b["upts"][5:] = rng.uniform(0.1, 1, (nvars - 5, N))
    b["jmat"] = rng.normal(0, 0.05, (2, 5, 5, nF))
    for r in range(5):
        b["jmat"][0, r, r] += b["fspr"]
        b["jmat"][1, r, r] -= b["fspr"]
    return b, color


def in_colour_order(b, color):
    new = np.empty(b["nlocal"], dtype=np.int64)
    new[np.argsort(color, kind="stable")] = np.arange(b["nlocal"])
    return mg.renumber_flowsys(b, new)


# colours of 108 and 4000 (lanes), 10976 (beyond them for more than four faces)
# and 17968 cells (a thread per active face up to eight); width 9 takes the loop
@pytest.mark.parametrize("width", [5, 7, 8, 9])
@pytest.mark.parametrize("m", [6, 20, 28, 33])
@pytest.mark.parametrize("nvars", [5, 7])
def test_scalar_sweeps(width, m, nvars, port, ucfd):
    from tests.test_gpu_lusgs import make_flowsys
    b, color = ragged(m, width, nvars, m + width)
    rans = nvars > 5
    br = in_colour_order(b, color)
    ref = port.flowsys_lusgs_step(br, b["upts"], b["rhs"], b["dt"], b["dsrc"], b["fspr"],
                                  b["tfspr"] if rans else None, kappa=1.01, a0=0.3, turb_factor=1.5, rans=rans)[0]
    # FP32: the bound of the box meshes' test; FMA mode: 1e-12 of the largest
    # change, and the two roundings of u + du
    for prec, tol in ((0, 0.0), (1, 1e-12), (2, 1e-5)):
        outs = []
        for variant, both in ((0, False), (5, False)) + (((0, True),) if rans else ()):
            S, e = make_flowsys(b, b, prec=prec, on_device=True, colored=color)
            S.set_launch_config(sweep_variant=variant)
            S.lusgs_pack(0, 1.5, 0.3)
            if both:
                S.lusgs_nsrans_prepare(1.01)
                S.lusgs_nsrans_lower(1.01)
                S.lusgs_nsrans_upper(1.01)
            else:
                S.lusgs_ns_prepare(1.01)
                S.lusgs_ns_lower(1.01)
                S.lusgs_ns_upper(1.01)
                if rans:
                    S.lusgs_rans_prepare(1.01)
                    S.lusgs_rans_lower(1.01)
                    S.lusgs_rans_upper(1.01)
            S.lusgs_update(0)
            outs.append(e["upts"].cpu().numpy())
        for up in outs:  # one kernel per level, face lists, both systems at once
            np.testing.assert_array_equal(up, outs[0])
        d, r = outs[0] - b["upts"], ref - b["upts"]
        if prec == 0:
            np.testing.assert_array_equal(outs[0], ref)
        else:
            assert np.abs(d - r).max() <= tol * np.abs(r).max() + np.spacing(np.abs(ref).max())


@pytest.mark.parametrize("width", [5, 7, 8, 9])
@pytest.mark.parametrize("m", [6, 27])
def test_block_sweeps(width, m, port, ucfd):
    """Against the oracle after two pairs of sweeps (bounds as above), and in calls of any order
    against sweeps that form every face (a Prepare before each)."""
    from tests.test_gpu_blusgs import make, run_sweeps
    b, color = ragged(m, width, 5, m + width)
    br = in_colour_order(b, color)
    up, _, res, _ = port.flowsys_blusgs(br, b["rhs"], b["dt"], b["jmat"], b["vol"], b["upts"], nsweeps=2)
    for prec, tol in ((0, 0.0), (1, 1e-12), (2, 1e-5)):
        S, e = make(b, prec=prec, on_device=True, colored=color)
        run_sweeps(S, 2)
        got = e["upts"].cpu().numpy()
        if prec == 0:
            np.testing.assert_array_equal(got, up)
            np.testing.assert_array_equal(e["res"].cpu().numpy(), res)
        else:
            d, r = got - b["upts"], up - b["upts"]
            assert np.abs(d - r).max() <= tol * np.abs(r).max() + np.spacing(np.abs(up).max())
        outs = []
        for stale in (False, True):
            S, e = make(b, prec=prec, on_device=True, colored=color)
            S.blusgs_pack(0, 0.0)
            S.blusgs_ns_prepare()
            S.blusgs_reset()
            for step in "luulluRul":
                if step == "R":
                    S.blusgs_reset()
                    continue
                if stale:
                    S.blusgs_ns_prepare()
                (S.blusgs_ns_lower if step == "l" else S.blusgs_ns_upper)()
            S.blusgs_update(0)
            outs.append(e["upts"].cpu().numpy())
        np.testing.assert_array_equal(outs[0], outs[1])


def array_case(m, width, ndims, floor, seed):
    """The array layout: width > 4 a ragged box, else a square of m x m cells;
    floor: every third cell's energy at half of what its momentum holds, so its
    pressure is raised to the floor."""
    rng = np.random.default_rng(seed)
    if ndims == 3:
        e, _ = pairs(m, width, rng)
        N = m ** 3
    else:
        c = np.arange(m * m)
        e = np.concatenate([np.stack([c[c % m < m - 1], c[c % m < m - 1] + 1], 1),
                            np.stack([c[c < m * (m - 1)], c[c < m * (m - 1)] + m], 1)])
        N = m * m
    nv = ndims + 2
    nei = np.tile(np.arange(N, dtype=np.int32), (width, 1))
    deg = np.zeros(N, dtype=int)
    for a, b in e:
        nei[deg[a], a], nei[deg[b], b] = b, a
        deg[a] += 1
        deg[b] += 1
    nei = np.take_along_axis(nei, rng.random((width, N)).argsort(0), 0)
    vec = rng.standard_normal((width, ndims, N))
    u = np.empty((nv, N))
    u[0] = rng.uniform(0.9, 1.1, N)
    u[1:-1] = rng.uniform(-0.5, 0.5, (ndims, N)) + 0.6
    ke = 0.5 * (u[1:-1] ** 2).sum(0) / u[0]
    u[-1] = 2.5 + ke
    if floor:
        u[-1, ::3] = 0.5 * ke[::3]
    icolor, ranges, lcolor = mg.greedy_coloring_np(nei, rng.permutation(N))  # more than the checkerboard's two
    return dict(neles=N, nface=width, nvars=nv, nei_ele=nei, fnorm_vol=rng.uniform(0.5, 1.5, (width, N)),
                vec_fnorm=vec / np.linalg.norm(vec, axis=1, keepdims=True), fspr=rng.uniform(0.5, 2, (width, N)),
                dt=rng.uniform(1e-2, 1e-1, N), rhs=rng.standard_normal((nv, N)) * 0.1, upts=u,
                lcolor=lcolor.astype(np.int32)), icolor.astype(np.int32), [int(r) for r in ranges]


@pytest.mark.parametrize("width,ndims,floor", [(5, 3, False), (7, 3, False), (8, 3, True), (9, 3, False),
                                               (13, 3, True), (4, 2, False), (4, 2, True)])
def test_gradients(width, ndims, floor, port, ucfd):
    """Gradients of the colored step against central differences of the oracle
    (h and relative bound of the box meshes' test), FP32 ones against FP64, and the
    forward values against the oracle."""
    from tests.test_gpu_adjoint import FD_H, FD_REL, T
    from ucfd_sparse_gb300.adjoint import ColoredMesh, lusgs_step
    c, icolor, ranges = array_case(5 if ndims == 3 else 11, width, ndims, floor, 3)
    nv = ndims + 2
    mesh = ColoredMesh(c["nei_ele"], c["fnorm_vol"], c["vec_fnorm"], icolor, ranges, nvars=nv, nfvars=nv, ndims=ndims)

    def oracle(rhs, dt, fspr):
        return port.legacy_step(dict(c, rhs=rhs, dt=dt, fspr=fspr), icolor, ranges, c["lcolor"], nfvars=nv,
                                ndims=ndims)[1]

    base = {k: c[k] for k in ("rhs", "dt", "fspr")}
    rng = np.random.default_rng(11)
    g = rng.standard_normal(c["rhs"].shape)
    grads = {}
    for dtype in (torch.float64, torch.float32):
        xs = {k: T(v, dtype).requires_grad_() for k, v in base.items()}
        dq = lusgs_step(xs["rhs"], xs["dt"], xs["fspr"], mesh, T(c["upts"], dtype))
        if dtype == torch.float64:
            np.testing.assert_array_equal(dq.detach().cpu().numpy(), oracle(**base))
        (dq * T(g, dtype)).sum().backward()
        grads[dtype] = {k: x.grad.double().cpu().numpy() for k, x in xs.items()}
    for name in base:
        for _ in range(3):
            v = rng.standard_normal(base[name].shape) * np.abs(base[name])
            lp = float((oracle(**dict(base, **{name: base[name] + FD_H * v})) * g).sum())
            lm = float((oracle(**dict(base, **{name: base[name] - FD_H * v})) * g).sum())
            fd = (lp - lm) / (2 * FD_H)
            ad = float((grads[torch.float64][name] * v).sum())
            # of the derivative's usual size: a direction may by chance give far less
            size = np.linalg.norm(grads[torch.float64][name] * v)
            assert abs(ad - fd) <= FD_REL * max(abs(fd), size), (name, ad, fd, size)
        a, b = grads[torch.float32][name], grads[torch.float64][name]
        assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max(), name
