"""The work that programs have this library do, as timed cases.

A case is one pass of one of the library's paths through its public entry
points: a colored or natural-order LU-SGS step, the pseudo-time loop, a block
LU-SGS step with a fixed number of sweeps or solved to a tolerance, a BSR
matvec, a preconditioner apply, a whole Krylov step on a newly assembled
matrix, and the differentiable step with its gradients.  The sizes run from
boxes of a few thousand cells to the 2.1M-cell and 5.3M-row systems of
bench.py; box sides need not be equal or even.

  listed()   the cases by name
  draw(rng)  one more case of the same ranges
  prepare    the inputs (on the GPU, from the seed) and the objects a program keeps
  run        one pass; its outputs whole
  work       bytes and operations a pass cannot do without
  exact      the outputs in 64 bits by plain torch, without the library
"""
import math

import numpy as np
import torch

from ucfd_sparse_gb300 import coloredlusgs as cl
from ucfd_sparse_gb300.adjoint import ColoredMesh, lusgs_step
from ucfd_sparse_gb300.flowsys import FlowSys
from ucfd_sparse_gb300.krylov import Precon, Solver, SpMat

DEV = "cuda"
F64, F32, I32 = torch.float64, torch.float32, torch.int32
GAMMA = 1.4
EXACT, FMA, FP32 = 0, 1, 2  # UCFD_PREC_*: the reference's arithmetic, fused multiply-adds, FP32 (with FP64 refinement)


def listed():
    return [
        # the reference's own example (examples/omp3d.py): 32^3 box, checkerboard, double arrays
        dict(name="array_32", kind="array", nx=32, ny=32, nz=32, prec=EXACT),
        # a caller that only changed the library it loads: natural order on a box numbered x-fastest, FP64
        dict(name="lusgs_natural_fp64", kind="lusgs", nx=41, ny=36, nz=33, permute=False, greedy=False, nvars=5, prec=EXACT),
        # mean flow and one turbulence equation, coloured, single precision, irregular numbering
        dict(name="lusgs_rans_fp32", kind="lusgs", nx=97, ny=95, nz=96, permute=True, greedy=True, nvars=6, prec=FP32),
        # the pseudo-time loop on the device
        dict(name="loop_rans_fp32", kind="loop", nx=128, ny=128, nz=128, permute=True, greedy=True, nvars=6, prec=FP32, iters=20),
        # smallest block LU-SGS step: a rank of a partitioned mesh, a few thousand cells
        dict(name="blusgs_small_fma", kind="blusgs", nx=19, ny=17, nz=15, permute=True, greedy=True, prec=FMA, sweeps=5),
        # block LU-SGS with the reference's arithmetic and call sequence
        dict(name="blusgs_fp64", kind="blusgs", nx=64, ny=61, nz=58, permute=True, greedy=True, prec=EXACT, sweeps=10),
        # bench.py's default: 2,097,152 cells, FP32 sweeps refined to 1e-10, launch shape tuned once
        dict(name="blusgs_solve_fp32", kind="solve", nx=128, ny=128, nz=128, permute=True, greedy=True, prec=FP32),
        # matvec on the dual graph of a tetrahedral mesh, FP64 in the reference's order
        dict(name="spmv_tets_fp64", kind="spmv", nx=47, ny=48, nz=49, prec=EXACT),
        # the coloured preconditioner of a Krylov method of the caller's own
        dict(name="precon_tets_fma", kind="precon", nx=48, ny=45, nz=44, prec=FMA, ilu=False),
        # one implicit step: new matrix values, preconditioner, GMRES(30) to 1e-10, mixed precision, 5.3M rows
        dict(name="gmres_tets_mixed", kind="gmres", nx=96, ny=96, nz=96, prec=FP32),
        # the same with BiCGSTAB and block ILU(0) on a small system
        dict(name="bicgstab_bilu_fp64", kind="bicgstab", nx=23, ny=25, nz=24, prec=EXACT),
        # gradients of one coloured step (adjoint sensitivities), 64^3
        dict(name="adjoint_64_fp64", kind="adjoint", nx=64, ny=64, nz=64, permute=True, fp32=False),
    ]


#: Per kind: the smallest and largest box (cells, or hexahedra that are split into six tetrahedra) that draw() gives.
RANGES = {"array": (2000, 300000), "lusgs": (4000, 1000000), "loop": (8000, 2000000), "blusgs": (3000, 300000),
          "solve": (8000, 2000000), "spmv": (1000, 110000), "precon": (1000, 100000), "gmres": (1000, 800000),
          "bicgstab": (1000, 60000), "adjoint": (4000, 262144)}


def draw(rng):
    kind = rng.choice(sorted(RANGES))
    lo, hi = RANGES[kind]
    prec = rng.choice([FMA, FP32])
    if kind == "gmres" and prec == FMA:
        hi //= 8  # FP64 cycles always run their 30 steps
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    side = n ** (1 / 3)
    nx, ny = max(4, round(side * a)), max(4, round(side * b))
    c = dict(kind=kind, nx=nx, ny=ny, nz=max(4, int(n / (nx * ny))))
    if kind in ("array", "spmv"):
        c.update(prec=rng.choice([EXACT, FMA] if kind == "array" else [EXACT, FMA, FP32]))
    elif kind in ("lusgs", "loop"):
        c.update(permute=rng.random() < 0.7, nvars=rng.choice([5, 6, 7]), prec=rng.choice([EXACT, FMA, FP32]))
        c.update(greedy=c["permute"] and rng.random() < 0.8)
        if kind == "loop":
            c.update(iters=rng.randint(3, 10))
    elif kind == "blusgs":
        c.update(permute=True, greedy=rng.random() < 0.8, prec=rng.choice([EXACT, FMA, FP32]), sweeps=rng.randint(2, 10))
    elif kind == "solve":
        c.update(permute=True, greedy=True, prec=rng.choice([FMA, FP32, FP32]))
    elif kind == "precon":
        c.update(prec=rng.choice([EXACT, FMA, FP32]), ilu=rng.random() < 0.3)
    elif kind == "gmres":
        c.update(prec=prec)
    elif kind == "bicgstab":
        c.update(prec=rng.choice([EXACT, FMA]))
    else:
        c.update(permute=rng.random() < 0.7, fp32=rng.random() < 0.5)
    return c


# ---- meshes ------------------------------------------------------------------
def _gen(seed, stream):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + stream) % (1 << 62))
    return g


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=F64) * (hi - lo) + lo


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _box_neighbours(nx, ny, nz):
    """[6, N] neighbours -x,+x,-y,+y,-z,+z of a box numbered x-fastest, -1 outside."""
    c = torch.arange(nx * ny * nz, device=DEV).reshape(nz, ny, nx)
    t = torch.full((6, nz, ny, nx), -1, dtype=torch.int64, device=DEV)
    t[0, :, :, 1:], t[1, :, :, :-1] = c[:, :, :-1], c[:, :, 1:]
    t[2, :, 1:], t[3, :, :-1] = c[:, :-1], c[:, 1:]
    t[4, 1:], t[5, :-1] = c[:-1], c[1:]
    return t.reshape(6, -1)


def _levels(tab, greedy):
    """Sweep order of a neighbour table [P, N] (-1: none): the colours of the
    greedy colouring in index order, or the levels of the natural order."""
    P, N = tab.shape
    lev = torch.full((N,), -1, dtype=torch.int64, device=DEV)
    me = torch.arange(N, device=DEV)
    lower = torch.where((tab >= 0) & (tab < me), tab, -1)
    left = me
    while left.numel():
        low = lower[:, left]
        known = torch.where(low >= 0, lev[low.clamp(min=0)], -2)  # -2: no such neighbour, -1: not known yet
        ready = (known != -1).all(0)
        k = known[:, ready]
        if greedy:
            used = torch.zeros(k.shape[1], dtype=torch.int64, device=DEV)
            for p in range(P):
                used |= torch.where(k[p] >= 0, torch.ones_like(used) << k[p].clamp(min=0), 0)
            free = ~used
            lev[left[ready]] = torch.round(torch.log2((free & -free).double())).long()
        else:
            lev[left[ready]] = k.clamp(min=-1).max(0).values + 1
        left = left[~ready]
    return lev


def _by_level(lev):
    order = torch.argsort(lev, stable=True)
    ends = torch.cumsum(torch.bincount(lev), 0).tolist()
    return [order[a:b] for a, b in zip([0] + ends[:-1], ends)]


def _free_stream(nvars, n, g):
    u = torch.zeros(nvars, n, dtype=F64, device=DEV)
    u[0], u[1], u[4] = GAMMA, GAMMA * 1.5, 1.0 / (GAMMA - 1) + 0.5 * GAMMA * 1.5 * 1.5
    u[:5] *= 1 + 0.02 * _uniform(g, -1, 1, 5, n)
    u[2:4] += 0.05 * _normal(g, 2, n)
    if nvars > 5:
        u[5:] = _uniform(g, 0.1, 1.0, nvars - 5, n)
    return u


def _flowsys_mesh(case, seed):
    """CSR of shared faces over a box of jittered hexahedra (boundary faces
    have no entry), ranks permuted at random where the case says so."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    N = nx * ny * nz
    g = _gen(seed, 1)
    tab = _box_neighbours(nx, ny, nz)
    perm = torch.randperm(N, generator=g, device=DEV) if case["permute"] else torch.arange(N, device=DEV)
    inv = torch.argsort(perm)
    has = tab[1::2] >= 0                                        # cells with a face in +x, +y, +z
    slot_up = torch.cumsum(has.reshape(-1), 0).reshape(3, N) - 1  # that face's number
    slot = torch.full((6, N), -1, dtype=torch.int64, device=DEV)
    slot[1::2] = torch.where(has, slot_up, -1)
    for a in range(3):
        below = tab[2 * a]
        slot[2 * a] = torch.where(below >= 0, slot_up[a][below.clamp(min=0)], -1)
    nF = int(has.sum())
    h = torch.tensor([1.0 / nx, 1.0 / ny, 1.0 / nz], dtype=F64, device=DEV)
    axis = torch.arange(3, device=DEV)[:, None].expand(3, N)[has]
    area = (h.prod() / h)[axis] * (1 + _uniform(g, -0.2, 0.2, nF))
    normal = 0.15 * _normal(g, 3, nF)
    normal[axis, torch.arange(nF, device=DEV)] += 1.0
    normal /= normal.norm(dim=0, keepdim=True)
    vol = h.prod() * (1 + _uniform(g, -0.2, 0.2, N))
    row_slot, row_nb = slot[:, inv].T, tab[:, inv].T            # [rank, 6]
    ok = row_slot >= 0
    rowptr = torch.zeros(N + 1, dtype=I32, device=DEV)
    rowptr[1:] = torch.cumsum(ok.sum(1), 0)
    side = torch.tensor([-1, 1, -1, 1, -1, 1], dtype=torch.int8, device=DEV).expand(N, 6)
    return dict(N=N, nF=nF, rowptr=rowptr, colidx=perm[row_nb[ok]].to(I32), slots=row_slot[ok].to(I32),
                sides=side[ok].contiguous(), area=area, normal=normal, rcp_vol=(1.0 / vol)[inv].contiguous(),
                ids=perm.to(I32), vol=vol, g=g)


def _flowsys(case, m, e):
    S = FlowSys(m["N"], case.get("nvars", 5), 5, 3, m["nF"], 1, m["rowptr"], m["colidx"], m["slots"], m["sides"],
                m["area"], m["normal"], m["rcp_vol"])
    if case["greedy"]:
        S.color_greedy()
    S.set_precision(case["prec"])
    S.set_element(0, m["N"], 6, m["ids"], e["upts"], e["rhs"], e["dt"], e["dsrc"], m["vol"], e["resid"])
    return S


def _flowsys_inputs(case, seed):
    m = _flowsys_mesh(case, seed)
    g, N, nv = m["g"], m["N"], case.get("nvars", 5)
    block = case["kind"] in ("blusgs", "solve")
    # scalar steps repeat on their own state: a right-hand side of 1e-3 keeps it physical for thousands of steps
    e = dict(upts=_free_stream(nv, N, g), rhs=_normal(g, nv, N) * (1.0 if block else 1e-3),
             dt=_uniform(g, 1e-3, 1e-2, N), dsrc=torch.zeros(nv, N, dtype=F64, device=DEV),
             resid=torch.zeros(nv, N, dtype=F64, device=DEV))
    if block:
        sigma = _uniform(g, 0.5, 2.0, m["nF"])
        e["jmat"] = 0.05 * _normal(g, 2, 5, 5, m["nF"])
        for r in range(5):
            e["jmat"][0, r, r] += sigma
            e["jmat"][1, r, r] -= sigma
    else:
        e["fspr"], e["tfspr"] = _uniform(g, 0.5, 2.0, m["nF"]), _uniform(g, 0.5, 2.0, m["nF"])
    return m, e


def _array_inputs(case, seed):
    """The array layout of the reference's examples: neighbour table with boundary faces pointing to the cell itself."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    N = nx * ny * nz
    g = _gen(seed, 2)
    tab = _box_neighbours(nx, ny, nz)
    me = torch.arange(N, device=DEV)
    nei = torch.where(tab >= 0, tab, me)
    if case["kind"] == "array":
        x, y, z = me % nx, me // nx % ny, me // (nx * ny)
        lev = (x + y + z) & 1  # the checkerboard of the reference's make_coloring
    else:
        if case["permute"]:
            perm = torch.randperm(N, generator=g, device=DEV)
            inv = torch.argsort(perm)
            tab = torch.where(tab[:, inv] >= 0, perm[tab[:, inv].clamp(min=0)], -1)
            nei = torch.where(tab >= 0, tab, me)
        lev = _levels(tab, True)
    scale = torch.tensor([nx, nx, ny, ny, nz, nz], dtype=F64, device=DEV)[:, None]
    vec = 0.15 * _normal(g, 6, 3, N)
    for f in range(6):
        vec[f, f // 2] += 1.0 if f % 2 else -1.0
    vec /= vec.norm(dim=1, keepdim=True)
    cells = _by_level(lev)
    return dict(N=N, nei=nei, lev=lev, cells=cells, icolor=torch.cat(cells).to(I32), lcolor=(lev + 1).to(I32),
                ranges=np.cumsum([c.numel() for c in cells]).tolist(),
                fnv=scale * (1 + _uniform(g, -0.2, 0.2, 6, N)), vec=vec, fspr=_uniform(g, 0.5, 2.0, 6, N),
                dt=_uniform(g, 1e-3, 1e-2, N), upts=_free_stream(5, N, g), rhs=_normal(g, 5, N) * 1e-3, g=g)


def _tet_neighbours(nx, ny, nz):
    """[4, 6 nx ny nz] face neighbours of a box whose hexahedra are split into
    the six tetrahedra of the axis orders (a, b, c), each along its diagonal."""
    orders = [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]
    h = torch.arange(nx * ny * nz, device=DEV)
    at = [h % nx, h // nx % ny, h // (nx * ny)]
    size, stride = (nx, ny, nz), (1, nx, nx * ny)
    t = torch.full((4, nx * ny * nz, 6), -1, dtype=torch.int64, device=DEV)
    for q, (a, b, c) in enumerate(orders):
        t[0, :, q] = torch.where(at[a] + 1 < size[a], 6 * (h + stride[a]) + orders.index((b, c, a)), -1)
        t[1, :, q] = 6 * h + orders.index((b, a, c))
        t[2, :, q] = 6 * h + orders.index((a, c, b))
        t[3, :, q] = torch.where(at[c] > 0, 6 * (h - stride[c]) + orders.index((c, a, b)), -1)
    return t.reshape(4, -1)


def _bsr_inputs(case, seed):
    """Diagonally dominant BSR 5x5 system on the tetrahedra's dual graph,
    rows numbered colour by colour of the greedy colouring."""
    g = _gen(seed, 3)
    tab = _tet_neighbours(case["nx"], case["ny"], case["nz"])
    n = tab.shape[1]
    cells = _by_level(_levels(tab, True))
    old = torch.cat(cells)
    new = torch.argsort(old)
    tab = torch.where(tab[:, old] >= 0, new[tab[:, old].clamp(min=0)], n)
    me = torch.arange(n, device=DEV)
    cols = torch.cat([tab, me[None]]).T.sort(dim=1).values       # [n, 5], missing ones last
    ok = cols < n
    rowptr = torch.zeros(n + 1, dtype=I32, device=DEV)
    rowptr[1:] = torch.cumsum(ok.sum(1), 0)
    colidx = cols[ok]
    rows = me[:, None].expand(n, 5)[ok]
    diag = torch.nonzero(colidx == rows).reshape(-1)
    vals = _normal(g, colidx.numel(), 5, 5)
    total = torch.zeros(n, 5, 5, dtype=F64, device=DEV)          # [row, slot, scalar row]
    total[rows, torch.arange(colidx.numel(), device=DEV) - rowptr[:-1].long()[rows]] = vals.abs().sum(2)
    total = total.sum(1)
    r = torch.arange(5, device=DEV)
    total -= vals[diag][:, r, r].abs()
    vals[diag[:, None], r, r] = total + _uniform(g, 0.1, 1.0, n, 5)
    return dict(n=n, rowptr=rowptr, colidx=colidx.to(I32), diag=diag.to(I32), vals=vals, rows=rows,
                ends=np.cumsum([0] + [c.numel() for c in cells]).astype(np.int32), vec=_normal(g, n * 5))


def _precon(m, values, ilu, prec):
    pc = Precon(m["rowptr"], m["colidx"], m["diag"], values)
    (pc.set_pbilu if ilu else pc.set_pblusgs)(m["n"], 5, len(m["ends"]) - 1, m["ends"])
    pc.set_precision(prec)
    pc.prepare()
    return pc


# ---- prepare and run -----------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("lusgs", "loop", "blusgs", "solve"):
        s["m"], s["e"] = m, e = _flowsys_inputs(case, seed)
        torch.cuda.synchronize()  # the library reads the arrays on a stream of its own
        s["S"] = S = _flowsys(case, m, e)
        if kind in ("lusgs", "loop"):
            S.set_lusgs(e["fspr"], e["tfspr"] if case["nvars"] > 5 else None)
        else:
            S.set_blusgs(e["jmat"])
        S.levels()  # the schedule of the sweeps, built once per mesh
        if kind == "solve":
            S.blusgs_pack(0, 0.0)
            S.blusgs_ns_prepare()
            S.autotune(reps=3)
    elif kind in ("array", "adjoint"):
        s["m"] = m = _array_inputs(case, seed)
        if kind == "array":
            m["nei32"] = m["nei"].to(I32)
            m["rhs0"] = m["rhs"].clone()
            m["diag"] = torch.zeros(m["N"], dtype=F64, device=DEV)
            m["dub"] = torch.zeros_like(m["rhs"])
            cl.set_dims(5, 5, 3)
        else:
            dt = F32 if case["fp32"] else F64
            s["mesh"] = ColoredMesh(m["nei"].cpu().numpy(), m["fnv"].cpu().numpy(), m["vec"].cpu().numpy(),
                                    m["icolor"].cpu().numpy(), m["ranges"])
            s["in"] = [m[k].to(dt).requires_grad_() for k in ("rhs", "dt", "fspr")]
            s["upts"] = m["upts"].to(dt)
            s["grad"] = _normal(m["g"], 5, m["N"]).to(dt)
    else:
        s["m"] = m = _bsr_inputs(case, seed)
        torch.cuda.synchronize()
        n = m["n"] * 5
        if kind != "precon":
            s["A"] = SpMat(m["n"], 5, m["rowptr"], m["colidx"], m["vals"], cuda=True)
        if kind == "spmv":
            s["y"] = torch.zeros(n, dtype=F64, device=DEV)
        elif kind == "precon":
            s["values"] = m["vals"].clone()  # ILU factors take the place of the values
            s["b"] = m["vec"].clone()
            torch.cuda.synchronize()
            s["pc"] = _precon(m, s["values"], case["ilu"], case["prec"])
        else:
            s["values"] = m["vals"].clone()
            s["x"] = torch.zeros(n, dtype=F64, device=DEV)
            torch.cuda.synchronize()
            s["pc"] = _precon(m, s["values"], kind == "bicgstab", case["prec"])
            s["solver"] = Solver(n, 30, 40, 1e-10 * float(m["vec"].norm()), cuda=True,
                                 kind="gmres" if kind == "gmres" else "bicgstab")
            s["solver"].set_precision(case["prec"])
    torch.cuda.synchronize()
    return s


def run(s):
    return globals()["_run_" + s["case"]["kind"]](s)


def _written():
    """What torch wrote on its stream is there before the library reads it on its own."""
    torch.cuda.current_stream().synchronize()


def _run_array(s):
    m, case = s["m"], s["case"]
    m["rhs"].copy_(m["rhs0"])  # the step's right-hand side; the sweeps leave dQ in its place
    _written()
    cl.set_precision(case["prec"])
    c = dict(neles=m["N"], nface=6, nei_ele=m["nei32"], lcolor=m["lcolor"], fnorm_vol=m["fnv"], vec_fnorm=m["vec"],
             upts=m["upts"], rhs=m["rhs"], dt=m["dt"], fspr=m["fspr"])
    cl.colored_step(c, m["icolor"], m["ranges"], m["diag"], m["dub"])
    return [m["upts"], m["rhs"], m["diag"]]


def _run_lusgs(s):
    S = s["S"]
    S.lusgs_pack(0, 1.0, 0.0)
    if s["case"]["nvars"] == 5:
        S.lusgs_ns_prepare()
        S.lusgs_ns_lower()
        S.lusgs_ns_upper()
    else:
        S.lusgs_nsrans_prepare()
        S.lusgs_nsrans_lower()
        S.lusgs_nsrans_upper()
    S.lusgs_update(0)
    return s["e"]["upts"]


def _run_loop(s):
    S, case = s["S"], s["case"]
    norms = np.zeros(case["iters"])
    S.lusgs_pack(0, 1.0, 0.0)
    S.lusgs_run(case["iters"], rans=case["nvars"] > 5, resid=norms)
    S.lusgs_update(0)
    return [s["e"]["upts"], norms]


def _run_blusgs(s):
    S = s["S"]
    S.blusgs_pack(0, 0.0)
    S.blusgs_ns_prepare()
    S.blusgs_reset()
    for _ in range(s["case"]["sweeps"]):
        S.blusgs_ns_lower()
        S.blusgs_ns_upper()
        S.blusgs_sub_residual(0)
    S.blusgs_update(0)
    return [s["e"]["upts"], s["e"]["resid"]]


def _run_solve(s):
    S = s["S"]
    S.blusgs_pack(0, 0.0)
    S.blusgs_ns_prepare()
    S.blusgs_reset()
    S.blusgs_solve(rtol=1e-10, max_sweeps=400, inner_sweeps=20)
    S.blusgs_update(0)
    return s["e"]["upts"]


def _run_spmv(s):
    s["A"].mult(1.0, s["m"]["vec"], 0.0, s["y"], precision=s["case"]["prec"])
    return s["y"]


def _run_precon(s):
    s["b"].copy_(s["m"]["vec"])
    _written()
    s["pc"].apply(s["b"])
    return s["b"]


def _run_gmres(s):
    s["values"].copy_(s["m"]["vals"])  # the step's assembled matrix (block ILU(0) factorises it in place)
    s["x"].zero_()
    _written()
    s["A"].update_values()
    s["pc"].prepare()
    s["solver"].solve(s["pc"], s["A"], s["x"], s["m"]["vec"])
    return s["x"]


_run_bicgstab = _run_gmres


def _run_adjoint(s):
    dq = lusgs_step(*s["in"], s["mesh"], s["upts"])
    return [dq, *torch.autograd.grad(dq, s["in"], s["grad"])]


# ---- what a pass cannot do without ------------------------------------------------
def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    kind, nv = case["kind"], case.get("nvars", 5)
    faces = 3 * n - case["nx"] * case["ny"] - case["ny"] * case["nz"] - case["nx"] * case["nz"]
    flux = 2 * (60 + 8 * (nv - 5))          # two fluxes and their difference, one face
    if kind == "array":                     # nei, fnorm_vol, vec, fspr, lcolor/icolor, dt; upts, rhs in and out; diag out
        return dict(bytes=n * (6 * 4 + 6 * 8 * 5 + 8 + 8 + 2 * 10 * 8 + 8.0), flops=n * (6 * flux + 60.0))
    if kind == "adjoint":
        w = 4 if case["fp32"] else 8
        return dict(bytes=n * (6 * 8 + 8 + w * (6 * 5 + 6 + 2 * 1 + 5 * 5 + 2.0)), flops=n * (6 * flux + 6 * 2 * 90.0))
    if kind in ("lusgs", "loop"):           # CSR, faces (area, normal, radius), state in and out, rhs, dt, source
        once = n * (4 + 8 + 4 + 8 + 8.0 * (4 * nv)) + faces * (2 * 9 + 8 * (5 + (nv > 5)))
        it = case.get("iters", 1)
        w = 4 if case["prec"] == FP32 else 8
        # every iteration needs each face's data and each cell's state, increment and right-hand side
        return dict(bytes=once + (it - 1) * (n * w * 4 * nv + faces * (2 * 4 + w * (5 + (nv > 5)))),
                    flops=it * n * (6.0 * flux + 60))
    if kind in ("blusgs", "solve"):         # the face Jacobians once, and the off-diagonal blocks once per sweep pair
        w = 4 if case["prec"] == FP32 else 8
        pairs = case["sweeps"] if kind == "blusgs" else 40
        pair = 2 * faces * (4 + 25 * w) + n * 5 * w * 6.0
        return dict(bytes=faces * (400 + 2 * 9 + 32.0) + n * 8 * (5 * 3 + 2) + pairs * pair,
                    flops=n * 2 * (150 + 100.0) + pairs * 2 * faces * 50.0)
    rows = 6 * n
    inner = 24 * n - 4 * (case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nx"] * case["nz"])  # off-diagonal blocks
    w = 4 if case["prec"] == FP32 else 8
    product = dict(bytes=(inner + rows) * (4 + 25.0 * w) + rows * 80, flops=(inner + rows) * 50.0)
    sweep = dict(bytes=inner * (4 + 25.0 * w) + rows * (25 * w + 80), flops=inner * 50.0 + rows * 100)
    if kind == "spmv":
        return product
    if kind == "precon":
        return sweep
    new = (inner + rows) * 200.0            # the matrix values are read once more than the solve reads them
    if kind == "gmres":                     # about nine Arnoldi steps, each vector orthogonalised against those before it
        return dict(bytes=new + 9 * (product["bytes"] + sweep["bytes"] + rows * 40 * 8),
                    flops=9 * (product["flops"] + sweep["flops"] + rows * 5 * 2 * 4 * 5.0))
    return dict(bytes=new + 3 * (2 * product["bytes"] + 2 * sweep["bytes"] + rows * 40 * 10),
                flops=3 * (2 * product["flops"] + 2 * sweep["flops"] + rows * 5 * 30.0))


# ---- the same in plain 64-bit torch -------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "array":
        m = _array_inputs(case, seed)
        dq, diag = _colored_step(m, m["rhs"], m["dt"], m["fspr"], m["upts"])
        return [m["upts"] + dq, dq, diag]
    if kind == "adjoint":
        m = _array_inputs(case, seed)
        dt = F32 if case["fp32"] else F64
        leaf = [m[k].to(dt).double().requires_grad_() for k in ("rhs", "dt", "fspr")]
        m["fnv"], m["vec"] = m["fnv"].to(dt).double(), m["vec"].to(dt).double()
        dq, _ = _colored_step(m, *leaf, m["upts"].to(dt).double())
        grads = torch.autograd.grad(dq, leaf, _normal(m["g"], 5, m["N"]).to(dt).double())
        return [dq.detach(), *grads]
    if kind in ("lusgs", "loop"):
        return _exact_lusgs(case, seed)
    if kind in ("blusgs", "solve"):
        return _exact_blusgs(case, seed)
    return _exact_bsr(case, seed)


def _flux(u, n):
    """Euler flux through unit normals n [3, ...] of states u [5, ...]."""
    c = (u[1:4] * n).sum(0) / u[0]
    p = (GAMMA - 1) * (u[4] - 0.5 * (u[1:4] ** 2).sum(0) / u[0])
    return torch.cat([(u[0] * c)[None], u[1:4] * c + n * p, ((u[4] + p) * c)[None]])


def _scalar_sums(cells, nb, act, u, d, n, lam, fa, turb):
    """Sum over the active faces of (F(u + d) - F(u) - lam d) fa; nb, act, lam, fa [P, k], n [3, P, k]."""
    uj, dj = u[:, nb], d[:, nb]
    if turb:
        df = dj * ((uj[1:4] * n).sum(0) / uj[0])
    else:
        df = _flux(uj[:5] + dj, n) - _flux(uj[:5], n)
    return ((df - lam * dj) * (fa * act)).sum(1)


def _colored_step(m, rhs, dt, fspr, upts):
    diag = 1.0 / dt + (0.5 * fspr * m["fnv"]).sum(0)
    d = torch.zeros_like(rhs)
    for upper in (False, True):
        for l in range(len(m["cells"])) if not upper else reversed(range(len(m["cells"]))):
            c = m["cells"][l]
            nb = m["nei"][:, c]
            act = (m["lev"][nb] > l) if upper else (m["lev"][nb] < l)
            df = _scalar_sums(c, nb, act, upts, d, m["vec"][:, :, c].transpose(0, 1), fspr[:, c], m["fnv"][:, c], False)
            new = d[:, c] - 0.5 * df / diag[c] if upper else (rhs[:, c] - 0.5 * df) / diag[c]
            d = d.index_copy(1, c, new)
    return d, diag


def _cell_faces(m):
    """The CSR as tables [6, N]: neighbour (-1: none), face, side, and area over volume."""
    N = m["N"]
    deg = (m["rowptr"][1:] - m["rowptr"][:-1]).long()
    row = torch.repeat_interleave(torch.arange(N, device=DEV), deg)
    at = torch.arange(row.numel(), device=DEV) - m["rowptr"][:-1].long()[row]
    nb = torch.full((6, N), -1, dtype=torch.int64, device=DEV)
    slot, side = torch.zeros_like(nb), torch.zeros(6, N, dtype=F64, device=DEV)
    nb[at, row], slot[at, row], side[at, row] = m["colidx"].long(), m["slots"].long(), m["sides"].double()
    return nb, slot, side, torch.where(nb >= 0, m["area"][slot], 0) * m["rcp_vol"]


def _exact_lusgs(case, seed):
    m, e = _flowsys_inputs(case, seed)
    nb, slot, side, fa = _cell_faces(m)
    lev = _levels(nb, case["greedy"])
    cells = _by_level(lev)
    ids = m["ids"].long()
    rank = torch.argsort(ids)  # element of each rank
    n = (m["normal"][:, slot] * side)  # [3, 6, N]
    u, rhs, dt = e["upts"][:, rank].clone(), e["rhs"][:, rank], e["dt"][rank]
    systems = [(slice(0, 5), e["fspr"][slot], False)]
    if case["nvars"] > 5:
        systems.append((slice(5, None), e["tfspr"][slot], True))
    norms = []
    for _ in range(case.get("iters", 1)):
        d = torch.zeros_like(u)
        for v, lam, turb in systems:
            diag = 1.0 / dt + (0.5 * lam * fa).sum(0)
            x = torch.zeros_like(rhs[v])
            for upper in (False, True):
                for l in range(len(cells)) if not upper else reversed(range(len(cells))):
                    c = cells[l]
                    g = nb[:, c]
                    k = lev[g.clamp(min=0)]
                    act = (g >= 0) & ((k > l) if upper else (k < l))
                    df = _scalar_sums(c, g.clamp(min=0), act, u, x, n[:, :, c], lam[:, c], fa[:, c], turb)
                    x[:, c] = x[:, c] - 0.5 * df / diag[c] if upper else (rhs[v][:, c] - 0.5 * df) / diag[c]
            d[v] = x
        u += d
        norms.append(float(d.norm()))
    up = u[:, ids]
    return up if case["kind"] == "lusgs" else [up, np.array(norms)]


def _exact_blusgs(case, seed):
    m, e = _flowsys_inputs(case, seed)
    nb, slot, side, fa = _cell_faces(m)
    lev = _levels(nb, case["greedy"])
    cells = _by_level(lev)
    ids = m["ids"].long()
    rank = torch.argsort(ids)
    N = m["N"]
    rhs, dt, vol = e["rhs"][:, rank].T.contiguous(), e["dt"][rank], m["vol"][rank]
    h = e["jmat"].permute(0, 3, 1, 2).reshape(2, m["nF"], 25).contiguous()
    D = (1.0 / dt)[:, None, None] * torch.eye(5, dtype=F64, device=DEV)
    J = torch.empty(6, N, 5, 5, dtype=F64, device=DEV)
    for p in range(6):
        pos = (side[p] > 0)[:, None]
        a, b = h[0][slot[p]], h[1][slot[p]]
        D += (torch.where(pos, a, -b) * fa[p][:, None]).reshape(N, 5, 5)
        J[p] = (torch.where(pos, b, -a) * fa[p][:, None]).reshape(N, 5, 5)
    del h
    inv = torch.linalg.inv(D)
    x, last = torch.zeros(N, 5, dtype=F64, device=DEV), torch.zeros(N, 5, dtype=F64, device=DEV)
    resid = None
    for k in range(case["sweeps"] if case["kind"] == "blusgs" else 120):
        for order in (range(len(cells)), reversed(range(len(cells)))):
            for l in order:
                c = cells[l]
                t = rhs[c].clone()
                for p in range(6):
                    t -= (J[p][c] @ x[nb[p][c].clamp(min=0)][:, :, None])[:, :, 0]
                x[c] = (inv[c] @ t[:, :, None])[:, :, 0]
        step = (x - last)
        resid = step ** 2 * vol[:, None]
        last = x.clone()
        if case["kind"] == "solve" and float(step.norm()) < 1e-15 * float(x.norm()):
            break
    up = e["upts"] + x.T[:, ids]
    return up if case["kind"] == "solve" else [up, resid.T[:, ids].contiguous()]


def _block_product(m, vals, x, keep=None):
    """Sum over the kept blocks of each row of block @ x."""
    t = torch.zeros(m["n"], 5, dtype=F64, device=DEV)
    step = 1 << 22
    for a in range(0, vals.shape[0], step):
        b = slice(a, a + step)
        y = (vals[b] * x[m["colidx"][b].long()][:, None, :]).sum(2)
        t.index_add_(0, m["rows"][b], y if keep is None else y * keep[b, None])
    return t


def _exact_bsr(case, seed):
    m = _bsr_inputs(case, seed)
    b, vals, col = m["vec"].reshape(-1, 5), m["vals"], m["colidx"].long()
    if case["kind"] == "spmv":
        return _block_product(m, vals, b).reshape(-1)
    if case["kind"] == "precon":
        return _exact_precon(case, m, b).reshape(-1)
    inv = torch.linalg.inv(vals[m["diag"].long()])
    x = torch.zeros_like(b)
    for _ in range(200):  # block Jacobi: strongly diagonally dominant rows
        r = b - _block_product(m, vals, x)
        x += (inv @ r[:, :, None])[:, :, 0]
        if float(r.norm()) < 1e-15 * float(b.norm()):
            break
    return x.reshape(-1)


def _exact_precon(case, m, b):
    """Symmetric Gauss-Seidel or block ILU(0) of the colour-ordered rows: colour by colour down, then up."""
    n, col, rows = m["n"], m["colidx"].long(), m["rows"]
    start = m["rowptr"].long()
    tab = torch.full((5, n), -1, dtype=torch.int64, device=DEV)  # slots of each row
    tab[torch.arange(col.numel(), device=DEV) - start[rows], rows] = torch.arange(col.numel(), device=DEV)
    vals, diag = m["vals"].clone(), m["diag"].long()
    ends = m["ends"].tolist()
    cells = [torch.arange(a, z, device=DEV) for a, z in zip(ends[:-1], ends[1:])]
    if case["ilu"]:
        for c in cells:  # rows of one colour are independent
            for p in range(5):
                q = tab[p, c]
                r = c[(q >= 0) & (col[q.clamp(min=0)] < c)]
                q = tab[p, r]
                k = col[q]
                f = vals[q] @ torch.linalg.inv(vals[diag[k]])
                vals[q] = f
                for j in range(p + 1, 5):
                    t = tab[j, r]
                    for i in range(5):
                        o = tab[i, k]
                        hit = (t >= 0) & (o >= 0) & (col[t.clamp(min=0)] == col[o.clamp(min=0)])
                        vals[t[hit]] -= f[hit] @ vals[o[hit]]
    inv = torch.linalg.inv(vals[diag])
    x = b.clone()
    for upper in (False, True):
        for c in reversed(cells) if upper else cells:
            t = torch.zeros(c.numel(), 5, dtype=F64, device=DEV)
            for p in range(5):
                q = tab[p, c]
                g = col[q.clamp(min=0)]
                use = (q >= 0) & ((g > c) if upper else (g < c))
                t += ((vals[q.clamp(min=0)] @ x[g][:, :, None])[:, :, 0]) * use[:, None]
            solve = lambda v: (inv[c] @ v[:, :, None])[:, :, 0]  # noqa: E731
            if case["ilu"]:
                x[c] = solve(x[c] - t) if upper else x[c] - t
            else:
                x[c] = x[c] - solve(t) if upper else solve(x[c] - t)
    return x
