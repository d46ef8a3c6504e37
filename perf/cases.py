"""Performance cases of the ADER-DG element path: what a user's program has it do.

Kinds (``kind``), each through the public entry points of adg_gb300 or the C ABI:

  evolve    state in from a device array, time step size, `steps` steps of the evolve loop
            (graph replay), state out to a device array
  patches   the zero-copy boundary: the state lives in per-(box, variable) device arrays with one
            ghost cell, as an AMReX host keeps it; read, step, write back
  host      the state lives in page-locked host memory: packed copy in, step, step readback
  transfer  L2 projections of a batch of cells between levels (gather of the children, scatter)
  train     epochs of Adam on the seed network, whole data set per batch

Layouts (``layout``): "single" one level; "boxes" refinement boxes given by the caller (a host that
owns the regrid); "regrid" the library's own tagging and clustering every 4 steps.
With ``seeded`` the predictor starts from the learned seed (two FP32 sweeps).

`exact` restates the method in 64 bits with dense matrices on dense level arrays.
"""
import ctypes
import itertools
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "ader-dg-amr_gb300"))
import adg_gb300 as G  # noqa: E402

DEV = "cuda"
F64 = torch.float64
GAMMA, C_DT = 1.4, 0.5


def listed():
    return [
        # benchmark configuration 1: smallest grid, 20 steps at once (launch-bound)
        dict(name="vortex_p1_32_20steps", kind="evolve", D=2, P=1, nx=32, ny=32, nz=1, ic="vortex", periodic=True,
             layout="single", levels=1, steps=20, seeded=False, limited=False),
        # a ragged grid with outflow boundaries, a few thousand elements
        dict(name="vortex_p2_45x61_outflow", kind="evolve", D=2, P=2, nx=45, ny=61, nz=1, ic="vortex", periodic=False,
             layout="single", levels=1, steps=2, seeded=False, limited=False),
        # benchmark configuration 2: single-level Kelvin-Helmholtz
        dict(name="kh_p3_256", kind="evolve", D=2, P=3, nx=256, ny=256, nz=1, ic="kh", periodic=True,
             layout="single", levels=1, steps=1, seeded=False, limited=False),
        # benchmark configuration 3: three levels with the library's own regrid every 4 steps
        dict(name="kh_p3_3levels_regrid", kind="evolve", D=2, P=3, nx=64, ny=64, nz=1, ic="kh", periodic=True,
             layout="regrid", levels=3, steps=4, seeded=False, limited=False),
        # the same hierarchy owned by an AMReX host: boxes from the host, state in its device arrays
        dict(name="kh_p3_3levels_patches", kind="patches", D=2, P=3, nx=64, ny=64, nz=1, ic="kh", periodic=True,
             layout="boxes", levels=3, steps=1, seeded=False, limited=False),
        # benchmark configuration 4 end to end: learned seed, state in and out of host memory every step
        dict(name="kh_p3_3levels_seeded_host", kind="host", D=2, P=3, nx=64, ny=64, nz=1, ic="kh", periodic=True,
             layout="boxes", levels=3, steps=1, seeded=True, limited=False),
        # the 3D blast of benchmark configuration 5 on one level
        dict(name="blast_p2_64cubed", kind="evolve", D=3, P=2, nx=64, ny=64, nz=64, ic="blast", periodic=False,
             layout="single", levels=1, steps=1, seeded=False, limited=False),
        # configuration 5: two levels, TVB limiter every step, regrid (32^3 -> 64^3)
        dict(name="blast_p2_32cubed_2levels_limited", kind="evolve", D=3, P=2, nx=32, ny=32, nz=32, ic="blast",
             periodic=False, layout="regrid", levels=2, steps=4, seeded=False, limited=True),
        # the highest degree the reference's thesis runs
        dict(name="vortex_p6_48", kind="evolve", D=2, P=6, nx=48, ny=48, nz=1, ic="vortex", periodic=True,
             layout="single", levels=1, steps=1, seeded=False, limited=False),
        # the highest 3D degree, ragged box
        dict(name="blast_p3_20x14x18", kind="evolve", D=3, P=3, nx=20, ny=14, nz=18, ic="blast", periodic=False,
             layout="single", levels=1, steps=1, seeded=False, limited=False),
        # a host's own FillPatch / average down: projections of a batch of cells
        dict(name="transfer_p3_60001", kind="transfer", D=2, P=3, cells=60001),
        # training the seed network (hidden width 128)
        dict(name="train_p3_16384", kind="train", D=2, P=3, pairs=16384, epochs=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    r = rng.random()
    if r < 0.1:
        D = rng.choice([2, 2, 3])
        P = rng.randint(1, 3) if D == 2 else rng.randint(1, 2)
        return dict(kind="transfer", D=D, P=P, cells=_log_int(rng, 300, 120000))
    if r < 0.18:
        return dict(kind="train", D=2, P=rng.choice([2, 3]), pairs=_log_int(rng, 1000, 20000), epochs=rng.randint(2, 8))
    if r < 0.5:  # AMR hierarchies in 2D
        kind = rng.choice(["evolve", "patches", "host"])
        layout = "regrid" if kind == "evolve" and rng.random() < 0.5 else "boxes"
        n = 16 * rng.randint(1, 5)
        levels = rng.randint(2, 3)
        return dict(kind=kind, D=2, P=rng.choice([1, 2, 3, 3]), nx=n, ny=max(32, n), nz=1, ic="kh", periodic=True,
                    layout=layout, levels=levels, steps=4 if layout == "regrid" else 1,
                    seeded=rng.random() < 0.4, limited=False)
    if r < 0.75:  # one level, 2D
        P = rng.choice([1, 2, 3, 3, 4, 5, 6])
        top = {1: 256, 2: 256, 3: 230, 4: 110, 5: 64, 6: 48}[P]
        ic = rng.choice(["kh", "vortex"])
        return dict(kind="evolve", D=2, P=P, nx=_log_int(rng, 8, top), ny=_log_int(rng, 8, top), nz=1, ic=ic,
                    periodic=ic == "kh" or rng.random() < 0.5, layout="single", levels=1, steps=rng.randint(1, 3),
                    seeded=P <= 3 and rng.random() < 0.3, limited=False)
    P = rng.choice([1, 2, 2, 3])  # one level, 3D
    top = {1: 60, 2: 40, 3: 16}[P]
    return dict(kind="evolve", D=3, P=P, nx=_log_int(rng, 5, top), ny=_log_int(rng, 5, top), nz=_log_int(rng, 5, top),
                ic="blast", periodic=rng.random() < 0.4, layout="single", levels=1, steps=1, seeded=False,
                limited=rng.random() < 0.3)


# --------------------------------------------------------------------------- geometry and inputs
def _dims(c, lev):
    return [c["nx"] << lev, c["ny"] << lev] + ([c["nz"] << lev] if c["D"] == 3 else [])


def _extent(c):
    s = 10.0 if c["ic"] == "vortex" else 1.0
    n = _dims(c, 0)
    return [s * k / max(n) for k in n] if c["ic"] != "kh" else [1.0] * c["D"]


def _boxes(c):
    """The caller's boxes of each level: level 0 whole; finer levels bands about the two shear layers."""
    out = []
    for lev in range(c["levels"]):
        nx, ny = _dims(c, lev)
        rows = [(0, ny)] if lev == 0 else [(ny // 4 - 8, ny // 4 + 8), (3 * ny // 4 - 8, 3 * ny // 4 + 8)]
        bx = []
        for lo, hi in rows:
            for j in range(lo, hi, 32):
                for i in range(0, nx, 32):
                    bx.append([i, j, 0, min(i + 32, nx) - 1, min(j + 32, hi) - 1, 0])
        out.append(np.array(bx, np.int32))
    return out


def _cells(boxes, n):
    """Cells (i, j, k) of a level's boxes in the order of the state arrays (x fastest over the level)."""
    mask = np.zeros(n[::-1], bool)
    for b in boxes:
        mask[tuple(slice(b[d], b[d + 3] + 1) for d in range(len(n)))[::-1]] = True
    idx = np.argwhere(mask)[:, ::-1]
    return torch.from_numpy(np.ascontiguousarray(idx)).to(DEV)


def _basis(D, P):
    x, w = np.polynomial.legendre.leggauss(P + 1)
    x, w = x[::-1].copy(), w[::-1].copy()  # node 0 is the largest one, where the time step is evaluated
    modes = [m for m in itertools.product(range(P + 1), repeat=D) if sum(m) <= P]
    val = np.stack([np.polynomial.legendre.legval(x, np.eye(P + 1)[k]) for k in range(P + 1)])
    return x, w, modes, val


def _primitive(c, x, seed):
    """(rho, v_1.., p) at points x [..., D]: the initial condition of the case, its free parameters from the seed."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    u = torch.rand(6, generator=g, device=DEV, dtype=F64)
    if c["ic"] == "kh":  # shear layer, perturbed, with noise at every point
        y = x[..., 1]
        inside = (y > 0.25) & (y < 0.75)
        rho = torch.where(inside, 2.0, 1.0).to(F64)
        noise = 2 * torch.rand(rho.shape, generator=g, device=DEV, dtype=F64) - 1
        v = [torch.where(inside, 0.5, -0.5).to(F64),
             0.01 * torch.sin(4 * math.pi * (x[..., 0] + u[0])) + 1e-3 * noise]
        return [rho] + v + [torch.full_like(rho, 2.5)]
    if c["ic"] == "vortex":  # isentropic vortex on a free stream
        e = _extent(c)
        dx, dy = x[..., 0] - e[0] * (0.45 + 0.1 * u[0]), x[..., 1] - e[1] * (0.45 + 0.1 * u[1])
        r2, b = dx * dx + dy * dy, 4.0 + 2.0 * u[2]
        rho = (1 - (GAMMA - 1) * b * b / (8 * GAMMA * math.pi ** 2) * torch.exp(1 - r2)) ** (1 / (GAMMA - 1))
        k = b / (2 * math.pi) * torch.exp((1 - r2) / 2)
        return [rho, 1 - dy * k, 0.5 + dx * k, rho ** GAMMA]
    # spherical blast at rest, its centre and pressure from the seed
    e = _extent(c)
    r = torch.sqrt(sum((x[..., d] - e[d] * (0.47 + 0.06 * u[d])) ** 2 for d in range(3)))
    p = torch.where(r < 0.1, 9.0 + 2.0 * u[3], 0.1).to(F64)
    return [torch.ones_like(p)] + [torch.zeros_like(p)] * 3 + [p]


def _state(c, lev, ijk, seed):
    """Modal coefficients [cells, Q, Np_s] of the initial condition on the given cells of a level."""
    D, P = c["D"], c["P"]
    x, w, modes, val = _basis(D, P)
    pts = list(itertools.product(range(P + 1), repeat=D))
    e, n = _extent(c), _dims(c, lev)
    dx = torch.tensor([e[d] / n[d] for d in range(D)], device=DEV, dtype=F64)
    ref = torch.tensor([[x[p[d]] for d in range(D)] for p in pts], device=DEV, dtype=F64)
    proj = torch.tensor([[math.prod(val[m[d]][p[d]] * w[p[d]] * (2 * m[d] + 1) / 2 for d in range(D)) for p in pts]
                         for m in modes], device=DEV, dtype=F64)
    pos = (ijk[:, None, :].to(F64) + 0.5 + 0.5 * ref[None]) * dx
    pr = _primitive(c, pos, 1000003 * seed + lev)
    rho, v, p = pr[0], pr[1:-1], pr[-1]
    u = [rho] + [rho * a for a in v] + [p / (GAMMA - 1) + 0.5 * rho * sum(a * a for a in v)]
    return torch.einsum("mp,ecp->ecm", proj, torch.stack(u, 1)).contiguous()


def _solver(c, seed):
    D = c["D"]
    s = G.AmrDG(P=c["P"], D=D)
    multi = c["layout"] != "single"
    s.setGeometrySettings(prob_lo=(0.0,) * 3, prob_hi=_extent(c) + [1.0], n_cell=_dims(c, 0) + [1],
                          max_level=c["levels"] - 1, periodic=(int(c["periodic"]),) * 3,
                          max_grid=32 if multi else 1 << 20, blocking_factor=8,
                          dtn_regrid=4 if c["layout"] == "regrid" else 0)
    s.setAmrSettings(tag_kind=1 if c["ic"] == "blast" else 0, tag_threshold=0.1,
                     reflux_box_quirk=0 if c["layout"] == "boxes" else 1)
    s.settings(c_dt=C_DT, **(dict(limiter_type="TVB", TVB_M=10.0, t_limit=1) if c["limited"] else {}))
    name = {"kh": "kh_noise", "vortex": "isentropic_vortex", "blast": "blast3d"}[c["ic"]]
    s.init(G.Compressible_Euler().settings(name, seed=seed & 0xFFFF))
    return s


# --------------------------------------------------------------------------- the learned seed's network
def _gelu(z):
    return 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))


def _features(U, dtdx):
    rho = U[:, :1, 0]
    return torch.cat([U.reshape(U.shape[0], -1) / rho, dtdx.reshape(-1, 1)], 1)


def _network(c, levels, dt, seed):
    """Network parameters in the library's order (float32): three random layers, the output layer fitted
    by least squares to converged predictors of a sample of the given states."""
    D, P = c["D"], c["P"]
    U, e = torch.cat(levels), _extent(c)
    dtdx = torch.cat([torch.full((u.shape[0],), dt * _dims(c, k)[0] / e[0], device=DEV, dtype=F64)
                      for k, u in enumerate(levels)])
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 77)
    op = _operators(D, P)
    at = torch.randperm(U.shape[0], generator=g, device=DEV)[:3000]
    U, dtdx = U[at], dtdx[at]
    X = _features(U, dtdx)
    H = _picard(op, U, dtdx[:, None].expand(-1, D), 8)
    T = ((H - U @ op["W"].T) / (U[:, :1, :1] * dtdx[:, None, None])).reshape(U.shape[0], -1)
    xm, xs = X.mean(0), X.std(0, unbiased=False)
    xi = 1.0 / torch.maximum(xs, 0.1 * xm.abs() + 1e-6)
    ym, ys = T.mean(0), torch.maximum(T.std(0, unbiased=False), 0.1 * T.mean(0).abs() + 1e-6)
    par, h, fan = [], (X - xm) * xi, X.shape[1]
    for k in range(3):
        W = torch.randn(fan, 128, generator=g, device=DEV, dtype=F64) * (0.7 / math.sqrt(fan))
        b = 0.1 * torch.randn(128, generator=g, device=DEV, dtype=F64)
        h, fan = _gelu(h @ W + b), 128
        par += [W, b]
    A = torch.cat([h, torch.ones_like(h[:, :1])], 1)
    S = torch.linalg.solve(A.T @ A + 1e-6 * A.shape[0] * torch.eye(A.shape[1], device=DEV, dtype=F64),
                           A.T @ ((T - ym) / ys))
    par += [S[:-1], S[-1], xm, xi, ym, ys]
    return [p.to(torch.float32) for p in par]


# --------------------------------------------------------------------------- prepare and run
def _transfer_inputs(c, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    D, n = c["D"], c["cells"]
    nps, kids = math.comb(c["P"] + D, D), 1 << D
    decay = torch.exp(-1.5 * torch.arange(nps, device=DEV, dtype=F64) / nps)
    fine = torch.randn(n, kids, D + 2, nps, generator=g, device=DEV, dtype=F64) * decay
    coarse = torch.randn(n, D + 2, nps, generator=g, device=DEV, dtype=F64) * decay
    child = torch.randint(0, kids, (n,), generator=g, device=DEV).to(torch.int8)
    return fine, coarse, child


def _train_inputs(c, seed):
    """A Kelvin-Helmholtz grid of about `pairs` elements, and starting weights."""
    n = int(math.sqrt(c["pairs"]))
    grid = dict(c, nx=n, ny=n, nz=1, ic="kh", periodic=True, layout="single", levels=1, limited=False)
    U = _state(grid, 0, _cells([[0, 0, 0, n - 1, n - 1, 0]], [n, n]), seed)
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 3)
    sizes = [U.shape[1] * U.shape[2] + 1, 128, 128, 128, (c["D"] + 2) * math.comb(c["P"] + c["D"] + 1, c["D"] + 1)]
    par = []
    for a, b in zip(sizes, sizes[1:]):
        par += [(torch.rand(a, b, generator=g, device=DEV) * 2 - 1) * math.sqrt(6.0 / (a + b)),
                0.02 * torch.randn(b, generator=g, device=DEV)]
    return grid, U, par, _time_step(grid, [U])


def _patch_layout(c, cells_of):
    """(level, cell index array of the box, offset, extents) of each box, and the doubles of all arrays:
    per (box, variable) one array with a ghost cell on every side and the modes as components."""
    Q, nps = c["D"] + 2, math.comb(c["P"] + c["D"], c["D"])
    out, off = [], 0
    for lev, bx in enumerate(_boxes(c)):
        n, ijk = _dims(c, lev), cells_of(lev)
        index = torch.full((n[1], n[0]), -1, device=DEV, dtype=torch.int64)
        index[ijk[:, 1], ijk[:, 0]] = torch.arange(ijk.shape[0], device=DEV)
        for b in bx:
            e0, e1 = int(b[3] - b[0] + 3), int(b[4] - b[1] + 3)
            out.append((lev, b, index[b[1]:b[4] + 1, b[0]:b[3] + 1], off, e0, e1))
            off += Q * nps * e0 * e1
    return out, off


def _into_patches(c, layout, total, levels):
    flat = torch.zeros(total, device=DEV, dtype=F64)
    Q, nps = levels[0].shape[1:]
    for lev, _, cells, o, e0, e1 in layout:
        v = flat[o:o + Q * nps * e0 * e1].view(Q, nps, e1, e0)
        v[:, :, 1:-1, 1:-1] = levels[lev][cells].permute(2, 3, 0, 1)
    return flat


def _register_patches(c, s, levels):
    layout, total = _patch_layout(c, lambda lev: _coords(s, lev))
    start = _into_patches(c, layout, total, levels)
    arrays, patches = start.clone(), []
    for lev, b, _, o, e0, e1 in layout:
        p = G.AdgPatch()
        p.level, p.nghost, p.jstride, p.kstride, p.nstride = lev, 1, e0, e0 * e1, e0 * e1
        p.lo[0], p.lo[1], p.hi[0], p.hi[1] = int(b[0]), int(b[1]), int(b[3]), int(b[4])
        for q in range(s.Q):
            p.U_w[q] = arrays.data_ptr() + 8 * (o + q * s.Np_s * e0 * e1)
        patches.append(p)
    s.set_patches(patches)
    return dict(start=start, arrays=arrays)


def _coords(s, lev):
    return torch.from_numpy(s.level_cell_coords(lev)[:, :s.D].astype(np.int64)).to(DEV)


def _ok(rc):
    if rc != G.ADG_OK:
        raise RuntimeError("status %d" % rc)


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "transfer":
        s = G.AmrDG(P=c["P"], D=c["D"])
        s.setGeometrySettings(prob_lo=(0,) * 3, prob_hi=(1,) * 3, n_cell=(4,) * 3)
        s.init(G.Compressible_Euler().settings("const"))
        fine, coarse, child = _transfer_inputs(c, seed)
        torch.cuda.synchronize()
        return dict(c=c, s=s, fine=fine, coarse=coarse, child=child, up=torch.empty_like(coarse),
                    down=torch.empty_like(coarse))
    if c["kind"] == "train":
        grid, U, par, dt = _train_inputs(c, seed)
        s = _solver(grid, seed)
        torch.cuda.synchronize()
        s.set_U_w_device(0, U.data_ptr())
        s.Dt = dt
        net = G.PredictorSeed(c["D"], c["P"], hidden=128, rng_seed=5)
        net.collect(s, target_sweeps=8)
        net.train(0, U.shape[0])  # standardises the pairs
        p = net.get_params()
        flat = np.concatenate([w.reshape(-1).cpu().numpy() for w in par])
        p[:flat.size] = flat
        return dict(c=c, s=s, net=net, par=p, pairs=U.shape[0])
    s = _solver(c, seed)
    st = dict(c=c, s=s)
    if c["layout"] == "boxes":
        s.set_layout(_boxes(c))
    elif c["layout"] == "regrid":  # the first step regrids on the real state
        U = torch.cat([_state(c, lev, _coords(s, lev), seed) for lev in range(s.num_levels())])
        torch.cuda.synchronize()
        s.set_U_w_device(G.ADG_ALL_LEVELS, U.data_ptr())
        s.set_Dt()
        s.advance(1)
        s.synchronize()
        st["boxes"] = [s.boxes(lev) for lev in range(s.num_levels())]
    levels = [_state(c, lev, _coords(s, lev), seed) for lev in range(s.num_levels())]
    U = torch.cat(levels).contiguous()
    torch.cuda.synchronize()
    s.set_U_w_device(G.ADG_ALL_LEVELS, U.data_ptr())
    dt = s.set_Dt()
    if c["seeded"]:
        net = G.PredictorSeed(c["D"], c["P"], hidden=128, rng_seed=5)
        net.set_params(torch.cat([p.reshape(-1) for p in _network(c, levels, dt, seed)]).cpu().numpy())
        net.attach(s, mode=2, sweeps=2, tol=1e-3)
        st["net"] = net
    if c["kind"] == "patches":
        st.update(_register_patches(c, s, levels))
    elif c["kind"] == "host":
        st["pin"], st["back"] = G.PinnedArray(tuple(U.shape)), G.PinnedArray(tuple(U.shape))
        st["pin"].array[...] = U.cpu().numpy()
        _ok(G.lib().adg_set_readback(s.ctx, G.ADG_ALL_LEVELS, st["back"].array.ctypes.data, U.shape[0]))
    else:
        st["U"], st["out"] = U, torch.empty_like(U)
    torch.cuda.synchronize()
    return st


def run(st):
    c, s = st["c"], st["s"]
    if c["kind"] == "transfer":
        L, vp, n = G.lib(), ctypes.c_void_p, c["cells"]
        _ok(L.adg_interp_gather(s.ctx, vp(st["fine"].data_ptr()), n, vp(st["up"].data_ptr()), G.ADG_MEM_DEVICE))
        _ok(L.adg_interp_scatter(s.ctx, vp(st["coarse"].data_ptr()), vp(st["child"].data_ptr()), n,
                                 vp(st["down"].data_ptr()), G.ADG_MEM_DEVICE))
        return dict(up=st["up"], down=st["down"])
    if c["kind"] == "train":
        st["net"].set_params(st["par"])
        loss = st["net"].train(c["epochs"], st["pairs"], 1e-3)
        return dict(params=st["net"].get_params(), loss=np.float32(loss))
    if c["kind"] == "patches":
        st["arrays"].copy_(st["start"])  # the host's own update of its arrays
        torch.cuda.current_stream().synchronize()
        s.read_patches()
        dt0 = s.set_Dt()
        s.advance(c["steps"])
        s.write_patches()
        s.synchronize()
        return dict(U=st["arrays"], dt0=dt0)
    if c["kind"] == "host":
        _ok(G.lib().adg_set_state(s.ctx, G.ADG_ALL_LEVELS, st["pin"].array.ctypes.data, G.ADG_MEM_HOST_ASYNC))
        dt0 = s.set_Dt()
        s.advance(c["steps"])
        s.synchronize()
        return dict(U=st["back"].array, dt0=dt0)
    if "boxes" in st:
        s.set_layout(st["boxes"])  # back to the boxes that the state lives on
    s.set_U_w_device(G.ADG_ALL_LEVELS, st["U"].data_ptr())
    dt0 = s.set_Dt()
    s.advance(c["steps"])
    n = sum(s.level_cells(k) for k in range(s.num_levels()))
    if n > st["out"].shape[0]:
        st["out"] = torch.empty((n,) + tuple(st["out"].shape[1:]), device=DEV, dtype=F64)
    s.get_U_w_device(G.ADG_ALL_LEVELS, st["out"].data_ptr())
    return dict(U=st["out"][:n], dt0=dt0, dt=s.Dt)


def work(case):
    c = case
    D, P = c["D"], c["P"]
    Q, N = D + 2, P + 1
    nps, npst = math.comb(P + D, D), math.comb(P + D + 1, D + 1)
    if c["kind"] == "transfer":
        n, k = c["cells"], 1 << D
        return dict(bytes=8 * n * Q * nps * (k + 3) + n, flops=n * Q * (k + 1) * 6 * nps)
    if c["kind"] == "train":
        n, i, o = c["pairs"], Q * nps + 1, Q * npst
        return dict(bytes=c["epochs"] * 4 * n * (i + o), flops=c["epochs"] * 6 * n * (128 * (i + o) + 2 * 128 * 128))
    cells = math.prod(_dims(c, 0))
    for lev in range(1, c["levels"]):  # 2D: two bands of 16 rows; 3D: a cube of a quarter of the edge
        cells += 32 * _dims(c, lev)[0] if D == 2 else math.prod(_dims(c, lev)) // 64
    sweeps = 2 if c["seeded"] else P
    line = (D + 1) * N ** (D + 2)  # one tensor-product transform of a variable, truncated basis
    per = Q * line * (sweeps * (1 + D) + 1 + D) + 20 * N ** (D + 1) * (sweeps + 1) + 2 * D * 30 * N ** D
    return dict(bytes=2 * 8 * cells * Q * nps, flops=c["steps"] * cells * per)


# --------------------------------------------------------------------------- 64-bit restatement
_OPS = {}


def _operators(D, P):
    """Dense matrices of the method: space-time evaluation V, predictor update A_d and W, corrector volume
    and boundary terms, face evaluation, mass diagonal, projections to and from the children."""
    if (D, P) in _OPS:
        return _OPS[D, P]
    x, w, ms, val = _basis(D, P)
    N, leg = P + 1, np.polynomial.legendre
    dval = np.stack([leg.legval(x, leg.legder(np.eye(N)[k])) if k else 0 * x for k in range(N)])
    end = np.array([[(-1.0) ** k, 1.0] for k in range(N)])
    mst = [m for m in itertools.product(range(N), repeat=D + 1) if sum(m) <= P]
    st, sp = list(itertools.product(range(N), repeat=D + 1)), list(itertools.product(range(N), repeat=D))

    def mass(k):
        return 2.0 / (2 * k + 1)

    def der(a, b):  # int P_a P_b'
        return 2.0 if b > a and (a + b) % 2 else 0.0

    V = np.array([[math.prod(val[m[d]][p[d]] for d in range(D + 1)) for m in mst] for p in st])
    Vi = np.linalg.pinv(V)
    Mh = np.array([[math.prod(map(mass, j[:D])) * (1 - der(i[D], j[D])) if j[:D] == i[:D] else 0.0 for i in mst]
                   for j in mst])
    Mp = np.array([[(-1.0) ** j[D] * math.prod(map(mass, j[:D])) if j[:D] == i else 0.0 for i in ms] for j in mst])
    A, vol, face, bd, half_bd = [], [], [], [], []
    for d in range(D):
        S = np.array([[der(j[d], i[d]) * math.prod(mass(j[a]) for a in range(D + 1) if a != d)
                       if all(j[a] == i[a] for a in range(D + 1) if a != d) else 0.0 for i in mst] for j in mst])
        A.append(np.linalg.solve(Mh, S) @ Vi)
        vol.append(np.array([[math.prod((dval if a == d else val)[m[a]][p[a]] * w[p[a]] for a in range(D)) * w[p[D]]
                              for p in st] for m in ms]))
        free = [a for a in range(D + 1) if a != d]
        at = [dict(zip(free, p)) for p in sp]
        for s in range(2):
            face.append(np.array([[math.prod(end[m[a]][s] if a == d else val[m[a]][q[a]] for a in range(D + 1))
                                   for m in mst] for q in at]))
            bd.append(np.array([[math.prod(w[q[a]] for a in free) *
                                 math.prod(end[m[a]][s] if a == d else val[m[a]][q[a]] for a in range(D))
                                 for q in at] for m in ms]))
            for k in range(2 if D == 2 else 0):  # a fine face covers half of the coarse one
                h = np.stack([leg.legval(0.5 * x + (0.5 if k else -0.5), np.eye(N)[j]) for j in range(N)])
                half_bd.append(np.array([[w[q[1 - d]] * w[q[2]] * end[m[d]][s] * h[m[1 - d]][q[1 - d]] for q in at]
                                         for m in ms]))
    kid, kidw = [], []
    Mi = np.array([1 / math.prod(map(mass, m)) for m in ms])[:, None]
    B = np.array([[math.prod(val[m[d]][p[d]] * w[p[d]] for d in range(D)) for p in sp] for m in ms])
    for l in range(1 << D):  # bit D-1-d of a child: the upper half in direction d
        h = [np.stack([leg.legval(0.5 * x + (0.5 if (l >> (D - 1 - d)) & 1 else -0.5), np.eye(N)[k])
                       for k in range(N)]) for d in range(D)]
        E = np.array([[math.prod(h[d][m[d]][p[d]] for d in range(D)) for m in ms] for p in sp])
        kid.append(Mi * (B @ E))
        kidw.append(Mi * (B @ E).T / (1 << D))

    def t(a):
        return torch.tensor(np.array(a), device=DEV, dtype=F64)

    _OPS[D, P] = dict(D=D, P=P, nps=len(ms), V=t(V), W=t(np.linalg.solve(Mh, Mp)), A=t(A), vol=t(vol), face=t(face),
                      bd=t(bd), half_bd=t(half_bd), kid=t(kid), kidw=t(kidw), M=1 / t(Mi)[:, 0],
                      pt0=t([math.prod(val[m[d]][0] for d in range(D)) for m in ms]))
    return _OPS[D, P]


def _flux(u, D):
    """Fluxes [D][e, Q, points], pressure and velocities of the states u [e, Q, points]."""
    v = [u[:, d + 1] / u[:, 0] for d in range(D)]
    p = (GAMMA - 1) * (u[:, D + 1] - 0.5 * sum(u[:, d + 1] * v[d] for d in range(D)))
    p = torch.clamp(p, min=10 * 2.220446049250313e-16)
    F = [torch.stack([u[:, d + 1]] + [u[:, k + 1] * v[d] + (p if k == d else 0) for k in range(D)] +
                     [(u[:, D + 1] + p) * v[d]], 1) for d in range(D)]
    return F, p, v


def _chunks(op, U):
    step = max(1, int(1e9 / (8 * U.shape[1] * op["V"].shape[0] * (op["D"] + 3))))
    return [slice(a, min(U.shape[0], a + step)) for a in range(0, U.shape[0], step)]


def _picard(op, U, c, sweeps, H=None, tol=None):
    """Predictor modes [e, Q, Np_st] (c: Dt/dx per element and direction).  With H the sweeps start there
    (the learned seed), and an element whose first change exceeds tol gets the plain P sweeps."""
    D = op["D"]
    out = torch.empty(U.shape[0], U.shape[1], op["V"].shape[1], device=DEV, dtype=F64)
    for a in _chunks(op, U):
        u, wu, bad = U[a], U[a] @ op["W"].T, None
        h = torch.zeros_like(wu) if H is None else H[a]
        if H is None:
            h[:, :, :op["nps"]] = u
        for k in range(sweeps):
            F, _, _ = _flux(h @ op["V"].T, D)
            n = wu - sum(c[a, d, None, None] * (F[d] @ op["A"][d].T) for d in range(D))
            if k == 0 and tol is not None:
                bad = (n - h).abs().amax((1, 2)) > tol * u[:, :, 0].abs().amax(1)
            h = n
        if bad is not None and bool(bad.any()):
            h[bad] = _picard(op, u[bad], c[a][bad], op["P"])
        out[a] = h
    return out


def _time_step(c, levels):
    op, D, e, rate = _operators(c["D"], c["P"]), c["D"], _extent(c), 0.0
    for lev, U in enumerate(levels):
        u = (U @ op["pt0"])[:, :, None]
        _, p, v = _flux(u, D)
        lam = torch.stack([x.abs() for x in v]).amax(0) + torch.sqrt(GAMMA * p / u[:, 0])
        dx = [e[d] / _dims(c, lev)[d] for d in range(D)]
        rate = max(rate, float(lam.max()) / (sum(dx) / D))
    return C_DT / (2 * op["P"] + 1) / D / rate


class _Level:
    """One level as a dense array over its whole index space, cells x fastest."""

    def __init__(self, c, lev, ijk):
        n, D = _dims(c, lev), c["D"]
        self.dx = [_extent(c)[d] / n[d] for d in range(D)]
        stride = [1, n[0], n[0] * n[1]]
        total = math.prod(n)
        self.cell = sum(ijk[:, d] * stride[d] for d in range(D))
        self.valid = torch.zeros(total, dtype=torch.bool, device=DEV)
        self.valid[self.cell] = True
        flat = torch.arange(total, device=DEV)
        pos = [(flat // stride[d]) % n[d] for d in range(D)]
        self.nbr = {}
        for d in range(D):
            for s in range(2):
                q = pos[d] + 2 * s - 1
                q = q % n[d] if c["periodic"] else q.clamp(0, n[d] - 1)
                self.nbr[d, s] = flat + (q - pos[d]) * stride[d]
        self.fine0 = sum(2 * pos[d] * (stride[d] << d) for d in range(D))  # lower corner child on the next level
        self.fine_stride = [stride[d] << d for d in range(D)]
        self.parent = sum((pos[d] // 2) * (stride[d] >> d) for d in range(D))
        self.child = sum((pos[d] % 2) << (D - 1 - d) for d in range(D))


def _step(c, op, L, U, dt, net):
    """One step of every level: U the valid cells' modes per level."""
    D, dense, flux, new = op["D"], [], [], []
    for k, lv in enumerate(L):
        u = torch.zeros(lv.valid.shape[0], *U[k].shape[1:], device=DEV, dtype=F64)
        u[lv.cell] = U[k]
        if k and not bool(lv.valid.all()):  # cells beside the fine region: the coarse solution there
            at = torch.nonzero(~lv.valid)[:, 0]
            for q in range(1 << D):
                b = at[lv.child[at] == q]
                u[b] = dense[k - 1][lv.parent[b]] @ op["kid"][q].T
        dense.append(u)
        cd = torch.tensor([dt / x for x in lv.dx], device=DEV, dtype=F64).expand(u.shape[0], D)
        if net is None:
            H = _picard(op, u, cd, op["P"])
        else:
            H = _picard(op, u, cd, 2, _network_seed(net, u, cd[:, 0]) + u @ op["W"].T, 1e-3)
        R = u * op["M"]
        for a in _chunks(op, u):
            F, _, _ = _flux(H[a] @ op["V"].T, D)
            R[a] += sum(cd[0, d] * (F[d] @ op["vol"][d].T) for d in range(D))
        tr = {(d, s): H @ op["face"][2 * d + s].T for d in range(D) for s in range(2)}
        f = {}
        for d in range(D):
            for s in range(2):
                left = tr[d, 1] if s else tr[d, 1][lv.nbr[d, 0]]
                right = tr[d, 0][lv.nbr[d, 1]] if s else tr[d, 0]
                (Fl, pl, vl), (Fr, pr, vr) = _flux(left, D), _flux(right, D)
                C = torch.maximum(vl[d].abs() + torch.sqrt(GAMMA * pl / left[:, 0]),
                                  vr[d].abs() + torch.sqrt(GAMMA * pr / right[:, 0]))[:, None]
                f[d, s] = 0.5 * (Fl[d] + Fr[d] - C * (right - left))
        flux.append(f)
        new.append(R)
    for k, lv in enumerate(L):
        covered = torch.zeros_like(lv.valid)
        if k + 1 < len(L):
            covered[L[k + 1].parent[L[k + 1].cell]] = True
        for d in range(D):
            for s in range(2):
                term = flux[k][d, s] @ op["bd"][2 * d + s].T
                edge = torch.nonzero(~covered & covered[lv.nbr[d, s]] & lv.valid)[:, 0]
                if edge.numel():  # the fine level's fluxes through the coarse cell's face
                    base = lv.fine0[lv.nbr[d, s][edge]] + (1 - s) * lv.fine_stride[d]
                    term[edge] = 0.5 * sum(flux[k + 1][d, 1 - s][base + h * lv.fine_stride[1 - d]] @
                                           op["half_bd"][4 * d + 2 * s + h].T for h in range(2))
                new[k] = new[k] + (-1 if s else 1) * (dt / lv.dx[d]) * term
        new[k] = new[k] / op["M"]
    for k in range(len(L) - 1, 0, -1):
        lv = L[k]
        total = torch.zeros_like(new[k - 1])
        for q in range(1 << D):
            b = lv.cell[lv.child[lv.cell] == q]
            total[lv.parent[b]] += new[k][b] @ op["kidw"][q].T
        par = torch.unique(lv.parent[lv.cell])
        new[k - 1][par] = total[par]
    return [u[lv.cell] for lv, u in zip(L, new)]


def _network_seed(par, U, dtdx):
    """The network's change of the predictor, from 32-bit parameters in 64-bit arithmetic."""
    W1, b1, W2, b2, W3, b3, W4, b4, xm, xi, ym, ys = [p.to(F64) for p in par]
    h = (_features(U, dtdx) - xm) * xi
    for W, b in ((W1, b1), (W2, b2), (W3, b3)):
        h = _gelu(h @ W + b)
    y = ((h @ W4 + b4) * ys + ym).reshape(U.shape[0], U.shape[1], -1)
    return y * (U[:, :1, :1] * dtdx[:, None, None])


def _train_exact(c, seed):
    """Full-batch Adam on the standardised pairs."""
    _, U, par, dt = _train_inputs(c, seed)
    op, D, n = _operators(c["D"], c["P"]), c["D"], int(math.sqrt(c["pairs"]))
    cd = torch.full((U.shape[0], D), dt * n, device=DEV, dtype=F64)
    H = _picard(op, U, cd, 8)
    X = _features(U, cd[:, 0])
    T = ((H - U @ op["W"].T) / (U[:, :1, :1] * dt * n)).reshape(U.shape[0], -1)
    xm, xs, ym, ys = X.mean(0), X.std(0, unbiased=False), T.mean(0), T.std(0, unbiased=False)
    xs = torch.stack([xs, 0.1 * xm.abs(), 1e-6 * (xm.abs() + xs).max().expand_as(xs)]).amax(0)
    still = ys < 1e-9 * ys.max()  # modes that the predictor does not change
    ym, ys = torch.where(still, 0.0, ym), torch.where(still, 1.0, ys)
    X, T = (X - xm) / xs, torch.where(still, 0.0, (T - ym) / ys)
    p = [q.to(F64).requires_grad_(True) for q in par]
    opt = torch.optim.Adam(p, lr=1e-3, betas=(0.9, 0.999), eps=1e-8)
    for _ in range(c["epochs"]):
        h = X
        for k in (0, 2, 4):
            h = _gelu(h @ p[k] + p[k + 1])
        loss = ((h @ p[6] + p[7] - T) ** 2).mean()
        opt.zero_grad()
        loss.backward()
        opt.step()
    flat = torch.cat([q.detach().reshape(-1) for q in p] + [xm, 1 / xs, ym, ys])
    return dict(params=flat, loss=float(loss.detach()))


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "transfer":
        fine, coarse, child = _transfer_inputs(c, seed)
        op = _operators(c["D"], c["P"])
        return dict(up=torch.einsum("kmn,ekqn->eqm", op["kidw"], fine),
                    down=(op["kid"][child.long()] @ coarse.transpose(1, 2)).transpose(1, 2))
    if c["kind"] == "train":
        return _train_exact(c, seed)
    if c["layout"] == "regrid" or c["limited"]:
        return None  # boxes of the clustering and the limiter's decisions are choices, not computed numbers
    op, n0 = _operators(c["D"], c["P"]), _dims(c, 0)
    boxes = _boxes(c) if c["layout"] == "boxes" else [[[0] * 3 + [n - 1 for n in n0] + [0] * (3 - c["D"])]]
    ijk = [_cells(b, _dims(c, k)) for k, b in enumerate(boxes)]
    U = [_state(c, k, x, seed) for k, x in enumerate(ijk)]
    L = [_Level(c, k, x) for k, x in enumerate(ijk)]
    dt0 = dt = _time_step(c, U)
    net = _network(c, U, dt0, seed) if c["seeded"] else None
    for _ in range(c["steps"]):
        U = _step(c, op, L, U, dt, net)
        dt = _time_step(c, U)
    if c["kind"] == "patches":
        layout, total = _patch_layout(c, lambda lev: ijk[lev])
        return dict(U=_into_patches(c, layout, total, U), dt0=dt0)
    if c["kind"] == "host":
        return dict(U=torch.cat(U), dt0=dt0)
    return dict(U=torch.cat(U), dt0=dt0, dt=dt)
