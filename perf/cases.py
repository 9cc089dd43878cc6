"""The work that users of the library have it do, as measurable cases.

Every case steps seeded discs through the C-ABI (the ctypes binding mhdgpu.py):
  run       one disc resident on the GPU, a few steps of mhd_run per pass and
            the conserved state back in host memory (precision and pair-state
            forms); downloads of the FP32 forms are kept in single precision on
            the GPU, for the program's own analysis
  step      one disc through mhd_step, the plain FP64 form: one main-loop pass
            of the reference program, U and V back in host memory
  exchange  a host code that owns the state: mhd_upload_state(U), a few steps,
            mhd_download(U) every pass
  batch     many independent discs of uneven sizes through mhd_batch_step

Physics: "free" (no gravity, beta 10), "cool" (cooling on, beta 1), "arms" (the
spiral force, beta 1, without the axisymmetric field and cooling: the disc
holds together over a long run), "shipped" (the reference's stretched grid,
model and knobs, cooling on).

exact() restates the scheme (reconstruction, HLLD / HLL, GLM, sources, boundary
fills, floors, TVD-RK) in 64-bit torch.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEV = "cuda" if torch.cuda.is_available() else "cpu"

_M = None


def binding():
    """mhdgpu.py (the package's folder name is no Python identifier)"""
    global _M
    if _M is None:
        path = os.path.join(ROOT, "171026-1-3dhlld-cyli-gal_gb300", "mhdgpu.py")
        spec = importlib.util.spec_from_file_location("mhdgpu", path)
        _M = importlib.util.module_from_spec(spec)
        sys.modules["mhdgpu"] = _M
        spec.loader.exec_module(_M)
    return _M


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _case(kind, form, physics, nr, nphi, nz, steps, limiter="minmod", solver="hlld", scheme=3, discs=1, branches=0):
    return dict(kind=kind, form=form, physics=physics, nr=nr, nphi=nphi, nz=nz, steps=steps, limiter=limiter,
                solver=solver, scheme=scheme, discs=discs, branches=branches)


def listed():
    return [
        # a parameter study's smallest disc, stepped and looked at one step at a time: launches and latency
        dict(_case("run", "fp32", "free", 16, 16, 16, 1), name="run fp32 16x16x16"),
        # the small reference grid kept on the GPU between looks
        dict(_case("run", "fp32", "free", 64, 64, 32, 20), name="run fp32 64x64x32"),
        # the precision configuration
        dict(_case("run", "fp32", "free", 256, 256, 128, 20), name="run fp32 256x256x128"),
        # the largest disc, the benchmark's configuration: cooling, beta 1
        dict(_case("run", "fp32", "cool", 512, 512, 256, 10), name="run fp32 512x512x256"),
        # ragged extents, MC reconstruction, spiral force
        dict(_case("run", "fp32", "arms", 151, 90, 77, 20, "mc"), name="run fp32 151x90x77 mc arms"),
        # the shipped production model in the precision form: stretched grid, live RK2
        dict(_case("exchange", "fp32", "shipped", 240, 64, 200, 2, scheme=2), name="exchange fp32 shipped rk2"),
        # a spiral disc with its state held as FP32 pairs
        dict(_case("run", "fp32x2", "arms", 256, 256, 128, 10, "mc"), name="run pair 256x256x128 mc arms"),
        # the drop-in for the reference's loop at its reference grid
        dict(_case("step", "fp64", "free", 64, 64, 32, 1), name="step fp64 64x64x32"),
        # the shipped production model as the reference computes it
        dict(_case("step", "fp64", "shipped", 240, 64, 200, 1, scheme=2), name="step fp64 shipped rk2"),
        # a large spiral disc in FP64
        dict(_case("step", "fp64", "arms", 256, 256, 128, 1, "mc"), name="step fp64 256x256x128 mc arms"),
        # a coupled host code that owns the state
        dict(_case("exchange", "fp32", "free", 256, 256, 128, 5), name="exchange fp32 256x256x128"),
        # a survey of uneven discs on parallel branches of one graph
        dict(_case("batch", "fp32", "arms", 0, 0, 0, 10, discs=16, branches=16), name="batch of 16 uneven discs"),
    ]


def _even(v):
    return max(4, 2 * int(round(v / 2.0)))


def draw(rng):
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    kind = rng.choice(["run", "run", "run", "run", "step", "step", "exchange", "batch"])
    limiter = rng.choice(["minmod", "minmod", "mc", "vanleer"])
    solver = rng.choice(["hlld", "hlld", "hlld", "hll"])
    scheme = rng.choice([3, 3, 2])
    if kind == "batch":
        return _case("batch", "fp32", "arms", 0, 0, 0, rng.randint(2, 10), limiter, solver, scheme,
                     discs=rng.randint(2, 16), branches=rng.choice([4, 8, 16]))
    form = "fp64" if kind == "step" else rng.choice(["fp32", "fp32", "fp32x2"])
    physics = rng.choice(["free", "cool", "arms", "arms", "shipped"])
    steps = 1 if kind == "step" else rng.randint(1, 20)
    nr, nphi, nz = int(log(14, 320)), _even(log(12, 320)), int(log(13, 160))
    if kind == "step":
        nr, nphi, nz = min(nr, 220), min(nphi, 220), min(nz, 120)
    if physics == "shipped":   # its own knobs and its live scheme
        nr, nphi, nz, limiter, solver, scheme = max(nr, 60), min(nphi, 96), max(nz, 60), "minmod", "hlld", 2
        if kind != "step":
            kind, steps = "exchange", rng.randint(1, 2)
    elif physics == "cool" and kind != "step":   # a short time from the start: it cools to dt = 0 in the end
        kind, steps = "exchange", min(steps, max(1, nphi // 6))
    return _case(kind, form, physics, nr, nphi, nz, steps, limiter, solver, scheme)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _grid_params(case, dims=None, **over):
    M = binding()
    dims = dims or (case["nr"], case["nphi"], case["nz"])
    knobs = dict(limiter=case["limiter"], solver=case["solver"], scheme=case["scheme"], precision=case["form"])
    if case["physics"] == "shipped":
        grid = M.Grid.shipped(*dims)
        grid.set_initial_gravity()
        return grid, M.default_params(**knobs), 0.0
    name = {"free": "disc1", "cool": "disc5", "arms": "disc2"}[case["physics"]]
    if case["physics"] == "arms":
        over = dict(dict(cooling=0, beta=1.0), **over)
    (nr, nphi, nz), params, ic = M.workload(name, nr=dims[0], nphi=dims[1], nz=dims[2], **dict(knobs, **over))
    return M.Grid.disc(nr, nphi, nz), params, ic["beta"]


def _noise(grid, seed, amp):
    """amp * (uniform in [-1, 1)) for rho and the three velocities"""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    return amp * (2.0 * torch.rand((4,) + grid.cell, dtype=torch.float64, device=DEV, generator=g) - 1.0)


def _vtou(grid, V):
    x = torch.as_tensor(grid.arr("x", grid.ixmax), device=V.device)[:, None, None]
    v2 = V[1] * V[1] + V[2] * V[2] + V[3] * V[3]
    b2 = V[4] * V[4] + V[5] * V[5] + V[6] * V[6]
    return torch.stack([V[0], V[0] * V[1], x * V[0] * V[2], V[0] * V[3], V[4], V[5], V[6],
                        0.5 * (V[0] * v2 + b2) + 1.5 * V[7], V[8]])


def _initial(case, grid, params, beta, seed):
    """U, V and what feeds the absorbing layers and floors (Uinit, Vinit,
    rhofloor; None: from U, V), on DEV in FP64"""
    M = binding()
    if case["physics"] == "shipped":
        U0, V0, Ui, Vi, rf = [torch.as_tensor(a, device=DEV) for a in grid.ic_galactic_disc3(params)]
        w = _noise(grid, seed, 1.0e-3)
        V = V0.clone()
        V[0] *= 1.0 + w[0]
        V[7] *= 1.0 + w[0]
        for m in (1, 2, 3):
            V[m] += w[m]
        return _vtou(grid, V), V, (Ui, Vi, rf)
    w = _noise(grid, seed, 0.01)
    z = torch.as_tensor(grid.arr("z", grid.kzmax), device=DEV)
    V = torch.zeros((9,) + grid.cell, dtype=torch.float64, device=DEV)
    V[0] = (torch.exp(-z * z / 0.02) + 1.0e-3) * (1.0 + w[0])
    V[1] = w[1]
    V[2] = 1.0 + w[2]
    V[3] = w[3]
    V[7] = 0.01 * V[0]
    V[5] = torch.sqrt(2.0 * V[7] / beta)
    return _vtou(grid, V), V, (None, None, None)


def _discs(case):
    """grid, params, beta of every disc of the case"""
    if case["kind"] != "batch":
        return [_grid_params(case)]
    out = []
    for (nr, nphi, nz), p, ic in binding().batch_workload(case["discs"], seed=7):
        out.append(_grid_params(case, (nr, nphi, nz), epssp0=p.epssp0, omegapattern=p.omegapattern, beta=ic["beta"]))
    return out


def _host(a):
    """a tensor's copy in page-locked host memory (where there is a GPU)"""
    if DEV == "cpu":
        return a
    h = torch.empty(a.shape, dtype=a.dtype, pin_memory=True)
    h.copy_(a)
    return h


class _State:
    """what a user's program keeps: the context, its time and its host buffers"""

    def __del__(self):
        for name in ("disc", "batch"):
            if getattr(self, name, None) is not None:
                getattr(self, name).close()


def prepare(case, seed):
    M = binding()
    s = _State()
    s.case, s.M, s.t, s.U, s.dev, s.out = case, M, 0.0, [], [], []
    discs = _discs(case)
    if case["kind"] == "batch":
        s.batch = M.Batch([d[0] for d in discs], [d[1] for d in discs])
        s.batch.set_mode(2, case["branches"])
        s.t = np.zeros(len(discs))
    else:
        s.disc = M.Disc(*discs[0][:2])
    for n, (grid, params, beta) in enumerate(discs):
        U, V, (Ui, Vi, rf) = _initial(case, grid, params, beta, seed * 100 + n)
        U, V = _host(U), _host(V)
        if case["kind"] == "batch":
            s.batch.upload(n, U.numpy(), V.numpy())
        elif Ui is None:
            s.disc.upload(U.numpy(), V.numpy())
        else:
            s.disc.upload(U.numpy(), V.numpy(), Ui.cpu().numpy(), Vi.cpu().numpy(), rf.cpu().numpy())
        if case["kind"] == "exchange":
            s.U0 = U.clone().pin_memory() if DEV == "cuda" else U.clone()
        s.U.append(U)                                     # the page-locked buffers downloads land in
        if case["form"] == "fp64":
            s.V = V
        else:
            s.dev.append(torch.zeros(U.shape, dtype=torch.float64, device=DEV))
            s.out.append(torch.zeros(U.shape, dtype=torch.float32, device=DEV))
    return s


def _single(s, n):
    """the downloaded state in single precision, on the GPU"""
    s.dev[n].copy_(s.U[n])
    s.out[n].copy_(s.dev[n])


def run(s):
    case = s.case
    if case["kind"] == "step":
        for _ in range(case["steps"]):
            rc, s.t, dt, ch, cnt = s.disc.step(s.t)
            s.M.check(rc, "mhd_step")
        s.disc.download_into(s.U[0].numpy(), s.V.numpy())
        return {"U": s.U[0], "V": s.V, "dt": dt, "ch": ch}
    if case["kind"] == "batch":
        s.t, status = s.batch.step(case["steps"], s.t)
        if np.any(status):
            raise RuntimeError("a disc's time step failed")
        for n, U in enumerate(s.U):
            s.M.check(s.M.lib().mhd_batch_download(s.batch.h, n, U.data_ptr(), None), "mhd_batch_download")
            _single(s, n)
        return list(s.out)
    if case["kind"] == "exchange":
        s.disc.upload_state(s.U0.numpy(), None)
        s.disc.run(case["steps"], 0.0)
    else:
        s.t = s.disc.run(case["steps"], s.t)
    s.disc.download_into(s.U[0].numpy(), None)
    _single(s, 0)
    return s.out[0]


def work(case):
    """Per step the state is read and written by every stage at least once: 75
    values per zone in RK3 (two stages with U^n and U^(k), one with U^n; V, U
    and the floor), 46 in RK2; an exchange or a download moves FP64 values.
    About 350 operations per face (reconstruction and Riemann solver) and 150
    per zone in the update."""
    zones = sum((g.ix * g.jy * g.kz) for g, _, _ in _discs(case))
    esz = {"fp64": 8, "fp32": 4, "fp32x2": 4}[case["form"]]
    per = (75 if case["scheme"] == 3 else 46) + (0 if case["form"] != "fp32x2" else 39 if case["scheme"] == 3 else 24)
    moved = 9 * 8 * (2 if case["kind"] in ("exchange", "step") else 1)
    return {"bytes": float(zones) * (case["steps"] * per * esz + moved),
            "flops": float(zones) * case["steps"] * case["scheme"] * 1200.0}


# ---------------------------------------------------------------------------
# the scheme in 64-bit torch
# ---------------------------------------------------------------------------

GM = 5.0 / 3.0


def _at(a, axis, lo, n):
    """cells lo .. lo+n-1 of a [9, i, j, k] array along a grid axis"""
    return a.narrow(axis + 1, lo, n)


def _fast(v, bn):
    b2 = v[4] ** 2 + v[5] ** 2 + v[6] ** 2
    g = GM * v[7]
    disc = ((b2 + g) ** 2 - 4.0 * g * bn * bn).clamp_min(0.0)
    return torch.sqrt(((b2 + g) + torch.sqrt(disc)) / (2.0 * v[0]))


class _Exact:
    def __init__(self, grid, params, U, V, extra):
        self.p, self.dev = params, U.device
        n3 = grid.cell
        self.n = n3
        T = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)  # noqa: E731
        self.x, self.xm = T(grid.arr("x", n3[0])), T(grid.arr("xm", n3[0]))
        self.ox, self.odx = T(grid.arr("oneox", n3[0])), T(grid.arr("oneodx", n3[0]))
        self.y, self.z, self.odz = T(grid.arr("y", n3[1])), T(grid.arr("z", n3[2])), T(grid.arr("oneodz", n3[2]))
        self.ody = float(grid.g.oneody)
        nf = (n3[0] - 1, n3[2] - 1)
        self.g = [T(grid.arr("g%d" % (s + 1), nf[0] * nf[1]).reshape(nf))[1:, 1:].unsqueeze(1) for s in range(6)]
        self.minl = T(grid.arr("minlength", n3[0] * n3[2]).reshape(n3[0], n3[2]))
        self.minmin = float(grid.g.minminlength)
        self.irin = grid.irin
        self.xabs, self.zabs = T(grid.arr("x_absorb_factor", 11)), T(grid.arr("z_absorb_factor", 11))
        self.cabs = T(grid.arr("c_absorb_factor", (grid.irin + 1) * n3[2]).reshape(grid.irin + 1, n3[2]))
        self.grax = [torch.zeros(1, 1, 1, dtype=torch.float64, device=self.dev).expand(n3[0], 1, n3[2])] * 3
        if grid.g.Grxaxi:
            self.grax = [T(grid.arr(a, n3[0] * n3[2]).reshape(n3[0], 1, n3[2])) for a in ("Grxaxi", "Gryaxi", "Grzaxi")]
        self.U, self.V = U.clone(), V.clone()
        self.Ui = U.clone() if extra[0] is None else extra[0]
        self.Vi = V.clone() if extra[1] is None else extra[1]
        self.rf = params.rhocr * U[0] if extra[2] is None else extra[2]
        self._ghosts()

    def _ghosts(self):
        """every cell's source cell and signs: the y, x, z fills in turn, later ones winning"""
        ni, nj, nk = self.n
        i, j, k = torch.meshgrid(*[torch.arange(m, device=self.dev) for m in self.n], indexing="ij")
        rk2 = self.p.scheme == 2
        sk = torch.where(k == 0, 2 if rk2 else nk - 2, torch.where(k == nk - 1, nk - 2 if rk2 else 1, k))
        half = (nj - 2) // 2
        axis = i == 0
        sj = torch.where(axis, torch.where(j < half + 1, j + half, j - half),
                         torch.where(j == 0, nj - 2, torch.where(j == nj - 1, 1, j)))
        si = torch.where(axis, 1, torch.where(i == ni - 1, ni - 2, i))
        self.src = ((si * nj + sj) * nk + sk).reshape(-1)
        self.axis_sign = torch.where(axis, -1.0, 1.0).to(torch.float64)
        self.vz_sign = torch.where((k == 0) & rk2, -1.0, 1.0).to(torch.float64)

    # -- time step ----------------------------------------------------------
    def cooling(self, v):
        te0 = (0.619047619 * 1.673e-24) * (1.0 / 1.3806504e-16) * 6.558e+6 * 6.558e+6
        T = v[7] / v[0]
        rate = torch.trunc(0.108e-37 * torch.pow(te0 * T.clamp(0.031, 0.054), 10.26))
        return torch.where((T > 0.031) & (T < 0.054), rate, torch.zeros_like(T))

    def timestep(self):
        v = self.V[:, 1:self.n[0] - 11, 1:-1, 1:-1]
        v2 = v[1] ** 2 + v[2] ** 2 + v[3] ** 2
        b2 = v[4] ** 2 + v[5] ** 2 + v[6] ** 2
        rate = torch.sqrt(v2 + (GM * v[7] + b2) / v[0]) / self.minl[1:self.n[0] - 11, None, 1:-1]
        if self.p.cooling:
            rate = torch.maximum(rate, 2.0 * (v[0] * v[0] * self.cooling(v)) / (1.5 * v[7]))
        top = float(rate.max())
        return self.p.cfl / top, self.minmin * top

    # -- fluxes -------------------------------------------------------------
    def slots(self, V, d, dt):
        """left (at c+1/2) and right (at c-1/2) states of the interior cells along d"""
        n = self.n[d] - 2
        for a in range(3):
            if a != d:
                V = _at(V, a, 1, self.n[a] - 2)
        vm, vc, vp = _at(V, d, 0, n), _at(V, d, 1, n), _at(V, d, 2, n)
        a, b = vc - vm, vp - vc
        same = a * b > 0.0
        lim = self.p.limiter
        if lim == 0:
            grad = torch.where(same, torch.where(a > 0, torch.minimum(a, b), torch.maximum(a, b)), 0.0)
            fast = _fast(vc, vc[4 + d])
            lmax, lmin = (vc[1 + d] + fast).clamp_min(0.0), (vc[1 + d] - fast).clamp_max(0.0)
            if d == 0:
                hi, lo = self.odx[1:-1, None, None], self.odx[:-2, None, None]
            elif d == 1:
                hi = lo = self.ox[1:-1, None, None] * self.ody
            else:
                hi, lo = self.odz[1:-1], self.odz[:-2]
            return vc + 0.5 * (1.0 - lmax * dt * hi) * grad, vc - 0.5 * (1.0 + lmin * dt * lo) * grad
        if lim == 1:
            c = 0.25 * (vp - vm)
            grad = torch.where(a > 0, torch.minimum(a, torch.minimum(b, c)), torch.maximum(a, torch.maximum(b, c)))
            grad = torch.where(same, grad, 0.0)
        elif lim == 2:
            grad = torch.where(same, a * b / torch.where(same, a + b, 1.0), 0.0)
        else:
            s = torch.sign(a)
            big = torch.maximum(torch.minimum(a.abs(), 2.0 * b.abs()), torch.minimum(2.0 * a.abs(), b.abs()))
            grad = torch.where(same, 0.5 * s * big, 0.0)
        return vc + grad, vc - grad

    def faces(self, V, d, dt):
        """left and right states of faces 0 .. N along d, with the limiters' own end fills"""
        n, lim = self.n[d] - 2, self.p.limiter
        Wl, Wr = self.slots(V, d, dt)
        first, last = (lambda w: _at(w, d, 0, 1)), (lambda w: _at(w, d, n - 1, 1))

        def ghost(c):
            W = self.Vi
            for a in range(3):
                W = _at(W, a, c, 1) if a == d else _at(W, a, 1, self.n[a] - 2)
            return W

        if lim == 2 and d != 1:
            L0, R0, LN, RN = first(Wr), first(Wr), last(Wl), last(Wl)
        elif (lim == 2 and d == 1) or (lim == 1 and d == 2):
            L0, R0, LN, RN = ghost(0), first(Wr), last(Wl), ghost(n + 1)
        elif lim == 0 and d == 2:
            L0 = _at(Wr, d, 1, 1).clone()
            L0[3] = -L0[3]
            R0, LN, RN = first(Wr), last(Wl), last(Wl)
        else:
            L0, R0, LN, RN = last(Wl), first(Wr), last(Wl), first(Wr)
        return (torch.cat([L0, _at(Wl, d, 0, n - 1), LN], d + 1), torch.cat([R0, _at(Wr, d, 1, n - 1), RN], d + 1))

    def physical(self, w, pt, en, d, r, vb=None):
        """flux of a state along d (U2 carries r)"""
        vn, bn = w[1 + d], w[4 + d]
        vb = w[1] * w[4] + w[2] * w[5] + w[3] * w[6]
        F = [w[0] * vn]
        for m in range(3):
            f = w[0] * w[1 + m] * vn - w[4 + m] * bn
            f = f + pt if m == d else f
            F.append(r * f if m == 1 else f)
        for m in range(3):
            F.append(torch.zeros_like(vn) if m == d else w[4 + m] * vn - w[1 + m] * bn)
        F.append((en + pt) * vn - vb * bn)
        return F

    def riemann(self, L, R, d, r):
        n, bn = 1 + d, 4 + d
        side = []
        for w in (L, R):
            v2 = w[1] ** 2 + w[2] ** 2 + w[3] ** 2
            b2 = w[4] ** 2 + w[5] ** 2 + w[6] ** 2
            side.append((w[7] + 0.5 * b2, 0.5 * (w[0] * v2 + b2) + 1.5 * w[7]))
        (ptl, el), (ptr, er) = side
        vf = torch.maximum(_fast(L, L[bn]), _fast(R, R[bn]))
        sl, sr = torch.minimum(L[n], R[n]) - vf, torch.maximum(L[n], R[n]) + vf
        if self.p.solver == 1:
            Fl, Fr = self.physical(L, ptl, el, d, r), self.physical(R, ptr, er, d, r)
            Ul = [L[0], L[0] * L[1], r * L[0] * L[2], L[0] * L[3], L[4], L[5], L[6], el]
            Ur = [R[0], R[0] * R[1], r * R[0] * R[2], R[0] * R[3], R[4], R[5], R[6], er]
            return [torch.where(sl >= 0, Fl[m], torch.where(
                sr >= 0, (sr * Fl[m] - sl * Fr[m] + sr * sl * (Ur[m] - Ul[m])) / (sr - sl), Fr[m])) for m in range(8)]
        dl, dr = (sl - L[n]) * L[0], (sr - R[n]) * R[0]
        sm = (dr * R[n] - dl * L[n] - ptr + ptl) / (dr - dl)
        pt = (dr * ptl - dl * ptr + dr * dl * (R[n] - L[n])) / (dr - dl)
        b = (sr * R[bn] - sl * L[bn]) / (sr - sl)
        tv = [1 + (d + 1) % 3, 1 + (d + 2) % 3]
        star = []
        for w, s, q, en, ptw in ((L, sl, dl, el, ptl), (R, sr, dr, er, ptr)):
            rho = q / (s - sm)
            X = q * (s - sm) - b * b
            ok = X.abs() > 1.0e-8 * b * b
            c = torch.where(ok, b * (sm - w[n]) / torch.where(ok, X, 1.0), 0.0)
            f = torch.where(ok, (q * (s - w[n]) - b * b) / torch.where(ok, X, 1.0), 1.0)
            vt = [w[t] - w[t + 3] * c for t in tv]
            bt = [w[t + 3] * f for t in tv]
            vb0 = w[1] * w[4] + w[2] * w[5] + w[3] * w[6]
            vb1 = sm * b + vt[0] * bt[0] + vt[1] * bt[1]
            e = ((s - w[n]) * en - ptw * w[n] + pt * sm + b * (vb0 - vb1)) / (s - sm)
            star.append((rho, vt, bt, e, vb1, torch.sqrt(rho)))
        (rl, vl, bl, e1, vb1, ql), (rr, vr, br, e2, vb2, qr) = star
        left = sm >= 0
        alone = torch.where(left, sm - b.abs() / ql >= 0, sm + b.abs() / qr <= 0)
        sg = torch.sign(b)
        o = 1.0 / (ql + qr)
        vi = [(ql * vl[m] + qr * vr[m] + (br[m] - bl[m]) * sg) * o for m in (0, 1)]
        bi = [(ql * br[m] + qr * bl[m] + ql * qr * (vr[m] - vl[m]) * sg) * o for m in (0, 1)]
        vbi = sm * b + vi[0] * bi[0] + vi[1] * bi[1]
        en = torch.where(left, e1, e2)
        en = torch.where(alone, en, torch.where(left, e1 - ql * (vb1 - vbi) * sg, e2 + qr * (vb2 - vbi) * sg))
        w = [None] * 8
        w[0], w[n], w[bn] = torch.where(left, rl, rr), sm, b
        for m in (0, 1):
            w[tv[m]] = torch.where(alone, torch.where(left, vl[m], vr[m]), vi[m])
            w[tv[m] + 3] = torch.where(alone, torch.where(left, bl[m], br[m]), bi[m])
        up, dn = sl >= 0, sr <= 0
        w[7] = pt
        w = [torch.where(up, L[m], torch.where(dn, R[m], w[m])) for m in range(8)]
        pt = torch.where(up, ptl, torch.where(dn, ptr, pt))
        en = torch.where(up, el, torch.where(dn, er, en))
        return self.physical(w, pt, en, d, r)

    def divergence(self, V, dt, ch):
        div = 0.0
        for d in range(3):
            L, R = self.faces(V, d, dt)
            r = (self.xm[:self.n[0] - 1] if d == 0 else self.x[1:-1])[:, None, None]
            F = self.riemann(L, R, d, r)
            F[4 + d] = F[4 + d] + 0.5 * (L[8] + R[8] + ch * (L[4 + d] - R[4 + d]))
            F.append(0.5 * ch * (ch * (L[4 + d] + R[4 + d]) + (L[8] - R[8])))
            F = torch.stack(F)
            n = self.n[d] - 2
            div = div + self.g[2 * d + 1] * _at(F, d, 1, n) - self.g[2 * d] * _at(F, d, 0, n)
            del L, R, F
        return div

    # -- sources ------------------------------------------------------------
    def gravity(self, t):
        if not self.p.gravity:
            return 0.0, 0.0, 0.0
        p = self.p
        sw = (t - p.tausp) / abs(t - p.tausp)
        eps = 0.5 * p.epssp0 * (t / p.tausp * (1.0 - sw) + (1.0 + sw))
        x, z = self.x[:, None, None], self.z[None, None, :]
        cot = 1.0 / math.tan(p.pitch)
        ph = p.armnum * (self.y[None, :, None] - (p.omegapattern - p.omegasp) * t + cot * torch.log(x / p.scalephase))
        s, c = torch.sin(ph), torch.cos(ph)
        q = torch.sqrt(z * z + 0.026 * 0.026)
        A = 1.0 / torch.sqrt(x * x + (0.65 + q) ** 2)
        u = (x / p.scaler) ** 2
        w = (1.0 / (1.0 + u)) ** 1.5
        C1, C2, D = x / p.scaler / p.scaler * w, u * w, (2.0 - u) / (1.0 + u)
        S, Q, Rz = p.scalez / torch.sqrt(z * z + p.scalez ** 2), 1.0 + 0.65 / q, 1.0 / (z * z + p.scalez ** 2)
        m1 = 10.0 * eps * (torch.arange(self.n[0], device=self.dev) >= self.irin)[:, None, None]
        gx = self.grax[0] - m1 * A * S * C1 * ((x * A * A - D) * c + p.armnum * cot * s)
        gy = self.grax[1] + m1 * A * S * C1 * p.armnum * s
        gz = self.grax[2] - m1 * A * z * S * C2 * (Q * A * A + Rz) * c
        return [g[1:-1, :, 1:-1] if g.shape[1] == 1 else g[1:-1, 1:-1, 1:-1] for g in (gx, gy, gz)]

    def source(self, V, g):
        v = V[:, 1:-1, 1:-1, 1:-1]
        x, ox, om = self.x[1:-1, None, None], self.ox[1:-1, None, None], self.p.omegasp
        S = torch.zeros_like(v)
        b2 = v[4] ** 2 + v[5] ** 2 + v[6] ** 2
        S[1] = ((v[0] * v[2] ** 2 - v[5] ** 2 + v[7] + 0.5 * b2) * ox + v[0] * g[0] + v[0] * om * om * x
                + 2.0 * v[0] * v[2] * om)
        S[2] = x * (v[0] * g[1] - 2.0 * v[0] * v[1] * om)
        S[3] = v[0] * g[2]
        S[5] = (v[5] * v[1] - v[2] * v[4]) * ox
        S[7] = v[0] * (v[1] * g[0] + v[2] * g[1] + v[3] * g[2]) + v[0] * x * v[1] * om * om
        if self.p.cooling:
            S[7] -= v[0] * v[0] * self.cooling(v)
        return S

    # -- one step -----------------------------------------------------------
    def tail(self, u, last):
        """fills, absorbing layers, primitives and floors of the raw updated state"""
        ni, nj, nk = self.n
        full = torch.zeros((9,) + self.n, dtype=torch.float64, device=self.dev)
        full[:, 1:-1, 1:-1, 1:-1] = u
        u = full.reshape(9, -1)[:, self.src].reshape(full.shape)
        for m in (1, 2, 4, 5):
            u[m] *= self.axis_sign
        u[3] *= self.vz_sign
        rk2 = self.p.scheme == 2
        if rk2:
            u[3, :, :, 1] = 0.0
        if last:
            du = lambda sl: u[sl] - self.Ui[sl]  # noqa: E731
            sx = (slice(None), slice(ni - 11, ni))
            u[sx] -= self.xabs[:, None, None] * du(sx)
            sc = (slice(None), slice(0, self.irin + 1))
            u[sc] -= self.cabs[:, None, :] * du(sc)
            if rk2:
                sz = (slice(None), slice(None), slice(None), slice(nk - 11, nk))
                u[sz] -= self.zabs * du(sz)
        x, ox, p = self.x[:, None, None], self.ox[:, None, None], self.p
        w = u.clone()
        b2 = u[4] ** 2 + u[5] ** 2 + u[6] ** 2
        w[1] = u[1] / u[0]
        w[2] = u[2] / u[0] * ox
        w[3] = u[3] / u[0]
        w[7] = 2.0 / 3.0 * (u[7] - 0.5 * ((u[1] ** 2 + (u[2] * ox) ** 2 + u[3] ** 2) / u[0] + b2))

        def reset(bad, rho, pr):
            w[0], w[7] = torch.where(bad, rho, w[0]), torch.where(bad, pr, w[7])
            for m in (1, 3):
                w[m] = torch.where(bad, 0.0, w[m])
                u[m] = torch.where(bad, 0.0, u[m])
            u[0] = torch.where(bad, w[0], u[0])
            u[2] = torch.where(bad, x * w[0] * w[2], u[2])
            u[7] = torch.where(bad, 0.5 * (w[0] * w[2] ** 2 + b2) + 1.5 * w[7], u[7])

        reset(w[0] < self.rf, self.rf, w[7])
        bad = w[7] < w[0] * p.prcr
        u0, u2 = u[0].clone(), u[2].clone()   # the pressure floor leaves these as they are
        reset(bad, w[0], w[0] * p.prcr)
        u[0], u[2] = u0, u2
        ob = 0.5 * b2 / w[7]
        reset(ob > 1.0 / p.betacr, p.betacr * ob * w[0], p.betacr * ob * w[7])
        return u, w

    def step(self, t):
        p = self.p
        dt, ch = self.timestep()
        psi = math.exp(-dt * ch / 0.18 * (0.5 if p.scheme == 2 else 1.0 / 3.0))
        g = self.gravity(t)
        inner = lambda a: a[:, 1:-1, 1:-1, 1:-1].clone()  # noqa: E731
        un = inner(self.U)
        U1, V = self.U, self.V
        stages = ((0, False), (3, True)) if p.scheme == 2 else ((0, False), (1, False), (2, True))
        for kind, last in stages:
            W = V.clone()
            W[8] *= psi
            inc = dt * (self.source(V, g) - self.divergence(W, dt, ch))
            del W
            a, b = un.clone(), inner(U1)
            a[8] *= psi
            b[8] *= psi
            raw = (a + inc if kind == 0 else 0.25 * (3.0 * a + b + inc) if kind == 1 else
                   (a + 2.0 * (b + inc)) / 3.0 if kind == 2 else 0.5 * (a + b + inc))
            U1, V = self.tail(raw, last)
        self.U, self.V = U1, V
        return t + dt, dt, ch


def exact(case, seed):
    discs = _discs(case)
    zones = sum(g.ix * g.jy * g.kz for g, _, _ in discs)
    if zones * case["steps"] * case["scheme"] > 700.0e6:   # over about 20 s
        return None
    out = []
    for n, (grid, params, beta) in enumerate(discs):
        e = _Exact(grid, params, *_initial(case, grid, params, beta, seed * 100 + n))
        t = 0.0
        for _ in range(case["steps"]):
            t, dt, ch = e.step(t)
        if case["kind"] == "step":
            return {"U": e.U.cpu(), "V": e.V.cpu(), "dt": dt, "ch": ch}
        out.append(e.U.cpu())
    return out if case["kind"] == "batch" else out[0]
