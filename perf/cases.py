"""The work that programs on this package have it do, as timed cases.

Every case names a ``kind`` (one public entry point or a short sequence of
them), its sizes and its data type.  ``listed`` holds one or two cases of
each kind; ``draw`` gives more of the same ranges.  Sizes are interior
cells; fields carry the one-cell ghost ring where the entry point wants it.

kind          what a program does with it
arakawa       right-hand side of an energy/enstrophy-conserving QG model:
              J(psi, q) and biharmonic diffusion of q
advect        flux-form tracer advection with a high-order upwind scheme,
              with or without a coastline
momentum      shallow-water momentum tendency: Coriolis and vector-invariant
              advection on a masked basin
qg_step       one RK3 step of the 1.5-layer QG model (advection + Helmholtz
              inversion three times)
helmholtz     Dirichlet / Neumann / periodic inversions, batched over layers
              or members, with a lambda per layer
vcycle, pcg   masked variable-coefficient Helmholtz problems: one multigrid
              V-cycle, and a whole multigrid-preconditioned solve
ensemble      one step of an ensemble of multi-layer QG members of uneven size
train         one training step of the learned preconditioner's network
"""

from __future__ import annotations

import math
from fractions import Fraction

import torch

import finitevolx_b200 as fvx
from finitevolx_b200 import learned

LX = 5.12e6       # domain width in x, m
BETA = 1.7e-11    # planetary vorticity gradient, 1/(m s)
F0 = 9.375e-5     # Coriolis parameter, 1/s
LD = 4.0e4        # deformation radius, m
H_LAYERS = (400.0, 1100.0, 2600.0)
G_PRIME = (9.81, 0.025, 0.0125)
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # the smallest calls: a teaching-size QG right-hand side, where launches and host time count
        {"name": "arakawa_f64_130x98", "kind": "arakawa", "dtype": "f64", "ny": 130, "nx": 98},
        # an ordinary large tracer field without coasts, single precision
        {"name": "advect_weno5_f32_2048", "kind": "advect", "dtype": "f32", "ny": 2048, "nx": 2048,
         "method": "weno5", "masked": False},
        # a regional basin with a coastline, odd sizes, the double-precision path
        {"name": "advect_weno5_f64_masked_1531x1019", "kind": "advect", "dtype": "f64", "ny": 1531, "nx": 1019,
         "method": "weno5", "masked": True},
        # shallow-water momentum on a masked basin
        {"name": "momentum_al_f64_1020x764", "kind": "momentum", "dtype": "f64", "ny": 1020, "nx": 764,
         "scheme": "al"},
        # the plain QG configuration: 256^2, double precision, its step captured in a CUDA graph
        {"name": "qg_step_f64_256", "kind": "qg_step", "dtype": "f64", "n": 256, "captured": True},
        # the large single-precision QG step
        {"name": "qg_step_f32_2048", "kind": "qg_step", "dtype": "f32", "n": 2048, "captured": False},
        # PV inversion of a three-layer model, a lambda per layer, double precision
        {"name": "helmholtz_dst_f64_3x1024x768", "kind": "helmholtz", "dtype": "f64", "bc": "dst", "batch": 3,
         "ny": 1024, "nx": 768, "layers": True},
        # many right-hand sides of one size, single precision
        {"name": "helmholtz_dst_f32_16x1024x1024", "kind": "helmholtz", "dtype": "f32", "bc": "dst", "batch": 16,
         "ny": 1024, "nx": 1024, "layers": False},
        # pressure on a quarter-degree-sized grid, Neumann walls
        {"name": "helmholtz_dct_f32_720x1440", "kind": "helmholtz", "dtype": "f32", "bc": "dct", "batch": 1,
         "ny": 720, "nx": 1440, "layers": False},
        # masked Helmholtz solve to 1e-8
        {"name": "pcg_mg_f32_512", "kind": "pcg", "dtype": "f32", "n": 512, "ld": LD},
        # uneven members, 1 to 3 layers
        {"name": "ensemble_f32_8", "kind": "ensemble",
         "members": "1024x1 512x3 512x2 256x3 256x1 128x3 128x2 128x1"},
        # one optimiser step of the preconditioner's network on a batch of level-sized problems
        {"name": "train_32x128", "kind": "train", "batch": 32, "n": 128},
    ]


def _log(rng, lo, hi, step=1):
    """A size spread over the logarithm of [lo, hi], a multiple of step."""
    return max(lo, min(hi, step * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)))


def draw(rng):
    kind = rng.choice(("arakawa", "advect", "advect", "momentum", "qg_step", "qg_step", "helmholtz", "helmholtz",
                       "helmholtz", "vcycle", "pcg", "ensemble", "train"))
    dtype = rng.choice(("f32", "f64"))
    if kind == "arakawa":
        return {"kind": kind, "dtype": dtype, "ny": _log(rng, 96, 4096), "nx": _log(rng, 96, 4096)}
    if kind == "advect":
        masked = rng.random() < 0.5
        method = rng.choice(("weno3", "weno5", "wenoz5", "van_leer") if masked
                            else ("weno5", "wenoz5", "weno7", "van_leer"))
        return {"kind": kind, "dtype": dtype, "ny": _log(rng, 96, 2600), "nx": _log(rng, 96, 2600),
                "method": method, "masked": masked}
    if kind == "momentum":
        return {"kind": kind, "dtype": dtype, "ny": _log(rng, 96, 2600), "nx": _log(rng, 96, 2600),
                "scheme": rng.choice(("energy", "enstrophy", "al"))}
    if kind == "qg_step":
        n = _log(rng, 128, 2048, 8) if dtype == "f32" else _log(rng, 96, 512)
        return {"kind": kind, "dtype": dtype, "n": n, "captured": n <= 512}
    if kind == "helmholtz":
        step = 8 if dtype == "f32" and rng.random() < 0.7 else 1
        layers = rng.random() < 0.4
        top = 1200 if dtype == "f32" and step == 8 else 700
        return {"kind": kind, "dtype": dtype, "bc": rng.choice(("dst", "dst", "dct", "fft")),
                "batch": rng.randint(2, 3) if layers else _log(rng, 1, 8), "ny": _log(rng, 64, top, step),
                "nx": _log(rng, 64, top, step), "layers": layers}
    if kind in ("vcycle", "pcg"):
        return {"kind": kind, "dtype": dtype, "n": rng.choice((128, 192, 256, 320, 384, 512)),
                "ld": round(LX / _log(rng, 32, 256), 1)}
    if kind == "ensemble":
        m = [(rng.choice((128, 256, 512)), rng.randint(1, 3)) for _ in range(rng.randint(3, 9))]
        return {"kind": kind, "members": " ".join("%dx%d" % x for x in m)}
    return {"kind": "train", "batch": _log(rng, 4, 32), "n": rng.choice((64, 96, 128))}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _spectrum(gen, ny, nx, amp, count=1):
    """count Gaussian random fields [count, ny, nx] (FP64, unit std) with Fourier amplitude amp(|k|), k in cycles per cell."""
    w = torch.randn((count, ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(nx, device="cuda", dtype=torch.float64)[None, :]
    k = torch.sqrt(kx ** 2 + ky ** 2)
    a = amp(k)
    a[0, 0] = 0.0
    f = torch.fft.irfft2(torch.fft.rfft2(w) * a, s=(ny, nx))
    return f / f.std(dim=(-2, -1), keepdim=True)


def _kminus3(gen, ny, nx, count=1):
    return _spectrum(gen, ny, nx, lambda k: torch.where(k > 0, k, torch.ones_like(k)) ** -1.5, count)


def _smooth(gen, ny, nx, cells):
    return _spectrum(gen, ny, nx, lambda k: torch.exp(-2.0 * (math.pi * cells * k) ** 2))[0]


def _ghosts(f):
    """Interior [..., ny, nx] -> periodic field [..., ny + 2, nx + 2]."""
    f = torch.cat((f[..., -1:, :], f, f[..., :1, :]), dim=-2)
    return torch.cat((f[..., :, -1:], f, f[..., :, :1]), dim=-1).contiguous()


def _velocities(gen, ny, nx, dx, dy):
    """Divergence-free C-grid (u, v), max |u| = 1 m/s, from a random streamfunction at the corners."""
    psi = _ghosts(_spectrum(gen, ny, nx, lambda k: torch.where(k > 0, k, torch.ones_like(k)) ** -2.5)[0])
    u = torch.zeros_like(psi)
    v = torch.zeros_like(psi)
    u[1:-1, 1:-1] = -(psi[1:-1, 1:-1] - psi[:-2, 1:-1]) / dy
    v[1:-1, 1:-1] = (psi[1:-1, 1:-1] - psi[1:-1, :-2]) / dx
    s = torch.maximum(u.abs().max(), v.abs().max())
    return _ghosts(u[1:-1, 1:-1] / s), _ghosts(v[1:-1, 1:-1] / s)


def _basin(gen, ny, nx):
    """Smooth random coastline, 30 % land, closed at the edges; bool [ny, nx]."""
    g = _smooth(gen, ny, nx, max(3.0, min(ny, nx) / 40.0))
    m = g > torch.sort(g.reshape(-1)).values[int(0.3 * g.numel())]
    m[0, :] = m[-1, :] = False
    m[:, 0] = m[:, -1] = False
    return m


def _grid(ny, nx):
    return fvx.ArakawaCGrid2D.from_interior(nx, ny, LX, LX * ny / nx)


def _members(case):
    return [tuple(int(p) for p in m.split("x")) for m in case["members"].split()]


def _lambdas(case):
    if not case["layers"]:
        return 0.0 if case["bc"] == "dct" else 1.0 / LD ** 2
    n = case["batch"]
    rr, _, _ = fvx.decompose_vertical_modes(fvx.build_coupling_matrix(H_LAYERS[:n], G_PRIME[:n]), F0)
    return [1.0 / float(r) ** 2 for r in rr]


def _inputs(case, seed):
    """The case's input arrays in FP64 on the GPU, before rounding to its data type."""
    g, kind = _gen(seed), case["kind"]
    if kind == "arakawa":
        ny, nx = case["ny"], case["nx"]
        return {"psi": _ghosts(_spectrum(g, ny, nx, lambda k: torch.where(k > 0, k, torch.ones_like(k)) ** -2.5)[0]) * 1e4,
                "q": _ghosts(_kminus3(g, ny, nx)[0]) * 1e-5}
    if kind in ("advect", "momentum"):
        ny, nx = case["ny"], case["nx"]
        gr = _grid(ny, nx)
        u, v = _velocities(g, ny, nx, gr.dx, gr.dy)
        d = {"h": _ghosts(_kminus3(g, ny, nx)[0]), "u": u, "v": v}
        if kind == "momentum":
            d["f"] = F0 + BETA * (torch.arange(ny + 2, device="cuda", dtype=torch.float64) * gr.dy)[:, None] + 0.0 * u
        if kind == "momentum" or case["masked"]:
            d["mask"] = _basin(g, ny + 2, nx + 2)
        return d
    if kind == "qg_step":
        return {"q": _ghosts(_kminus3(g, case["n"], case["n"])[0]) * 1e-5}
    if kind == "helmholtz":
        f = _kminus3(g, case["ny"], case["nx"], case["batch"]) * 1e-5
        if case["bc"] != "dst":
            f = f - f.mean(dim=(-2, -1), keepdim=True)
        return {"rhs": f if case["batch"] > 1 else f[0]}
    if kind in ("vcycle", "pcg"):
        n = case["n"]
        m = _basin(g, n, n)
        c = torch.exp(0.5 * _smooth(g, n, n, max(3.0, n / 40.0)))
        b = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64) * m
        return {"mask": m.double(), "coeff": c, "b": b}
    if kind == "ensemble":
        return {"q": [_ghosts(_kminus3(g, n, n, nl)) * 1e-6 for n, nl in _members(case)]}
    n, b = case["n"], case["batch"]
    x = torch.randn((b, 3, n, n), generator=g, device="cuda", dtype=torch.float64)
    m = torch.stack([_basin(g, n, n) for _ in range(4)]).double()[torch.arange(b, device="cuda") % 4]
    x[:, 0] *= m
    x[:, 1] = m
    x[:, 2] = 0.5 * x[:, 2] * m
    return {"x": x, "target": 0.3 * torch.randn((b, 1, n, n), generator=g, device="cuda", dtype=torch.float64)}


def prepare(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    t = DTYPES.get(case.get("dtype", "f32"))
    s = {"case": case}
    if kind == "arakawa":
        gr = _grid(case["ny"], case["nx"])
        s.update(grid=gr, psi=d["psi"].to(t), q=d["q"].to(t), bih=fvx.BiharmonicDiffusion2D(gr), nu=1e-3 * gr.dx ** 4 / 86400)
    elif kind == "advect":
        gr = _grid(case["ny"], case["nx"])
        mask = fvx.Mask2D.from_mask(d["mask"]) if case["masked"] else None
        s.update(adv=fvx.Advection2D(gr, mask), h=d["h"].to(t), u=d["u"].to(t), v=d["v"].to(t))
    elif kind == "momentum":
        gr = _grid(case["ny"], case["nx"])
        mask = fvx.Mask2D.from_mask(d["mask"])
        s.update(cor=fvx.Coriolis2D(gr, mask), mom=fvx.MomentumAdvection2D(gr, mask), u=d["u"].to(t), v=d["v"].to(t),
                 f=d["f"].to(t))
    elif kind == "qg_step":
        gr = _grid(case["n"], case["n"])
        model = fvx.QGModel(gr, BETA, 1.0 / LD ** 2, method="weno5", dtype=t)
        s.update(model=model, q=d["q"].to(t), dt=0.5 * gr.dx)
        if case["captured"]:
            s["out"] = torch.empty_like(s["q"])
            model.step(s["q"], s["dt"], out=s["out"])
            torch.cuda.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                model.step(s["q"], s["dt"], out=s["out"])
    elif kind == "helmholtz":
        s.update(rhs=d["rhs"].to(t), lam=_lambdas(case))
    elif kind in ("vcycle", "pcg"):
        dx = LX / case["n"]
        s["mg"] = fvx.build_multigrid_solver(d["mask"], dx, dx, lambda_=1.0 / case["ld"] ** 2, coeff=d["coeff"], dtype=t)
        s["b"] = d["b"].to(t)
        if kind == "pcg":
            s["pcg"] = fvx.MaskedHelmholtzPCG(s["mg"])
        else:
            s["precond"] = fvx.make_multigrid_preconditioner(s["mg"])
    elif kind == "ensemble":
        s["ens"] = fvx.QGEnsemble(_members(case), Lx=LX, beta=BETA, f0=F0, H=H_LAYERS, gprime=G_PRIME, umax=10.0)
        for m, q in enumerate(d["q"]):
            for layer in range(q.shape[0]):
                s["ens"].set_layer(m, layer, q[layer].float())
    else:
        s.update(net=learned.UNet(case["n"], case["n"], batch_max=case["batch"], seed=0), x=d["x"].float(),
                 target=d["target"].float(), loss=torch.zeros(1, dtype=torch.float64, device="cuda"))
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "arakawa":
        g = state["grid"]
        return fvx.arakawa_jacobian(state["psi"], state["q"], g.dx, g.dy), state["bih"](state["q"], state["nu"])
    if kind == "advect":
        return state["adv"](state["h"], state["u"], state["v"], method=case["method"])
    if kind == "momentum":
        return (state["cor"](state["u"], state["v"], state["f"]),
                state["mom"](state["u"], state["v"], scheme=case["scheme"]))
    if kind == "qg_step":
        if case["captured"]:
            state["graph"].replay()
            return state["out"]
        return state["model"].step(state["q"], state["dt"])
    if kind == "helmholtz":
        gr = _grid(case["ny"], case["nx"])
        if case["layers"]:
            return fvx.pv_inversion(state["rhs"], gr.dx, gr.dy, state["lam"], bc=case["bc"])
        return fvx.streamfunction_from_vorticity(state["rhs"], gr.dx, gr.dy, bc=case["bc"], lambda_=state["lam"])
    if kind == "vcycle":
        return state["precond"](state["b"])
    if kind == "pcg":
        return state["pcg"].solve(state["b"], rtol=1e-8, precond="mg", graph=True)[0]
    if kind == "ensemble":
        ens = state["ens"]
        ens.step(1)
        return [ens.get_layer(m, k) for m, (_, nl) in enumerate(ens.members) for k in range(nl)]
    net = state["net"]
    net.train_step(state["x"], state["target"], lr=1e-3, loss_out=state["loss"])
    return {"gradient": net.grad(), "parameters": net.params(), "loss": state["loss"]}


def _fft_flops(rows, n):
    return 2.5 * rows * n * math.log2(n)


def work(case):
    """Each input read once, each output written once; the least arithmetic (a fast transform for the inversions)."""
    kind = case["kind"]
    e = {"f32": 4, "f64": 8}[case.get("dtype", "f32")]
    if kind == "arakawa":
        p = (case["ny"] + 2) * (case["nx"] + 2)
        return {"bytes": 4 * p * e, "flops": 60 * p}
    if kind == "advect":
        p = (case["ny"] + 2) * (case["nx"] + 2)
        per = {"van_leer": 40, "weno3": 60, "weno5": 140, "wenoz5": 150, "weno7": 300}[case["method"]]
        return {"bytes": p * (4 * e + 2 * case["masked"]), "flops": per * p}
    if kind == "momentum":
        p = (case["ny"] + 2) * (case["nx"] + 2)
        return {"bytes": p * (7 * e + 4), "flops": 100 * p}

    def solve(ny, nx):
        return 2 * _fft_flops(ny, nx) + 2 * _fft_flops(nx, ny) + ny * nx

    if kind == "qg_step":
        p = case["n"] ** 2
        return {"bytes": 2 * p * e, "flops": 3 * (solve(case["n"], case["n"]) + 170 * p)}
    if kind == "helmholtz":
        return {"bytes": 2 * case["batch"] * case["ny"] * case["nx"] * e,
                "flops": case["batch"] * solve(case["ny"], case["nx"])}
    if kind == "vcycle":  # rhs, mask, cx, cy, 1/diagonal read, result written; 12 sweeps on every level
        return {"bytes": 6 * case["n"] ** 2 * e, "flops": 12 * 4 / 3 * 12 * case["n"] ** 2}
    if kind == "pcg":  # a V-cycle and the vector updates for each of about eight iterations
        return {"bytes": case["n"] ** 2 * (5 * e + 8), "flops": 8 * (12 * 4 / 3 * 12 + 40) * case["n"] ** 2}
    if kind == "ensemble":
        m = _members(case)
        return {"bytes": sum(8 * n * n * nl for n, nl in m),
                "flops": sum(3 * nl * (solve(n, n) + (170 + 4 * nl) * n * n) for n, nl in m)}
    p = case["n"] ** 2
    macs = 9 * (3 * 16 + 16 * 16 / 4 + 16 * 32 / 16 + 32 * 32 / 64 + 32 * 32 / 16 + 32 * 16 / 4 + 16 * 16 + 16) * p
    return {"bytes": 4 * 4 * case["batch"] * p + 16 * 33000, "flops": 3 * 2 * macs * case["batch"]}


# --------------------------------------------------------------------------
# the same results in plain 64-bit arithmetic
# --------------------------------------------------------------------------


def _weno_tables(r):
    """Candidate weights, linear weights and smoothness matrices of the order 2r - 1 scheme (cell averages -> right face), exact."""
    F = Fraction

    def poly(k):  # cell averages of cells k-r+1 .. k -> monomial coefficients of the reconstruction about cell 0
        lo = k - r + 1
        a = [[(F(2 * (lo + i) + 1, 2) ** (m + 1) - F(2 * (lo + i) - 1, 2) ** (m + 1)) / (m + 1) for m in range(r)]
             + [F(int(i == j)) for j in range(r)] for i in range(r)]
        for i in range(r):
            p = next(q for q in range(i, r) if a[q][i] != 0)
            a[i], a[p] = a[p], a[i]
            a[i] = [x / a[i][i] for x in a[i]]
            for q in range(r):
                if q != i:
                    a[q] = [x - a[q][i] * y for x, y in zip(a[q], a[i])]
        return [row[r:] for row in a]

    cand, beta = [], []
    for k in range(r):
        c = poly(k)
        cand.append([sum(c[m][j] * F(1, 2) ** m for m in range(r)) for j in range(r)])
        b = [[F(0)] * r for _ in range(r)]
        for deg in range(1, r):
            d = [[c[m][j] * math.perm(m, deg) for j in range(r)] for m in range(deg, r)]
            for p in range(len(d)):
                for q in range(len(d)):
                    w = F(1, p + q + 1) * (F(1, 2) ** (p + q + 1) - F(-1, 2) ** (p + q + 1))
                    for i in range(r):
                        for j in range(r):
                            b[i][j] += d[p][i] * d[q][j] * w
        beta.append(b)
    # linear weights: the combination that gives the 2r-1 cell reconstruction, from the outermost cells inwards
    full = _central(r)
    lin = []
    for k in range(r):
        lin.append((full[k] - sum(lin[m] * cand[m][k - m] for m in range(k))) / cand[k][0])
    return ([[float(x) for x in row] for row in cand], [float(x) for x in lin],
            [[[float(x) for x in row] for row in b] for b in beta])


def _central(r):
    """Weights of cells -r+1 .. r-1 in the order 2r - 1 value at the right face of cell 0."""
    n, out = 2 * r - 1, []
    for j in range(n):
        s = Fraction(0)
        for m in range(j + 1, n + 1):
            num = Fraction(0)
            for a in range(n + 1):
                if a != m:
                    t = Fraction(1)
                    for b in range(n + 1):
                        if b not in (a, m):
                            t *= r - b
                    num += t
            den = Fraction(1)
            for a in range(n + 1):
                if a != m:
                    den *= m - a
            s += num / den
        out.append(s)
    return out


def _weno(v, r, z=False):
    """Order 2r - 1 value at the downstream face from the 2r - 1 cells v, upstream first."""
    cand, lin, beta = _weno_tables(r)
    num = den = 0.0
    b = [sum(v[k + i] * sum(beta[k][i][j] * v[k + j] for j in range(r)) for i in range(r)) for k in range(r)]
    if r == 2:  # beta as the plain squares
        b = [(v[1] - v[0]) ** 2, (v[2] - v[1]) ** 2]
    if r == 3:
        b = [13 / 12 * (v[k] - 2 * v[k + 1] + v[k + 2]) ** 2 + 0.25 * d ** 2 for k, d in
             ((0, v[0] - 4 * v[1] + 3 * v[2]), (1, v[1] - v[3]), (2, 3 * v[2] - 4 * v[3] + v[4]))]
    for k in range(r):
        c = sum(cand[k][j] * v[k + j] for j in range(r))
        w = lin[k] * (1 + (b[0] - b[-1]).abs() / (b[k] + {2: 1e-14, 3: 1e-16}.get(r))) if z else lin[k] / (b[k] + 1e-8) ** 2
        num, den = num + w * c, den + w
    return num / den


def _upwind_faces(h, scheme):
    """Values at faces 1 .. N-2 of each row of h for flow to the right and to the left."""
    n = h.shape[-1]
    z = scheme == "wenoz5"
    order = {"upwind1": 0, "weno3": 1, "weno5": 2, "wenoz5": 2, "wenoz3": 1, "weno7": 3, "van_leer": -1}[scheme]
    z = z or scheme == "wenoz3"
    pos, neg = torch.empty_like(h[..., 1:-1]), torch.empty_like(h[..., 1:-1])
    if order < 0:
        d = h[..., 1:] - h[..., :-1]
        lim = lambda r: (r + r.abs()) / (1 + r.abs())  # noqa: E731
        pos = h[..., 1:-1] + 0.5 * lim(d[..., :-1] / (d[..., 1:] + 1e-8)) * d[..., 1:]
        neg[..., -1] = h[..., -1]
        neg[..., :-1] = h[..., 2:-1] - 0.5 * lim(-d[..., 2:] / (-d[..., 1:-1] + 1e-8)) * d[..., 1:-1]
        return pos, neg
    for out, first, sign in ((pos, 1, 1), (neg, 2, -1)):  # upwind cell of face i: i, or i + 1
        for reach in range(order + 1):
            # cells at exactly `reach` from an end, or at least that for the full scheme
            at = [c for c in range(first, first + n - 2) if min(c, n - 1 - c, order) == reach]
            if not at:
                continue
            c = torch.tensor(at, device=h.device)
            if reach == 0:
                out[..., c - first] = h[..., c]
            else:
                out[..., c - first] = _weno([h[..., c + sign * k] for k in range(-reach, reach + 1)], reach + 1, z)
    return pos, neg


def _face_flux(h, u, scheme, tier=None):
    """East-face fluxes with a zero ring; tier: 0 .. 3 per cell (dry, first order, third, fifth), or None."""
    out = torch.zeros_like(h)
    right = u[1:-1, 1:-1] >= 0
    if tier is None:
        pos, neg = _upwind_faces(h[1:-1], scheme)
        out[1:-1, 1:-1] = torch.where(right, pos, neg) * u[1:-1, 1:-1]
        return out
    low = {"weno5": "weno3", "wenoz5": "wenoz3"}.get(scheme, scheme)
    t = torch.where(right, tier[1:-1, 1:-1], tier[1:-1, 2:])
    acc = torch.zeros_like(h[1:-1, 1:-1])
    for k, s in ((1, "upwind1"), (2, low), (3, scheme)):
        pos, neg = _upwind_faces(h[1:-1], s)
        acc = torch.where(t == k, torch.where(right, pos, neg), acc)
    out[1:-1, 1:-1] = acc * u[1:-1, 1:-1]
    return out


def _tiers(m):
    """Tier per cell from the run of wet cells on both sides along x."""
    t = torch.zeros(m.shape, dtype=torch.int64, device=m.device)
    ok = m.clone()
    for k in range(3):
        t[ok] = k + 1
        near = torch.zeros_like(m)
        if k < 2:
            near[:, k + 1:m.shape[1] - k - 1] = m[:, :m.shape[1] - 2 * k - 2] & m[:, 2 * k + 2:]
        ok = ok & near
    return t


def _advection(h, u, v, dx, dy, scheme, mask=None):
    tx = ty = None
    if mask is not None:
        tx, ty = _tiers(mask), _tiers(mask.T)
    fe = _face_flux(h, u, scheme, tx)
    fn = _face_flux(h.T, v.T, scheme, ty).T
    out = torch.zeros_like(h)
    out[2:-2, 2:-2] = -((fe[2:-2, 2:-2] - fe[2:-2, 1:-3]) / dx + (fn[2:-2, 2:-2] - fn[1:-3, 2:-2]) / dy)
    return out if mask is None else out * mask


def _ring(x):
    out = torch.zeros((x.shape[0] + 2, x.shape[1] + 2), dtype=x.dtype, device=x.device)
    out[1:-1, 1:-1] = x
    return out


def _momentum(u, v, f, mask, dx, dy, scheme):
    p = torch.nn.functional.pad
    k = mask.double()
    e, n = p(k, (0, 1))[:, 1:], p(k, (0, 0, 0, 1))[1:]
    ne = p(k, (0, 1, 0, 1))[1:, 1:]
    mu, mv, mx = ((k + e) > 1.5).double(), ((k + n) > 1.5).double(), ((k + e + n + ne) > 3.5).double()
    C, E, W, N, S = (slice(1, -1), slice(1, -1)), (slice(1, -1), slice(2, None)), (slice(1, -1), slice(0, -2)), \
        (slice(2, None), slice(1, -1)), (slice(0, -2), slice(1, -1))
    NE, NW, SE = (slice(2, None), slice(2, None)), (slice(2, None), slice(0, -2)), (slice(0, -2), slice(2, None))
    v_u = _ring(0.25 * (v[C] + v[S] + v[E] + v[SE]))
    u_v = _ring(0.25 * (u[C] + u[N] + u[W] + u[NW]))
    cu = _ring(0.5 * (f[C] + f[E])) * v_u * mu
    cv = -_ring(0.5 * (f[C] + f[N])) * u_v * mv
    zeta = _ring((v[E] - v[C]) / dx - (u[N] - u[C]) / dy) * mx
    ke = _ring(0.5 * ((0.5 * (u[C] + u[W]) * k[C]) ** 2 + (0.5 * (v[C] + v[S]) * k[C]) ** 2))
    kx, ky = _ring((ke[E] - ke[C]) / dx) * mu, _ring((ke[N] - ke[C]) / dy) * mv
    on_u = lambda x: _ring(0.5 * (x[C] + x[S])) * mu  # noqa: E731
    on_v = lambda x: _ring(0.5 * (x[C] + x[W])) * mv  # noqa: E731
    energy = on_u(zeta) * v_u * mu, on_v(zeta) * u_v * mv
    enstrophy = on_u(zeta * _ring(0.5 * (v[C] + v[E])) * mx), on_v(zeta * _ring(0.5 * (u[C] + u[N])) * mx)
    a = {"energy": 1.0, "enstrophy": 0.0, "al": 1.0 / 3.0}[scheme]
    du = (a * energy[0] + (1 - a) * enstrophy[0] - kx) * mu
    dv = (-(a * energy[1] + (1 - a) * enstrophy[1]) - ky) * mv
    return (cu, cv), tuple(torch.nn.functional.pad(x[2:-2, 2:-2], (2, 2, 2, 2)) for x in (du, dv))


def _transform(x, bc, inverse=False):
    """Sine, cosine or Fourier transform along the last axis, by an FFT of the periodic extension."""
    n = x.shape[-1]
    if bc == "fft":
        return torch.fft.ifft(x) if inverse else torch.fft.fft(x)
    if bc == "dst":
        z = torch.zeros_like(x[..., :1])
        y = -torch.fft.rfft(torch.cat((z, x, z, -x.flip(-1)), dim=-1)).imag[..., 1:n + 1]
        return y / (2 * (n + 1)) if inverse else y
    k = torch.arange(n, device=x.device, dtype=torch.float64)
    w = torch.exp(-0.5j * math.pi * k / n)
    if not inverse:
        return (torch.fft.rfft(torch.cat((x, x.flip(-1)), dim=-1))[..., :n] * w).real
    return torch.fft.irfft(torch.cat((x / w, torch.zeros_like(x[..., :1])), dim=-1), n=2 * n)[..., :n]


def _eigenvalues(n, d, bc, device):
    k = torch.arange(n, device=device, dtype=torch.float64)
    a = {"dst": 0.5 * (k + 1) / (n + 1), "dct": 0.5 * k / n, "fft": k / n}[bc]
    return -4.0 / d ** 2 * torch.sin(math.pi * a) ** 2


def _invert(f, dx, dy, lam, bc):
    ny, nx = f.shape[-2:]
    g = _transform(_transform(f, bc).transpose(-1, -2), bc).transpose(-1, -2)
    lam = torch.as_tensor(lam, dtype=torch.float64, device=f.device).reshape(-1, 1, 1)
    d = _eigenvalues(ny, dy, bc, f.device)[:, None] + _eigenvalues(nx, dx, bc, f.device)[None, :] - lam
    g = torch.where(d == 0, torch.zeros_like(g), g / torch.where(d == 0, torch.ones_like(d), d))
    g = _transform(_transform(g, bc, True).transpose(-1, -2), bc, True).transpose(-1, -2)
    return (g.real if bc == "fft" else g).reshape(f.shape)


def _qg_rhs(q, psi_interior, dx, dy):
    psi = _ring(psi_interior)
    x = _ring(0.25 * (psi[1:-1, 1:-1] + psi[1:-1, 2:] + psi[2:, 1:-1] + psi[2:, 2:]))
    u = _ring(-(x[1:-1, 1:-1] - x[:-2, 1:-1]) / dy)
    v = _ring((x[1:-1, 1:-1] - x[1:-1, :-2]) / dx)
    return _advection(q, u, v, dx, dy, "weno5") - BETA * _ring(0.5 * (v[1:-1, 1:-1] + v[:-2, 1:-1]))


def _qg_step(q, dx, dt, lam, l2m, m2l):
    """RK3 step of the layers q [nl, n + 2, n + 2]."""
    def rhs(y):
        y = _ghosts(y[:, 1:-1, 1:-1])
        psi = torch.einsum("kl,lyx->kyx", m2l, _invert(torch.einsum("kl,lyx->kyx", l2m, y[:, 1:-1, 1:-1]), dx, dx, lam, "dst"))
        return torch.stack([_qg_rhs(a, b, dx, dx) for a, b in zip(y, psi)])

    y1 = q + dt * rhs(q)
    y2 = 0.75 * q + 0.25 * y1 + 0.25 * dt * rhs(y1)
    return _ghosts((q / 3 + 2 / 3 * y2 + 2 / 3 * dt * rhs(y2))[:, 1:-1, 1:-1])


def _masked_solve(mask, c, b, dx, lam):
    """(div c grad - lambda) x = b with zero flux at coasts, by conjugate gradients to rounding."""
    c = c * mask
    cx, cy = torch.zeros_like(c), torch.zeros_like(c)
    cx[:, :-1] = 0.5 * (c[:, :-1] + c[:, 1:]) * mask[:, :-1] * mask[:, 1:]
    cy[:-1] = 0.5 * (c[:-1] + c[1:]) * mask[:-1] * mask[1:]

    def apply(x):  # the negative operator, positive definite on wet cells
        fx, fy = torch.zeros_like(x), torch.zeros_like(x)
        fx[:, :-1] = cx[:, :-1] * (x[:, 1:] - x[:, :-1])
        fy[:-1] = cy[:-1] * (x[1:] - x[:-1])
        out = fx + fy
        out[:, 1:] -= fx[:, :-1]
        out[1:] -= fy[:-1]
        return (lam * x - out / dx ** 2) * mask

    w, s = torch.zeros_like(c), torch.zeros_like(c)
    w[:, 1:], s[1:] = cx[:, :-1], cy[:-1]
    inv = mask / ((cx + w + cy + s) / dx ** 2 + lam)
    x, r = torch.zeros_like(b), -b * mask
    z = inv * r
    p, rz, stop = z, (r * z).sum(), 1e-15 * r.norm()
    for k in range(6000):
        ap = apply(p)
        a = rz / (p * ap).sum()
        x, r = x + a * p, r - a * ap
        if k % 25 == 0 and r.norm() < stop:
            break
        z = inv * r
        new = (r * z).sum()
        p, rz = z + new / rz * p, new
    return x


def _train(theta, x, target):
    """Loss and gradient of the network (weights in bf16, everything else in 64 bits) and its first optimiser step."""
    nn = torch.nn.functional
    w, at = [], 0
    theta = torch.as_tensor(theta, device=x.device)
    for ci, co in learned.LAYERS:
        k = theta[at:at + co * ci * 9].bfloat16().double().reshape(co, ci, 3, 3).requires_grad_()
        at += co * ci * 9
        b = theta[at:at + co].double().requires_grad_()
        at += co
        w += [k, b]
    conv = lambda i, a: nn.conv2d(a, w[2 * i], w[2 * i + 1], padding=1)  # noqa: E731
    pool = lambda a: nn.avg_pool2d(a, 2)  # noqa: E731
    up = lambda a: a.repeat_interleave(2, dim=-1).repeat_interleave(2, dim=-2)  # noqa: E731
    e0 = conv(0, x).relu()
    e1 = conv(1, pool(e0)).relu()
    e2 = conv(2, pool(e1)).relu()
    d = conv(3, pool(e2)).relu()
    for i, skip in ((4, e2), (5, e1), (6, e0)):
        d = (conv(i, up(d)) + skip).relu()
    y = conv(7, d)
    loss = (((y - target) * x[:, 1:2]) ** 2).sum() / y.numel()
    g = torch.cat([a.reshape(-1) for a in torch.autograd.grad(loss, w)])
    return {"gradient": g, "parameters": theta.double() - 1e-3 * g / (g.abs() + 1e-8), "loss": loss.detach().reshape(1)}


def exact(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    t = DTYPES.get(case.get("dtype", "f32"))
    d = {k: (v.to(t).double() if isinstance(v, torch.Tensor) and v.is_floating_point() and k not in ("mask", "coeff") else v)
         for k, v in d.items()}
    if kind == "arakawa":
        gr = _grid(case["ny"], case["nx"])
        f, g = d["psi"], d["q"]
        a = lambda x, j, i: x[1 + j:x.shape[0] - 1 + j, 1 + i:x.shape[1] - 1 + i]  # noqa: E731
        jpp = (a(f, 0, 1) - a(f, 0, -1)) * (a(g, 1, 0) - a(g, -1, 0)) - (a(f, 1, 0) - a(f, -1, 0)) * (a(g, 0, 1) - a(g, 0, -1))
        jpx = (a(f, 0, 1) * (a(g, 1, 1) - a(g, -1, 1)) - a(f, 0, -1) * (a(g, 1, -1) - a(g, -1, -1))
               - a(f, 1, 0) * (a(g, 1, 1) - a(g, 1, -1)) + a(f, -1, 0) * (a(g, -1, 1) - a(g, -1, -1)))
        jxp = (a(g, 1, 0) * (a(f, 1, 1) - a(f, 1, -1)) - a(g, -1, 0) * (a(f, -1, 1) - a(f, -1, -1))
               - a(g, 0, 1) * (a(f, 1, 1) - a(f, -1, 1)) + a(g, 0, -1) * (a(f, 1, -1) - a(f, -1, -1)))

        def lap(h):  # no flux through the outer faces of the interior
            fx = (h[1:-1, 2:-1] - h[1:-1, 1:-2]) / gr.dx
            fy = (h[2:-1, 1:-1] - h[1:-2, 1:-1]) / gr.dy
            pad = torch.nn.functional.pad
            return _ring((pad(fx, (0, 1)) - pad(fx, (1, 0))) / gr.dx + (pad(fy, (0, 0, 0, 1)) - pad(fy, (0, 0, 1, 0))) / gr.dy)

        return (jpp + jpx + jxp) / (12.0 * gr.dx * gr.dy), -(1e-3 * gr.dx ** 4 / 86400) * lap(lap(g))
    if kind == "advect":
        gr = _grid(case["ny"], case["nx"])
        return _advection(d["h"], d["u"], d["v"], gr.dx, gr.dy, case["method"], d.get("mask"))
    if kind == "momentum":
        gr = _grid(case["ny"], case["nx"])
        return _momentum(d["u"], d["v"], d["f"], d["mask"], gr.dx, gr.dy, case["scheme"])
    if kind == "qg_step":
        dx = LX / case["n"]
        one = torch.ones((1, 1), dtype=torch.float64, device="cuda")
        return _qg_step(d["q"][None], dx, 0.5 * dx, 1.0 / LD ** 2, one, one)[0]
    if kind == "helmholtz":
        gr = _grid(case["ny"], case["nx"])
        return _invert(d["rhs"], gr.dx, gr.dy, _lambdas(case), case["bc"])
    if kind == "vcycle":
        return None
    if kind == "pcg":
        return _masked_solve(d["mask"], d["coeff"], d["b"], LX / case["n"], 1.0 / case["ld"] ** 2)
    if kind == "ensemble":
        out = []
        for (n, nl), q in zip(_members(case), d["q"]):
            a = fvx.build_coupling_matrix(H_LAYERS[:nl], G_PRIME[:nl])
            rr, l2m, m2l = fvx.decompose_vertical_modes(a, F0)
            l2m, m2l = (torch.as_tensor(x, device="cuda") for x in (l2m, m2l))
            dx = LX / n
            out += list(_qg_step(q.float().double(), dx, 0.05 * dx, [1.0 / float(r) ** 2 for r in rr], l2m, m2l))
        return out
    return _train(learned.init_params(0), d["x"].float().double(), d["target"].float().double())
