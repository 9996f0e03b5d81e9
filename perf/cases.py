"""What is timed: the runs a user of wfe_b200 makes, and what they should give.

Every case goes through the package's public entry points.  A forecast keeps
its Case between passes, as a driver loop does: one pass runs ``steps`` large
steps (``Case.run``) and reads the state back into page-locked arrays
(``snapshot_begin`` / ``snapshot_wait``), the model's output step.  An ensemble
does the same for its members.  A gradient pass is one inner iteration of a
variational analysis, the tangent-linear run and the adjoint run about the same
trajectory (``wfe_b200.adjoint``), or the adjoint run alone.

The set-ups are those of ``cases/`` and of the tests (warm bubble, Straka density
current, Schaer mountain waves, WK82 supercell) and a regional forecast (terrain,
lateral relaxation, positive-definite moisture, Kessler, surface physics) on the
ensemble generator's grids.  The seed makes the initial perturbations: smooth
noise on the wind, theta' and moisture, and for the moist set-ups a cloud with a
rain shaft, so that every branch of the microphysics has work.

``exact`` restates the model in 64-bit torch operations, whole arrays at a time.
"""

import math

import numpy as np
import torch

G, CP, RD, LV, LS, RV, EPS = 9.81, 1004.5, 287.04, 2.5e6, 2.5e6 + 3.34e5, 461.5, 0.61
CV, P00, NG = CP - RD, 1.0e5, 3
FIELDS = ("u", "v", "w", "thp", "pip", "qv", "qc", "qr")
SURFACE = ("tsk", "pblh", "t2m", "u10")

#: Case keys by set-up, beside the grid; lengths that follow the grid are made in settings().
SETUPS = {
    "bubble": dict(dx=250, dy=250, dt=1.5, profile="isentropic", theta0=300, bc_x="open", bc_y="open",
                   rayleigh_alpha=0.03),
    "straka": dict(dx=100, dy=100, dt=0.5, profile="isentropic", theta0=300, diff_K=75),
    "schaer": dict(dx=500, dy=500, dt=4, profile="constant_N", theta0=280, bv_N=0.01, wind_u=10,
                   terrain="schaer", mtn_h0=250, mtn_a=5000, mtn_lambda=4000, bc_x="open",
                   rayleigh_alpha=0.05),
    "storm": dict(dx=1000, dy=1000, dt=6, stretch="geometric", dz_max=1000, profile="wk82",
                  wind_profile="linear", wind_us=35, wind_zs=6000, bc_x="open", bc_y="open",
                  rayleigh_alpha=0.03),
    "region": dict(dx=12000, dy=12000, dt=60, profile="wk82", wind_profile="linear", wind_us=20, wind_zs=9000,
                   terrain="gauss", mtn_h0=1800, mtn_a=150000, coriolis_f=1e-4, bc_x="open", bc_y="open",
                   w_damping="on", pd_moist="on", rayleigh_alpha=0.02),
}


def listed():
    return [
        # the small moist column of the tests, limiter and w damping on: launches and their gaps are all of it
        dict(name="storm 16x16x16 limited", kind="forecast", setup="storm", nx=16, ny=16, nz=16, steps=20,
             precision="f32", pd=True),
        # the shipped idealised benchmarks at their own sizes
        dict(name="bubble 80x80x40", kind="forecast", setup="bubble", nx=80, ny=80, nz=40, steps=40,
             precision="f32", pd=False),
        dict(name="straka 512x4x64", kind="forecast", setup="straka", nx=512, ny=4, nz=64, steps=40,
             precision="f32", pd=False),
        dict(name="schaer 400x4x65", kind="forecast", setup="schaer", nx=400, ny=4, nz=65, steps=40,
             precision="f32", pd=False),
        dict(name="storm 160x160x40", kind="forecast", setup="storm", nx=160, ny=160, nz=40, steps=20,
             precision="f32", pd=False),
        # the same storm as a verification run in 64 bits
        dict(name="storm 160x160x40 f64", kind="forecast", setup="storm", nx=160, ny=160, nz=40, steps=10,
             precision="f64", pd=False),
        # sizes that fit no tile, a deeper column
        dict(name="storm 181x203x53", kind="forecast", setup="storm", nx=181, ny=203, nz=53, steps=10,
             precision="f32", pd=False),
        # regional forecasts, the smallest and the largest grid of the ensemble generator
        dict(name="region 120x90x45", kind="forecast", setup="region", nx=120, ny=90, nz=45, steps=15,
             precision="f32", pd=True),
        dict(name="region 300x200x45", kind="forecast", setup="region", nx=300, ny=200, nz=45, steps=10,
             precision="f32", pd=True),
        # members of uneven grids stepped together
        dict(name="ensemble of 3", kind="ensemble", setup="region", nx=120, ny=90, nz=45, steps=20,
             precision="f32", pd=True),
        # one inner iteration of a variational analysis on the mountain-wave slab
        dict(name="schaer gradient", kind="inner", setup="schaer", nx=400, ny=4, nz=65, steps=20,
             precision="f32", pd=False),
        # the moist adjoint of a storm
        dict(name="storm gradient 96x96x40", kind="adjoint", setup="storm", nx=96, ny=96, nz=40, steps=5,
             precision="f32", pd=False),
    ]


def draw(rng):
    """Any of the set-ups on any grid of its range: the regional grids from half the generator's smallest, the slabs and
    boxes from far smaller, all up to the largest listed case."""
    setup = rng.choice(("bubble", "straka", "schaer", "storm", "storm", "region", "region"))
    kind = rng.choice(("forecast",) * 5 + ("ensemble",)) if setup == "region" else "forecast"
    if setup in ("schaer", "storm") and rng.random() < 0.3:
        kind = rng.choice(("inner", "adjoint"))
    nz = rng.randint(24, 50) if kind == "ensemble" else rng.randint(16, 80)
    if setup in ("straka", "schaer"):
        nx, ny = int(math.exp(rng.uniform(math.log(128), math.log(1024)))), rng.randint(4, 9)
    else:
        least = {"forecast": 5400, "ensemble": 10500}[kind] if setup == "region" else 256
        most = {"forecast": 2.4e6, "ensemble": 6e5, "inner": 4e5, "adjoint": 4e5}[kind] / nz
        area, ratio = math.exp(rng.uniform(math.log(least), math.log(most))), rng.uniform(0.6, 1.6)
        nx, ny = math.ceil(math.sqrt(area * ratio)), math.ceil(math.sqrt(area / ratio))
    if kind in ("inner", "adjoint"):
        steps, precision = rng.randint(3, 6), rng.choice(("f32", "f32", "f64"))
    elif kind == "ensemble":
        steps, precision = 20, "f32"
    else:
        steps, precision = rng.randint(5, 15), rng.choice(("f32", "f32", "f32", "f64"))
    if kind == "forecast":  # the largest listed case is 27 million cell-steps in 32 bits
        most = 2.7e7 if precision == "f32" else 1.3e7
        steps = max(3, min(steps, int(most / (nx * ny * nz))))
    pd = setup == "region" or (setup == "storm" and kind == "forecast" and rng.random() < 0.3)
    return dict(kind=kind, setup=setup, nx=nx, ny=ny, nz=nz, steps=steps, precision=precision, pd=pd)


def moist(case):
    return case["setup"] in ("storm", "region")


def work(case):
    cells = sum(m["nx"] * m["ny"] * m["nz"] for m in members(case))
    size = 4 if case["precision"] == "f32" else 8
    fields = 8 if moist(case) else 5
    # a large step reads the state of time n and writes the next; its three tendency evaluations and ten
    # acoustic substeps are about 4600 operations a cell with moisture, 2700 without
    passes = {"forecast": 1, "ensemble": 1, "adjoint": 4, "inner": 7}[case["kind"]]
    return {"bytes": cells * case["steps"] * passes * 2 * fields * size,
            "flops": cells * case["steps"] * passes * (4600 if moist(case) else 2700)}


def tolerance(case):
    """About four times the largest distance from exact() over the listed and two dozen drawn cases.  In 32 bits a point
    where the limiter, the saturation adjustment or the boundary layer's top takes the other branch shows in the
    maximum, and in the condensate's norm; the 64-bit runs differ by the 1 m table's interpolation in the base state."""
    if case["precision"] == "f64":
        return {"rel": 2e-7, "max": 1e-5}
    if case["setup"] == "region":
        return {"rel": 9e-3, "max": 0.99}
    if case["kind"] in ("inner", "adjoint"):
        return {"rel": 5e-3, "max": 0.99} if moist(case) else {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1e-4, "max": 2e-2} if moist(case) else {"rel": 3e-5, "max": 2e-4}


# ------------------------------------------------------------------ inputs
def members(case):
    """The grids of a case: its own, or three uneven ones."""
    if case["kind"] != "ensemble":
        return [case]
    return [dict(case, nx=int(case["nx"] * s), ny=int(case["ny"] * s), nz=case["nz"] - d)
            for s, d in ((1.0, 0), (0.85, 3), (0.7, 0))]


def settings(case):
    """The keys of the case file."""
    kv = dict(SETUPS[case["setup"]], nx=case["nx"], ny=case["ny"], nz=case["nz"], acoustic_ns=6)
    if case["pd"]:
        kv.update(pd_moist="on", w_damping="on")
    top = {"bubble": 10000.0, "straka": 6400.0}.get(case["setup"], 20000.0)
    # in sixteenths: the base state's 1 m table, which starts 16 dz below ground, has a point at z = 0
    kv["dz"] = round(16 * top / case["nz"]) / 16
    if kv.get("stretch"):
        # layers from 0.4 of the mean, growing by one ratio up to dz_max to the same top (or near it)
        kv["dz0"] = 0.4 * kv["dz"]
        kv["dz_max"] = max(kv["dz_max"], 1.6 * kv["dz"])
        lo, hi = 1.0, 1.5
        for _ in range(60):
            r = 0.5 * (lo + hi)
            h = sum(min(kv["dz0"] * r ** k, kv["dz_max"]) for k in range(case["nz"]))
            lo, hi = (r, hi) if h < top else (lo, r)
        kv["dz_ratio"] = r
    if "rayleigh_alpha" in kv:
        kv["rayleigh_zd"] = {"bubble": 0.7, "schaer": 0.5, "storm": 0.8, "region": 0.75}[case["setup"]] * top
    if case["setup"] == "schaer":
        kv["mtn_xc"] = case["nx"] * kv["dx"] / 2
    if case["setup"] == "region":
        kv["mtn_ya"] = 120000
    # all digits: the model and exact() read the same numbers
    return {k: repr(float(v)) if isinstance(v, float) else v for k, v in kv.items()}


def noise(rng, shape):
    """Smooth noise of unit variance."""
    a = rng.standard_normal(shape, dtype=np.float32)
    for axis in range(3):
        for _ in range(3):
            a = 0.25 * (np.roll(a, 1, axis) + np.roll(a, -1, axis)) + 0.5 * a
    return (a / a.std()).astype(np.float64)


def perturb(case, seed, state):
    """The perturbed initial state: `state` is the set-up's own, in the boxes of the prognostic points."""
    rng = np.random.default_rng([seed, case["nx"], case["ny"], case["nz"]])
    nz, ny, nx = state["thp"].shape
    s = {k: np.array(v) for k, v in state.items()}
    s["u"][:, :, :nx] += 0.5 * noise(rng, (nz, ny, nx))
    s["v"][:, :ny] += 0.5 * noise(rng, (nz, ny, nx))
    s["w"][1:nz] += 0.2 * noise(rng, (nz - 1, ny, nx))
    s["thp"] += 0.5 * noise(rng, (nz, ny, nx))
    s["pip"] += 1e-5 * noise(rng, (nz, ny, nx))
    if moist(case):
        s["qv"] *= 1 + 0.05 * np.clip(noise(rng, (nz, ny, nx)), -3, 3)
        # a cloud over a rain shaft, off the centre
        z, y, x = np.meshgrid((np.arange(nz) + 0.5) / nz, (np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx,
                              indexing="ij")
        xc, yc = rng.uniform(0.3, 0.7, 2)
        r2 = ((x - xc) / 0.12) ** 2 + ((y - yc) / 0.12) ** 2
        s["qc"] += 2e-3 * np.exp(-r2 - ((z - 0.25) / 0.08) ** 2)
        s["qr"] += 3e-3 * np.exp(-r2 - (z / 0.2) ** 2)
        s["thp"] += 2.0 * np.exp(-r2 - ((z - 0.12) / 0.1) ** 2)
        # an edge, not a tail: where the condensate is 1e-40 its gradient is a matter of the type's smallest value
        s["qc"][s["qc"] < 1e-6] = 0
        s["qr"][s["qr"] < 1e-6] = 0
    else:
        s["qv"][:] = s["qc"][:] = s["qr"][:] = 0
    return {k: v.astype(np.float32).astype(np.float64) for k, v in s.items()}


def surface_inputs(case, seed):
    rng = np.random.default_rng([seed, 7, case["nx"], case["ny"]])
    ny, nx = case["ny"], case["nx"]
    smooth = [noise(rng, (1, ny, nx))[0] for _ in range(3)]
    y, x = np.meshgrid(np.linspace(-8, 8, ny), np.linspace(-12, 12, nx), indexing="ij")
    out = dict(tsk=299 + 2 * smooth[0], land=(smooth[1] > -0.3) * 1.0, lat=40 + y, lon=30 + x,
               soilw=0.25 + 0.08 * np.tanh(smooth[2]))
    return {k: v.astype(np.float32).astype(np.float64) for k, v in out.items()}


def box(case, name):
    """The slices of a field's prognostic points in the padded layout."""
    return (slice(NG, NG + case["nz"] + (name == "w")), slice(NG, NG + case["ny"] + (name == "v")),
            slice(NG, NG + case["nx"] + (name == "u")))


def padded(case, name, a):
    out = np.zeros((case["nz"] + 2 * NG + 1, case["ny"] + 2 * NG, case["nx"] + 2 * NG))
    out[box(case, name)] = a
    return out


def cotangent(case, seed, names):
    """A field over the prognostic points, the gradient of a smooth cost of the final state."""
    rng = np.random.default_rng([seed, 3, case["nx"], case["ny"], case["nz"]])
    shape = (case["nz"], case["ny"], case["nx"])
    # each field in the units of one over its own size
    size = dict(u=1, v=1, w=1, thp=1, pip=1e3, qv=1e3, qc=1e3, qr=1e3)
    out = {}
    for k in names:
        a = np.zeros([s.stop - s.start for s in box(case, k)])
        a[1 if k == "w" else 0:case["nz"], :case["ny"], :case["nx"]] = (size[k] * noise(rng, shape))[1 if k == "w" else 0:]
        out[k] = a.astype(np.float32).astype(np.float64)
    return out


def prepare(case, seed):
    import wfe_b200 as W

    state = {"case": case, "t": 0.0, "cases": [], "bufs": []}
    for n, m in enumerate(members(case)):
        text = "".join("%s = %s\n" % kv for kv in settings(m).items())
        c = W.Case(text=text, precision=m["precision"], device=0)
        own = {k: c.field(k)[box(m, k)] for k in FIELDS}
        x0 = perturb(m, seed + 101 * n, own)
        for k in FIELDS:
            c.set_field(k, padded(m, k, x0[k]))
        if m["setup"] == "region":
            # lateral relaxation toward the unperturbed state over a six-hour interval, surface physics
            targets = [padded(m, k, own[k]) for k in ("u", "v", "thp", "pip", "qv")]
            c.set_boundary(targets, targets, c.bdy_weights(5, 600.0), 0.0, 21600.0)
            c.set_physics(*surface_inputs(m, seed + 101 * n).values(), 9.0, 172, True)
        state["cases"].append(c)
        if m["kind"] in ("forecast", "ensemble"):
            names = (FIELDS + ("rain",) if moist(m) else FIELDS[:5]) + (SURFACE if m["setup"] == "region" else ())
            state["bufs"].append(c.snapshot_buffers(names, np.float32 if m["precision"] == "f32" else np.float64))
        else:
            names = FIELDS if moist(m) else FIELDS[:5]
            state["x0"] = {k: padded(m, k, x0[k]) for k in names}
            state["dx"] = {k: padded(m, k, v) for k, v in increment(m, seed, names).items()}
            state["ybar"] = {k: padded(m, k, v) for k, v in cotangent(m, seed, names).items()}
    if case["kind"] == "ensemble":
        state["ensemble"] = W.Ensemble(state["cases"])
    return state


def increment(case, seed, names):
    """An analysis increment: the cotangent's shapes in the fields' own sizes."""
    size = dict(u=0.1, v=0.1, w=0.02, thp=0.1, pip=1e-8, qv=1e-8, qc=1e-8, qr=1e-8)
    return {k: (size[k] * v).astype(np.float32).astype(np.float64)
            for k, v in cotangent(case, seed + 1, names).items()}


def run(state):
    import wfe_b200.adjoint as A

    case, cases = state["case"], state["cases"]
    if case["kind"] in ("inner", "adjoint"):
        c, cut = cases[0], lambda d: {k: a[box(case, k)] for k, a in d.items()}
        out = {}
        if case["kind"] == "inner":
            out["tangent"] = cut(A.tangent(c, state["x0"], state["dx"], case["steps"]))
        out["adjoint"] = cut(A.adjoint(c, state["x0"], state["ybar"], case["steps"]))
        return out
    dt = cases[0].dt
    if case["kind"] == "ensemble":
        state["ensemble"].run(case["steps"], dt, state["t"])
    else:
        cases[0].run(case["steps"], dt, state["t"])
    state["t"] += case["steps"] * dt
    for c, b in zip(cases, state["bufs"]):
        c.snapshot_begin(b)
    for c in cases:
        c.snapshot_wait()
    return state["bufs"]


# ---------------------------------------------------- the model in 64 bits
class Exact:
    """The model on padded (NZ, NY, NX) arrays in torch float64.  A neighbour is a rolled array; what rolls in from the
    far side only reaches points outside the boxes that are kept."""

    def __init__(self, case):
        kv = settings(case)
        num = lambda k, d=0.0: float(kv.get(k, d))  # noqa: E731
        self.case, self.kv = case, kv
        self.nx, self.ny, self.nz = nx, ny, nz = case["nx"], case["ny"], case["nz"]
        self.dx, self.dy, self.dt = num("dx"), num("dy"), num("dt")
        self.ox, self.oy = kv.get("bc_x") == "open", kv.get("bc_y") == "open"
        self.moist, self.pd, self.damp = moist(case), kv.get("pd_moist") == "on", kv.get("w_damping") == "on"
        self.K, self.beta, self.smdiv, self.cstar = num("diff_K"), 0.2, 0.1, 30.0
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        # levels
        zw = np.arange(nz + 1) * num("dz")
        if kv.get("stretch"):
            d, zw = num("dz0"), [0.0]
            for _ in range(nz):
                zw.append(zw[-1] + d)
                d = min(d * num("dz_ratio"), num("dz_max"))
            zw = np.array(zw)
        q = np.arange(-NG, nz + 2 + NG)
        ext = np.where(q < 0, q * zw[1], np.where(q > nz, zw[nz] + (q - nz) * (zw[nz] - zw[nz - 1]), zw[np.clip(q, 0, nz)]))
        zeta_w, zeta_c = ext[:-1], 0.5 * (ext[:-1] + ext[1:])
        zt = zw[nz]
        dzc = np.append(np.diff(zeta_w), zeta_w[-1] - zeta_w[-2])
        dzw = np.insert(np.diff(zeta_c), 0, zeta_c[1] - zeta_c[0])
        # terrain
        x = (np.arange(-NG, nx + NG) + 0.5) * self.dx
        y = (np.arange(-NG, ny + NG) + 0.5) * self.dy
        Y, X = np.meshgrid(y, x, indexing="ij")

        def height(x, y):
            if kv.get("terrain") == "schaer":
                r = x - num("mtn_xc", nx * self.dx / 2)
                return num("mtn_h0") * np.exp(-(r / num("mtn_a")) ** 2) * np.cos(np.pi * r / num("mtn_lambda")) ** 2
            if kv.get("terrain") == "gauss":
                r, s = (x - nx * self.dx / 2) / num("mtn_a"), (y - ny * self.dy / 2) / num("mtn_ya")
                return num("mtn_h0") * np.exp(-r * r - s * s)
            return np.zeros_like(x)

        h = height(X, Y)
        jac = (zt - h) / zt
        self.h, self.zeta_np, self.zt = h, zeta_c, zt
        # base state on a 1 m table, at each point's height
        zmin = -(NG + 1) * num("dz") * 4 - 100.0
        n = int(zt + (NG + 1) * num("dz") * 4 + 100.0 - zmin) + 2
        i0 = int(-zmin)
        ztab = zmin + np.arange(n)

        def theta(z):
            z = np.maximum(z, 0) if kv["profile"] == "wk82" else z
            if kv["profile"] == "wk82":
                return np.where(z <= 12000, 300 + 43 * (np.minimum(z, 12000) / 12000) ** 1.25,
                                343 * np.exp(G * (z - 12000) / (CP * 213)))
            if kv["profile"] == "constant_N":
                return num("theta0") * np.exp(num("bv_N") ** 2 * z / G)
            return np.full_like(z, num("theta0"))

        def exner(thv):
            d = G / (CP * 0.5 * (thv[:-1] + thv[1:]))
            return np.concatenate([1 + np.cumsum(d[:i0][::-1])[::-1], [1.0], 1 - np.cumsum(d[i0:])])

        th, qt = theta(ztab), np.zeros(n)
        pit = exner(th)
        if self.moist:
            rh = np.where(ztab <= 12000, 1 - 0.75 * (np.clip(ztab, 0, 12000) / 12000) ** 1.25, 0.25)
            for _ in range(5):
                T, p = th * pit, P00 * pit ** (CP / RD)
                es = 610.78 * np.exp(17.269 * (T - 273.16) / (T - 35.86))
                qt = np.where(ztab < 0, 0, np.minimum(rh * 0.622 * es / (p - es), 0.014))
                pit = exner(th * (1 + EPS * qt))
        at = lambda z: h[None] + z[:, None, None] * (zt - h[None]) / zt  # noqa: E731
        zc, zwp = at(zeta_c), at(zeta_w)
        tab = lambda a, z: np.interp(z, ztab, a)  # noqa: E731
        qvb, qvw = (tab(qt, zc), tab(qt, zwp)) if self.moist else (0 * zc, 0 * zc)
        rho = lambda pi, thv: P00 * pi ** (CV / RD) / (RD * thv)  # noqa: E731
        pib, piw = tab(pit, zc), tab(pit, zwp)
        thb, thbw = theta(zc), theta(zwp)
        thvb, thvbw = thb * (1 + EPS * qvb), thbw * (1 + EPS * qvw)
        z = np.maximum(zeta_c, 0)
        ub = {"tanh": num("wind_us") * np.tanh(z / num("wind_zs", 1)),
              "linear": num("wind_us") * np.minimum(z / num("wind_zs", 1), 1)}.get(kv.get("wind_profile"), 0 * z + num("wind_u"))
        self.ub_np, self.qvb_np = ub, qvb
        lev, col = lambda a: self.t(a)[:, None, None], lambda a: self.t(a)[None]  # noqa: E731
        slope = lambda a, b, d: (a - b) / d  # noqa: E731
        self.jac, self.hx, self.hy = col(jac), col(slope(height(X + self.dx, Y), height(X - self.dx, Y), 2 * self.dx)), col(
            slope(height(X, Y + self.dy), height(X, Y - self.dy), 2 * self.dy))
        self.hxu, self.hyv = col(slope(h, height(X - self.dx, Y), self.dx)), col(slope(h, height(X, Y - self.dy), self.dy))
        self.fcor = num("coriolis_f")
        self.zc, self.zw, self.dzc, self.dzw, self.ub = lev(zeta_c), lev(zeta_w), lev(dzc), lev(dzw), lev(ub)
        self.thb, self.pib, self.rhob, self.dthb = self.t(thb), self.t(pib), self.t(rho(pib, thvb)), self.t((theta(zc + 1) - theta(zc - 1)) / 2)
        self.thbw, self.rhobw, self.qvb = self.t(thbw), self.t(rho(piw, thvbw)), self.t(qvb)
        zd, alpha = num("rayleigh_zd", -1), num("rayleigh_alpha")

        def sponge(zeta):
            s = np.sin(np.pi / 2 * np.clip((zeta - zd) / (zt - zd), 0, 1)) if zt > zd >= 0 else 0 * zeta
            return lev(alpha * s * s)

        self.sc, self.sw = sponge(zeta_c), sponge(zeta_w)
        # acoustic coefficients
        rtj = self.rhob * self.t(thvb) * self.jac
        self.rtjx, self.rtjy = 0.5 * (self.X(rtj, -1) + rtj), 0.5 * (self.Y(rtj, -1) + rtj)
        self.kt3 = RD * self.pib / (CV * rtj)
        self.aw = self.rhobw * self.t(thvbw)
        # lateral and vertical source points of the ghost fill
        m = lambda n, last, o: (np.clip(np.arange(-NG, n + NG), 0, last) if o else np.arange(-NG, n + NG) % n)  # noqa: E731
        ix = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
        self.mx, self.mxu = ix(m(nx, nx - 1, self.ox)), ix(m(nx, nx, self.ox))
        self.my, self.myv = ix(m(ny, ny - 1, self.oy)), ix(m(ny, ny, self.oy))
        self.mz = ix(np.clip(np.arange(-NG, nz + 1 + NG), 0, nz - 1))
        k = np.arange(-NG, nz + 1 + NG)
        self.inner_w = lev(((k >= 1) & (k < nz)) * 1.0)
        self.rj = self.rhob * self.jac
        self.bdy = self.sfc = None

    # neighbours: X(a, n)[.., i] = a[.., i + n]
    def X(self, a, n):
        return torch.roll(a, -n, 2)

    def Y(self, a, n):
        return torch.roll(a, -n, 1)

    def Z(self, a, n):
        return torch.roll(a, -n, 0)

    def cut(self, a, name="c"):
        return a[box(self.case, name)]

    def fill(self, f, name="c"):
        """Ghosts of the field on its box: z, then x, then y."""
        if name == "w":
            f = torch.cat([f[:self.nz], 0 * f[:1]])
            f = torch.cat([torch.stack([2 * f[0] - f[m] for m in (3, 2, 1)]), f, torch.stack([-f[self.nz - m] for m in (1, 2, 3)])])
        else:
            f = f[self.mz]
        f = f[:, :, self.mxu if name == "u" else self.mx]
        return f[:, self.myv if name == "v" else self.my]

    def initial(self):
        """The set-up's own state (its bubble apart, which no case has), boxes in numpy."""
        nx, ny, nz = self.nx, self.ny, self.nz
        s = {k: np.zeros([c.stop - c.start for c in box(self.case, k)]) for k in FIELDS}
        s["u"] += self.ub_np[NG:NG + nz, None, None]
        if self.moist:
            s["qv"] += self.qvb_np[box(self.case, "c")]
        return s

    def face(self, S, q, vel):
        """5th-order upwind value on the lower face of q's points, S the shift along the axis."""
        a, b, c, d, e, f = S(q, -3), S(q, -2), S(q, -1), q, S(q, 1), S(q, 2)
        cen = 37 * (c + d) - 8 * (b + e) + (a + f)
        upw = (f - a) - 5 * (e - b) + 10 * (d - c)
        return vel * torch.where(vel >= 0, cen - upw, cen + upw) / 60

    def tendencies(self, s, dt, tf):
        """Slow tendencies on padded arrays of the filled state s."""
        X, Y, Z = self.X, self.Y, self.Z
        u, v, w = s["u"], s["v"], s["w"]
        mx, my = 0.5 * (X(self.rj, -1) + self.rj) * u, 0.5 * (Y(self.rj, -1) + self.rj) * v
        uw = 0.25 * (Z(u, -1) + X(Z(u, -1), 1) + u + X(u, 1))
        vw = 0.25 * (Z(v, -1) + Y(Z(v, -1), 1) + v + Y(v, 1))
        mz = self.inner_w * self.rhobw * (w - (uw * self.hx + vw * self.hy) * (1 - self.zw / self.zt))
        div = (X(mx, 1) - mx) / self.dx + (Y(my, 1) - my) / self.dy + (Z(mz, 1) - mz) / self.dzc

        def flux_div(F, dz, axes):
            # axes: the shifts from the lower to the upper face of the point along x, y, z
            (Sx, Sy, Sz), (fx, fy, fz) = axes, F
            return (Sx(fx) - fx) / self.dx + (Sy(fy) - fy) / self.dy + (Sz(fz) - fz) / dz

        up = (lambda a: X(a, 1), lambda a: Y(a, 1), lambda a: Z(a, 1))
        t = {}
        # u: the face fluxes averaged to u's own cell
        fx, fy, fz = 0.5 * (X(mx, -1) + mx), 0.5 * (X(my, -1) + my), 0.5 * (X(mz, -1) + mz)
        F = self.face(X, u, fx), self.face(Y, u, fy), self.face(Z, u, fz)
        va = 0.25 * (X(v, -1) + X(Y(v, 1), -1) + v + Y(v, 1))
        t["u"] = (-flux_div(F, self.dzc, up) + u * 0.5 * (X(div, -1) + div)) / (0.5 * (X(self.rj, -1) + self.rj)) + self.fcor * va - self.sc * (u - self.ub)
        fx, fy, fz = 0.5 * (Y(mx, -1) + mx), 0.5 * (Y(my, -1) + my), 0.5 * (Y(mz, -1) + mz)
        F = self.face(X, v, fx), self.face(Y, v, fy), self.face(Z, v, fz)
        ua = 0.25 * (Y(u, -1) + Y(X(u, 1), -1) + u + X(u, 1))
        t["v"] = (-flux_div(F, self.dzc, up) + v * 0.5 * (Y(div, -1) + div)) / (0.5 * (Y(self.rj, -1) + self.rj)) - self.fcor * (ua - self.ub) - self.sc * v
        fx, fy, fz = 0.5 * (Z(mx, -1) + mx), 0.5 * (Z(my, -1) + my), 0.5 * (Z(mz, -1) + mz)
        F = self.face(X, w, fx), self.face(Y, w, fy), self.face(Z, w, fz)
        t["w"] = (-flux_div(F, self.dzw, up) + w * 0.5 * (Z(div, -1) + div)) / (self.rhobw * self.jac) - self.sw * w
        if self.damp:
            cr = w.abs() * dt / (self.dzw * self.jac)
            t["w"] = t["w"] - torch.where(cr > 1, 0.3 * (cr - 1) * w / dt, 0 * w)
        for k in ("thp", "qv", "qc", "qr") if self.moist else ("thp",):
            q = s[k]
            F = self.face(X, q, mx), self.face(Y, q, my), self.face(Z, q, mz)
            if self.pd and k != "thp":
                out = sum((S(f).clamp(min=0) + (-f).clamp(min=0)) / d for S, f, d in zip(up, F, (self.dx, self.dy, self.dzc)))
                r = torch.where(dt * out > 1e-20, self.rj * q.clamp(min=0) / (dt * out).clamp(min=1e-20), torch.ones_like(q)).clamp(max=1)
                r = self.fill(self.cut(r))
                F = tuple(f * torch.where(f >= 0, S(r, -1), r) for S, f in zip((X, Y, Z), F))
            t[k] = (-flux_div(F, self.dzc, up) + q * div) / self.rj
            if k == "thp":
                t[k] = t[k] - self.sc * q
        if self.K:
            for k in ("u", "v", "w", "thp"):
                f, dz = s[k], (self.dzw if k == "w" else self.dzc) * self.jac
                t[k] = t[k] + self.K * sum((S(f, 1) - 2 * f + S(f, -1)) / d ** 2 for S, d in ((X, self.dx), (Y, self.dy), (Z, dz)))
        t["pip"] = torch.zeros_like(u)
        if self.bdy:
            for k, target in self.bdy["targets"].items():
                t[k] = t[k] + self.bdy["weight"] * (target - s[k])
        return t

    def acoustic(self, n, t, dtau, ns):
        """ns acoustic substeps from the filled state n under the tendencies t: the boxes of u v w theta' pi'."""
        X, Y, Z, cut, nz = self.X, self.Y, self.Z, self.cut, self.nz
        u, v, w, th, pi, prev = n["u"], n["v"], cut(n["w"], "w"), n["thp"], n["pip"], n["pip"]
        mask = torch.zeros_like(u)
        mask[box(self.case, "c")] = 1.0
        pad = lambda a: torch.nn.functional.pad(a, (NG, NG, NG, NG, NG, NG + 1))  # noqa: E731
        c1, c2 = (1 + self.beta) / 2, (1 - self.beta) / 2
        moisture = 1 + EPS * n["qv"] if self.moist else 1.0
        dzc2 = Z(self.zc, 1) - Z(self.zc, -1)
        fc, fw = 1 - self.zc / self.zt, 1 - self.zw / self.zt
        jac, hx, hy = (cut(a.expand_as(u))[:1] for a in (self.jac, self.hx, self.hy))
        aw, kt, dthb = cut(self.aw), cut(self.kt3), cut(self.dthb)
        dzc = self.dzc[NG:NG + nz]
        inner = slice(1, nz)
        mid = lambda a: 0.5 * (a[:-1] + a[1:])  # noqa: E731
        thbw, dzw = cut(self.thbw)[inner], self.dzw[NG + 1:NG + nz]
        vap = 1.0
        buoy_q = 0.0
        if self.moist:
            q, c, r, b = (cut(a) for a in (n["qv"], n["qc"], n["qr"], self.qvb))
            vap = 1 + EPS * mid(q)
            buoy_q = G * (EPS * (mid(q) - mid(b)) - (mid(c) + mid(r)))
        rows = lambda a, name, lo: a[NG:NG + nz, NG:NG + self.ny + (lo == "y"), NG:NG + self.nx + (lo == "x")]  # noqa: E731
        for _ in range(ns):
            ps = pi + self.smdiv * (pi - prev)
            thv = (self.thb + th) * moisture
            grad = lambda S, d, slope: (ps - S(ps, -1)) / d - slope * fc / (0.5 * (S(self.jac, -1) + self.jac)) * 0.5 * (  # noqa: E731
                (S(Z(ps, 1), -1) - S(Z(ps, -1), -1)) + (Z(ps, 1) - Z(ps, -1))) / dzc2
            un = u + dtau * (-CP * 0.5 * (X(thv, -1) + thv) * grad(X, self.dx, self.hxu) + t["u"])
            vn = v + dtau * (-CP * 0.5 * (Y(thv, -1) + thv) * grad(Y, self.dy, self.hyv) + t["v"])
            ub, vb = un[NG:NG + nz, NG:NG + self.ny, NG:NG + self.nx], vn[NG:NG + nz, NG:NG + self.ny, NG:NG + self.nx]
            if self.ox:
                lo, hi = rows(u, "u", "x")[:, :, 0], rows(u, "u", "x")[:, :, self.nx]
                ref = self.ub[NG:NG + nz, :, 0]
                lo = torch.where(lo >= 0, ref.expand_as(lo), lo - dtau * (lo - self.cstar) * (ub[:, :, 1] - lo) / self.dx)
                hi = torch.where(hi <= 0, ref.expand_as(hi), hi - dtau * (hi + self.cstar) * (hi - ub[:, :, -1]) / self.dx)
                ub = torch.cat([lo[:, :, None], ub[:, :, 1:], hi[:, :, None]], 2)
            else:
                ub = torch.cat([ub, ub[:, :, :1]], 2)
            if self.oy:
                lo, hi = rows(v, "v", "y")[:, 0], rows(v, "v", "y")[:, self.ny]
                lo = torch.where(lo >= 0, 0 * lo, lo - dtau * (lo - self.cstar) * (vb[:, 1] - lo) / self.dy)
                hi = torch.where(hi <= 0, 0 * hi, hi - dtau * (hi + self.cstar) * (hi - vb[:, -1]) / self.dy)
                vb = torch.cat([lo[:, None], vb[:, 1:], hi[:, None]], 1)
            else:
                vb = torch.cat([vb, vb[:, :1]], 1)
            u, v = self.fill(ub, "u"), self.fill(vb, "v")
            # w - pi' columns: A on levels 0..nz, zero at both ends
            zero = torch.zeros_like(aw[:1])
            A = torch.cat([zero, aw[inner], zero])
            uc, vc = ub[:, :, :-1] + ub[:, :, 1:], vb[:, :-1] + vb[:, 1:]
            S = torch.cat([zero, aw[inner] * (0.5 * mid(uc) * hx + 0.5 * mid(vc) * hy) * fw[NG + 1:NG + nz], zero])
            Fx, Fy = rows(self.rtjx, "u", "x") * ub, rows(self.rtjy, "v", "y") * vb
            Dh = (Fx[:, :, 1:] - Fx[:, :, :-1]) / self.dx + (Fy[:, 1:] - Fy[:, :-1]) / self.dy
            p0, th0 = cut(pi), cut(th)
            P = p0 + dtau * cut(t["pip"]) - dtau * kt * (Dh - (S[1:] - S[:-1]) / dzc + c2 * (A[1:] * w[1:] - A[:-1] * w[:-1]) / dzc)
            E = dtau * kt * c1 / dzc
            thvw = (thbw + mid(th0)) * vap
            Gk = dtau * CP * thvw * c1 / (jac * dzw)
            lower, upper = -Gk * E[:-1] * A[:nz - 1], -Gk * E[1:] * A[2:]
            diag = 1 + Gk * A[1:nz] * (E[1:] + E[:-1])
            rhs = w[inner] + dtau * (G * mid(th0) / thbw + buoy_q + cut(t["w"])[inner]) - dtau * CP * thvw * c2 * (p0[1:] - p0[:-1]) / (jac * dzw)
            D = rhs - Gk * (P[1:] - P[:-1])
            cs, ds = [upper[0] / diag[0]], [D[0] / diag[0]]
            for k in range(1, nz - 1):
                m = diag[k] - lower[k] * cs[-1]
                cs.append(upper[k] / m)
                ds.append((D[k] - lower[k] * ds[-1]) / m)
            W, above = [], torch.zeros_like(ds[0])
            for c, d in zip(reversed(cs), reversed(ds)):
                above = d - c * above
                W.append(above)
            bottom = 0.5 * uc[0] * hx[0] + 0.5 * vc[0] * hy[0]
            w = torch.stack([bottom] + W[::-1] + [torch.zeros_like(bottom)])
            pib = P - E * (A[1:] * w[1:] - A[:-1] * w[:-1])
            thn = th0 + dtau * (cut(t["thp"]) - mid(w) * dthb)
            prev = torch.where(mask > 0, pi, n["pip"])
            th = torch.where(mask > 0, pad(thn), n["thp"])
            pi = self.fill(pib)
        return {"u": ub, "v": vb, "w": w, "thp": thn, "pip": pib}

    def step(self, s, rain, t):
        """One large step of the boxes s."""
        n = {k: self.fill(v, k) for k, v in s.items()}
        est = n
        for dts, ns in ((self.dt / 3, 1), (self.dt / 2, 3), (self.dt, 6)):
            tend = self.tendencies(est, self.dt, t)
            x = self.acoustic(n, tend, dts / ns, ns)
            for k in ("qv", "qc", "qr"):
                x[k] = s[k] + dts * self.cut(tend[k]) if self.moist else s[k]
            est = {k: self.fill(v, k) for k, v in x.items()}
        if self.moist:
            x, rain = self.kessler(x, rain)
        if self.sfc:
            x = self.surface(x, t + self.dt)
        return x, rain

    def qsat(self, p, T, ice):
        a, b = (21.875, 7.66) if ice else (17.269, 35.86)
        es = 610.78 * torch.exp(a * (T - 273.16) / (T - b))
        return 0.622 * es / (p - es).clamp(min=1.0)

    def kessler(self, s, rain):
        cut, nz, dt = self.cut, self.nz, self.dt
        rho, pi, thb = cut(self.rhob), cut(self.pib) + s["pip"], cut(self.thb)
        T = (thb + s["thp"]) * pi
        dz = self.dzc[NG:NG + nz] * cut(self.jac.expand_as(self.thb))
        slow = torch.where(T < 273.15, 0.35, 1.0)
        speed = lambda rq: torch.where(rq > 1e-9, 36.34 * rq.clamp(min=1e-9) ** 0.1364 * torch.sqrt(rho[:1] / rho) * slow, 0 * rq)  # noqa: E731
        # selections as the branches of the model make them, at equality too: the gradients need that
        pos = lambda a: torch.where(a > 0, a, 0 * a)  # noqa: E731
        least = lambda a, b: torch.where(a > b, b, a)  # noqa: E731
        qr = pos(s["qr"])
        vr = speed(rho * qr)
        nsub = 1 + torch.floor(vr.detach().amax(0) * dt / (0.8 * dz.amin(0)))
        dts = dt / nsub
        acc = torch.zeros_like(rain)
        for b in range(int(nsub.max())):
            on = b < nsub
            flux = rho * qr * vr
            acc = acc + torch.where(on, dts * flux[0], 0 * dts)
            top = torch.cat([flux[1:], 0 * flux[:1]])
            qr = torch.where(on, qr + dts * (top - flux) / (rho * dz), qr)
            vr = torch.where(b + 1 < nsub, speed(rho * pos(qr)), vr)
        p = P00 * pi ** (CP / RD)
        blend = lambda T: ((T - 233.15) / 40).clamp(0, 1)  # noqa: E731

        def sat(T):
            f = blend(T)
            return f * self.qsat(p, T, False) + (1 - f) * self.qsat(p, T, True)

        f, qs = blend(T), sat(T)
        L = f * LV + (1 - f) * LS
        qv, qc, qr = pos(s["qv"]), pos(s["qc"]), pos(qr)
        d = least(dt * (0.001 * pos(qc - 0.001) + 2.2 * qc * torch.where(qr > 1e-9, qr, 1e-9 + 0 * qr) ** 0.875), qc)
        qc, qr = qc - d, qr + d
        dry = (qv < qs) & (qr > 0)
        rq = rho * torch.where(dry, qr, torch.ones_like(qr))
        ern = (1.6 + 124.9 * rq ** 0.2046) * rq ** 0.525 / (2.55e8 / (p * qs) + 5.4e5) * (qs - qv) / (rho * qs)
        e = torch.where(dry, least(least(dt * ern, qr), qs - qv), 0 * qr)
        qr, qv = qr - e, qv + e
        th = s["thp"] - L * e / (CP * pi)
        T = torch.where(dry, (thb + th) * pi, T)
        qs = torch.where(dry, sat(T), qs)
        dq = (qv - qs) / (1 + L * L * qs / (CP * RV * T * T))
        dq = torch.where(dq < 0, -least(-dq, qc), dq)
        out = dict(s, thp=th + L * dq / (CP * pi), qv=pos(qv - dq), qc=pos(qc + dq), qr=pos(qr))
        return out, rain + acc

    # ---------------------------------------- lateral relaxation, surface
    def set_region(self, own, inputs):
        nx, ny = self.nx, self.ny
        self.bdy = {"targets": {k: self.t(padded(self.case, k, own[k])) for k in ("u", "v", "thp", "pip", "qv")}}
        i, j = np.minimum(np.arange(nx), np.arange(nx)[::-1]), np.minimum(np.arange(ny), np.arange(ny)[::-1])
        d = np.minimum(j[:, None], i[None])
        wgt = np.where(d < 5, np.cos(1.5707963267948966 * d / 5) ** 2 / 600.0, 0.0)
        self.bdy["weight"] = self.t(np.pad(wgt, NG, mode="edge"))[None]
        self.sfc = {k: self.t(v) for k, v in inputs.items()}
        self.sfc.update(tdeep=self.sfc["tsk"], soil=[self.sfc["tsk"]] * 4)

    def diffuse(self, phi, rho, rhow, dzc, dzw, K, source, cg=None):
        """Implicit vertical mixing; K on the inner w levels."""
        n, dt = self.nz, self.dt
        a = rhow[1:] * K / dzw[1:]
        m = rho * dzc / dt
        zero = torch.zeros_like(a[:1])
        B = m + torch.cat([zero, a]) + torch.cat([a, zero])
        D = m * phi
        if cg is not None:
            D = D + torch.cat([zero, cg]) - torch.cat([cg, zero])
        D[0] += source
        b, d = [B[0]], [D[0]]
        for k in range(1, n):
            f = -a[k - 1] / b[-1]
            b.append(B[k] + f * a[k - 1])
            d.append(D[k] - f * d[-1])
        x = [d[-1] / b[-1]]
        for k in range(n - 2, -1, -1):
            x.append((d[k] + a[k] * x[-1]) / b[k])
        return torch.stack(x[::-1])

    def surface(self, s, t):
        cut, nz, dt, sf = self.cut, self.nz, self.dt, self.sfc
        sigma, kappa = 5.67e-8, 0.4
        J = cut(self.jac.expand_as(self.thb))
        rho, rhow, pi = cut(self.rhob), cut(self.rhobw), cut(self.pib) + s["pip"]
        dzc, dzw = self.dzc[NG:NG + nz] * J, self.dzw[NG:NG + nz] * J
        zc, zw = self.zc[NG:NG + nz] * J, self.zw[NG:NG + nz] * J
        uc, vc = 0.5 * (s["u"][:, :, :-1] + s["u"][:, :, 1:]), 0.5 * (s["v"][:, :-1] + s["v"][:, 1:])
        th, qv = cut(self.thb) + s["thp"], s["qv"]
        thv = th * (1 + EPS * qv)
        du, dl = rho * qv * dzc, rho * s["qc"].clamp(min=0) * dzc * 1000
        lwp = dl.sum(0)
        # surface layer
        land = sf["land"] > 0.5
        wet = ((sf["soilw"] - 0.08) / (0.32 - 0.08)).clamp(0, 1)
        z0 = torch.where(land, 0 * wet + 0.1, 0 * wet + 2e-4)
        alb = torch.where(land, 0 * wet + 0.2, 0 * wet + 0.08)
        beta = torch.where(land, (wet * wet).clamp(min=0.05), 0 * wet + 1)
        z1, V = 0.5 * dzc[0], torch.sqrt(uc[0] ** 2 + vc[0] ** 2).clamp(min=0.5)
        p1, Ts = P00 * pi[0] ** (CP / RD), sf["tsk"]
        ths = Ts / (pi[0] + G * z1 / (CP * thv[0]))
        qss = self.qsat(p1, Ts, False)
        thvs = ths * (1 + EPS * (beta * qss + (1 - beta) * qv[0]))
        Rib = G * z1 * (thv[0] - thvs) / (thvs * V * V)
        ln = torch.log(z1 / z0)
        a2 = (kappa / ln) ** 2
        sq = torch.sqrt((-Rib).clamp(min=0) * z1 / z0)
        stable = 1 / (1 + 4.7 * Rib.clamp(min=0)) ** 2
        Fm = torch.where(Rib < 0, 1 - 9.4 * Rib / (1 + 7.4 * 9.4 * a2 * sq), stable)
        Fh = torch.where(Rib < 0, 1 - 9.4 * Rib / (1 + 5.3 * 9.4 * a2 * sq), stable)
        Cd, Ch = a2 * Fm, a2 * Fh
        cdv = Cd * V

        def psi(zeta, heat):
            x = (1 - 16 * zeta.clamp(max=0)) ** 0.25
            if heat:
                un = 2 * torch.log((1 + x * x) / 2)
            else:
                un = 2 * torch.log((1 + x) / 2) + torch.log((1 + x * x) / 2) - 2 * torch.atan(x) + math.pi / 2
            return torch.where(zeta >= 0, -5 * zeta.clamp(max=2), un)

        zeta = torch.where(Rib >= 0, Rib * ln / (1 - 5 * Rib.clamp(max=0.19)), Rib * ln).clamp(-8, 2)
        zol = zeta / z1
        r10 = ((torch.log(10 / z0) - psi(10 * zol, 0) + psi(z0 * zol, 0)) / (ln - psi(zeta, 0) + psi(z0 * zol, 0)).clamp(min=0.1)).clamp(0, 1.2)
        zh = 0.1 * z0
        r2 = ((torch.log(2 / zh) - psi(2 * zol, 1) + psi(zh * zol, 1)) / (torch.log(z1 / zh) - psi(zeta, 1) + psi(zh * zol, 1)).clamp(min=0.1)).clamp(0, 1.2)
        sf["u10"], sf["t2m"] = V * r10, (ths + (th[0] - ths) * r2) * pi[0]
        shf, qflx = Ch * V * (ths - th[0]), Ch * V * beta * (qss - qv[0])
        qflx = torch.where(land, qflx, qflx.clamp(min=0))
        # radiation
        utc = (9.0 + t / 3600) % 24
        decl, lat = 0.40928 * math.sin(6.2832 * (284 + 172) / 365), sf["lat"] * 0.0174533
        cosz = (torch.sin(lat) * math.sin(decl) + torch.cos(lat) * math.cos(decl) * torch.cos(0.2618 * (utc + sf["lon"] / 15 - 12))).clamp(min=0)
        black = sigma * (th * pi) ** 4
        eps = 1 - torch.exp(-(0.22 * du + 0.30 * dl))
        dn, up = [torch.zeros_like(Ts)], None
        for k in range(nz - 1, -1, -1):
            dn.append(dn[-1] * (1 - eps[k]) + eps[k] * black[k])
        dn = torch.stack(dn[::-1])
        up = [0.97 * sigma * Ts ** 4 + 0.03 * dn[0]]
        for k in range(nz):
            up.append(up[-1] * (1 - eps[k]) + eps[k] * black[k])
        up = torch.stack(up)
        sun = 1361 * cosz * 0.95 * (1 - lwp / (lwp + 60))
        tau = torch.exp(-(0.008 * du + 0.15 * dl) / cosz.clamp(min=0.05))
        absorbed = [None] * nz
        for k in range(nz - 1, -1, -1):
            absorbed[k] = sun * (1 - tau[k])
            sun = sun * tau[k]
        heat = ((dn[1:] - dn[:-1]) + (up[:-1] - up[1:]) + torch.stack(absorbed)) / (rho * CP * dzc) / pi
        # soil
        ground = sun * (1 - alb) + 0.97 * dn[0] - 0.97 * sigma * Ts ** 4 - rho[0] * CP * shf * pi[0] - rho[0] * LV * qflx
        w4 = sf["soilw"].clamp(0, 0.4)
        Cso, Kso, depth = 1.2e6 + 3.2e6 * w4, 0.25 + 3.0 * w4, (0.1, 0.3, 0.6, 1.0)
        kl = [Kso / (0.5 * (depth[q] + depth[q + 1])) for q in range(3)] + [Kso / depth[3]]
        B = [Cso * depth[q] / dt + kl[q] + (kl[q - 1] if q else 0) for q in range(4)]
        D = [Cso * depth[q] / dt * sf["soil"][q] for q in range(4)]
        D[0], D[3] = D[0] + ground, D[3] + kl[3] * sf["tdeep"]
        for q in range(1, 4):
            f = -kl[q - 1] / B[q - 1]
            B[q], D[q] = B[q] + f * kl[q - 1], D[q] - f * D[q - 1]
        soil = [D[3] / B[3]]
        for q in (2, 1, 0):
            soil.append((D[q] + kl[q] * soil[-1]) / B[q])
        sf["soil"] = [torch.where(land, x.clamp(200, 350), o) for x, o in zip(soil[::-1], sf["soil"])]
        sf["tsk"] = torch.where(land, sf["soil"][0], Ts)
        # eddy diffusivity
        ust, wth = torch.sqrt(Cd) * V, shf * (1 + EPS * qv[0]) + EPS * th[0] * qflx
        warm = wth > 0
        ws = ust.clamp(min=0.1)
        cbrt = lambda a: a.clamp(min=0) ** (1 / 3)  # noqa: E731
        for _ in range(3):
            ths_v = thv[0] + torch.where(warm, 6.8 * wth / ws, 0 * ws)
            hp, found, prev = zc[nz - 1], torch.zeros_like(land), 0 * ws
            for k in range(1, nz):
                Rb = G * (thv[k] - ths_v) * zc[k] / (thv[0] * (uc[k] ** 2 + vc[k] ** 2 + 0.1))
                hit = (Rb >= 0.25) & ~found
                f = ((0.25 - prev) / (Rb - prev + 1e-9)).clamp(0, 1)
                hp = torch.where(hit, zc[k - 1] + f * (zc[k] - zc[k - 1]), hp)
                found, prev = found | hit, Rb
            hp = torch.maximum(hp, zc[0])
            wst = cbrt(torch.where(warm, G / thv[0] * wth * hp, 0 * ws))
            ws = cbrt(ust ** 3 + 0.6 * wst ** 3).clamp(min=0.1)
        sf["pblh"] = hp
        gth, gqv = (torch.where(warm, 6.8 * a / (ws * hp), 0 * ws) for a in (shf, qflx))
        lo, hi = slice(0, nz - 1), slice(1, nz)
        dz, z = dzw[hi], zw[hi]
        S2 = ((uc[hi] - uc[lo]) / dz) ** 2 + ((vc[hi] - vc[lo]) / dz) ** 2 + 1e-8
        Ri = G / (0.5 * (thv[lo] + thv[hi])) * (thv[hi] - thv[lo]) / dz / S2
        mix = kappa * z / (1 + kappa * z / 150)
        local = mix ** 2 * torch.sqrt(S2) * torch.where(Ri < 0, torch.sqrt(1 - 16 * Ri.clamp(max=0)), 1 / (1 + 5 * Ri.clamp(min=0)) ** 2)
        within = warm & (z < hp)
        K0 = torch.where(within, kappa * ws * z * (1 - z / hp) ** 2, local)
        cg = torch.where(within, rhow[hi] * K0, 0 * K0)
        K = K0.clamp(0.1, 1000)
        th = self.diffuse(th, rho, rhow, dzc, dzw, K, rho[0] * shf, cg * gth)
        q = self.diffuse(qv, rho, rhow, dzc, dzw, K, rho[0] * qflx, cg * gqv).clamp(min=0)
        out = dict(s, thp=th - cut(self.thb) + (dt * heat).clamp(-0.02, 0.02), qv=q)
        # momentum on the inner faces
        for name, ax in (("u", 2), ("v", 1)):
            n = self.nx if ax == 2 else self.ny
            av = lambda a: 0.5 * (a.narrow(a.dim() - 3 + ax, 0, n - 1) + a.narrow(a.dim() - 3 + ax, 1, n - 1))  # noqa: E731
            f = s[name].narrow(ax, 1, n - 1)
            mixed = self.diffuse(f, av(rho), av(rhow), self.dzc[NG:NG + nz] * av(J), self.dzw[NG:NG + nz] * av(J), av(K), -av(rho)[0] * av(cdv) * f[0])
            out[name] = torch.cat([s[name].narrow(ax, 0, 1), mixed, s[name].narrow(ax, n, 1)], ax)
        return out


def exact(case, seed):
    outs = []
    for n, m in enumerate(members(case)):
        e = Exact(m)
        own = e.initial()
        s = {k: e.t(v) for k, v in perturb(m, seed + 101 * n, own).items()}
        if m["kind"] in ("inner", "adjoint"):
            return exact_gradients(e, m, seed, s)
        if m["setup"] == "region":
            e.set_region(own, surface_inputs(m, seed + 101 * n))
        rain, dt = torch.zeros_like(s["thp"][0]), e.dt
        with torch.no_grad():
            for k in range(m["steps"]):
                s, rain = e.step(s, rain, k * dt)
        names = (FIELDS + ("rain",) if e.moist else FIELDS[:5]) + (SURFACE if e.sfc else ())
        every = dict(s, rain=rain, **(e.sfc or {}))
        # the snapshot's boxes leave out the last face
        outs.append({k: every[k][..., :m["ny"], :m["nx"]] for k in names})
    return outs


def exact_gradients(e, case, seed, s):
    """M dx by forward and M^T ybar by reverse differentiation of the steps."""
    names = FIELDS if e.moist else FIELDS[:5]
    rest = {k: s[k] for k in FIELDS if k not in names}
    rain = torch.zeros_like(s["thp"][0])

    def step(*x):
        y = e.step(dict(zip(names, x), **rest), rain, 0.0)[0]
        return tuple(y[k] for k in names)

    x, states = tuple(s[k] for k in names), []
    dx = tuple(e.t(v) for v in increment(case, seed, names).values())
    for _ in range(case["steps"]):
        states.append(x)
        if case["kind"] == "inner":
            x, dx = torch.func.jvp(step, x, dx)
        else:
            with torch.no_grad():
                x = step(*x)
    out = {"tangent": dict(zip(names, dx))} if case["kind"] == "inner" else {}
    bar = tuple(e.t(v) for v in cotangent(case, seed, names).values())
    for x in reversed(states):
        x = tuple(a.detach().requires_grad_(True) for a in x)
        g = torch.autograd.grad(step(*x), x, bar, allow_unused=True)
        bar = tuple(torch.zeros_like(a) if b is None else b for a, b in zip(x, g))
        del g
    out["adjoint"] = dict(zip(names, bar))
    return out
