"""Full RK3 steps of the CUDA path against the oracle, and the reference's
guarantees (GPU).

Tolerances (scaled error = max |diff| / max |oracle| per field):
  FP64 build vs FP64 oracle after 8 steps: <= 1e-10 (rounding only).
  FP32 build vs FP64 oracle after 8 steps: relative L2 <= 1e-4 for u, v, w,
  theta' (<= 1e-3 for pi') and max-norm <= 1e-3 of the field magnitude.
"""

import numpy as np
import pytest

import oracle as O
import wfe_b200 as W
from helpers import CASES, make_file_small, rel_l2, scaled_err

pytestmark = pytest.mark.gpu

RUN_CASES = ["bubble_open", "straka_periodic", "schaer_open", "wk82_small", "moist_blob"]
NSTEPS = 8


# The deepest column each acoustic variant holds, in FP32 and FP64 (over terrain,
# moist, without relaxation where its shared memory depends on them); forced on
# a deeper one, the tuner's pick stands.
DEEPEST = {7: (132, 66), 8: (265, 132), 9: (265, 132), 10: (167, 71), 11: (83, 47), 12: (191, 95), 13: (95, 47),
           14: (255, 127), 15: (335, 143), 16: (47, 47), 17: (95, 95), 18: (63, 63), 19: (47, 41), 20: (47, 47),
           21: (47, 47), 22: (41, 41)}


def _held(c, v):
    """whether the case's column fits variant v, which then is the one that ran"""
    fits = c.nz <= DEEPEST[v][c.precision == "f64"]
    assert (c.variants()["column"] == v) == fits, (v, c.nz, c.variants())
    return fits


def _oracle_run(name, nsteps, overrides=None):
    o = O.Case(CASES / f"{name}.ini", overrides)
    it = o.integrator()
    it.set_state(o.initial_state())
    for s in range(nsteps):
        it.step(o.dt, s * o.dt)
    return o, it


def _interior(c, a, k):
    return c.interior(a, "w" if k == "w" else "c")


@pytest.mark.parametrize("name", RUN_CASES)
def test_fp64_steps_match_oracle(name):
    o, it = _oracle_run(name, NSTEPS)
    c = W.Case(CASES / f"{name}.ini", precision="f64")
    for s in range(NSTEPS):
        c.step(c.dt, s * c.dt)
    for k in W.FIELDS:
        e = scaled_err(_interior(c, c.field(k), k), _interior(o, it.field(k), k))
        assert e <= 1e-10, (name, k, e)
    if c.moisture:
        assert scaled_err(c.rain(), it.rain().reshape(c.NY, c.NX)) <= 1e-10


@pytest.mark.parametrize("name", RUN_CASES)
def test_fp32_steps_within_tolerance(name):
    o, it = _oracle_run(name, NSTEPS)
    c = W.Case(CASES / f"{name}.ini", precision="f32")
    c.run(NSTEPS, c.dt, 0.0)
    c.sync()
    # horizontal winds are judged against the wind-speed scale (in the 2D
    # slabs v is a rounding-level field)
    speed = max(np.abs(_interior(o, it.field(k), k)).max() for k in ("u", "v"))
    for k in ["u", "v", "w", "thp", "pip"]:
        a, b = _interior(c, c.field(k), k), _interior(o, it.field(k), k)
        if np.abs(b).max() == 0:
            assert np.abs(a).max() <= 1e-6, k
            continue
        if k in ("u", "v"):
            rl2 = np.sqrt(((a - b) ** 2).mean()) / speed
            smax = np.abs(a - b).max() / speed
        else:
            rl2, smax = rel_l2(a, b), scaled_err(a, b)
        assert rl2 <= (1e-3 if k == "pip" else 1e-4), (name, k, rl2)
        assert smax <= 1e-3, (name, k, smax)


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_graph_replay_equals_direct_steps(prec):
    a = W.Case(CASES / "wk82_small.ini", precision=prec)
    b = W.Case(CASES / "wk82_small.ini", precision=prec)
    for s in range(7):
        a.step(a.dt, s * a.dt)
    b.run(7, b.dt, 0.0)
    b.sync()
    for k in W.FIELDS:
        assert np.array_equal(a.field(k), b.field(k)), k
    assert np.array_equal(a.rain(), b.rain())
    assert b.launches_per_step() > 0


def test_uv_mirror_symmetry_fp32():
    """x <-> y symmetric set-up: u(k, j, i) == v(k, i, j) to <= 2e-6 relative RMS
    (the reference gates 1e-4, tools/run_tests.py:61-78, and claims 2e-6)."""
    c = W.Case(CASES / "bubble_open.ini", precision="f32")
    c.run(40, c.dt, 0.0)
    u = c.field("u", interior=True)
    v = c.field("v", interior=True)
    rms = np.sqrt((u ** 2).mean())
    assert rms > 1e-3
    asym = np.sqrt(((u - np.transpose(v, (0, 2, 1))) ** 2).mean()) / rms
    assert asym <= 2e-6, asym


@pytest.mark.parametrize("prec,tol", [("f64", 1e-12), ("f32", 1e-6)])
def test_resting_atmosphere_over_terrain(prec, tol):
    """schaer_rest (tools/run_tests.py:83-85): no wind, terrain, stratified:
    |w| and |theta'| stay at rounding level."""
    c = W.Case(CASES / "schaer_open.ini", {"wind_u": 0, "coriolis_f": 0}, precision=prec)
    c.run(60, c.dt, 0.0)
    c.sync()
    assert c.field_absmax("w") <= tol
    assert c.field_absmax("thp") <= tol


def test_positive_definite_moisture_fp32():
    """moist_blob (tools/run_tests.py:97-98): PD transport keeps qv >= 0."""
    c = W.Case(CASES / "moist_blob.ini", precision="f32")
    c.run(200, c.dt, 0.0)
    qv = c.field("qv", interior=True)
    assert qv.min() >= -1e-9, qv.min()
    assert qv.max() > 4e-3


def test_no_spurious_precipitation():
    """Subsaturated moisture with microphysics on: no condensate, no rain."""
    c = W.Case(CASES / "moist_blob.ini", {"microphysics": "on", "qvbub_dq": 0.002},
               precision="f32")
    c.run(50, c.dt, 0.0)
    assert c.field_absmax("qc") == 0.0
    assert c.field_absmax("qr") == 0.0
    assert np.abs(c.rain()).max() == 0.0


def test_dry_mass_fp64_matches_oracle_and_is_reproducible():
    o, it = _oracle_run("straka_periodic", 4)
    c = W.Case(CASES / "straka_periodic.ini", precision="f64")
    for s in range(4):
        c.step(c.dt, s * c.dt)
    m1, m2 = c.dry_mass(), c.dry_mass()
    assert m1 == m2
    ref = o.dry_mass(it.state())
    assert abs(m1 - ref) <= 1e-12 * abs(ref)


def test_watchdog_absmax_reports_nan():
    c = W.Case(CASES / "bubble_open.ini", precision="f32")
    w = c.field("w")
    w[5, 5, 5] = np.nan
    c.set_field("w", w)
    assert c.field_absmax("w") > 1e30 or np.isnan(c.field_absmax("w"))


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_interior_transfers_roundtrip(prec):
    """Writer-layout uploads/downloads (src/io/writer.cpp:89-107) keep ghosts
    and agree with the padded transfers."""
    c = W.Case(CASES / "bubble_open.ini", precision=prec)
    rng = np.random.default_rng(3)
    for k in ("u", "w", "qv"):
        before = c.field(k)
        nzl = c.nz + 1 if k == "w" else c.nz
        a = rng.standard_normal((nzl, c.ny, c.nx)).astype(np.float32)
        c.set_field(k, a, interior=True)
        back = c.field(k, interior=True, dtype=np.float32)
        assert np.array_equal(back, a)
        pad = c.field(k)
        g = c.ng
        assert np.array_equal(pad[g:g + nzl, g:g + c.ny, g:g + c.nx].astype(np.float32), a)
        mask = np.ones(c.shape, bool)
        mask[g:g + nzl, g:g + c.ny, g:g + c.nx] = False
        assert np.array_equal(pad[mask], before[mask])


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_async_snapshot_equals_interior_download(prec):
    c = W.Case(CASES / "wk82_small.ini", precision=prec)
    c.run(3)
    names = list(W.FIELDS) + ["rain"]
    for dt in (np.float32, np.float64):
        bufs = c.snapshot_buffers(names, dtype=dt)
        c.snapshot_begin(bufs)
        c.run(2)  # steps issued after the snapshot do not change it
        c.snapshot_wait()
        c2 = None
        for k in names:
            assert bufs[k].dtype == dt
        # the state 2 steps ago: redo on a twin case for the reference values
        c2 = W.Case(CASES / "wk82_small.ini", precision=prec)
        c2.run(3 if dt is np.float32 else 5)
        for k in W.FIELDS:
            assert np.array_equal(bufs[k], c2.field(k, interior=True, dtype=dt)), k
        assert np.array_equal(bufs["rain"], c2.rain(interior=True).astype(dt))
        c2.close()
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["wk82_small", "schaer_open", "bubble_open", "straka_periodic",
                                  "ops_periodic", "moist_blob"])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_acoustic_variants_are_bit_identical(name, prec, monkeypatch):
    """The fused substep kernel that computes its tile's u, v faces itself
    (variants 7-9: three tile shapes) and the column kernel with every level's
    inputs in registers (10-15: six shapes), with ragged tiles where nx is no
    multiple of the tile width, give the same values, bit for bit, as the u, v
    kernel + shared-memory column tile kernel (variant 0)."""
    out = {}
    for v in (0, *range(7, 16)):
        monkeypatch.setenv("WFE_COLUMN_VARIANT", str(v))
        c = W.Case(CASES / f"{name}.ini", precision=prec)
        for s in range(4):
            c.step(c.dt, s * c.dt)
        c.run(3, t0=4 * c.dt)
        out[v] = {k: c.field(k) for k in W.FIELDS}
        assert c.variants()["column"] == v
        kt = c.kernel_times()  # one more step, timed per kernel: which kernels ran
        assert ("acoustic_fused" in kt) == (v in (7, 8, 9)), (v, sorted(kt))
        c.close()
    for v in range(7, 16):
        for k in W.FIELDS:
            assert np.array_equal(out[0][k], out[v][k]), (v, k)


@pytest.mark.gpu
def test_column_variant_6_is_the_first_tile_shape(monkeypatch):
    """Number 6 has no kernel of its own: it runs the first tile shape and is
    reported as that."""
    monkeypatch.setenv("WFE_COLUMN_VARIANT", "6")
    c = W.Case(CASES / "wk82_small.ini")
    c.step(c.dt, 0.0)
    assert c.variants()["column"] == 0
    c.close()


def _surface_w_error(c):
    """largest |w - (u h_x + v h_y)| of the surface points, from the run's own u
    and v (the last substep's), over the largest |u h_x| + |v h_y|"""
    g = slice(3, 3 + c.ny), slice(3, 3 + c.nx)
    u, v, w = (c.field(k)[3] for k in ("u", "v", "w"))
    us = 0.5 * (u[g] + u[3:3 + c.ny, 4:4 + c.nx])
    vs = 0.5 * (v[g] + v[4:4 + c.ny, 3:3 + c.nx])
    hx, hy = (c.metric(k).reshape(c.NY, c.NX)[g] for k in ("hx", "hy"))
    assert np.abs(vs * hy).max() > 0.1 and np.abs(us * hx).max() > 0.1
    return np.abs(w[g] - (us * hx + vs * hy)).max() / (np.abs(us * hx) + np.abs(vs * hy)).max()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("nx,ny,nz", [(16, 25, 44), (33, 20, 45), (17, 9, 31), (40, 12, 64), (9, 8, 5), (24, 6, 96),
                                      (21, 18, 41), (40, 12, 63), (19, 7, 47)])
def test_column_variants_over_a_hill_in_both_directions(nx, ny, nz, prec, monkeypatch):
    """Terrain sloping in x and in y under columns deeper and shallower than 32
    levels, ragged tiles, wind in both directions.  Every acoustic variant that
    holds the column gives the surface w = u h_x + v h_y of its own u and v
    within four roundings (the mean of the faces, the slope, a product, the
    sum), and the column above it bit for bit as the column
    tile kernel (7-15) or to rounding (the parallel solves, 16-22: relative L2
    as in test_parallel_solve_column_agrees_to_rounding)."""
    ov = {"nx": str(nx), "ny": str(ny), "nz": str(nz), "dz": "312.5", "dt": "2", "stretch": "none"}
    monkeypatch.setenv("WFE_TUNE", "0")
    eps, tol = (2.0**-53, 1e-11) if prec == "f64" else (2.0**-24, 1e-4)
    ref = {}
    for v in (0, *DEEPEST):
        monkeypatch.setenv("WFE_COLUMN_VARIANT", str(v))
        c = W.Case(CASES / "ops_open.ini", ov, precision=prec)
        c.set_field("v", c.field("v") + 15.0)
        for s in range(2):
            c.step(c.dt, s * c.dt)
        if v == 0 or _held(c, v):
            got = {k: c.field(k) for k in W.FIELDS}
            assert np.isfinite(got["w"]).all()
            assert _surface_w_error(c) <= 4 * eps, v
            ref = ref or got
            speed = np.abs(ref["u"]).max()
            for k in W.FIELDS:
                if v < 16:
                    assert np.array_equal(ref[k], got[k]), (v, k)
                elif k in ("u", "v"):
                    assert np.sqrt(((got[k] - ref[k]) ** 2).mean()) <= tol * speed, (v, k)
                else:
                    assert rel_l2(got[k], ref[k]) <= tol, (v, k)
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("moist", [True, False])
@pytest.mark.parametrize("terrain", ["gauss", "none"])
@pytest.mark.parametrize("nx,ny,nz", [(35, 9, 45), (13, 10, 44)])
def test_column_variants_under_relaxation(nx, ny, nz, terrain, moist, prec, monkeypatch):
    """Lateral relaxation adds a slow pi' tendency to the column: the register-
    held kernels (10-15) give the column tile kernel's values bit for bit, in
    steps (moist: with the step's moisture terms) and in operator-level
    substeps (moist: with the moisture fields), over a hill and on flat ground."""
    ov = {"nx": str(nx), "ny": str(ny), "nz": str(nz), "dz": "312.5", "dt": "2", "stretch": "none", "terrain": terrain,
          "profile": "wk82" if moist else "constant_N", "wind_profile": "tanh" if moist else "const",
          "wind_u": "12"}
    monkeypatch.setenv("WFE_TUNE", "0")
    ref = None
    for v in (0, *range(10, 16)):
        monkeypatch.setenv("WFE_COLUMN_VARIANT", str(v))
        c = W.Case(CASES / "ops_open.ini", ov, precision=prec)
        assert bool(c.moisture) == moist
        x = [c.field(k) for k in ("u", "v", "thp", "pip", "qv")]
        rng = np.random.default_rng(3)
        amp = (2.0, 2.0, 1.0, 1e-4, 0.0)
        c.set_boundary([a + s * rng.standard_normal(a.shape) for a, s in zip(x, amp)], x, c.bdy_weights(3, 60.0), 0.0, 60.0)
        for s in range(2):
            c.step(c.dt, s * c.dt)
        if v == 0 or _held(c, v):
            got = {k: c.field(k) for k in W.FIELDS}
            c.acoustic_substeps(c.dt / 6, 3)
            got.update({"op " + k: c.field(k, "work") for k in W.FIELDS[:5]})
            if v == 0:
                ref = got
                plain = W.Case(CASES / "ops_open.ini", ov, precision=prec)
                for s in range(2):
                    plain.step(plain.dt, s * plain.dt)
                assert not np.array_equal(plain.field("pip"), got["pip"])  # the relaxation acts
                plain.close()
            for k in got:
                assert np.array_equal(ref[k], got[k]), (v, k)
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["wk82_small", "schaer_open", "bubble_open", "straka_periodic",
                                  "ops_periodic", "moist_blob"])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_uv_variants_are_bit_identical(name, prec, monkeypatch):
    """The forward u, v kernel in column marches of two levels and of one (1 and
    3: interior points in the march, edge points -- radiation or periodic -- in
    blocks of their own; ragged tiles, terrain, moisture) and in slab-shaped
    blocks (2: 32 x 2 x 4) gives the same values, bit for bit, as in square
    blocks (0)."""
    out = {}
    for v in ("0", "1", "2", "3"):
        monkeypatch.setenv("WFE_UV_VARIANT", v)
        c = W.Case(CASES / f"{name}.ini", precision=prec)
        for s in range(3):
            c.step(c.dt, s * c.dt)
        c.run(3, t0=3 * c.dt)
        out[v] = {k: c.field(k) for k in W.FIELDS}
        assert c.variants()["uv"] == int(v)
        c.close()
    for v in ("1", "2", "3"):
        for k in W.FIELDS:
            assert np.array_equal(out["0"][k], out[v][k]), (v, k)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("bc", ["open", "periodic"])
@pytest.mark.parametrize("nx,ny,nz", [(33, 9, 10), (34, 17, 11), (7, 8, 12), (64, 5, 9), (3, 4, 8), (40, 26, 4)])
def test_uv_marches_over_a_hill(nx, ny, nz, bc, prec, monkeypatch):
    """The column marches of the forward u, v step (1: two levels, 3: one) at the
    edges of their 32 x 8 tiles and level pairs, with terrain sloping in x and y,
    moisture, open and periodic boundaries, down to grids of the ghost width and
    two interior levels: the same values, bit for bit, as the thread-per-face kernel (0)."""
    ov = {"nx": str(nx), "ny": str(ny), "nz": str(nz), "dz": "500", "dt": "2", "stretch": "none", "bc_x": bc, "bc_y": bc}
    out = {}
    for v in ("0", "1", "2", "3"):
        monkeypatch.setenv("WFE_UV_VARIANT", v)
        c = W.Case(CASES / "ops_open.ini", ov, precision=prec)
        for s in range(2):
            c.step(c.dt, s * c.dt)
        out[v] = {k: c.field(k) for k in W.FIELDS}
        assert c.variants()["uv"] == int(v)
        c.close()
    assert np.isfinite(out["0"]["u"]).all()
    for v in ("1", "2", "3"):
        for k in W.FIELDS:
            assert np.array_equal(out["0"][k], out[v][k]), (v, k)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["wk82_small", "schaer_open", "straka_periodic", "bubble_open"])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_tendency_variants_are_bit_identical(name, prec, monkeypatch):
    """The fused (0) and split (1) tendency kernels, the variant with
    TMA-staged scalar tiles (2: each face flux computed once) and the fused
    kernel with two cells per thread (3) give the same values, bit for bit."""
    ov = {"pd_moist": "off"} if name == "wk82_small" else None
    out = {}
    for v in ("0", "1", "2", "3"):
        monkeypatch.setenv("WFE_TEND_VARIANT", v)
        c = W.Case(CASES / f"{name}.ini", overrides=ov, precision=prec)
        for s in range(4):
            c.step(c.dt, s * c.dt)
        out[v] = {k: c.field(k) for k in W.FIELDS}
        c.close()
    for v in ("1", "2", "3"):
        for k in W.FIELDS:
            assert np.array_equal(out["0"][k], out[v][k]), (v, k)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["wk82_small", "moist_blob", "ops_open", "ops_periodic", "file_small"])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_tendency_variants_bit_identical_with_limiter_and_relaxation(name, prec, monkeypatch, tmp_path):
    """The fused (0), split (1) and two-cells-per-thread (3) tendency kernels
    where the TMA variant does not run: positive-definite moisture (limited
    fluxes with the upwind cells' outflow ratios, at open and periodic edges),
    diffusion, Davies relaxation and surface physics (the file-mode case)."""
    ini = make_file_small(tmp_path) if name == "file_small" else CASES / f"{name}.ini"
    out = {}
    for v in ("0", "1", "3"):
        monkeypatch.setenv("WFE_TEND_VARIANT", v)
        c = W.Case(ini, precision=prec)
        for s in range(6):
            c.step(c.dt, s * c.dt)
        out[v] = {k: c.field(k) for k in W.FIELDS}
        c.close()
    for v in ("1", "3"):
        for k in W.FIELDS:
            assert np.array_equal(out["0"][k], out[v][k]), (v, k)


@pytest.mark.gpu
def test_tuned_variants_are_kept_by_terrain_and_tables(monkeypatch, tmp_path):
    """Cases of one grid and physics on flat ground, on flat ground without the
    per-level tables and over a hill are tuned each for itself: the kernels'
    ranking differs, and a pick is kept on disk."""
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("WFE_TUNE_CACHE", str(cache))
    keys = []
    for terrain, tables in (("none", "1"), ("none", "0"), ("gauss", "1"), ("none", "1")):
        monkeypatch.setenv("WFE_LEVEL_TABLES", tables)
        c = W.Case(CASES / "ops_open.ini", {"nx": "29", "ny": "11", "terrain": terrain})
        c.step(c.dt, 0.0)
        var = c.variants()
        c.close()
        line = cache.read_text().splitlines()[-1].split()
        keys.append(line[0])
        if len(keys) < 4:
            assert [int(x) for x in line[1:3]] == [var["tendencies"], var["column"]] and int(line[4]) == var["uv"]
    assert len(cache.read_text().splitlines()) == len(set(keys)) == 3


@pytest.mark.gpu
def test_moisture_terms_take_one_field_of_memory():
    """A moist case holds one field more than a dry one of its grid, the second
    of the column's moisture terms (the first lies where only the fused substep
    keeps theta')."""
    import torch

    used = {}
    for profile in ("constant_N", "wk82", "constant_N", "wk82"):  # the first pair warms the context up
        before = torch.cuda.mem_get_info()[0]
        c = W.Case(CASES / "ops_open.ini", {"nx": "152", "ny": "150", "nz": "50", "dz": "300", "stretch": "none",
                                            "profile": profile, "wind_profile": "const", "pd_moist": "off"})
        c.step(c.dt, 0.0)
        c.sync()
        used[profile] = before - torch.cuda.mem_get_info()[0]
        c.close()
    field = 4 * 160 * 156 * 57
    assert used["wk82"] - used["constant_N"] < 1.6 * field, used


@pytest.mark.gpu
def test_watchdog_absmax_begin_end_matches_blocking_call():
    """The non-blocking watchdog (two page-locked slots, read one step behind)
    returns exactly what the blocking field_absmax returns for each step."""
    c = W.Case(CASES / "wk82_small.ini", precision="f32")
    seen = []
    for s in range(1, 5):
        c.run(1, c.dt, (s - 1) * c.dt)
        c.absmax_begin("w", s & 1)
        ref = c.field_absmax("w")
        seen.append((s, ref))
        if s > 1:
            assert c.absmax_end((s - 1) & 1) == seen[-2][1]
    assert c.absmax_end(4 & 1) == seen[-1][1]
    c.close()


@pytest.mark.gpu
def test_cases_of_different_depths_share_the_kernels(monkeypatch):
    """A shallower case set up after a deeper one must not lower the shared-
    memory limit of the kernels the deeper case launches (FP64 column tiles
    of 30 levels need more than the default 48 KB)."""
    monkeypatch.setenv("WFE_COLUMN_VARIANT", "0")
    deep = {"nz": "30"}
    a = W.Case(CASES / "bubble_open.ini", deep, precision="f64")
    ref = W.Case(CASES / "bubble_open.ini", deep, precision="f64")
    ref.run(2)
    ref.sync()
    shallow = W.Case(CASES / "bubble_open.ini", {"nz": "8"}, precision="f64")
    shallow.run(2)
    shallow.sync()
    for s in range(2):
        a.step(a.dt, s * a.dt)
    for k in W.FIELDS:
        assert np.array_equal(a.field(k), ref.field(k)), k
    for c in (a, ref, shallow):
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["wk82_small", "schaer_open", "moist_blob"])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_pipelined_parallel_solve_equals_parallel_solve(name, prec, monkeypatch):
    """The pipelined parallel-solve column kernels with 16 level lanes
    (variants 19-21: tiles streamed into shared memory by a producer warp)
    evaluate the parallel-solve kernel's expressions (variant 16) on the same
    values: the same fields, bit for bit, after five steps."""
    out = {}
    for v in ("16", "19", "20", "21"):
        monkeypatch.setenv("WFE_COLUMN_VARIANT", v)
        c = W.Case(CASES / f"{name}.ini", precision=prec)
        c.run(5, c.dt, 0.0)
        c.sync()
        out[v] = {k: c.field(k) for k in W.FIELDS}
        c.close()
    for v in ("19", "20", "21"):
        for k in W.FIELDS:
            assert np.array_equal(out["16"][k], out[v][k]), (v, k)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["wk82_small", "moist_blob", "bubble_open", "schaer_open"])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_level_tables_equal_fields(name, prec, monkeypatch):
    """On flat ground the column coefficients (rtjx, rtjy, aw, kt3, theta_b^w,
    dtheta_b/dz, qv_b) and the base state hold one value per level: the
    register-held column kernels (10-15) and the pipelined parallel solves
    (19-22) read the coefficients from per-level tables instead of a field of
    each, and the mass-flux, Kessler and u, v kernels the base state
    (thb, pib, rhob, rhobw).  The same fields, bit for bit, as from the 3D
    fields (WFE_LEVEL_TABLES=0) after five steps, for those variants and the
    plain column tile (0).  With terrain (schaer_open) no table is built."""
    for v in ("0", "10", "11", "12", "13", "14", "15", "19", "20", "21", "22"):
        monkeypatch.setenv("WFE_COLUMN_VARIANT", v)
        out = {}
        for prof in ("1", "0"):
            monkeypatch.setenv("WFE_LEVEL_TABLES", prof)
            c = W.Case(CASES / f"{name}.ini", precision=prec)
            c.run(5, c.dt, 0.0)
            c.sync()
            out[prof] = {k: c.field(k) for k in W.FIELDS}
            var = c.variants()
            assert var["column"] == int(v)
            assert var["level_tables"] == (prof == "1" and name != "schaer_open"), (v, var)
            assert var["base_tables"] == (prof == "1" and name != "schaer_open"), (v, var)
            c.close()
        for k in W.FIELDS:
            assert np.array_equal(out["1"][k], out["0"][k]), (v, k)


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [("f64", 1e-11), ("f32", 1e-4)])
def test_parallel_solve_columns_with_relaxation_and_surface_physics(prec, tol, monkeypatch, tmp_path):
    """The file-mode case (Davies relaxation, whose slow pi' tendency is one
    more box in the pipelined kernels' stages, surface physics, terrain,
    a Lambert map): the pipelined parallel-solve kernels with 16 level lanes
    (19-21) equal the parallel-solve kernel (16) bit for bit, and every
    parallel-solve variant (16-22) agrees with the Thomas kernel (0) to
    rounding after six steps (relative L2 <= 1e-11 FP64 / 1e-4 FP32)."""
    ini = make_file_small(tmp_path)
    out = {}
    for v in ("0", "16", "17", "18", "19", "20", "21", "22"):
        monkeypatch.setenv("WFE_COLUMN_VARIANT", v)
        c = W.Case(ini, precision=prec)
        c.run(6, c.dt, 0.0)
        c.sync()
        out[v] = {k: c.field(k) for k in W.FIELDS}
        c.close()
    for v in ("19", "20", "21"):
        for k in W.FIELDS:
            assert np.array_equal(out["16"][k], out[v][k]), (v, k)
    ref = out["0"]
    speed = max(np.abs(ref["u"]).max(), np.abs(ref["v"]).max(), 1e-30)
    for v in ("16", "17", "18", "22"):
        for k in W.FIELDS:
            a, b = out[v][k], ref[k]
            if k in ("u", "v"):
                err = np.sqrt(((a - b) ** 2).mean()) / speed
            else:
                err = rel_l2(a, b) if np.abs(b).max() > 0 else np.abs(a).max()
            assert err <= tol, (v, k, err)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["wk82_small", "schaer_open", "bubble_open", "straka_periodic",
                                  "ops_periodic", "moist_blob"])
@pytest.mark.parametrize("prec,tol", [("f64", 1e-11), ("f32", 1e-4)])
def test_parallel_solve_column_agrees_to_rounding(name, prec, tol, monkeypatch):
    """The column kernels with the parallel tridiagonal solve (variants 16-18:
    each level lane eliminates its own rows, cyclic reduction over the lanes;
    19-22: the same fed by the pipelined bulk-tensor-load ring) solve the
    same rows as the Thomas-sweep kernels: after seven steps the
    fields agree to rounding -- relative L2 <= 1e-11 (FP64) / 1e-4 (FP32, the
    FP32 step-parity bound against the oracle; measured up to 1.2e-5 on the
    moist convective case) of the field (u, v against the wind-speed
    scale) -- and the FP64 steps stay within 1e-10 of the FP64 oracle."""
    out = {}
    variants = ["0"] + [v for v in ("16", "17", "18", "19", "20", "21", "22")]
    for v in variants:
        monkeypatch.setenv("WFE_COLUMN_VARIANT", v)
        c = W.Case(CASES / f"{name}.ini", precision=prec)
        c.run(7, c.dt, 0.0)
        c.sync()
        out[v] = {k: c.field(k) for k in W.FIELDS}
        kt = c.kernel_times()
        assert "acoustic_column" in kt
        c.close()
    ref = out["0"]
    speed = max(np.abs(ref["u"]).max(), np.abs(ref["v"]).max(), 1e-30)
    for v in variants[1:]:
        for k in W.FIELDS:
            a, b = out[v][k], ref[k]
            if k in ("u", "v"):
                err = np.sqrt(((a - b) ** 2).mean()) / speed
            else:
                err = rel_l2(a, b) if np.abs(b).max() > 0 else np.abs(a).max()
            assert err <= tol, (v, k, err)
    if prec == "f64":
        o, it = _oracle_run(name, 7)
        for k in W.FIELDS:
            c = W.Case(CASES / f"{name}.ini", precision="f64", device=-1)
            e = scaled_err(_interior(c, out["16"][k], k), _interior(o, it.field(k), k))
            c.close()
            assert e <= 1e-10, (k, e)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("nx,ny,nz", [(18, 18, 12), (61, 40, 40), (70, 41, 90)])
def test_padded_transfers_roundtrip(nx, ny, nz, prec):
    """A padded upload converted by one thread and by several (fields of 0.1, 1.2
    and 2.7 MB) and its download give every point back, ghosts included."""
    ov = {"nx": str(nx), "ny": str(ny), "nz": str(nz)}
    c = W.Case(CASES / "bubble_open.ini", ov, precision=prec)
    a = np.random.default_rng(nz).standard_normal(c.shape)
    want = a if prec == "f64" else a.astype(np.float32).astype(np.float64)
    for dtype in (np.float64, np.float32):
        c.set_field("thp", a.astype(dtype))
        got = c.field("thp")
        assert np.array_equal(got, want if dtype == np.float64 else a.astype(np.float32).astype(np.float64))
    c.close()
