"""The register-held regions of the single-launch 2D solve (64 columns by 32 to
64 rows) at the sizes where their tiling can go wrong: one region exactly, one
cell more, the last size of two tiles and one more, odd sizes, shallow and deep
passes, different sweep counts of u and v, several tiles per CTA, values that
leave the range of the precomputed reciprocals.  Tolerance: exact, every value
equal to the oracle's after whole outer iterations."""
import numpy as np
import pytest

import ifc
import oracle as O
from helpers import assert_bitwise, load_both, rel_l2, seeded_state, to_oracle_cfg

pytestmark = pytest.mark.gpu


def check(cfg, iters, scale=None, seed=3):
    prec = "d" if cfg.get("precision") == "d" else "f"
    o = O.Oracle(to_oracle_cfg(cfg), prec)
    s = ifc.Solver(cfg)
    st = seeded_state(cfg, seed, s.dtype)
    if scale is not None:
        st = {k: (v * scale).astype(s.dtype) for k, v in st.items()}
    load_both(o, s, st)
    for it in range(iters):
        r = s.iterate(1)
        assert r["kernel_launches"] == 3, r  # begin, face BCs, the one cooperative launch
        o.outer_iteration()
        o.bc_face_vel()
        for k in ("u", "v", "p", "uf", "vf"):
            assert_bitwise(s.get(k), o.field(k), f"it{it} {k}")
    s.close()


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("nx,ny", [(64, 32), (65, 33), (108, 64), (109, 65), (3, 64), (152, 36), (66, 107), (31, 3)])
def test_region_edges(gpu_ok, nx, ny, prec):
    check(dict(ifc.channel2d(nx, ny), precision=prec), 2)


@pytest.mark.parametrize("ks,nu,nv,np_", [(2, 3, 5, 7), (10, 10, 10, 20), (5, 4, 11, 6), (3, 0, 2, 4), (8, 0, 0, 1)])
def test_pass_depths_and_counts(gpu_ok, ks, nu, nv, np_):
    check(dict(ifc.cavity2d(97, ny=70), sweeps_per_pass=ks, nIter_u=nu, nIter_v=nv, nIter_p=np_), 2)


@pytest.mark.parametrize("case", ["f", "d", "quick", "early_exit"])
def test_several_tiles_per_cta(gpu_ok, monkeypatch, case):
    monkeypatch.setenv("IFC_PERSIST_MAX_CTAS", "2")
    cfg = dict(ifc.channel2d(150, 101), precision="d" if case == "d" else "f")
    if case == "quick":
        cfg["convection_scheme"] = "quick"
    if case == "early_exit":  # loose tolerances: passes end before their sweeps are used up
        cfg.update(tol_u=0.3, tol_v=0.05, tol_p=0.3, sweeps_per_pass=2)
        s = ifc.Solver(cfg)
        load = seeded_state(cfg, 3, s.dtype)
        monkeypatch.setenv("IFC_PERSIST_MAX_CTAS", "148")
        t = ifc.Solver(cfg)
        for k, v in load.items():
            s.set(k, v)
            t.set(k, v)
        a, b = s.iterate(2), t.iterate(2)
        assert a["sweeps"] == b["sweeps"] and min(a["sweeps"][0], a["sweeps"][3]) < 10, (a, b)
        for k in ("u", "v", "p", "uf", "vf"):
            assert np.array_equal(s.get(k), t.get(k)), k
        return
    check(cfg, 2)


@pytest.mark.parametrize("scale", [1e-22, 1e-30, 3e-38])
def test_values_outside_the_reciprocal_range(gpu_ok, scale):
    # velocities and pressures whose quotients are tiny, subnormal or zero
    check(dict(ifc.cavity2d(70, ny=40), velBC_val=[[0.0] * 3] * 6), 2, scale=scale)


@pytest.mark.parametrize("mu", [1e-20, 1e15])
def test_diagonals_outside_the_reciprocal_range(gpu_ok, mu):
    check(dict(ifc.cavity2d(40, ny=36), dynamicViscosity=mu, density=1e-20 if mu < 1 else 1.0), 1)


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("nx,ny,sweeps,tol", [(64, 32, 23, 0.0), (65, 33, 7, 0.0), (109, 65, 60, 0.2), (24, 150, 40, 0.05)])
def test_stored_coefficient_sweeps(gpu_ok, monkeypatch, nx, ny, sweeps, tol, prec):
    """The temperature's sweeps in one launch (with the early exit in the middle
    of them) against the per-pass launches: the same temperature and counts."""
    cfg = dict(ifc.channel2d(nx, ny), precision=prec)
    rng = np.random.default_rng(5)
    state = {"uf": rng.uniform(-1e-3, 1e-3, (nx + 1) * ny), "vf": rng.uniform(-1e-3, 1e-3, nx * (ny + 1)),
             "T": rng.uniform(280, 340, nx * ny)}
    out = []
    for off in ("0", "1"):
        monkeypatch.setenv("IFC_PERSIST_OFF", off)
        s = ifc.Solver(cfg)
        for k, v in state.items():
            s.set(k, v)
        r = s.solve_energy(max_sweeps=sweeps, tol=tol)
        out.append((r["sweeps"], r["converged"], s.get("T")))
        s.close()
    assert out[0][:2] == out[1][:2] and (tol == 0.0 or out[0][0] < sweeps), [o[:2] for o in out]
    assert_bitwise(out[0][2], out[1][2], "T")


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("nx,ny,nz,bc", [(73, 12, 11, "cavity"), (77, 31, 30, "cavity"), (80, 3, 3, "cavity"), (128, 13, 14, "channel"),
                                         (151, 20, 9, "channel"), (154, 3, 40, "cavity")])
def test_3d_pressure_rows(gpu_ok, monkeypatch, nx, ny, nz, bc, prec):
    """The 3D p' solve with its row links in shared memory, at odd and even rows,
    one and two warps of cells per row, blocks of a single row, with the early
    exit in the middle, against the per-half-sweep kernels: the same p' and
    sweep count.  Tolerance: exact (the same updates in the same order)."""
    base = ifc.cavity3d(16) if bc == "cavity" else ifc.channel2d(16, 16)
    cfg = dict(base, dim=3, nx=nx, ny=ny, nz=nz, precision=prec, nIter_w=base["nIter_u"])
    for tol in (0.0, 0.3):
        out = []
        for off in ("0", "1"):
            monkeypatch.setenv("IFC_PC3D_OFF", off)
            s = ifc.Solver(dict(cfg, tol_p=tol, nIter_p=9))
            for k, v in seeded_state(cfg, 4, s.dtype).items():
                s.set(k, v)
            s.iterate(2)
            out.append([s.get(k) for k in ("pc", "p", "u", "v", "w", "uf")])
            s.close()
        for k, a, b in zip(("pc", "p", "u", "v", "w", "uf"), *out):
            assert_bitwise(a, b, f"tol {tol} {k}")


@pytest.mark.parametrize("variant", ["1", "2"])
@pytest.mark.parametrize("prec", ["f", "d"])
def test_batch_regions(gpu_ok, monkeypatch, variant, prec):
    """Batched cases of one region, one cell more, several regions per CTA and
    different sweep counts of u and v, against the oracle over a fixed number of
    outer iterations.  Tolerance: relative L2 1e-6 (every update is the oracle's;
    only an inner exit decided on differently summed norms may move)."""
    monkeypatch.setenv("IFC_BATCH_VARIANT", variant)
    cases = [ifc.channel2d(64, 32), ifc.channel2d(65, 33), ifc.channel2d(3, 70), ifc.channel2d(230, 131)]
    cases[1].update(nIter_u=3, nIter_v=11, nIter_p=7)
    cases = [dict(c, precision=prec, numOuterIter=6, tol_u=1e-12, tol_v=1e-12, tol_p=1e-12) for c in cases]
    res, fields, _ = ifc.batch_solve(cases)
    for c, r, f in zip(cases, res, fields):
        o = O.Oracle(to_oracle_cfg(dict(c, sweep_mode=O.GS_REDBLACK, check_every=r["sweeps_per_pass"])), prec)
        n, _ = o.solve()
        assert r["outer_iterations"] == n == 6
        for k in ("u", "v", "p"):
            a, b = f[k].astype(np.float64), o.field(k).astype(np.float64)
            err = np.linalg.norm(a - b) / np.linalg.norm(b)
            assert err < 1e-6, (c["nx"], c["ny"], k, err)


@pytest.mark.parametrize("nu,nv,tu,tv", [(15, 10, 2.0, 0.0), (10, 15, 0.0, 2.0), (15, 10, 0.0, 0.0), (5, 5, 2.0, 2.0)])
def test_sweep_counts_without_pressure_sweeps(gpu_ok, monkeypatch, nu, nv, tu, tv):
    """nIter_p = 0 with one component's sweeps ended early and the other's in an
    earlier pass than the last: the counts of the per-pass launches, and the
    same fields."""
    cfg = dict(ifc.channel2d(97, 70), nIter_u=nu, nIter_v=nv, nIter_p=0, tol_u=tu, tol_v=tv)
    out = []
    for off in ("0", "1"):
        monkeypatch.setenv("IFC_PERSIST_OFF", off)
        s = ifc.Solver(cfg)
        for k, v in seeded_state(cfg, 6, s.dtype).items():
            s.set(k, v)
        r = s.iterate(1)
        out.append((list(r["sweeps"]), r["cell_updates"], [s.get(k) for k in ("u", "v", "p", "uf", "vf")]))
        s.close()
    assert out[0][:2] == out[1][:2], [o[:2] for o in out]
    for a, b in zip(out[0][2], out[1][2]):
        assert_bitwise(a, b)


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("spp,every,nx,ny,cap", [(6, 6, 97, 70, 0), (7, 6, 150, 101, 2), (8, 8, 64, 64, 0), (8, 8, 150, 101, 2),
                                                 (9, 8, 33, 31, 0), (10, 10, 97, 70, 0), (16, 10, 300, 37, 3)])
@pytest.mark.parametrize("tol", [0.0, 0.3])
def test_deep_passes(gpu_ok, monkeypatch, prec, spp, every, nx, ny, cap, tol):
    """Six to sixteen sweeps per pass: one launch, and the early exit taken after
    every 6, 8 or 10 sweeps, whatever the passes are split into.  Tolerance: exact."""
    if cap:
        monkeypatch.setenv("IFC_PERSIST_MAX_CTAS", str(cap))
    cfg = dict(ifc.channel2d(nx, ny), precision=prec, sweeps_per_pass=spp, nIter_u=17, nIter_v=9, nIter_p=23, tol_u=tol,
               tol_v=tol / 3, tol_p=2 * tol)
    o = O.Oracle(dict(to_oracle_cfg(cfg), check_every=every), prec)
    s = ifc.Solver(cfg)
    load_both(o, s, seeded_state(cfg, 8, s.dtype))
    for it in range(2):
        r = s.iterate(1)
        assert r["kernel_launches"] == 3, r
        want = o.outer_iteration()["sweeps"]
        o.bc_face_vel()
        assert list(r["sweeps"]) == list(want), (it, r["sweeps"], want)
        for k in ("u", "v", "p", "uf", "vf"):
            assert_bitwise(s.get(k), o.field(k), f"it{it} {k}")
    s.close()


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("nx,ny,spp", [(33, 31, 5), (64, 20, 4), (65, 21, 4), (40, 23, 2), (29, 621, 5), (64, 28, 5), (70, 29, 5)])
def test_small_and_narrow_regions(gpu_ok, nx, ny, spp, prec):
    """Regions of 20 and 28 rows: filled exactly, one row more, and the tall
    narrow grid that takes them at the default depth."""
    check(dict(ifc.channel2d(nx, ny), precision=prec, sweeps_per_pass=spp), 2)


@pytest.mark.parametrize("prec,bound", [("f", 1e-6), ("d", 1e-11)])
def test_several_tiles_per_cta_closed(gpu_ok, monkeypatch, prec, bound):
    """Several tiles per CTA with the p' mean removal of a closed domain (150
    columns are at least three tiles, on two CTAs).  Relative L2 against the
    oracle: the values differ by the order of the mean's FP64 sum only, at most
    15150 terms times the rounding unit (FP64), less than one FP32 rounding."""
    monkeypatch.setenv("IFC_PERSIST_MAX_CTAS", "2")
    cfg = dict(ifc.cavity2d(150, ny=101), precision=prec)
    o = O.Oracle(to_oracle_cfg(cfg), prec)
    s = ifc.Solver(cfg)
    load_both(o, s, seeded_state(cfg, 3, s.dtype))
    for it in range(3):
        assert s.iterate(1)["kernel_launches"] == 3
        o.outer_iteration()
        o.bc_face_vel()
        for k in ("u", "v", "p", "uf", "vf"):
            assert rel_l2(s.get(k), o.field(k)) < bound, (it, k)


def test_several_tiles_per_cta_converged(gpu_ok, monkeypatch):
    """A cavity to convergence with several tiles per CTA (130 columns are at
    least three tiles) against one tile per CTA: the per-sweep FP64 sums are
    grouped by CTA, so only their rounding can differ."""
    cfg = ifc.cavity2d(130, ny=40)
    one = ifc.Solver(cfg)
    a = one.solve()
    monkeypatch.setenv("IFC_PERSIST_MAX_CTAS", "2")
    several = ifc.Solver(cfg)
    b = several.solve()
    assert a["converged"] and b["converged"] and abs(a["outer_iterations"] - b["outer_iterations"]) <= 2
    for k in ("u", "v"):
        assert rel_l2(several.get(k), one.get(k)) < 1e-6, k


@pytest.mark.parametrize("nx,ny,nz,prec", [(80, 128, 128, "f"), (77, 100, 103, "d")])
def test_3d_pressure_blocks(gpu_ok, monkeypatch, nx, ny, nz, prec):
    """The 3D p' solve on blocks with inner rows (ny*nz rows on at most 148 blocks:
    70 and more rows each, 10x12 and 8x9), so rows whose four neighbours are in
    shared memory, and the sweep of inner rows between the two halves of the
    grid barrier; against the per-half-sweep kernels.  Tolerance: exact."""
    cfg = dict(ifc.cavity3d(16), nx=nx, ny=ny, nz=nz, precision=prec, nIter_p=9)
    state = seeded_state(cfg, 4, np.float32 if prec == "f" else np.float64)
    for tol in (0.0, 0.3):
        out = []
        for off in ("0", "1"):
            monkeypatch.setenv("IFC_PC3D_OFF", off)
            s = ifc.Solver(dict(cfg, tol_p=tol, pin_pressure=0))
            for k, v in state.items():
                s.set(k, v)
            r = s.iterate(1)
            out.append((list(r["sweeps"]), [s.get(k) for k in ("pc", "p", "u", "v", "w", "uf")]))
            s.close()
        assert out[0][0] == out[1][0]
        for k, a, b in zip(("pc", "p", "u", "v", "w", "uf"), out[0][1], out[1][1]):
            assert_bitwise(a, b, f"tol {tol} {k}")


@pytest.mark.parametrize("prec,conv", [("f", "upwind"), ("d", "upwind"), ("d", "quick")])
@pytest.mark.parametrize("nx,ny,cap", [(32, 40, 0), (33, 40, 0), (46, 25, 0), (307, 19, 0), (64, 22, 0), (64, 64, 7), (111, 30, 5)])
def test_narrow_tiles(gpu_ok, monkeypatch, nx, ny, cap, prec, conv):
    """Tiles made narrower to use more CTAs: columns that just do not and just do
    split into tiles of twelve, an odd last tile, one row of tiles, a cap on
    the CTAs that leaves room for some of them."""
    if cap:
        monkeypatch.setenv("IFC_PERSIST_MAX_CTAS", str(cap))
    check(dict(ifc.channel2d(nx, ny), precision=prec, convection_scheme=conv), 2)
