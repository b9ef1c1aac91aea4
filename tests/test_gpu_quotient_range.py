"""Quotients outside the range in which the precomputed reciprocal of the
diagonal is used (ifc_tile2d.cuh): diagonals too large and too small for it, in
both precisions, quotients far below it, in the 2D solve and in the 3D p' solve.
Tolerance: exact -- the quotient is the division's in every range."""
import numpy as np
import pytest

import ifc
import oracle as O
from helpers import assert_bitwise, load_both, seeded_state, to_oracle_cfg

pytestmark = pytest.mark.gpu


def still(cfg, **kw):
    # without the p' mean removal, whose FP64 sum depends on the order of its terms
    return dict(cfg, velBC_val=[[0.0] * 3] * 6, pin_pressure=0, **kw)


# mu, rho, scale of the start fields.  The p' diagonal is about rho A^2 / mu: in
# the first case 1e-28 under numerators of 1e-8, whose quotients are finite.
@pytest.mark.parametrize("prec,mu,rho,scale", [("f", 1e24, 1.0, 1e-6), ("f", 1e28, 1.0, 1e-9), ("d", 1e70, 1.0, 1.0),
                                               ("d", 1e70, 1.0, 1e-20), ("d", 1e-70, 1e-70, 1.0), ("d", 0.01, 1.0, 1e-215)])
def test_2d_solve(gpu_ok, prec, mu, rho, scale):
    cfg = still(ifc.cavity2d(70, ny=40), dynamicViscosity=mu, density=rho, precision=prec)
    o = O.Oracle(to_oracle_cfg(cfg), prec)
    s = ifc.Solver(cfg)
    load_both(o, s, {k: (v * scale).astype(s.dtype) for k, v in seeded_state(cfg, 3, np.float64).items()})
    s.iterate(1)
    o.outer_iteration()
    o.bc_face_vel()
    for k in ("u", "v", "p", "uf", "vf"):
        assert np.isfinite(o.field(k)).all(), k
        assert_bitwise(s.get(k), o.field(k), k)


@pytest.mark.parametrize("prec,mu,rho,scale", [("f", 1e24, 1.0, 1e-4), ("f", 1e15, 1.0, 1.0), ("d", 1e70, 1.0, 1.0),
                                               ("d", 1e-70, 1e-70, 1.0), ("f", 0.01, 1.0, 1e-30), ("d", 0.01, 1.0, 1e-215)])
def test_3d_pressure_rows(gpu_ok, monkeypatch, prec, mu, rho, scale):
    """k_psolve3d (rows of 77 cells) against the per-half-sweep kernels."""
    cfg = still(ifc.cavity3d(16), nx=77, ny=31, nz=30, dynamicViscosity=mu, density=rho, precision=prec, nIter_p=9)
    out = []
    for off in ("0", "1"):
        monkeypatch.setenv("IFC_PC3D_OFF", off)
        s = ifc.Solver(cfg)
        for k, v in seeded_state(cfg, 4, np.float64).items():
            s.set(k, (v * scale).astype(s.dtype))
        s.iterate(1)
        out.append([s.get(k) for k in ("pc", "p", "u", "v", "w", "uf")])
        s.close()
    for k, a, b in zip(("pc", "p", "u", "v", "w", "uf"), *out):
        assert np.isfinite(b).all(), k
        assert_bitwise(a, b, k)


@pytest.mark.parametrize("prec,scale", [("f", 1e-30), ("f", 1e-36), ("f", 2e-38), ("f", 1e-41), ("d", 1e-306),
                                        ("d", 3e-308), ("d", 1e-312)])
def test_small_and_subnormal_quotients(gpu_ok, prec, scale):
    """Ordinary diagonals under numerators whose quotients are near the smallest
    normal number or below it."""
    cfg = still(ifc.cavity2d(70, ny=40), precision=prec)
    o = O.Oracle(to_oracle_cfg(cfg), prec)
    s = ifc.Solver(cfg)
    load_both(o, s, {k: (v * scale).astype(s.dtype) for k, v in seeded_state(cfg, 5, np.float64).items()})
    for it in range(2):
        s.iterate(1)
        o.outer_iteration()
        o.bc_face_vel()
        for k in ("u", "v", "p", "uf", "vf"):
            assert_bitwise(s.get(k), o.field(k), f"it{it} {k}")


@pytest.mark.parametrize("prec,iters", [("f", 3), ("d", 9)])
def test_front_from_rest(gpu_ok, prec, iters):
    """A channel flow developing from rest: the front of u, v and p' passes
    through every magnitude down to zero (FP32: 1e-45, FP64: 1e-324)."""
    cfg = dict(ifc.channel2d(900, 40), precision=prec)
    o = O.Oracle(to_oracle_cfg(cfg), prec)
    o.init_face_vel()
    o.bc_face_vel()
    s = ifc.Solver(cfg)
    for it in range(iters):
        s.iterate(1)
        o.outer_iteration()
        o.bc_face_vel()
        for k in ("u", "v", "p", "uf", "vf"):
            assert_bitwise(s.get(k), o.field(k), f"it{it} {k}")
    u = abs(o.field("u"))
    tiny = np.finfo(u.dtype).tiny
    assert (u == 0).any() and ((u > 0) & (u < tiny)).any()
