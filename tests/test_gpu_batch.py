"""The batched form (ifc_batch_solve): many independent 2D cases of uneven
size, Reynolds number and boundary type in one persistent launch, each checked
against the CPU oracle run on its own (same red-black ordering, inner
early-exit rule at the granularity the case ran with: after every sweep for
whole-row sweeps, after every pass of sweeps_per_pass sweeps for the
temporally blocked variants).  Every variant is run forced
(IFC_BATCH_VARIANT) and as chosen by the autotuner.  Tolerance: relative L2
1e-6 against the oracle with the same ordering (FP64 norms summed in a
different order can move a convergence decision by one iteration), and the
converged-solution bound of 1e-4 against the FP64 lexicographic oracle."""
import numpy as np
import pytest

import ifc
import oracle as O
from helpers import rel_l2, to_oracle_cfg

pytestmark = pytest.mark.gpu


def mixed_cases():
    cases = [ifc.cavity2d(16, re=50.0, ny=24), ifc.cavity2d(32, re=400.0), ifc.cavity2d(24, re=1000.0, ny=9),
             ifc.channel2d(40, 12), ifc.cavity2d(8, re=10.0, ny=33)]
    for c in cases:
        c["numOuterIter"] = 3000
    return cases


def oracle_fields(cfg, sweep_mode=O.GS_REDBLACK, prec="f", check_every=1):
    o = O.Oracle(to_oracle_cfg(dict(cfg, sweep_mode=sweep_mode, check_every=check_every)), prec)
    n, nm = o.solve()
    p = o.field("p").astype(np.float64)
    return n, nm, {"u": o.field("u").copy(), "v": o.field("v").copy(), "p": p}


@pytest.fixture(params=["0", "1", "2", "tuned"])
def batch_variant(request, monkeypatch):
    if request.param == "tuned":
        monkeypatch.delenv("IFC_BATCH_VARIANT", raising=False)
    else:
        monkeypatch.setenv("IFC_BATCH_VARIANT", request.param)
    return request.param


def test_batch_matches_oracle(gpu_ok, batch_variant):
    cases = mixed_cases()
    res, fields, ms = ifc.batch_solve(cases)
    assert ms > 0
    for c, r, f in zip(cases, res, fields):
        if batch_variant != "tuned":
            assert r["sweeps_per_pass"] == {"0": 1, "1": 3, "2": 5}[batch_variant]
        n, nm, ref = oracle_fields(c, check_every=r["sweeps_per_pass"])
        assert r["converged"] == nm["converged"] == 1, (r, nm)
        assert abs(r["outer_iterations"] - n) <= 1, (r["outer_iterations"], n)
        closed = all(t != ifc.OUTLET for t in c["velBC_type"][:4])
        for k in ("u", "v", "p"):
            a, b = f[k].astype(np.float64), ref[k]
            if k == "p" and closed:
                a, b = a - a.mean(), b - b.mean()
            assert rel_l2(a, b) < 1e-6, (c["nx"], c["ny"], k, rel_l2(a, b))


def test_batch_is_deterministic_and_order_independent(gpu_ok, batch_variant):
    cases = mixed_cases()
    r1, f1, _ = ifc.batch_solve(cases)
    r2, f2, _ = ifc.batch_solve(list(reversed(cases)))
    for a, b in zip(f1, reversed(f2)):
        for k in ("u", "v", "p"):
            assert np.array_equal(a[k], b[k])
    assert [x["outer_iterations"] for x in r1] == [x["outer_iterations"] for x in reversed(r2)]


def test_batch_case_against_fp64_oracle(gpu_ok):
    c = ifc.cavity2d(32, re=100.0)
    res, fields, _ = ifc.batch_solve([c])
    _, _, ref = oracle_fields(c, O.GS_LEX, "d", res[0]["sweeps_per_pass"])
    for k in ("u", "v", "p"):
        a, b = fields[0][k].astype(np.float64), ref[k]
        if k == "p":
            a, b = a - a.mean(), b - b.mean()
        assert rel_l2(a, b) < 1e-4


def test_batch_rejects_3d_and_mixed_precision():
    import ctypes as C
    cfgs = [ifc.cavity3d(8), ifc.cavity2d(8)]
    arr = (ifc.IfcConfig * 2)()
    keep = []
    for k, c in enumerate(cfgs):
        arr[k], kp = ifc.make_struct(c)
        keep.append(kp)
    res = (ifc.IfcBatchResult * 2)()
    assert ifc.load().ifc_batch_solve(arr, 2, res, None, None) == ifc.UNSUPPORTED


def loose(cfg, **kw):
    """Open domain (no p' mean, whose FP64 sum depends on the order of its terms)
    and inner tolerances that end the sweeps early, at changing places."""
    return dict(cfg, numOuterIter=3, nIter_u=13, nIter_v=11, nIter_p=23, tol_u=0.6, tol_v=0.6, tol_p=0.9,
                criterion=O.CRIT_PER_FIELD, tol_mass=0.0, **kw)


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("check", [1, 2, 3, 4, 5, 7])
def test_exit_interval_of_every_variant(gpu_ok, monkeypatch, prec, check):
    """The inner early exit after every `check` sweeps, deeper and shallower than
    the variants' passes: the oracle's sweep counts, and the same values from
    every variant.  Tolerance: exact."""
    monkeypatch.setenv("IFC_BATCH_CHECK", str(check))
    cases = [loose(c, precision=prec) for c in (ifc.channel2d(64, 32), ifc.channel2d(97, 40), ifc.channel2d(30, 70))]
    out = []
    for variant in "012":
        monkeypatch.setenv("IFC_BATCH_VARIANT", variant)
        res, fields, _ = ifc.batch_solve(cases)
        out.append((res, fields))
    ended = 0
    for k, c in enumerate(cases):
        o = O.Oracle(to_oracle_cfg(dict(c, sweep_mode=O.GS_REDBLACK, check_every=check)), prec)
        o.init_face_vel()
        o.bc_face_vel()
        done = 0
        while done < out[0][0][k]["outer_iterations"]:
            want = o.outer_iteration()["sweeps"]
            o.bc_face_vel()
            done += 1
        ended += sum(want) < 13 + 11 + 23
        for res, fields in out:
            assert res[k]["sweeps_per_pass"] == check
            assert res[k]["outer_iterations"] == done and list(res[k]["sweeps"]) == list(want), (k, res[k], want)
            for f in ("u", "v", "p"):
                assert np.array_equal(fields[k][f].ravel(), o.field(f)), (k, f)
    assert ended  # some inner solves did end early


@pytest.mark.parametrize("prec", ["f", "d"])
def test_a_case_does_not_depend_on_its_batch(gpu_ok, monkeypatch, prec):
    """The same cases in a small batch and among many others, which run them in
    other variants: the same values and counts.  Tolerance: exact."""
    monkeypatch.delenv("IFC_BATCH_VARIANT", raising=False)
    cases = [loose(c, precision=prec) for c in (ifc.channel2d(64, 40), ifc.channel2d(140, 130), ifc.channel2d(230, 131))]
    others = [loose(ifc.channel2d(150 + 3 * k, 140), precision=prec) for k in range(28)] * 5
    r1, f1, _ = ifc.batch_solve(cases)
    r2, f2, _ = ifc.batch_solve(others + cases)
    for a, b, fa, fb in zip(r1, r2[len(others):], f1, f2[len(others):]):
        assert (a["outer_iterations"], list(a["sweeps"]), a["sweeps_per_pass"]) == \
               (b["outer_iterations"], list(b["sweeps"]), b["sweeps_per_pass"])
        for f in ("u", "v", "p"):
            assert np.array_equal(fa[f], fb[f]), f
    assert any(a["tile_y"] != b["tile_y"] for a, b in zip(r1, r2[len(others):]))  # other variants did run them
