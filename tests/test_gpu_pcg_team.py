"""The PCG with one team of CTAs per model (csrc/pcg_team.cu, what auto takes
wherever every model's rows fit) against the grid-wide kernel of
B200FEM_OPT_PCG_SPLIT 1 on the same step: both end at a true relative residual
of 1e-12, so velocities agree to the condition of the solve matrix times that
(1e-8 relative holds for condition numbers up to 1e4), positions to h times
the velocities' difference (1e-9).

The sizes sit at the edges of the kernel's layout: one CTA (up to 96 rows) and
several, rows just below and above the ten-row warps, the 60-row step of the
lane rule and the 150 rows of one component set (PCG_CTAS bounds the number of
CTAs, so that a CTA takes more), teams beyond 16 and 80 members (rounds of the
partial sums), rows longer than a lane's register blocks.
"""
import numpy as np
import pytest

from artisynth_core_b200 import _lib as L
from artisynth_core_b200 import workloads as W
from artisynth_core_b200.femmodel import (FemPack, LinearMaterial, MechSystemSolver, MooneyRivlinMaterial,
                                          NeoHookeanMaterial)

from helpers import rel_err

pytestmark = pytest.mark.gpu

NH, LIN = NeoHookeanMaterial(5e4, 0.4), LinearMaterial(1e5, 0.33, True)
MR = MooneyRivlinMaterial(1000.0, 500.0, 0.0, 0.0, 0.0, 1e5)


def _beam(elem, cells, mat):
    wl = W.Workload("beam", elem, cells, tuple(0.05 * c for c in cells), 0.04, 5, mat, 1000.0, "xmin",
                    (0.0, 0.0, -9.81), 0.005, 1)
    return wl.build_mesh()


def _state(wl):
    rng = np.random.default_rng(3)
    x = wl.rest.copy()
    s = (x[:, 0] - x[:, 0].min()) / np.ptp(x[:, 0])
    x[:, 2] += 1e-3 * s ** 2
    v = 0.05 * s[:, None] * rng.standard_normal(x.shape)
    v[wl.fixed != 0] = 0
    return x, v


def _step(wl, precision, options, steps=1, variant=0, setup=None, integrator=0):
    m = wl.model(precision=precision)
    m.options = options
    if setup:
        setup(m)
    ms = MechSystemSolver(m, tol=1e-12, max_iter=20000, pcg_variant=variant, integrator=integrator)
    x, v = _state(wl)
    m.setState(x, v)
    ms.backwardEuler(wl.h, steps)
    assert ms.stats.rel_residual <= 1e-12
    return m.getState(), ms


CASES = {
    "8_rows": (L.ELEM_TET, (2, 1, 1), NH, {}),
    "90_rows": (L.ELEM_TET, (10, 2, 2), LIN, {}),
    "96_rows": (L.ELEM_TET, (6, 3, 3), NH, {}),
    "99_rows": (L.ELEM_HEX, (11, 2, 2), NH, {}),
    "two_ctas_of_60": (L.ELEM_HEX, (5, 3, 5), NH, {}),
    "team_of_17": (L.ELEM_TET, (20, 6, 6), NH, {}),
    "team_of_100": (L.ELEM_HEX, (45, 11, 10), NH, {}),
    "long_rows": (L.ELEM_QUADHEX, (4, 3, 2), NH, {}),
    "element_pressure": (L.ELEM_HEX, (6, 4, 3), MR, {}),
    "nodal_one_cta": (L.ELEM_TET, (5, 3, 3), MR, {}),
    "nodal_team": (L.ELEM_TET, (12, 6, 5), MR, {}),
    "150_rows_in_one": (L.ELEM_TET, (6, 4, 4), NH, {L.OPT_PCG_CTAS: 1}),
    "two_sets": (L.ELEM_TET, (9, 5, 5), NH, {L.OPT_PCG_CTAS: 2}),
    "two_sets_nodal": (L.ELEM_TET, (7, 4, 4), MR, {L.OPT_PCG_CTAS: 2}),
}


@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_MIXED])
@pytest.mark.parametrize("name", list(CASES))
def test_step_matches_grid_wide_kernel(name, precision, b200):
    elem, cells, mat, opts = CASES[name]
    wl = _beam(elem, cells, mat)
    (xt, vt), _ = _step(wl, precision, dict(opts))
    (xg, vg), _ = _step(wl, precision, {L.OPT_PCG_SPLIT: L.SPLIT_CONTIGUOUS})
    assert rel_err(xt, xg) <= 1e-9, rel_err(xt, xg)
    assert rel_err(vt, vg) <= 1e-8, rel_err(vt, vg)


@pytest.mark.parametrize("variant", [L.PCG_CLASSIC, L.PCG_PIPELINED])
@pytest.mark.parametrize("mat", [NH, MR])
def test_variants(variant, mat, b200):
    wl = _beam(L.ELEM_TET, (9, 4, 4), mat)
    (xt, vt), _ = _step(wl, L.PREC_FP64, {}, variant=variant)
    (xg, vg), _ = _step(wl, L.PREC_FP64, {L.OPT_PCG_SPLIT: L.SPLIT_CONTIGUOUS})
    assert rel_err(xt, xg) <= 1e-9 and rel_err(vt, vg) <= 1e-8


def test_plane_constraints_in_two_sets(b200):
    wl = _beam(L.ELEM_TET, (9, 5, 5), NH)
    tip = np.where(wl.rest[:, 0] >= wl.rest[:, 0].max() - 1e-9)[0]
    nrm = np.tile(np.array([0.0, 0.6, 0.8]), (tip.size, 1))
    off = (nrm * wl.rest[tip]).sum(axis=1)
    out = [_step(wl, L.PREC_FP64, opts, setup=lambda m: m.setPlaneConstraints(tip, nrm, off),
                 integrator=L.INTEGRATOR_CONSTRAINED_BACKWARD_EULER)[0]
           for opts in ({L.OPT_PCG_CTAS: 2}, {}, {L.OPT_PCG_SPLIT: L.SPLIT_CONTIGUOUS})]
    for x, v in out[:2]:
        assert rel_err(x, out[2][0]) <= 1e-9 and rel_err(v, out[2][1]) <= 1e-8
        assert np.abs((nrm * x[tip]).sum(axis=1) - off).max() <= 1e-12


@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_MIXED])
def test_pack_more_slots_than_ctas(precision, b200):
    """Teams of different sizes queue for few CTAs; left-out models keep their state; repeated solves (the packet tags
    run on) give the same bits."""
    cells = [(12, 4, 4), (3, 2, 2), (9, 5, 5), (6, 3, 3), (20, 2, 2), (4, 4, 4)]
    wls = [_beam(L.ELEM_TET, c, NH) for c in cells]
    xs, vs = zip(*(_state(w) for w in wls))
    active = np.array([1, 1, 0, 1, 1, 1])
    runs = []
    for opts in ({L.OPT_PCG_CTAS: 3}, {}, {L.OPT_PCG_SPLIT: L.SPLIT_CONTIGUOUS}):
        p = FemPack([w.model() for w in wls], precision=precision, options=opts)
        p.setActive(active)
        got = []
        for _ in range(3):
            p.setStates(xs, vs)
            p.backwardEuler(wls[0].h, 1, tol=1e-12)
            got.append(p.getStates())
        for other in got[1:]:
            assert all(np.array_equal(a, b) for s, t in zip(got[0], other) for a, b in zip(s, t))
        runs.append(got[0])
    for i in range(len(wls)):
        for r in runs[:2]:
            assert rel_err(r[i][0], runs[2][i][0]) <= 1e-9 and rel_err(r[i][1], runs[2][i][1]) <= 1e-8
    assert np.array_equal(runs[0][2][0], xs[2]) and np.array_equal(runs[0][2][1], vs[2])


@pytest.mark.parametrize("skip", [1, 2])
def test_missing_member_times_out_and_recovers(skip, b200):
    """A CTA that never publishes: the team's waits run out, the state stays, and the handle then steps as a fresh one."""
    wl = _beam(L.ELEM_HEX, (8, 4, 4), NH)
    m, ref = wl.model(), wl.model()
    e = m.engine()
    e.call("b200fem_set_option", L.OPT_BARRIER_TIMEOUT_MS, 200)
    e.call("b200fem_set_option", L.OPT_TEST_SKIP_ARRIVAL, skip)
    ms = MechSystemSolver(m, tol=1e-12)
    x, v = _state(wl)
    m.setState(x, v)
    with pytest.raises(L.B200FemError) as ei:
        ms.backwardEuler(wl.h, 2)
    assert ei.value.status == L.ERR_TIMEOUT
    assert np.array_equal(m.getState()[0], x) and np.array_equal(m.getState()[1], v)
    e.call("b200fem_set_option", L.OPT_TEST_SKIP_ARRIVAL, 0)
    m.setState(x, v)
    ms.backwardEuler(wl.h, 2)
    ref.setState(x, v)
    MechSystemSolver(ref, tol=1e-12).backwardEuler(wl.h, 2)
    assert all(np.array_equal(a, b) for a, b in zip(m.getState(), ref.getState()))


def test_short_wait_limit_with_queued_teams(b200):
    """A limit of 1 ms bounds waits within a team, not the wait for CTAs that solve other models: packs that queue for
    two CTAs step as with the default limit."""
    wls = [_beam(L.ELEM_TET, c, NeoHookeanMaterial(E, 0.4))
           for c, E in (((9, 4, 4), 1e9), ((9, 4, 4), 1e9), ((9, 5, 5), 1e3), ((6, 3, 3), 1e8))]
    xs, vs = zip(*(_state(w) for w in wls))
    out = []
    for ms in (1, 5000):
        p = FemPack([w.model() for w in wls], precision=L.PREC_FP64,
                    options={L.OPT_PCG_CTAS: 2, L.OPT_BARRIER_TIMEOUT_MS: ms})
        p.setStates(xs, vs)
        p.backwardEuler(wls[0].h, 2, tol=1e-12, max_iter=20000)
        out.append(p.getStates())
    assert all(np.array_equal(a, b) for s, t in zip(*out) for a, b in zip(s, t))


@pytest.mark.parametrize("resident", [1, 2])
def test_explicit_residency_keeps_the_grid_wide_kernel(resident, b200):
    """PCG_RESIDENT asks for a layout of the contiguous split: it is the one that runs."""
    wl = _beam(L.ELEM_HEX, (8, 4, 4), NH)
    out = []
    for opts in ({L.OPT_PCG_RESIDENT: resident}, {L.OPT_PCG_RESIDENT: resident, L.OPT_PCG_SPLIT: L.SPLIT_CONTIGUOUS}):
        p = FemPack([wl.model()], precision=L.PREC_FP64, options=opts)
        p.engine()
        assert p.option(L.OPT_PCG_SPLIT) == L.SPLIT_CONTIGUOUS and p.option(L.OPT_PCG_RESIDENT) == resident
        p.setStates(*([a] for a in _state(wl)))
        p.backwardEuler(wl.h, 2, tol=1e-12)
        out.append(p.getStates()[0])
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("cells", [(10, 2, 2), (20, 6, 6)])
def test_teams_hold_no_arrays_of_the_grid_wide_kernel(cells, b200):
    """Where S fits the CTAs, the teams' tables take less device memory than the vectors and lists they replace."""
    wl = _beam(L.ELEM_TET, cells, NH)
    team, grid = (FemPack([wl.model()], precision=L.PREC_FP64, options=o)
                  for o in ({}, {L.OPT_PCG_SPLIT: L.SPLIT_CONTIGUOUS}))
    assert team.deviceBytes() < grid.deviceBytes(), (team.deviceBytes(), grid.deviceBytes())


def test_grid_wide_kernel_where_teams_exceed_the_memory(b200):
    """A large model's teams hold a copy of the blocks that stream: with device memory for the grid-wide kernel's arrays
    but not for that copy, the model builds and steps as it does with that kernel."""
    import torch

    wl = _beam(L.ELEM_HEX, (60, 30, 30), NH)
    x, v = _state(wl)

    def step(options):
        p = FemPack([wl.model()], precision=L.PREC_FP64, options=options)
        p.setStates([x], [v])
        p.backwardEuler(wl.h, 1, tol=1e-8)
        out = p.getStates()[0], p.option(L.OPT_PCG_SPLIT), p.deviceBytes()
        p.close()
        return out

    _, split, team_bytes = step({})
    ref, _, grid_bytes = step({L.OPT_PCG_SPLIT: L.SPLIT_CONTIGUOUS})
    assert split == L.SPLIT_TEAM and team_bytes - grid_bytes > 64 << 20, (team_bytes, grid_bytes)
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (team_bytes + grid_bytes) // 2, dtype=torch.uint8, device="cuda")
    got, split, _ = step({})
    del hold
    torch.cuda.empty_cache()
    assert split == L.SPLIT_CONTIGUOUS
    assert all(np.array_equal(a, b) for a, b in zip(got, ref))


# what a CTA takes with few CTAs allowed: three component sets (324 and 310 rows in one), steps of S beyond the shared
# memory, in both precisions and with the factored NODAL matrix
FULL_CTAS = {
    "three_sets": (L.ELEM_TET, (9, 5, 5), NH, 1),
    "three_sets_streamed": (L.ELEM_HEX, (11, 5, 4), NH, 1),
    "two_ctas_streamed": (L.ELEM_HEX, (16, 5, 5), NH, 2),
    "quadratic_streamed": (L.ELEM_QUADHEX, (5, 2, 2), NH, 1),
    "three_sets_nodal": (L.ELEM_TET, (31, 4, 1), MR, 1),
    "nodal_streamed": (L.ELEM_TET, (12, 5, 5), MR, 2),
}


@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_MIXED])
@pytest.mark.parametrize("name", list(FULL_CTAS))
def test_full_ctas_match_grid_wide_kernel(name, precision, b200):
    elem, cells, mat, ctas = FULL_CTAS[name]
    wl = _beam(elem, cells, mat)
    out = []
    for opts in ({L.OPT_PCG_CTAS: ctas}, {L.OPT_PCG_SPLIT: L.SPLIT_CONTIGUOUS}):
        p = FemPack([wl.model()], precision=precision, options=opts)
        p.engine()
        assert p.option(L.OPT_PCG_SPLIT) == opts.get(L.OPT_PCG_SPLIT, L.SPLIT_TEAM)
        p.setStates(*([a] for a in _state(wl)))
        p.backwardEuler(wl.h, 2, tol=1e-12)
        out.append(p.getStates()[0])
    (xt, vt), (xg, vg) = out
    assert rel_err(xt, xg) <= 1e-9 and rel_err(vt, vg) <= 1e-8, (rel_err(xt, xg), rel_err(vt, vg))


@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_MIXED])
def test_pack_of_nodal_and_other_models(precision, b200):
    """The factored matrix holds for the whole pack: models without NODAL incompressibility run through it beside those
    with it, queued for few CTAs."""
    wls = [_beam(e, c, m) for e, c, m in ((L.ELEM_TET, (9, 4, 4), MR), (L.ELEM_TET, (6, 3, 3), NH),
                                          (L.ELEM_TET, (3, 2, 2), MR), (L.ELEM_TET, (10, 5, 4), NH))]
    xs, vs = zip(*(_state(w) for w in wls))
    out = []
    for opts in ({L.OPT_PCG_CTAS: 3}, {}, {L.OPT_PCG_SPLIT: L.SPLIT_STRIDED}):
        p = FemPack([w.model() for w in wls], precision=precision, options=opts)
        p.setStates(xs, vs)
        p.backwardEuler(wls[0].h, 2, tol=1e-12)
        out.append(p.getStates())
    for i in range(len(wls)):
        for r in out[:2]:
            assert rel_err(r[i][0], out[2][i][0]) <= 1e-9 and rel_err(r[i][1], out[2][i][1]) <= 1e-8, i
