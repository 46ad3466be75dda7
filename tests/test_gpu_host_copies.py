"""Host arrays of every size come back as they went in: below and above the 6 MiB of x and v together from which
pageable arrays are staged in chunks of 1 MiB, a last chunk of a few values, page-locked arrays; a non-finite value anywhere is refused before
the device's state changes; the stiffness arrays of an update equal the ones of the device's other exports."""
import numpy as np
import pytest

from artisynth_core_b200 import _lib as L
from artisynth_core_b200 import workloads as W
from artisynth_core_b200.femmodel import FemPack, LinearMaterial, MechSystemSolver, NeoHookeanMaterial

pytestmark = pytest.mark.gpu


def _model(n_nodes):
    """A tetrahedron and nodes that belong to nothing."""
    rest = np.zeros((n_nodes, 3))
    rest[:4] = [[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]]
    rest[4:, 0] = 2.0 + np.arange(n_nodes - 4)
    fixed = np.ones(n_nodes, dtype=np.int32)
    fixed[1:4] = 0
    wl = W.Workload("t", L.ELEM_TET, (1, 1, 1), (1, 1, 1), 0, 0, LinearMaterial(1e5, 0.3), 1000.0, "xmin", (0, 0, 0),
                    0.01, 1)
    wl.rest, wl.conn, wl.fixed = rest, np.array([[0, 1, 2, 3]], dtype=np.int32), fixed
    return wl.model()


@pytest.mark.parametrize("n", [5, 43691, 131072, 131073, 174763])
def test_state_round_trip(n, b200):
    m = _model(n)
    rng = np.random.default_rng(n)
    x, v = rng.standard_normal((n, 3)), rng.standard_normal((n, 3))
    m.setState(x, v)
    xg, vg = m.getState()
    assert np.array_equal(xg, x) and np.array_equal(vg, v)
    for which in (0, 1):
        for at in (0, 3 * n // 2, 3 * n - 1):
            bad = [x + 1, v + 1]
            bad[which].reshape(-1)[at] = np.nan
            with pytest.raises(L.B200FemError) as ei:
                m.setState(*bad)
            assert ei.value.status == L.ERR_INVALID_ARG
    assert all(np.array_equal(a, b) for a, b in zip(m.getState(), (x, v)))


def test_page_locked_arrays(b200):
    import torch

    n = 140000
    m = _model(n)
    x = torch.randn(3 * n, dtype=torch.float64).pin_memory().numpy()
    v = torch.randn(3 * n, dtype=torch.float64).pin_memory().numpy()
    e = m.engine()
    e.call("b200fem_set_state", L.dptr(x), L.dptr(v))
    out = [torch.zeros(3 * n, dtype=torch.float64).pin_memory().numpy() for _ in range(2)]
    e.call("b200fem_get_state", L.dptr(out[0]), L.dptr(out[1]))
    assert np.array_equal(out[0], x) and np.array_equal(out[1], v)


@pytest.mark.parametrize("cells", [(4, 2, 2), (24, 10, 10)])
def test_update_exports_agree(cells, b200):
    """Blocks and scalar CRS values hold the same numbers (the CRS rows are the blocks' rows side by side), in both
    precisions."""
    for precision in (L.PREC_FP64, L.PREC_MIXED):
        wl = W.Workload("t", L.ELEM_HEX, cells, tuple(0.05 * c for c in cells), 0.03, 1, NeoHookeanMaterial(5e4, 0.4),
                        1000.0, "xmin", (0, 0, 0), 0.01, 1).build_mesh()
        m = wl.model(precision)
        f, K, crs = m.updateStressAndStiffness(wl.rest, want_crs=True)
        f2, K2 = m.updateStressAndStiffness(wl.rest)
        assert np.array_equal(f, f2) and np.array_equal(K, K2)
        rp, _ = m.getBlockPattern()
        for r in (0, len(rp) // 2, len(rp) - 2):
            rows = K[rp[r]:rp[r + 1]].transpose(1, 0, 2).reshape(-1)
            assert np.array_equal(crs[9 * rp[r]:9 * rp[r + 1]], rows)


def test_pack_states_reuse_their_buffer(b200):
    wls = W.batched_beams(count=3)
    ms = [w.build_mesh().model() for w in wls]
    p = FemPack(ms, precision=L.PREC_FP64)
    rng = np.random.default_rng(0)
    for _ in range(2):
        xs = [w.rest + 1e-3 * rng.standard_normal(w.rest.shape) for w in wls]
        vs = [rng.standard_normal(w.rest.shape) for w in wls]
        p.setStates(xs, vs)
        for (x, v), xe, ve in zip(p.getStates(), xs, vs):
            assert np.array_equal(x, xe) and np.array_equal(v, ve)
    alone = ms[0]
    alone.setState(xs[0], vs[0])
    assert np.array_equal(alone.getState()[0], xs[0])
    MechSystemSolver(alone, tol=1e-10).backwardEuler(0.01, 1)
