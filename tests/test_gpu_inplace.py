"""RK stages in place (csrc/solver.cuh k_inplace_wet): steps of the reference decode with under
a tenth of the leaves wet leave the dry leaves that a stage does not change as they stand.

Against the CPU oracle, which writes every leaf in both stages: leaves, neighbours and flags
bit-exact, states within 1e-10 relative to max(1, |value|) (FP64; the bound of the other
oracle tests), over catchments with and without friction (which clears the dry leaves'
discharges) and limiter, on levels walked by bands only and on levels above them. The state
is read by the getters that need U^n of the standing leaves, which those steps do not store:
leaf state, water volume, stage points; a switch to the keep-values decode and back changes
the route of the stages and keeps the state."""
import numpy as np
import pytest

import cases
import mwdg2_b200
import oracle_py
from gpu_util import assert_same_topology, rel_err

pytestmark = pytest.mark.gpu


# (11, 0.0, True, 1e-3) is left out: at its step 6 a limiter decision sits on its threshold and
# the CUDA path and the oracle part by 1.6e-8, in place or with every leaf written
# (test_gpu_inplace_routes.py holds the two routes to each other there)
@pytest.mark.parametrize("L,manning,limit,eps", [(7, 0.0, True, 1e-3), (8, 0.03, True, 1e-3), (9, 0.03, False, 1e-2),
                                                 (11, 0.03, False, 1e-3)])
def test_in_place_stages_match_oracle(tmp_path, L, manning, limit, eps):
    z = cases.fbm_surface(1 << L, 0.8, 20261203 + L, 29.37)
    level = float(np.sort(z.ravel())[int(0.02 * z.size)])
    c = cases.fbm_catchment(str(tmp_path), L=L, eps=eps, relief=29.37, seed=20261203 + L, manning=manning, limitslopes=limit,
                            start_depth=np.maximum(0.0, np.round(level, 3) + 0.00037 - z), sim_time=600.0, t_peak=60.0)
    sim, orc = mwdg2_b200.Simulation(c.par, precision=64), oracle_py.Oracle(c.par, 64)
    try:
        wet, leaves, in_place = 1, 1, 0
        for s in range(1, 11 if L > 9 else 19):
            if s in (8, 10):   # the keep-values decode for two steps
                sim.set_decode_mode("keep" if s == 8 else "reference")
                orc.set_keep_values(s == 8)
            expected = 10 * wet < leaves and s not in (8, 9)   # the rule, from the step before
            ok, dt, n = sim.step()
            ok2, dt2, n2 = orc.step()
            assert ok and ok2 and n == n2, f"step {s}: {n} leaves, {n2} in the oracle"
            assert abs(dt - dt2) <= 1e-9 * dt2, f"step {s}: dt {dt}, {dt2} in the oracle"
            k = sim.last_step_counters()
            assert k["in_place"] == expected, f"step {s}: in place {k['in_place']}"
            in_place += k["in_place"]
            wet, leaves = max(k["wet_stage1"], k["wet_stage2"]), k["leaves"]
            if s % 3 != 0:
                continue       # two steps between reads of the state
            vol = sim.volume()
            lf = sim.leaves()
            assert_same_topology(lf, orc.leaves(), f"step {s}")
            np.testing.assert_array_equal(sim.sig(), orc.sig(), err_msg=f"step {s}: significance")
            a, b = sim.state(), orc.state()
            for f in a:
                assert rel_err(a[f], b[f]) <= 1e-10, f"step {s}: {f}"
            cells = 4 ** (L - lf["lvl"].astype(np.int64))
            assert abs(vol - float((a["h0"] * cells).sum()) * c.cellsize ** 2) <= 1e-9 * abs(vol)
            # the stage points stand at cells (n/4, n/2) and (n/2, n/2): Z codes 2/4 + 1/16 and 3/4 of 4^L
            at = np.searchsorted(np.cumsum(cells), [9 * 4 ** L // 16, 3 * 4 ** L // 4], side="right")
            assert np.max(np.abs(sim.stage(2) - a["h0"][at])) <= 1e-12
        assert in_place >= 6, f"{in_place} of {s} steps ran in place"
    finally:
        sim.close()
        orc.close()


def test_in_place_stages_without_epsilon(tmp_path):
    """With epsilon 0 only the first step builds the leaf list (every finest cell), before any step
    can run in place; the later steps' in-place stages use its parent marks, also after steps of
    the keep-values decode between them. Against the oracle as above."""
    L, n = 7, 128
    z = cases.fbm_surface(n, 0.8, 5, 29.37)
    level = float(np.sort(z.ravel())[int(0.02 * z.size)])
    c = cases.fbm_catchment(str(tmp_path), L=L, relief=29.37, seed=5, limitslopes=True, sim_time=600.0, t_peak=60.0,
                            start_depth=np.maximum(0.0, np.round(level, 3) + 0.00037 - z))
    sim, orc = mwdg2_b200.Simulation(c.par, precision=64, epsilon=0.0), oracle_py.Oracle(c.par, 64, epsilon=0.0)
    try:
        for s in range(1, 13):
            if s in (1, 3, 6, 8):   # the keep-values decode in steps 1 to 2 and 6 to 7
                sim.set_decode_mode("keep" if s in (1, 6) else "reference")
                orc.set_keep_values(s in (1, 6))
            ok, dt, nl = sim.step()
            ok2, dt2, nl2 = orc.step()
            assert ok and ok2 and nl == nl2 == n * n, f"step {s}: {nl} leaves, {nl2} in the oracle"
            assert abs(dt - dt2) <= 1e-9 * dt2, f"step {s}: dt {dt}, {dt2} in the oracle"
            if s % 2:
                continue
            assert sim.last_step_counters()["in_place"] == (s not in (2, 6)), f"step {s}"
            assert_same_topology(sim.leaves(), orc.leaves(), f"step {s}")
            a, b = sim.state(), orc.state()
            for f in a:
                assert rel_err(a[f], b[f]) <= 1e-10, f"step {s}: {f}"
    finally:
        sim.close()
        orc.close()


@pytest.mark.parametrize("precision", [32, 64])
def test_in_place_stages_take_no_memory_of_their_own(tmp_path, precision):
    """What an MWDG2 simulation holds on the device, as its arrays' sizes give it: two hierarchies
    (12 and 9 coefficient arrays), the flags, and per finest cell the leaf list (25 bytes with the
    four neighbour ids and the wet list), two dry marks and nine state values. The in-place
    stages use these arrays only. cudaMalloc hands out large arrays in units of 2 MiB; 12 MiB are
    left for everything small (streams, events, scalars), where one more index per finest cell
    would take 18."""
    import torch

    L, unit = 11, 2 << 20
    F, n_det, P = 4 ** L, (4 ** L - 1) // 3 + 3, precision // 8
    n_all = n_det + F
    arrays = 21 * [n_all * P] + 9 * [F * P] + 6 * [4 * F] + 3 * [F] + [n_det]
    want = sum(-(-(a + 64) // unit) * unit for a in arrays)
    warm = cases.fbm_catchment(str(tmp_path / "small"), L=7)
    c = cases.fbm_catchment(str(tmp_path / "case"), L=L)
    mwdg2_b200.Simulation(warm.par, precision=precision).close()   # the context and the modules
    before = torch.cuda.mem_get_info()[0]
    sim = mwdg2_b200.Simulation(c.par, precision=precision)
    held = before - torch.cuda.mem_get_info()[0]
    sim.close()
    print(f"held {held}, arrays {want}, rest {held - want}")
    assert held - want <= 12 << 20, f"{held - want} bytes beyond the arrays"
