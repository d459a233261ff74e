"""RK stages in place (csrc/solver.cuh k_inplace_wet) beside the other routes of a step: a
simulation that runs in place against the same case in a batch's size class, which writes every
dry leaf in both stages. Every kernel is deterministic, so the two give the same bits:

* dt, leaves, flags, states and stage points, with and without friction and limiter, in both
  precisions, on levels walked by bands only and on levels above them, for a member that
  alternates between its class and steps of its own (in place; U^n of the leaves that stand is
  not stored by those steps and stored again by the class);
* the raster, VTK and c-prop files written after steps in place, character for character.

With the refinement proposal switched on, off and on again between steps in place, the leaf state
of every leaf is the one that its hierarchy slot holds: no frozen leaf has a U^n from before.

The step counters say which route a step took."""
import os

import numpy as np
import pytest

import cases
import mwdg2_b200

pytestmark = pytest.mark.gpu


def _lake(root, L, seed, manning, limit, **kw):
    """A catchment with 2 % of its cells under water and a point inflow."""
    z = cases.fbm_surface(1 << L, 0.8, seed, 29.37)
    level = float(np.sort(z.ravel())[int(0.02 * z.size)])
    return cases.fbm_catchment(root, L=L, relief=29.37, seed=seed, manning=manning, limitslopes=limit, sim_time=600.0,
                               t_peak=60.0, start_depth=np.maximum(0.0, np.round(level, 3) + 0.00037 - z), **kw)


# (11, 64, 0.0, True) has a limiter decision on its threshold at step 6, where the CUDA path and
# the CPU oracle part by 1.6e-8 on either route: here the two routes are held to each other
@pytest.mark.parametrize("L,precision,manning,limit", [(11, 64, 0.0, True), (11, 32, 0.03, True), (10, 32, 0.0, False),
                                                       (9, 64, 0.03, True), (8, 32, 0.03, True)])
def test_in_place_equals_size_class(tmp_path, L, precision, manning, limit):
    pars = [_lake(str(tmp_path / f"m{i}"), L, 20261203 + L, manning, limit).par for i in range(2)]
    sim = mwdg2_b200.Simulation(pars[0], precision=precision)
    with mwdg2_b200.Batch(pars, precision=precision) as b:
        m = b.member(0)
        for s in range(1, 13):
            classes = s in (2, 3, 4, 7, 8, 11)
            b.group_max_level(L if classes else 0)
            ok, dt, n = sim.step()
            _, dts, leaves = b.step()
            assert ok and dt == dts[0] and n == leaves[0], f"step {s}"
            assert sim.last_step_counters()["in_place"] == (s > 1), f"step {s}"
            assert m.last_step_counters()["in_place"] == (s > 1 and not classes), f"step {s}"
            np.testing.assert_array_equal(sim.stage(2), m.stage(2), err_msg=f"step {s}: stage points")
            if s not in (4, 6, 8, 9, 12):
                continue
            np.testing.assert_array_equal(sim.sig(), m.sig(), err_msg=f"step {s}: significance")
            lf, want = sim.leaves(), m.leaves()
            for key in want:
                np.testing.assert_array_equal(lf[key], want[key], err_msg=f"step {s}: {key}")
            st, want = sim.state(), m.state()
            for key in want:
                np.testing.assert_array_equal(st[key], want[key], err_msg=f"step {s}: {key}")
    sim.close()


@pytest.mark.parametrize("precision", [32, 64])
def test_files_written_after_steps_in_place(tmp_path, precision):
    kw = dict(saveint=0.4, extra=["raster_out", "vtk", "c_prop", "voutput", "qoutput"])
    roots = [str(tmp_path / r) for r in ("alone", "m0", "m1")]
    pars = [_lake(r, 8, 5, 0.03, True, **kw).par for r in roots]
    sim = mwdg2_b200.Simulation(pars[0], precision=precision, write_outputs=True)
    with mwdg2_b200.Batch(pars[1:], precision=precision, write_outputs=True) as b:
        b.group_max_level(8)
        for s in range(1, 31):
            sim.run(1)
            b.run(1)
            assert sim.last_step_counters()["in_place"] == (s > 1), f"step {s}"
            assert b.member(0).last_step_counters()["in_place"] == 0, f"step {s}"
    sim.close()

    def written(root):
        out = {}
        for folder, _, names in os.walk(root):
            for f in names:
                rel = os.path.relpath(os.path.join(folder, f), root)
                if rel.startswith("res"):
                    with open(os.path.join(folder, f), "rb") as fp:
                        out[rel] = fp.read()
        return out

    mine, want = written(roots[0]), written(roots[1])
    assert sorted(mine) == sorted(want)
    maps = [f for f in want if f.endswith((".wd", ".vtk", ".csv", ".elev", ".Qx", ".vx"))]
    assert sum(f.endswith(".vtk") for f in maps) >= 3 and len(maps) > 10, sorted(want)
    for f in want:
        if not f.endswith(".cumu"):   # (holds run times)
            assert mine[f] == want[f], f


def test_proposal_between_steps_in_place(tmp_path):
    L = 9
    sim = mwdg2_b200.Simulation(_lake(str(tmp_path), L, 5, 0.03, False).par, precision=64)
    nothing = np.zeros(mwdg2_b200.MLP_PARAMS, np.float32)
    nothing[-4:] = -20.0
    frozen = 0
    for s in range(1, 20):
        if s in (5, 12):
            sim.proposal_enable(nothing, judge_every=0, threshold=0.0, miss_bound=1.0)
        if s in (9, 16):
            sim.proposal_enable(None)
        on = 5 <= s < 9 or 12 <= s < 16
        ok, _, _ = sim.step()
        k = sim.last_step_counters()
        assert ok and k["in_place"] == (s > 1 and not on), f"step {s}"
        frozen += k["frozen_leaves"]
        if s % 2 == 0 and not on:
            continue       # two steps in place between reads of the state
        act, st = sim.leaves()["act"], sim.state()
        eta, z = sim.hierarchy(0, 0)[act], sim.hierarchy(3, 0)[act]
        # up to rounding: the surface is stored as h + z, and a frozen leaf whose parent is decoded
        # has the decode's rounding in its slot
        for got, slot in ((st["h0"] + z, eta), (st["qx0"], sim.hierarchy(1, 0)[act]), (st["qy0"], sim.hierarchy(2, 0)[act])):
            assert np.max(np.abs(got - slot)) <= 1e-13 * 30.0, f"step {s}"
    assert frozen > 0
    sim.close()
