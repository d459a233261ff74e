"""Boundary segments on a mostly dry DEM: RK stages in place (csrc/solver.cuh k_inplace_wet)
against the writers of every dry leaf.

A segment resets the depth of the border leaves that it covers, dry ones too. The reset depth
is the leaf's U^n and stays its state, but over a bed of tens of metres the elevation keeps only
part of its digits, so an elevation that a stage would put back unchanged does not say that
the depth is unchanged. A batch's size class always runs the writers; a simulation on its own
runs in place here. Every kernel is deterministic, so both give the same bits: dt, leaves, states
and stage points (and the volume up to its order of summation), in both precisions, over QFIX, QVAR and HFIX segments."""
import os

import numpy as np
import pytest

import cases
import mwdg2_b200

pytestmark = pytest.mark.gpu


def _dry_with_segments(root, L, manning):
    """A catchment, 2 % of it under water, whose segments give depths below the dry threshold
    (1 mm): north QFIX, east QVAR, south HFIX over a level margin."""
    n, dx = 1 << L, 2.0
    z = np.round(cases.fbm_surface(n, 0.8, 77, 30.0), 3)
    z[:2, :] = 11.3
    level = float(np.sort(z.ravel())[int(0.02 * z.size)])
    c = cases.fbm_catchment(root, L=L, cellsize=dx, sim_time=600.0, manning=manning, peak_q=0.0,
                            start_depth=np.maximum(0.0, np.round(level, 3) + 0.00037 - z),
                            stage_points=[(n * dx / 2 + dx / 2, n * dx - dx / 2), (n * dx - dx / 2, n * dx / 2 + dx / 2),
                                          (n * dx / 2 + dx / 2, dx / 2)])
    cases.write_esri_ascii(os.path.join(root, "case.dem"), z[::-1], dx, decimals=3)
    a, b = n * dx / 4, 3 * n * dx / 4
    with open(os.path.join(root, "case.bci"), "w") as f:
        f.write(f"N {a!r} {b!r} QFIX 0.00071\nE {a!r} {b!r} QVAR HYD\nS {a!r} {b!r} HFIX 11.30047\n")
    with open(os.path.join(root, "case.bdy"), "w") as f:
        f.write("series\nHYD\n3 seconds\n0.00031 0\n0.00093 2400\n0.00093 4800\n")
    return c.par


@pytest.mark.parametrize("precision,manning", [(32, 0.03), (32, 0.0), (64, 0.03)])
def test_segments_that_reset_dry_leaves(tmp_path, precision, manning):
    L = 8
    pars = [_dry_with_segments(str(tmp_path / f"m{i}"), L, manning) for i in range(2)]
    sim = mwdg2_b200.Simulation(pars[0], precision=precision)
    reset = 0
    with mwdg2_b200.Batch(pars, precision=precision) as b:
        b.group_max_level(L)
        for s in range(1, 13):
            ok, dt, n = sim.step()
            _, dts, leaves = b.step()
            assert ok and dt == dts[0] and n == leaves[0], f"step {s}"
            assert sim.last_step_counters()["in_place"] == (s > 1), f"step {s}"
            assert b.member(0).last_step_counters()["in_place"] == 0, f"step {s}"
            if s % 3:
                continue       # two steps between reads of the state
            m = b.member(0)
            # the volume's at most 256 blocks add their sums in any order, 2^-53 relative each
            assert abs(sim.volume() - m.volume()) <= 1e-13 * m.volume(), f"step {s}: volume"
            np.testing.assert_array_equal(sim.stage(3), m.stage(3), err_msg=f"step {s}: stage points")
            lf, want = sim.leaves(), m.leaves()
            for key in want:
                np.testing.assert_array_equal(lf[key], want[key], err_msg=f"step {s}: {key}")
            st, want = sim.state(), m.state()
            for key in want:
                np.testing.assert_array_equal(st[key], want[key], err_msg=f"step {s}: {key}")
            # dry leaves on the segments whose depth the elevation does not give back
            t = np.float32 if precision == 32 else np.float64
            h, z = want["h0"].astype(t), want["z0"].astype(t)
            edge = (lf["lvl"] == L) & (lf["nb_ids"] == -1).any(axis=0) & (h > 0) & (h < 1e-3)
            reset += int(np.count_nonzero(edge & ((h + z) - z != h)))
    assert reset > 100, f"only {reset} dry border leaves hold a reset depth"
    sim.close()
