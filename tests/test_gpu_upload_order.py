"""A new simulation or trainer depends on its inputs alone, not on what its device memory held.

Its uploads and clears are on the stream of the kernels that read them. A copy from pageable host
memory and a memset return before they are done, and the legacy stream does not order with the
non-blocking streams that the library uses, so on the legacy stream a kernel could read memory
that its upload had not reached. Here the free device memory is filled with NaNs before each
creation, and the first step's results are compared bit for bit with the first run's; the
trainer's parameters move by at most the learning rate in its first Adam step (plus rounding),
whatever the sums' order."""
import numpy as np
import pytest

import cases
import mwdg2_b200

pytestmark = pytest.mark.gpu


def _fill_free_memory():
    import torch

    # blocks of the sizes that small simulations and the trainer take, from both of the driver's pools
    junk = [torch.full((n,), 0xFF, dtype=torch.uint8, device="cuda") for n in [64 << 20] + 40 * [2 << 20]]
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()


@pytest.mark.parametrize("solver,precision", [("mwdg2", 64), ("mwdg2", 32), ("hwfv1", 64)])
def test_first_step_depends_on_the_inputs_alone(tmp_path, solver, precision):
    par = cases.bc_edges(str(tmp_path), "b", L=7, solver=solver).par
    first = None
    for r in range(25):
        _fill_free_memory()
        sim = mwdg2_b200.Simulation(par, precision=precision)
        if solver == "mwdg2" and r % 5 == 4:
            sim.proposal_record(True)   # its buffers are cleared just before the step
        ok, dt, n = sim.step()
        got = {"dt": np.array(dt), "sig": sim.sig(), **sim.leaves(), **sim.state()}
        sim.close()
        assert ok
        first = first or got
        for key in first:
            np.testing.assert_array_equal(got[key], first[key], err_msg=f"run {r}: {key}")


def test_trainer_starts_from_its_parameters():
    rng = np.random.default_rng(5)
    feats = rng.normal(0, 1, (512, mwdg2_b200.MLP_FEATURES)).astype(np.float32)
    labels = rng.integers(0, 16, 512).astype(np.uint8)
    p0 = mwdg2_b200.mlp_init(3)
    for r in range(10):
        _fill_free_memory()
        t = mwdg2_b200.Trainer(p0, lr=1e-3)
        loss = t.step(feats, labels)
        p = t.params()
        t.close()
        assert np.isfinite(loss), f"run {r}: loss {loss}"
        assert np.max(np.abs(p - p0)) <= 1e-3 * (1 + 1e-4) + 1e-6, f"run {r}"
