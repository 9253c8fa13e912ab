"""Error paths of the device checks, made to fail from the host
(include/hyowon_debug.h): no GPU fault, trap or hang is involved.

* A pipeline wait of the five-pass potential solve that is given zero polls
  gives up at once: each block drains its own copies in flight, sets
  ST_PIPELINE and returns; the solve fails with the runtime error the status
  maps to, nothing is published, and with the default limit restored the same
  handle solves again with the same forces as a fresh handle.
* A CIC mass-conservation target moved off the deposited mass makes the
  solve fail with the reference's runtime error (src/math/cic_mass_conservation.cpp:41-59);
  with the target restored the handle solves again.
Both forms, on a power-of-two mesh (the five-pass solve) of 64^3 cells.
* A gradient of more steps than host memory holds checkpoints for is an
  out-of-memory error of the call, stateless or on a handle; the handle works on.
* A solve whose particles cannot be keyed (1LPT of non-finite noise) is refused
  after the sort was already enqueued: the particle arrays stay as they were.
"""
import numpy as np
import pytest

import hyowon_b200 as hb
from hyowon_b200 import _native as nat
from hyowon_b200 import adjoint, ic

pytestmark = pytest.mark.gpu

DEFAULT_WAIT = 16777216


def state(n=20000, L=50.0, seed=4):
    rng = np.random.default_rng(seed)
    return L, [rng.uniform(0.0, L, n) for _ in range(3)]


@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_pipeline_wait_timeout_is_reported_and_recovered(form):
    L, pos = state()
    with hb.PMSolver(hb.MeshGeometry(L, 64), hb.PMForceMethod.pure_pm(False), form) as fresh:
        fresh.upload(*pos, uniform_mass=1.0)
        fresh.solve_forces()
        want = fresh.download()
    with hb.PMSolver(hb.MeshGeometry(L, 64), hb.PMForceMethod.pure_pm(False), form) as s:
        s.upload(*pos, uniform_mass=1.0)
        assert nat.lib().hyowon_pm_debug_set_wait_limit(s.handle, 0) == 0
        with pytest.raises(RuntimeError, match="pipeline wait timed out"):
            s.solve_forces()
        assert nat.lib().hyowon_pm_debug_set_wait_limit(s.handle, DEFAULT_WAIT) == 0
        s.solve_forces()
        got = s.download()
    for k in ("ax", "ay", "az"):
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_mass_conservation_violation_is_reported_and_recovered(form):
    L, pos = state(seed=5)
    with hb.PMSolver(hb.MeshGeometry(L, 64), hb.PMForceMethod.pure_pm(False), form) as s:
        s.upload(*pos, uniform_mass=1.0)
        s.solve_forces()
        want = s.download()
        # binary64: 1e-6 of the total mass, far outside the forward-error bound;
        # precision form: one fixed-point unit off the exact integer sum
        assert nat.lib().hyowon_pm_debug_offset_mass_target(s.handle, 0.02 if form == "fp64" else 1.0) == 0
        with pytest.raises(RuntimeError, match="mass"):
            s.solve_forces()
        assert nat.lib().hyowon_pm_debug_offset_mass_target(s.handle, 0.0) == 0
        s.solve_forces()
        got = s.download()
    for k in ("ax", "ay", "az"):
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_gradient_of_too_many_steps_is_an_error(form):
    box, n, N = 60.0, 16, 32
    rng = np.random.default_rng(2)
    noise, target = rng.standard_normal(n ** 3), 0.3 * rng.standard_normal(N ** 3)

    class Endless(adjoint.DifferentiablePM):
        def _cfg(self):   # refused before the schedule is read
            c = super()._cfg()
            c.n_steps = 1 << 60
            return c

    args = (box, n, N, 0.05, 3, form, 1)
    with pytest.raises(MemoryError):
        Endless(*args).loss_and_grad(noise, target)
    with hb.PMSolver(hb.MeshGeometry(box, N), hb.PMForceMethod.pure_pm(False), form) as s:
        with pytest.raises(MemoryError):
            Endless(*args, solver=s).loss_and_grad(noise, target)
        got = adjoint.DifferentiablePM(*args, solver=s).loss_and_grad(noise, target)
    assert np.isfinite(got[0]) and np.all(np.isfinite(got[1]))


@pytest.mark.parametrize("mesh", [32, 27, 256])
def test_unkeyable_particles_leave_the_state_as_it_was(mesh):
    """Meshes whose deposit form the device picks (five-pass and cuFFT) and one where the
    host reads the densest bucket between the sort and the deposit."""
    L, pos = state(n=4096, seed=6)
    noise = np.random.default_rng(6).standard_normal(16 ** 3)
    noise[5] = np.nan
    with hb.PMSolver(hb.MeshGeometry(L, mesh), hb.PMForceMethod.pure_pm(False)) as s:
        s.upload(*pos, uniform_mass=1.0)
        s.solve_forces()
        want = s.download()
        ic.lpt_on_device(s, noise, 16, 0.05, 1.0)
        before = s.download(acc=False)
        for _ in range(2):
            with pytest.raises(ValueError, match="finite"):
                s.solve_forces()
            after = s.download(acc=False)
            for k in before:
                assert np.array_equal(before[k], after[k], equal_nan=True), k
        s.upload(*pos, uniform_mass=1.0)
        s.solve_forces()
        got = s.download()
    for k in ("ax", "ay", "az"):
        assert np.array_equal(got[k], want[k]), k
