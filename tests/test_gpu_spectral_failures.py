"""What a bounded wait that ran out in the FP64 spectral products leaves: a code
that every engine reports, NaN instead of old values, and a solver that works
again with the next call. The codes are set by the tests; no wait runs out."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CUDA_BIT = 1 << 2


def set_word(plan, value, offset=0):
    plan[offset:offset + 4].copy_(torch.tensor([value], dtype=torch.int32).view(torch.uint8))


def test_solver_reports_an_earlier_failure_and_solves_again():
    from pyaxisymflow_gb300.kernels.FastDiagonalisationStokesSolver import (
        FastDiagonalisationStokesSolver)
    s = FastDiagonalisationStokesSolver(200, 136, 0.01)
    w = torch.tensor(np.random.default_rng(0).standard_normal((200, 136))).cuda()
    ref, psi = torch.zeros_like(w), torch.zeros_like(w)
    s.solve(ref, w)
    assert s.engine.status() == 0
    set_word(s.engine.plan, 9)
    assert s.engine.status() == 9          # the last call's
    s.solve(psi, w)
    assert torch.equal(psi, ref)           # the next one starts afresh,
    assert int(s.engine.plan[:4].cpu().view(torch.int32)) == 0
    assert s.engine.status() == 9          # and the failure stays on record


@pytest.mark.parametrize("dct", [False, True])
def test_soft_engine_reports_a_failed_solve(dct):
    from pyaxisymflow_gb300.simulation import SoftCase, SoftSphereEngine
    eng = SoftSphereEngine(SoftCase(nz=64, nr=32, dx=1.0 / 64, z_cm=0.5, r_ball=0.15), dct=dct)
    eng.step(2)
    assert eng.status() == 0
    set_word(eng.plan_dct if dct else eng.sim.solver.engine.plan, 8)
    eng.step(1)
    assert eng.status() == CUDA_BIT


def test_sphere_loop_raises_on_a_failed_solve(monkeypatch):
    from pyaxisymflow_gb300.engine import RigidBodyCase
    from pyaxisymflow_gb300.simulation import RigidSphereSimulation
    sim = RigidSphereSimulation(RigidBodyCase(nz=64, nr=32, dx=2.0 / 64, r_sphere=0.2, z_cm=0.5))
    sim.step()
    solve = sim.solver.solve

    def fail(psi, w):
        solve(psi, w)
        psi.fill_(math.nan)
        set_word(sim.solver.engine.plan, 9)

    monkeypatch.setattr(sim.solver, "solve", fail)
    with pytest.raises(RuntimeError, match="solve failed"):
        sim.step()


@pytest.mark.parametrize("nz,nr", [(128, 64), (512, 256), (1024, 512)])
def test_engine_products_after_a_failure_are_right_or_nan(nz, nr):
    """With the plan's word set (it is not cleared there) waits may give up: psi
    holds no value that is neither the product's nor NaN, with narrow tiles (two
    sizes) and wide ones."""
    from pyaxisymflow_gb300.engine import RigidBodyCase, RigidEnsemble
    w0 = np.random.default_rng(nz).standard_normal((nr, nz))
    psi = []
    for word in (0, 9):
        e = RigidEnsemble([RigidBodyCase(nz=nz, nr=nr, dx=2.0 / nz, ramp=False)],
                          precision="f64", initial_vorticity=[w0])
        (info, plan, _, _), = e.plans
        set_word(plan, word, int(info.bytes) - 16)
        assert e.status()[0] == (CUDA_BIT if word else 0)
        e.fields[0]["psi"].fill_(7.0)
        for phase in (0, 1):
            e.phase(phase)
        torch.cuda.synchronize()
        psi.append(e.fields[0]["psi"])
    assert bool(((psi[1] == psi[0]) | torch.isnan(psi[1])).all())
