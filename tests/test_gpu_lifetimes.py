"""Tensors whose addresses go into a C call are alive until it returns."""
import weakref

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def watched(monkeypatch):
    """Every address taken with ptr() since the last call must belong to a living
    tensor when the next call is made."""
    from pyaxisymflow_gb300 import _native as N
    taken, calls = [], []
    ptr, call = N.ptr, N.call

    def watch(t, *args):
        if isinstance(t, torch.Tensor):
            # (a view's memory is its base's)
            taken.append(weakref.ref(t if t._base is None else t._base))
        return ptr(t, *args)

    def checked(name, *args):
        calls.append(name)
        assert all(r() is not None for r in taken), name
        taken.clear()
        return call(name, *args)

    monkeypatch.setattr(N, "ptr", watch)
    monkeypatch.setattr(N, "call", checked)
    return calls


@pytest.mark.parametrize("dct", [False, True])
def test_soft_engine(watched, dct):
    from pyaxisymflow_gb300.simulation import SoftCase, SoftSphereEngine
    eng = SoftSphereEngine(SoftCase(nz=64, nr=32, dx=1.0 / 64, z_cm=0.5, r_ball=0.15), dct=dct)
    eng.step(2)
    assert eng.status() == 0 and "axi_sliced_transform_plan" in watched


def test_loops_and_solvers(watched):
    from pyaxisymflow_gb300.engine import RigidBodyCase
    from pyaxisymflow_gb300.kernels.FastDiagonalisationStokesSolver import (
        FastDiagonalisationStokesSolver)
    from pyaxisymflow_gb300.simulation import RigidSphereSimulation, SoftCase, SoftSphereSimulation
    RigidSphereSimulation(RigidBodyCase(nz=64, nr=32, dx=2.0 / 64, r_sphere=0.2, z_cm=0.5)).step()
    SoftSphereSimulation(SoftCase(nz=64, nr=32, dx=1.0 / 64, z_cm=0.5, r_ball=0.15)).step()
    for real in (np.float32, np.float64):
        s = FastDiagonalisationStokesSolver(32, 64, 0.01, real_dtype=real)
        w = torch.ones((32, 66), dtype=torch.float64, device="cuda")[:, 1:65]
        s.solve(torch.zeros((32, 64), dtype=torch.float64, device="cuda"), w)
        assert s.engine.status() == 0
    assert len(watched) > 20
