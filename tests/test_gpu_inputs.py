"""Inputs at the border of what the entry points take.

* a prescribed value of zero moves nothing to the rhs, whatever the stiffness entry
  (src/fem/assembly.cpp:95 skips it): one element with a modulus that is not a number leaves
  the rhs exactly the load where all prescribed values are zero;
* a nodal flux and a rhs in the same memory.

Bars: bit equality where both sides take the same steps, else 1e-12 relative Frobenius in
FP64 (sums of at most a few hundred products whose error is cond(J) eps <= 2e2 x 1.1e-16)."""
import numpy as np
import pytest
import torch

from calculixpp_b200 import Plan, ThermalPlan
from calculixpp_b200 import meshgen as mg
from tests.helpers import box_model, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("etype", [mg.C3D8, mg.C3D10])
def test_zero_prescribed_values_move_nothing(cuda, etype, precision):
    model = box_model(etype, 3, 2, 2)
    model.mesh.young[0] = np.nan  # at the clamped face
    f = np.random.default_rng(0).normal(size=3 * model.mesh.n_nodes)
    with Plan(model, precision) as plan:
        vals, rhs = plan.assemble_linear(f)
        assert torch.isnan(vals).any()
        assert np.array_equal(to_np(rhs), f[plan.dof_eq >= 0])


def test_zero_prescribed_temperatures_move_nothing(cuda):
    mesh = box_model(mg.C3D15, 3, 2, 2).mesh
    held = mg.face_nodes(mesh, 0, 0.0)
    k = np.ones(mesh.n_elems)
    k[0] = np.inf
    q = np.random.default_rng(0).normal(size=mesh.n_nodes)
    with ThermalPlan(mesh, held, np.zeros(held.size)) as plan:
        vals, rhs = plan.assemble_conduction(k, q)
        assert not torch.isfinite(vals).all()
        assert np.array_equal(to_np(rhs), q[plan.t_dof_eq >= 0])


def test_flux_in_the_memory_of_the_rhs(cuda):
    mesh = box_model(mg.C3D8, 9, 8, 7).mesh
    held = mg.face_nodes(mesh, 0, 0.0)
    rng = np.random.default_rng(0)
    k, flux = rng.uniform(10.0, 50.0, mesh.n_elems), rng.normal(size=mesh.n_nodes)
    with ThermalPlan(mesh, held, rng.uniform(280.0, 320.0, held.size)) as plan:
        vals, rhs = plan.assemble_conduction(k, flux)
        both = torch.as_tensor(flux, device=cuda)
        v, r = plan.assemble_conduction(k, both, rhs=both[:plan.n_free])
        assert torch.equal(v, vals) and torch.equal(r, rhs)
