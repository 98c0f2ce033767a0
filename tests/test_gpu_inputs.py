"""Inputs at the border of what the entry points take.

* a prescribed value of zero moves nothing to the rhs, whatever the stiffness entry
  (src/fem/assembly.cpp:95 skips it): one element with a modulus that is not a number leaves
  the rhs exactly the load where all prescribed values are zero;
* a nodal flux and a rhs in the same memory;
* device buffers that start between two doubles, for the history and the nodal flux;
* accumulation onto any values: each entry the rounded sum of what was there and what an
  assembly alone gives, in rows with and without prescribed columns;
* an edge with 4096 and 4200 elements around it: candidate lists that fill the shared memory of
  a block, and longer ones;
* elements that name a node two or three times: hexahedra collapsed to wedges, against the
  oracle. In mixed precision 1e-5: FP32 blocks of about 2e2 x 6e-8.

Bars: bit equality where both sides take the same steps, else 1e-12 relative Frobenius in
FP64 (sums of at most a few hundred products whose error is cond(J) eps <= 2e2 x 1.1e-16)."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from calculixpp_b200 import Batch, Material, Model, Plan, ThermalPlan, _lib
from calculixpp_b200 import meshgen as mg
from oracle.oracle import make_material
from tests.test_gpu_edges import check_linear, constrained, shuffled
from tests.helpers import ISO_TABLE, box_model, per_element_materials, rel_fro, to_np

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


def collapsed(etype, jitter=0.05, cells=(2, 2, 3)):
    """Wedges written as hexahedra whose fourth edge has collapsed onto the third."""
    quadratic = etype in (mg.C3D20, mg.C3D20R)
    w = mg.box_mesh(mg.C3D15 if quadratic else mg.C3D6, *cells, jitter=jitter, seed=1, straight_edges=True)
    local = [0, 1, 2, 2, 3, 4, 5, 5] + ([6, 7, 2, 8, 9, 10, 5, 11, 12, 13, 14, 14] if quadratic else [])
    m = mg.Mesh(w.coords, np.ascontiguousarray(w.conn[:, local]), etype)
    m.young = np.random.default_rng(2).uniform(70e3, 210e3, m.n_elems)
    m.poisson = np.full(m.n_elems, 0.3)
    top = mg.face_nodes(m, 2, 1.0)
    sn, sc, sv = mg.clamp_face_spc(m, 2, 0.0)
    return Model(m, [Material(210000.0, 0.3)], None, (sn, sc, sv + 1e-3),
                 (top, np.zeros(top.size, int), np.ones(top.size)))


@pytest.mark.parametrize("precision,bar", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("jitter", [0.0, 0.05])
@pytest.mark.parametrize("etype", [mg.C3D8, mg.C3D8R, mg.C3D20, mg.C3D20R])
def test_elements_that_name_a_node_twice(cuda, port, etype, jitter, precision, bar):
    model = collapsed(etype, jitter)
    mats, em = per_element_materials(model)
    dof_eq, pre, nf = model.dof_map()
    f = model.external_load_vector()
    rp, ci, v, rhs = port.assemble_linear(model.mesh, mats, em, dof_eq, pre, nf, f)
    with Plan(model, precision) as plan:
        vals, r = plan.assemble_linear(f)
        A = sp.csr_matrix((to_np(vals), *(to_np(t) for t in reversed(plan.pattern()))), shape=(nf, nf))
        O = sp.csr_matrix((v, ci, rp), shape=(nf, nf))
        assert np.linalg.norm((A - O).data) <= bar * np.linalg.norm(v)
        assert rel_fro(to_np(r), rhs) <= bar
        plan.use_reference_pattern()
        assert all(np.array_equal(to_np(a), b) for a, b in zip(plan.pattern(), (rp, ci)))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_elements_that_name_a_node_twice_in_windows_and_batches(cuda, precision):
    models = [collapsed(mg.C3D8, cells=(2, 2, 24)), box_model(mg.C3D20, 2, 2, 2)]
    with Plan(models[0], precision) as plan:
        want = plan.assemble_linear()
        plan.set_ring_bytes(72 * 36 * (72 if precision == "fp64" else 36))
        got = plan.assemble_linear()
        assert plan.windows()[0] > 1
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    batch = Batch(models, precision)
    for mode in ("per_group", "one_launch"):
        batch.set_launch(mode)
        got = batch.slices(0, *batch.assemble())
        assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_plastic_elements_that_name_a_node_twice(cuda, port):
    model = collapsed(mg.C3D8)
    model.mesh.young[:] = 210000.0
    model.materials = [Material(210000.0, 0.3, ISO_TABLE)]
    dof_eq, pre, nf = model.dof_map()
    u = np.einsum("ij,nj->ni", np.random.default_rng(3).uniform(-0.01, 0.01, (3, 3)), model.mesh.coords).reshape(-1)
    with Plan(model) as plan:
        state = np.zeros((plan.n_gauss, 13))
        mats = [make_material(210000.0, 0.3, ISO_TABLE, 0, 0.0)]
        rp, ci, v, rhs, fi, _ = port.assemble_tangent(model.mesh, mats, None, dof_eq, pre, nf, u, state)
        vals, f_int, r = plan.assemble_tangent(u)
        assert (to_np(plan.state(committed=False))[:, 6] > 0).any()
        assert rel_fro(to_np(vals), v) <= 1e-12
        assert rel_fro(to_np(f_int), fi) <= 1e-12


def between_doubles(values):
    """A device copy of the values four bytes off their alignment: (buffer, address)."""
    raw = torch.zeros(8 * values.size + 8, dtype=torch.uint8, device="cuda")
    raw[4:-4] = torch.as_tensor(np.ascontiguousarray(values).reshape(-1).view(np.uint8), device="cuda")
    return raw, raw.data_ptr() + 4


def test_buffers_between_two_doubles(cuda):
    model = box_model(mg.C3D8, 2, 2, 2)
    with Plan(model) as plan:
        want = np.random.default_rng(0).normal(size=(plan.n_gauss, 13))
        for slot in (0, 1):
            raw, at = between_doubles(want)
            _lib.check(plan.lib.cxg_state_set(plan.h, slot, at))
            back, at = between_doubles(np.zeros_like(want))
            _lib.check(plan.lib.cxg_state_get(plan.h, slot, at))
            assert np.array_equal(to_np(back)[4:-4].view(np.float64).reshape(want.shape), want)
    q = np.random.default_rng(1).normal(size=model.mesh.n_nodes)
    k = torch.ones(model.mesh.n_elems, dtype=torch.float64, device=cuda)
    with ThermalPlan(model.mesh, [0], [300.0]) as plan:
        vals, rhs = plan.assemble_conduction(k, q)
        raw, at = between_doubles(q)
        v, r = torch.empty_like(vals), torch.empty_like(rhs)
        _lib.check(plan.lib.cxg_assemble_conduction(plan.h, k.data_ptr(), at, v.data_ptr(), r.data_ptr(), None))
        plan.check()
        assert torch.equal(v, vals) and torch.equal(r, rhs)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("etype", [mg.C3D8, mg.C3D10, mg.C3D20])
def test_accumulation_is_the_sum(cuda, etype, precision):
    model = box_model(etype, 5, 3, 3, prescribe=1e-3)
    rng = np.random.default_rng(etype)
    with Plan(model, precision) as plan:
        vals, rhs = plan.assemble_linear()
        v0 = torch.as_tensor(rng.normal(size=plan.nnz) * float(vals.abs().max()), device=cuda)
        r0 = torch.as_tensor(rng.normal(size=plan.n_free) * float(rhs.abs().max()), device=cuda)
        v, r = v0.clone(), r0.clone()
        plan.accumulate_linear(v, r)
        assert torch.equal(v, v0 + vals) and torch.equal(r, r0 + rhs)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_accumulation_in_windows(cuda, precision):
    model = box_model(mg.C3D8, 32, 2, 3, prescribe=1e-3)
    with Plan(model, precision) as plan:
        vals, rhs = plan.assemble_linear()
        plan.set_ring_bytes(192 * 36 * (72 if precision == "fp64" else 36))
        v, r = vals.clone(), rhs.clone()
        plan.accumulate_linear(v, r)
        assert plan.windows()[0] > 1
        assert torch.equal(v, vals + vals) and torch.equal(r, rhs + rhs)


@pytest.mark.parametrize("count", [4096, 4200])
def test_large_fan_around_an_edge(cuda, port, count):
    rng = np.random.default_rng(count)
    a = 2.0 * np.pi * np.arange(count) / count
    ring = np.stack([np.cos(a), np.sin(a), np.zeros(count)], axis=1)
    i = np.arange(count)
    conn = np.stack([np.zeros_like(i), 2 + i, 2 + (i + 1) % count, np.ones_like(i)], axis=1).astype(np.int32)
    fan = mg.Mesh(np.concatenate([[[0.0, 0.0, -0.5], [0.0, 0.0, 0.5]], ring]), conn, mg.C3D4)
    check_linear(port, constrained(shuffled(fan, rng), rng, 0.1))
