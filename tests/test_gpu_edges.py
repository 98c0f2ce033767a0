"""Edges of the kernels' batches, records and lists, against the oracle.

* meshes of 1 to 7 elements with shuffled node numbers and single components constrained
  at random: partly filled element batches, blocks stored in either node order, compressed
  rows, and the product over them;
* a fan of tetrahedra around one edge: nodes with 3 to 600 elements, whose candidate lists
  are ordered in shared memory up to 2048 entries and in global memory beyond;
* calls queued behind one another on a side stream, and work buffers shared by two streams:
  the same bits as from one stream with a wait after each call.

Bar: 1e-12 relative Frobenius. Both sides round in FP64 along different orders: a sum of at
most 600 x 27 products of gradients whose error is cond(J) eps <= 2e2 x 1.1e-16."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from calculixpp_b200 import Plan
from calculixpp_b200 import meshgen as mg
from calculixpp_b200.assembly import Material, Model
from tests.helpers import ALL_TYPES, box_model, per_element_materials, rel_fro, to_np

pytestmark = pytest.mark.gpu


def shuffled(mesh, rng):
    """The same mesh with its nodes renumbered at random."""
    to = rng.permutation(mesh.n_nodes)
    coords = np.empty_like(mesh.coords)
    coords[to] = mesh.coords
    return mg.Mesh(coords, to[mesh.conn].astype(np.int32), mesh.etype)


def constrained(mesh, rng, share):
    """A model with that share of all DOFs prescribed, and a load on every node."""
    mesh.young = rng.uniform(70e3, 210e3, mesh.n_elems)
    mesh.poisson = np.full(mesh.n_elems, 0.3)
    dof = np.flatnonzero(rng.random(3 * mesh.n_nodes) < share)
    nodes = np.arange(mesh.n_nodes)
    return Model(mesh, [Material(210000.0, 0.3)], None,
                 ((dof // 3).astype(np.int32), (dof % 3).astype(np.int32), rng.uniform(-1e-2, 1e-2, dof.size)),
                 (nodes, nodes % 3, rng.normal(size=nodes.size)))


def check_linear(port, model):
    mats, em = per_element_materials(model)
    dof_eq, pre, nf = model.dof_map()
    f = model.external_load_vector()
    rp, ci, v, rhs = port.assemble_linear(model.mesh, mats, em, dof_eq, pre, nf, f)
    with Plan(model) as plan:
        vals, r = plan.assemble_linear(f)
        A = sp.csr_matrix((to_np(vals), *(to_np(t) for t in reversed(plan.pattern()))), shape=(nf, nf))
        O = sp.csr_matrix((v, ci, rp), shape=(nf, nf))
        assert np.linalg.norm((A - O).data) <= 1e-12 * np.linalg.norm(v)
        assert rel_fro(to_np(r), rhs) <= 1e-12
        x = np.linspace(-1.0, 1.0, nf)
        assert rel_fro(to_np(plan.spmv(vals, torch.as_tensor(x, device=plan.device))), O @ x) <= 1e-12


@pytest.mark.parametrize("cells", [1, 2, 3, 5, 7])
@pytest.mark.parametrize("etype", ALL_TYPES)
def test_few_elements_any_numbering(cuda, port, etype, cells):
    rng = np.random.default_rng(100 * etype + cells)
    mesh = shuffled(mg.box_mesh(etype, cells, 1, 1, float(cells), jitter=0.05, seed=cells), rng)
    check_linear(port, constrained(mesh, rng, 0.3))


@pytest.mark.parametrize("count", [3, 11, 12, 128, 512, 513, 600])
def test_fan_around_an_edge(cuda, port, count):
    rng = np.random.default_rng(count)
    a = 2.0 * np.pi * np.arange(count) / count
    ring = np.stack([np.cos(a), np.sin(a), np.zeros(count)], axis=1)
    coords = np.concatenate([[[0.0, 0.0, -0.5], [0.0, 0.0, 0.5]], ring])
    i = np.arange(count)
    conn = np.stack([np.zeros_like(i), 2 + i, 2 + (i + 1) % count, np.ones_like(i)], axis=1).astype(np.int32)
    check_linear(port, constrained(shuffled(mg.Mesh(coords, conn, mg.C3D4), rng), rng, 0.1))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("etype", [mg.C3D8, mg.C3D20R])
def test_queued_calls_give_the_same_bits(cuda, etype, precision):
    model = box_model(etype, 3, 2, 2, jitter=0.05, seed=3)
    n = model.mesh.n_nodes
    rng = np.random.default_rng(1)
    loads = [torch.as_tensor(rng.normal(size=3 * n), device=cuda) for _ in range(4)]
    us = [torch.as_tensor(rng.uniform(-1e-3, 1e-3, 3 * n), device=cuda) for _ in range(4)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    with Plan(model, precision) as plan:
        def step(k):
            return (*plan.assemble_linear(loads[k], check=False), *plan.recover_fields(us[k], loads[k]),
                    plan.recover_gauss_stress(us[k]))

        want = []
        for k in range(4):
            want.append(step(k))
            torch.cuda.synchronize()
        for rounds in (streams[:1], streams):
            got = []
            for k in range(4):
                s = rounds[k % len(rounds)]
                s.wait_stream(rounds[(k - 1) % len(rounds)])
                with torch.cuda.stream(s):
                    got.append(step(k))
            torch.cuda.synchronize()
            for a, b in zip(want, got):
                assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_plans_come_and_go(cuda):
    """Plans of many sizes, alive together and freed in turn, give what a plan alone does."""
    models = [box_model(mg.C3D10, k, 2, 1, seed=k) for k in (1, 4, 2, 6)]
    alone = []
    for m in models:
        with Plan(m) as plan:
            alone.append([to_np(t).copy() for t in plan.assemble_linear(m.external_load_vector())])
    for _ in range(3):
        plans = [Plan(m) for m in models]
        for k in (2, 0, 3, 1):
            got = plans[k].assemble_linear(models[k].external_load_vector())
            assert all(np.array_equal(to_np(a), b) for a, b in zip(got, alone[k]))
            plans[k].close()
