"""The mixed-precision kernels of wave and Euler (CUDA cores) and Maxwell (tensor
cores) at element counts around their tiles: within the mixed path's bound of the
FP64 result, and the same on both grids (Maxwell: as the general kernel's too)."""

from __future__ import annotations

import pytest
import torch

from tests._helpers import jittered_box_mesh, make_problem

pytestmark = pytest.mark.gpu

MIXED_RTOL = 1e-5


#: elements per SM from which the plans take the 32-element tiles
PER_SM = {"wave": (540, 350, 120, 120), "euler": (800, 100, 72, 72)}


@pytest.mark.parametrize("equation,order,extra", [
    ("wave", 1, 1), ("wave", 2, 1), ("euler", 1, 1), ("euler", 2, 1), ("euler", 2, 31),
    *[(eq, o, x) for eq in ("wave", "euler") for o in (3, 4) for x in (0, 1, 31)]])
def test_mixed_tile_edges(equation, order, extra):
    from actx_dgfem_suite_gb300.mesh import TetMesh
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    nel = PER_SM[equation][order - 1] * nsm + extra
    n = 2
    while 6 * n**3 < nel:
        n += 1
    mesh = jittered_box_mesh(n)
    mesh = TetMesh(vertices=mesh.vertices, elements=mesh.elements[:nel])
    prob = make_problem(equation, mesh, order, seed=extra)
    dm = DeviceMesh(prob.disc, "cuda:0")
    q = torch.from_numpy(prob.fields).cuda()
    scale = torch.linspace(0.8, 1.2, nel, dtype=torch.float64, device="cuda")
    got = {}
    for prec, variant in (("fp64", 0), ("fp32-mixed", 0), ("fp32-mixed", 2)):
        plan = DevicePlan(dm, equation, prob.params, prec)
        plan.set_variant(variant)
        if prec != "fp64":
            assert plan.info()["block"] != 256
        r = plan.rhs(q)
        plan.set_element_scale(scale)
        res, qo, un = 0.5 * q, torch.empty_like(q), torch.empty_like(q)
        plan.rk_stage(q, qo, res, 0.3, 0.7, 1e-2, rhs_unscaled=un)
        plan.finish()
        got[prec, variant] = (r, res, qo, un)
    for ref, a, b in zip(*got.values()):
        assert torch.equal(a, b)
        assert float(torch.linalg.norm(a - ref)) <= MIXED_RTOL * float(torch.linalg.norm(ref))


@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("extra", [0, 1, 9])
def test_maxwell_warp_tile_edges(order, extra):
    """Warps of 8 elements: variants 1 and 3 from 450 or 300 elements per SM on."""
    from actx_dgfem_suite_gb300.mesh import TetMesh
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    nel = {2: 450, 3: 300}[order] * nsm + extra
    n = 2
    while 6 * n**3 < nel:
        n += 1
    mesh = jittered_box_mesh(n)
    mesh = TetMesh(vertices=mesh.vertices, elements=mesh.elements[:nel])
    prob = make_problem("maxwell", mesh, order, seed=extra)
    dm = DeviceMesh(prob.disc, "cuda:0")
    q = torch.from_numpy(prob.fields).cuda()
    scale = torch.linspace(0.8, 1.2, nel, dtype=torch.float64, device="cuda")
    got = {}
    for prec, variant in (("fp64", 0), ("fp32-mixed", 7), ("fp32-mixed", 1), ("fp32-mixed", 3)):
        plan = DevicePlan(dm, "maxwell", (0.8, 1.3, 0.7), prec)
        plan.set_variant(variant)
        if variant in (1, 3):
            assert plan.info()["block"] == {2: 512, 3: 384}[order]
        r = plan.rhs(q)
        plan.set_element_scale(scale)
        res, qo, un = 0.5 * q, torch.empty_like(q), torch.empty_like(q)
        plan.rk_stage(q, qo, res, 0.3, 0.7, 1e-2, rhs_unscaled=un)
        first = torch.full_like(q, float("nan"))   # a = 0 does not read it
        plan.rk_stage(q, qo, first, 0.0, 0.7, 1e-2)
        plan.finish()
        got[prec, variant] = (r, res, qo, un, first)
    for ref, a, b, c in zip(*got.values()):
        assert torch.equal(a, b) and torch.equal(a, c)
        assert float(torch.linalg.norm(a - ref)) <= MIXED_RTOL * float(torch.linalg.norm(ref))


@pytest.mark.parametrize("equation,order,variants", [
    *[(eq, o, (0, 2)) for eq in ("wave", "euler") for o in (1, 2, 3, 4)],
    ("maxwell", 2, (1, 3)), ("maxwell", 3, (1, 3))])
def test_members_of_a_large_mesh_have_their_own_meshs_bits(equation, order, variants):
    """The kernels that plans take from some size on give the bits of the general
    kernel, which serves each member's own mesh: copies of one mesh of 750 elements
    (no multiple of any tile) side by side, each with a state of its own, RHS and RK
    stage."""
    from actx_dgfem_suite_gb300.discretization import union_discretization
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    per_sm = {2: 450, 3: 300}[order] if equation == "maxwell" else PER_SM[equation][order - 1]
    params = {"wave": (0.9,), "euler": (1.4,), "maxwell": (0.8, 1.3, 0.7)}[equation]
    prob = make_problem(equation, jittered_box_mesh(5), order, seed=order)
    other = make_problem(equation, jittered_box_mesh(5), order, seed=order + 7)
    nel = prob.disc.nelements
    count = per_sm * nsm // nel + 1
    union, offsets = union_discretization([prob.disc] * count)
    # convex combinations of two admissible states
    t = torch.linspace(0.0, 1.0, count, dtype=torch.float64, device="cuda")[:, None, None, None]
    both = [torch.from_numpy(p.fields).cuda() for p in (prob, other)]
    states = (1.0 - t) * both[0] + t * both[1]
    scale = torch.linspace(0.8, 1.2, nel * count, dtype=torch.float64, device="cuda")

    def evaluate(plan, q, scale):
        plan.set_element_scale(None)
        r = plan.rhs(q)
        plan.set_element_scale(scale)
        res, qo, un = 0.5 * q, torch.empty_like(q), torch.empty_like(q)
        plan.rk_stage(q, qo, res, 0.3, 0.7, 1e-2, rhs_unscaled=un)
        first, qf = torch.full_like(q, float("nan")), torch.empty_like(q)
        plan.rk_stage(q, qf, first, 0.0, 0.7, 1e-2)
        plan.finish()
        return r, res, qo, un, first, qf

    small = DevicePlan(DeviceMesh(prob.disc, "cuda:0"), equation, params, "fp32-mixed")
    small.set_variant(variants[0])
    assert small.info()["block"] == 256
    want = [torch.cat(x, dim=1) for x in zip(*[
        evaluate(small, states[k].contiguous(), scale[k * nel:(k + 1) * nel].contiguous())
        for k in range(count)])]
    large = DevicePlan(DeviceMesh(union, "cuda:0"), equation, params, "fp32-mixed")
    q = torch.cat(list(states), dim=1).contiguous()
    assert list(offsets) == [nel * k for k in range(count + 1)]
    for variant in variants:
        large.set_variant(variant)
        assert large.info()["block"] != 256
        for a, b in zip(evaluate(large, q, scale), want):
            assert torch.equal(a, b)


def test_euler_plan_holds_one_table_per_node():
    """Node records (32 bytes) and pressures (4 bytes) of a mixed Euler plan serve
    different variants, so the plan holds room for one of them."""
    from actx_dgfem_suite_gb300.device_setup import DeviceBoxDiscretization
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    disc = DeviceBoxDiscretization(4, 28, -0.5, 0.5, with_nodes=False)
    mesh = DeviceMesh(disc, "cuda:0")
    used = []
    for _ in range(2):                           # the first loads the kernels
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        plan = DevicePlan(mesh, "euler", (1.4,), "fp32-mixed")
        used.append(before - torch.cuda.mem_get_info()[0])
        plan.close()
    nodes = mesh.nelements * mesh.np_            # 4.6 million: 147.5 and 18.4 MB
    # operator blocks and allocation granularity: 8 MB
    assert used[1] <= 32 * nodes + 8 * 2**20


@pytest.mark.parametrize("equation,order,variant", [
    *[(eq, o, 0) for eq in ("wave", "euler") for o in (1, 2, 3, 4)],
    ("maxwell", 2, 1), ("maxwell", 3, 1)])
def test_extreme_states_have_the_general_kernels_bits(equation, order, variant):
    """Values outside the normal floats (and NaN, infinities, zeros) in whole elements
    and in single nodes of a member: the same values, signs and NaNs on both kernels."""
    from actx_dgfem_suite_gb300.discretization import union_discretization
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    per_sm = {2: 450, 3: 300}[order] if equation == "maxwell" else PER_SM[equation][order - 1]
    prob = make_problem(equation, jittered_box_mesh(5), order, seed=order)
    nel = prob.disc.nelements
    count = per_sm * nsm // nel + 1
    q = torch.from_numpy(prob.fields).cuda()
    values = [float("nan"), float("inf"), -float("inf"), 0.0, -0.0, 1e300, -1e300, 1e-300,
              1e38, 3.5e38, 1.1e-38, 1e-39, 1e-44, -1.1e-38, 1.7e38, -2.5]
    item = 0
    for value in values:
        for k in range(q.shape[0]):
            for node in (slice(None), item % q.shape[2]):
                q[k, (37 * item + 5) % nel, node] = value
                item += 1
    big = torch.cat([q] * count, dim=1).contiguous()
    union, _ = union_discretization([prob.disc] * count)
    got = []
    for disc, x in ((prob.disc, q), (union, big)):
        plan = DevicePlan(DeviceMesh(disc, "cuda:0"), equation, prob.params, "fp32-mixed")
        plan.set_variant(variant)
        r = plan.rhs(x)
        res, qo = torch.zeros_like(x), torch.empty_like(x)
        plan.rk_stage(x, qo, res, 0.3, 0.7, 1e-2)
        plan.finish()
        got.append([y[:, -nel:] for y in (r, res, qo)] + [plan.info()["kernel"]])
    assert got[0][3] != got[1][3]
    for a, b in zip(got[0][:3], got[1][:3]):
        nan = torch.isnan(a)
        assert torch.equal(nan, torch.isnan(b))
        assert torch.equal(a[~nan].view(torch.int64), b[~nan].view(torch.int64))
        assert bool(torch.isfinite(a).any())
