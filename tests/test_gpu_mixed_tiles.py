"""The CUDA-core mixed-precision kernels of wave and Euler at element counts
around their 32-element tile: within the mixed path's bound of the FP64 result,
and the same on both grids."""

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
