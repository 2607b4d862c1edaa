"""Launch variants and the autotuner: the mixed-precision kernel with its
contractions on the tensor cores (3xTF32, FP32 accumulation; warp-level
mma.sync at three tile shapes, or one tcgen05 product per tile) keeps the
mixed path's accuracy; the one-CTA-per-tile grid gives identical results."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests._helpers import jittered_box_mesh, make_problem

pytestmark = pytest.mark.gpu

MIXED_RTOL = 1e-5
# the 3xTF32 tcgen05 variant: FP32-class accuracy, with the tensor core's own
# accumulation order (the bounded autotuner decides where it is admissible)
TF32_RTOL = 5e-5
RTOL = {4: MIXED_RTOL, 5: TF32_RTOL, 6: TF32_RTOL}


def _plans(equation, order, seed=0):
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    prob = make_problem(equation, jittered_box_mesh(4), order, seed=seed)
    dm = DeviceMesh(prob.disc, "cuda:0")
    ref = DevicePlan(dm, equation, prob.params, "fp64")
    mixed = DevicePlan(dm, equation, prob.params, "fp32-mixed")
    return prob, ref, mixed


@pytest.mark.parametrize("equation", ["wave", "euler", "maxwell"])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_tensor_core_mixed_matches_fp64(equation, order):
    prob, ref, mixed = _plans(equation, order, seed=order)
    q = torch.from_numpy(prob.fields).cuda()
    r64 = ref.rhs(q)
    mixed.set_variant(0)
    r0 = mixed.rhs(q)
    mixed.set_variant(1)
    assert mixed.info()["tensor_cores"]
    r1 = mixed.rhs(q)
    mixed.set_variant(3)
    r3 = mixed.rhs(q)
    shaped = {}
    for v in (7, 8, 9, 10):   # 128- and 512-thread tiles, both grids
        mixed.set_variant(v)
        info = mixed.info()
        assert info["tensor_cores"] and info["block"] == (128 if v <= 8 else 512)
        shaped[v] = mixed.rhs(q)
    mixed.finish()
    n64 = float(torch.linalg.norm(r64))
    assert float(torch.linalg.norm(r1 - r64)) <= MIXED_RTOL * n64
    assert float(torch.linalg.norm(r1 - r0)) <= MIXED_RTOL * n64
    assert torch.equal(r1, r3)            # same tiles, same arithmetic
    for v, r in shaped.items():
        assert float(torch.linalg.norm(r - r64)) <= MIXED_RTOL * n64, v
    assert torch.equal(shaped[7], shaped[8])
    assert torch.equal(shaped[9], shaped[10])


@pytest.mark.parametrize("variant", [1, 7, 10])
def test_tensor_core_mixed_rk_stage(variant):
    prob, ref, mixed = _plans("euler", 3, seed=4)
    q = torch.from_numpy(prob.fields).cuda()
    outs = []
    for plan, v in ((ref, 0), (mixed, variant)):
        plan.set_variant(v)
        res = torch.zeros_like(q)
        qo = torch.empty_like(q)
        plan.rk_stage(q, qo, res, 0.0, 0.5, 1e-3)
        plan.finish()
        outs.append((qo, res))
    dres = float(torch.linalg.norm(outs[1][1] - outs[0][1]))
    assert dres <= MIXED_RTOL * float(torch.linalg.norm(outs[0][1]))


def test_autotune_picks_a_supported_variant():
    prob, ref, mixed = _plans("maxwell", 3)
    q = torch.from_numpy(prob.fields).cuda()
    res = mixed.autotune(q, reps=2)
    assert res["chosen"] in range(len(mixed.VARIANTS))
    assert all(v is not None and v > 0 for v in res["ms"].values())
    res64 = ref.autotune(q, reps=2)
    assert res64["chosen"] in (0, 2)
    assert res64["ms"]["tensor-core, persistent"] is None
    assert all(res64["ms"][mixed.VARIANTS[v]] is None for v in (7, 8, 9, 10))
    from actx_dgfem_suite_gb300._lib import DGError
    for v in (1, 7, 10):
        with pytest.raises(DGError):
            ref.set_variant(v)


def test_bounded_autotune_respects_the_error_budget():
    """dg_plan_autotune_bounded: every reported error is the variant's true
    relative L2 distance from the FP64 result, and the chosen variant lies
    within the budget (or is the most accurate when none does)."""
    prob, ref, mixed = _plans("wave", 3, seed=2)
    q = torch.from_numpy(prob.fields).cuda()
    r64 = ref.rhs(q)
    ref.finish()
    names = {v: k for k, v in mixed.VARIANTS.items()}
    for budget in (1e-3, 0.0):
        res = mixed.autotune(q, reps=1, ref=r64, max_rel_l2=budget)
        errs = {names[k]: v for k, v in res["rel_l2"].items() if v is not None}
        assert set(errs) == set(range(len(mixed.VARIANTS)))
        for v, e in errs.items():  # the reported errors are the real ones
            mixed.set_variant(v)
            got = mixed.rhs(q)
            true = float(torch.linalg.norm(got - r64) / torch.linalg.norm(r64))
            assert abs(true - e) <= 1e-3 * true + 1e-15, (v, e, true)
        inside = [v for v, e in errs.items() if e <= budget]
        if inside:
            ms = {names[k]: v for k, v in res["ms"].items() if v is not None}
            assert res["chosen"] in inside
            assert ms[res["chosen"]] == min(ms[v] for v in inside)
        else:  # nothing meets a zero budget: the most accurate is kept
            assert res["chosen"] == min(errs, key=errs.get)
    mixed.finish()


@pytest.mark.parametrize("variant", [4, 5, 6])
@pytest.mark.parametrize("equation", ["wave", "euler", "maxwell"])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_tcgen05_mixed_matches_fp64(equation, order, variant):
    """Variants 4 and 5: [A_0 A_1 A_2 | LIFT] applied to the metric-combined
    inputs and face values as one tcgen05 product per tile (partial last
    tile), exact digit pairs or 3xTF32."""
    prob, ref, mixed = _plans(equation, order, seed=20 + order)
    q = torch.from_numpy(prob.fields).cuda()
    r64 = ref.rhs(q)
    mixed.set_variant(0)
    r0 = mixed.rhs(q)
    mixed.set_variant(variant)
    assert mixed.info()["tensor_cores"]
    r4 = mixed.rhs(q)
    mixed.finish()
    n64 = float(torch.linalg.norm(r64))
    assert float(torch.linalg.norm(r4 - r64)) <= RTOL[variant] * n64
    assert float(torch.linalg.norm(r4 - r0)) <= RTOL[variant] * n64


@pytest.mark.parametrize("variant", [4, 5, 6])
@pytest.mark.parametrize("equation,order", [("maxwell", 3), ("euler", 2), ("wave", 4)])
def test_tcgen05_mixed_many_tiles_per_cta(equation, order, variant):
    """More tiles than CTAs: every CTA runs the persistent loop several times."""
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    prob = make_problem(equation, jittered_box_mesh(20), order, seed=3)
    dm = DeviceMesh(prob.disc, "cuda:0")
    ref = DevicePlan(dm, equation, prob.params, "fp64")
    mixed = DevicePlan(dm, equation, prob.params, "fp32-mixed")
    mixed.set_variant(variant)
    tile = 128 // prob.fields.shape[0]   # elements per tile
    assert prob.disc.nelements > 2 * mixed.info()["grid"] * tile
    q = torch.from_numpy(prob.fields).cuda()
    r64 = ref.rhs(q)
    r4 = mixed.rhs(q)
    mixed.finish()
    n64 = float(torch.linalg.norm(r64))
    assert float(torch.linalg.norm(r4 - r64)) <= RTOL[variant] * n64


@pytest.mark.parametrize("variant", [4, 5, 6])
def test_tcgen05_mixed_rk_stage_and_element_scale(variant):
    prob, ref, mixed = _plans("wave", 3, seed=5)
    q = torch.from_numpy(prob.fields).cuda()
    nel = prob.disc.nelements
    scale = torch.linspace(0.8, 1.2, nel, dtype=torch.float64, device="cuda:0")
    res0 = torch.rand(q.shape, dtype=q.dtype, device=q.device,
                      generator=torch.Generator(device=q.device).manual_seed(7))
    outs = []
    for plan, v in ((ref, 0), (mixed, variant)):
        plan.set_variant(v)
        plan.set_element_scale(scale)
        res = res0.clone()
        qo = torch.empty_like(q)
        unscaled = torch.empty_like(q)
        plan.rk_stage(q, qo, res, 0.3, 0.5, 1e-3, rhs_unscaled=unscaled)
        plan.finish()
        outs.append((qo, res, unscaled))
    for k in range(3):
        ref_k = outs[0][k]
        assert float(torch.linalg.norm(outs[1][k] - ref_k)) <= \
            RTOL[variant] * float(torch.linalg.norm(ref_k))


@pytest.mark.parametrize("variant", [4, 5, 6])
def test_tcgen05_nan_stays_local(variant):
    """A NaN in one element's state reaches that element and its face
    neighbours only: X's padding columns, which share bytes with the other
    phase's layout and (3xTF32) with the previous tile's staged results, are
    rewritten with zeros before every product reads them."""
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    prob = make_problem("maxwell", jittered_box_mesh(12), 3, seed=4)
    dm = DeviceMesh(prob.disc, "cuda:0")
    mixed = DevicePlan(dm, "maxwell", prob.params, "fp32-mixed")
    q = torch.from_numpy(prob.fields).cuda()
    mixed.set_variant(0)
    ref = mixed.rhs(q)
    bad = 7
    qn = q.clone()
    qn[2, bad, 3] = float("nan")
    mixed.set_variant(variant)
    out = mixed.rhs(qn)
    mixed.finish()
    # elements sharing a face with the bad one (or the bad one itself)
    gather = prob.disc.gather_index()          # (Nel, 4, Nfp) flat exterior index
    np_ = prob.disc.np_
    ext_el = (gather.astype(np.int64) & 0x7FFFFFFF) // np_
    bdry = (gather >> 31).astype(bool)
    touched = {bad}
    touched |= set(np.nonzero(((ext_el == bad) & ~bdry).any(axis=(1, 2)))[0].tolist())
    finite = torch.isfinite(out).all(dim=(0, 2)).cpu().numpy()
    assert not finite[bad]
    others = np.array([e for e in range(prob.disc.nelements) if e not in touched])
    assert finite[others].all()
    n = float(torch.linalg.norm(ref[:, others]))
    assert float(torch.linalg.norm(out[:, others] - ref[:, others])) <= RTOL[variant] * n


def test_bounded_autotune_at_mid_size_wave_p3():
    """Wave P3 on the benchmark definition at n = 24 (82,944 tets, where the
    3xTF32 mma.sync variants exceed 1e-5 on the largest meshes): the
    variant the bounded autotuner keeps is within 1e-5 of the FP64 RHS."""
    from actx_dgfem_suite_gb300.array_context import GB300DGArrayContext
    from actx_dgfem_suite_gb300.rhs_builder import get_rhs
    actx = GB300DGArrayContext("cuda:0")
    rhs, args = get_rhs("wave", actx, 3, 3, definition="baseline", nel_1d=24,
                        device_setup=True)
    op = rhs.dg_operator
    q = actx.compile(rhs).stage(args[-1])
    r64 = op.plan_for(actx).rhs(q)
    op.precision = "fp32-mixed"
    mixed = op.plan_for(actx)
    res = mixed.autotune(q, reps=2, ref=r64, max_rel_l2=MIXED_RTOL)
    chosen_err = res["rel_l2"][mixed.VARIANTS[res["chosen"]]]
    assert chosen_err is not None and chosen_err <= MIXED_RTOL
    out = mixed.rhs(q)
    mixed.finish()
    assert float(torch.linalg.norm(out - r64) / torch.linalg.norm(r64)) <= MIXED_RTOL


@pytest.mark.parametrize("equation,order,precision,small,large", [
    ("wave", 3, "fp64", "dg_rhs_kernel", "dg_rhs_sym_kernel"),
    ("euler", 2, "fp64", "dg_rhs_kernel", "dg_rhs_sym_kernel"),
    ("maxwell", 4, "fp64", "dg_rhs_sym_kernel", "dg_rhs_sym_kernel"),
    ("euler", 3, "fp64-tc", "dg_rhs_tc_kernel", "dg_rhs_tc_kernel"),
    ("euler", 4, "fp32-mixed", "dg_rhs_kernel", "dg_rhs_mixed_kernel")])
def test_info_names_the_kernel(equation, order, precision, small, large):
    """Small meshes and large ones; and operators without the symmetry."""
    from actx_dgfem_suite_gb300.discretization import make_box_discretization
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    params = {"wave": (1.0,), "euler": (1.4,), "maxwell": (1.0, 1.0, 1.0)}[equation]
    for n, name in ((2, small), (13, large)):
        mesh = DeviceMesh(make_box_discretization(order, n), "cuda:0")
        plan = DevicePlan(mesh, equation, params, precision)
        assert plan.info()["kernel"] == name
        if precision == "fp32-mixed":
            for variant, other in ((1, "dg_rhs_kernel"), (5, "dg_rhs_tcm_kernel"),
                                   (7, "dg_rhs_kernel")):
                plan.set_variant(variant)
                assert plan.info()["kernel"] == other
        if precision == "fp64":
            mesh._weak, mesh._strong = 1.01 * mesh._weak, 1.01 * mesh._strong
            mesh._weak.reshape(-1)[0] = mesh._strong.reshape(-1)[0] = 0.0
            assert DevicePlan(mesh, equation, params).info()["kernel"] == "dg_rhs_kernel"
