"""The symmetry-adapted operator blocks (``pack_sym_ops``): applied to the
transformed inputs they reproduce the dense derivative and LIFT products, and
operators without the tetrahedron's symmetry are refused (such plans keep the
general kernels).  The block product is restated here in NumPy."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from actx_dgfem_suite_gb300 import _lib
from actx_dgfem_suite_gb300.refelem import reference_tet

EPS = np.finfo(np.float64).eps


def _pack(order, diff, lift, face_nodes, strong=None, reduce=False):
    """The block of the forward (``strong`` given) or adjoint operators; ``reduce``:
    products through coefficients of one degree less."""
    lib = ctypes.CDLL(str(_lib.library_path()))
    if strong is None:
        f, extra = lib._ZN2dg16pack_sym_adj_opsEiPKdS1_PKibPhi, []
    else:
        f, extra = lib._ZN2dg12pack_sym_opsEiPKdS1_PKibbPhi, [ctypes.c_bool(strong)]
    extra.append(ctypes.c_bool(reduce))
    f.restype = ctypes.c_int
    diff, lift = np.ascontiguousarray(diff), np.ascontiguousarray(lift)
    fn = np.ascontiguousarray(face_nodes, dtype=np.int32)
    args = [ctypes.c_int(order)] + [ctypes.c_void_p(x.ctypes.data) for x in (diff, lift, fn)]
    size = f(*args, *extra, None, 0)
    buf = np.zeros(size, dtype=np.uint8)
    got = f(*args, *extra, ctypes.c_void_p(buf.ctypes.data), size)
    return buf if got == size else None


class _Blocks:
    """The operator block of order N read back in the kernel's layout."""

    def __init__(self, order, buf, adjoint=False, reduced=None):
        self.np_ = (order + 1) * (order + 2) * (order + 3) // 6
        self.nfp = (order + 1) * (order + 2) // 2
        npr, nsg = int(order % 2 == 0), int(order == 4)
        self.no4 = (self.np_ - 6 * npr - nsg) // 4
        self.npr, self.db, self.da = npr, self.no4 + npr, self.no4 + 3 * npr + nsg
        even = lambda n: (n + 1) & ~1  # noqa: E731
        pitch = [even(self.da)] + 3 * [even(self.db)]
        dim = [self.da] + 3 * [self.db]
        self.slot0 = [0] + [self.da + k * self.db for k in range(3)]
        x = buf.view(np.float64) if buf.size % 8 == 0 else None
        pos = 0
        self.vol, self.lift = {}, {}
        # the space of degree N - 1 in every part: the blocks' outputs ("out") or inputs
        rank = {2: (1, 1), 3: (4, 2), 4: (5, 5)}.get(order, (0, 0))
        rank = [rank[0]] + 3 * [rank[1]]
        nin, nout = (rank if reduced == "in" else dim), (rank if reduced == "out" else dim)
        for r in range(4):
            for k in range(1, 4):
                n = nin[r ^ k] * even(nout[r])
                self.vol[r, k] = x[pos:pos + n].reshape(-1, even(nout[r]))[:, :nout[r]].T
                pos += n
        more = {}
        for r in range(4 if reduced else 0):
            rows, cols = (dim[r], rank[r]) if reduced == "in" else (rank[r], dim[r])
            n = rows * even(cols)
            more[r] = x[pos:pos + n].reshape(-1, even(cols))[:, :cols].T
            pos += n
        for r, k in self.vol if reduced else ():
            self.vol[r, k] = (self.vol[r, k] @ more[r ^ k] if reduced == "in"
                              else more[r] @ self.vol[r, k])
        if adjoint:                              # chunks of orbits, rows by node slot
            ch = self.nfp if order == 1 else (self.nfp + 1) // 2
            nch = -(-self.nfp // ch)
            n = nch * self.np_ * even(ch)
            t = x[pos:pos + n].reshape(nch, self.np_, even(ch))[:, :, :ch]
            t = t.transpose(1, 0, 2).reshape(self.np_, -1)
            assert not t[:, self.nfp:].any()
            for r in range(4):
                self.lift[r] = t[self.slot0[r]:self.slot0[r] + dim[r], :self.nfp].T
            pos += n
        for r in range(0 if adjoint else 4):
            n = self.nfp * pitch[r]
            self.lift[r] = x[pos:pos + n].reshape(-1, pitch[r])[:, :dim[r]].T
            pos += n
        tab = buf.view(np.int32)
        pos *= 2
        self.node_slot = tab[pos:pos + self.np_]
        pos += (self.np_ + 3) // 4 * 4
        self.slot_node = tab[pos:pos + self.np_]
        pos += (self.np_ + 3) // 4 * 4
        self.face_point = tab[pos:pos + 4 * self.nfp]
        self.dim = dim

    def transform(self, x):
        """In place on slots (last axis); applying it twice scales by 4, 2, 1."""
        h = np.array([[1, 1, 1, 1], [1, 1, -1, -1], [1, -1, 1, -1], [1, -1, -1, 1.0]])
        for o in range(self.no4):
            s = [o] + [self.slot0[k] + o for k in (1, 2, 3)]
            x[..., s] = x[..., s] @ h
        for k in range(3 * self.npr):
            s = [self.no4 + k, self.slot0[k + 1] + self.no4]
            x[..., s] = x[..., s] @ np.array([[1, 1], [1, -1.0]])
        return x

    def part(self, r):
        return slice(self.slot0[r], self.slot0[r] + self.dim[r])


@pytest.mark.parametrize("reduce", [False, True])
@pytest.mark.parametrize("strong", [False, True])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_blocks_reproduce_the_dense_operators(order, strong, reduce):
    ref = reference_tet(order)
    diff = ref.diff if strong else ref.weak_diff
    b = _Blocks(order, _pack(order, diff, ref.lift, ref.face_nodes, strong, reduce),
                reduced=("out" if strong else "in") if reduce and order > 1 else None)
    assert sorted(b.node_slot) == list(range(b.np_))
    assert list(b.slot_node[b.node_slot]) == list(range(b.np_))
    assert sorted(b.face_point) == list(range(4 * b.nfp))
    rng = np.random.default_rng(order)
    x = rng.standard_normal((7, b.np_))
    g = rng.standard_normal((3, 7, 1))           # one metric row per direction
    xs = np.empty_like(x)
    xs[:, b.node_slot] = x
    xs = b.transform(xs)
    h = [g[1] + g[2], g[0] + g[2], g[0] + g[1]]
    ys = np.zeros_like(xs)
    for r in range(4):
        for k in (1, 2, 3):
            if order == 1 and (r if strong else r ^ k) != 0:
                continue                         # not evaluated by the kernel
            ys[:, b.part(r)] += h[k - 1] * (xs[:, b.part(r ^ k)] @ b.vol[r, k].T)
    y = b.transform(ys)[:, b.node_slot]
    dense = sum(g[r] * (x @ diff[r].T) for r in range(3))
    # sums of 3 Np products of unit-size entries on either side
    scale = sum(np.abs(g[r]) * (np.abs(x) @ np.abs(diff[r]).T) for r in range(3))
    assert np.all(np.abs(y - dense) <= 3 * b.np_ * EPS * scale.max())

    f = rng.standard_normal((7, 4 * b.nfp))
    h4 = np.array([[1, 1, 1, 1], [1, 1, -1, -1], [1, -1, 1, -1], [1, -1, -1, 1.0]])
    fs = np.einsum("rg,ego->ero", h4, f[:, b.face_point].reshape(7, 4, b.nfp))
    ys = np.zeros_like(xs)
    for r in range(4):
        ys[:, b.part(r)] = fs[:, r] @ b.lift[r].T
    y = b.transform(ys)[:, b.node_slot]
    lift = ref.lift.reshape(b.np_, -1)
    scale = (np.abs(f) @ np.abs(lift).T).max()
    assert np.all(np.abs(y - f @ lift.T) <= 4 * b.nfp * EPS * scale)


@pytest.mark.parametrize("reduce", [False, True])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_adjoint_blocks_are_the_transposed_blocks(order, reduce):
    ref = reference_tet(order)
    args = (order, ref.weak_diff, ref.lift, ref.face_nodes)
    fwd = _Blocks(order, _pack(*args, strong=False))
    adj = _Blocks(order, _pack(*args, reduce=reduce), adjoint=True,
                  reduced="out" if reduce and order > 1 else None)
    assert np.array_equal(fwd.node_slot, adj.node_slot)
    assert np.array_equal(fwd.face_point, adj.face_point)
    for r in range(4):
        assert np.array_equal(adj.lift[r], fwd.lift[r].T)
        for k in (1, 2, 3):
            # the same sums rounded once to FP64, in another order of summation; reduced:
            # products of at most 5 terms, basis rows of unit length times columns of at
            # most 11 entries, each at most 1.5 times the largest derivative
            atol = (2 + 48 * reduce) * EPS * np.abs(ref.weak_diff).max()
            assert np.allclose(adj.vol[r, k], fwd.vol[r ^ k, k].T, rtol=0, atol=atol)
    bad = ref.weak_diff.copy()
    bad[0, 1, 0] += 1e-9
    assert _pack(order, bad, ref.lift, ref.face_nodes) is None


@pytest.mark.parametrize("order", [2, 3, 4])
def test_operators_that_keep_the_degree_are_refused(order):
    """Weak derivatives reach all of degree N, strong ones read it."""
    ref = reference_tet(order)
    for diff, strong in ((ref.weak_diff, True), (ref.diff, False)):
        assert _pack(order, diff, ref.lift, ref.face_nodes, strong) is not None
        assert _pack(order, diff, ref.lift, ref.face_nodes, strong, reduce=True) is None


@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_operators_without_the_symmetry_are_refused(order):
    ref = reference_tet(order)
    fn = ref.face_nodes
    for which in ("diff", "lift", "nodes", "nan"):
        diff, lift, nodes = ref.weak_diff.copy(), ref.lift.copy(), fn.copy()
        if which == "diff":
            diff[1, 0, -1] += 1e-9 * np.abs(diff).max()
        elif which == "lift":
            lift.reshape(-1)[3] += 1e-9 * np.abs(lift).max()
        elif which == "nan":
            diff[2, -1, 0] = np.nan
        else:                                    # a face that is not one
            nodes[0] = nodes[1]
        assert _pack(order, diff, lift, nodes, False) is None, which
    # another node order: the symmetry does not hold in this order's group action
    p = np.roll(np.arange(ref.np_), 1)
    diff = ref.weak_diff[:, p][:, :, p]
    lift = ref.lift[p]
    inv = np.argsort(p)
    got = _pack(order, diff, lift, inv[fn], False)
    if got is not None:                          # order 1: any order of four vertices
        assert order == 1


@pytest.mark.parametrize("table", ["one vertex", "first node twice"])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_faces_that_list_a_node_twice_are_refused(order, table):
    """With LIFT zero such a table commutes with the group, but its points are not
    four to an orbit; the general kernel evaluates it as given."""
    ref = reference_tet(order)
    full = np.asarray(ref.face_nodes).reshape(4, -1)
    fn = full.copy()
    for f in range(4):
        others = [set(full[g].tolist()) for g in range(4) if g != f]
        vertex = set.intersection(*others).pop()      # the one opposite face f
        if table == "one vertex":
            nodes = [vertex] * fn.shape[1]
        else:
            nodes = [fn[f, 0], *fn[f, :-1]]
        fn[f] = nodes
    zero = np.zeros_like(ref.lift)
    assert _pack(order, ref.weak_diff, zero, fn, False) is None
    assert _pack(order, ref.weak_diff, zero, fn) is None


@pytest.mark.gpu
@pytest.mark.parametrize("equation,order", [("wave", 1), ("wave", 4), ("euler", 2),
                                            ("euler", 3), ("maxwell", 3), ("maxwell", 4)])
def test_asymmetric_operators_take_the_general_kernel(equation, order):
    """An FP64 plan on the face-shared path whose operators lack the symmetry
    still evaluates them as given: equal to the fused kernel's result."""
    import torch

    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    from tests._helpers import jittered_box_mesh, make_problem
    prob = make_problem(equation, jittered_box_mesh(3), order, seed=order)
    q = torch.from_numpy(prob.fields).cuda()
    out = []
    for partner in (True, False):
        dm = DeviceMesh(prob.disc, "cuda:0", with_partner=partner)
        for name in ("_weak", "_strong", "_lift"):
            ops = getattr(dm, name).copy()
            ops.reshape(-1)[::7] *= 1.01
            setattr(dm, name, ops)
        plan = DevicePlan(dm, equation, prob.params, "fp64")
        out.append(plan.rhs(q))
        plan.finish()
    sym = DevicePlan(DeviceMesh(prob.disc, "cuda:0"), equation, prob.params, "fp64").rhs(q)
    norm = float(torch.linalg.norm(out[1]))
    assert float(torch.linalg.norm(out[0] - out[1])) <= 1e-12 * norm
    assert float(torch.linalg.norm(sym - out[1])) > 1e-6 * norm   # not the same operator


@pytest.mark.gpu
@pytest.mark.parametrize("equation", ["wave", "euler", "maxwell"])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("extra", [0, 1, 15, 17, 31, 33])
def test_tile_edges_match_the_general_kernel(equation, order, extra):
    """Element counts around the tile sizes (16 and 32 elements) from the smallest
    mesh that takes the kernel, RHS and RK stage with element scale: equal to the
    fused general kernel."""
    import torch

    from actx_dgfem_suite_gb300.mesh import TetMesh
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    from tests._helpers import jittered_box_mesh, make_problem
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    nel = 1 if order == 1 or equation == "maxwell" else (9 if order == 4 else 13) * nsm
    nel += extra
    mesh = jittered_box_mesh(3 if nel < 100 else 7)
    mesh = TetMesh(vertices=mesh.vertices, elements=mesh.elements[:nel])
    prob = make_problem(equation, mesh, order, seed=nel)
    q = torch.from_numpy(prob.fields).cuda()
    scale = torch.linspace(0.8, 1.2, nel, dtype=torch.float64, device="cuda")
    got = []
    for partner in (True, False):
        plan = DevicePlan(DeviceMesh(prob.disc, "cuda:0", with_partner=partner), equation,
                          prob.params, "fp64")
        r = plan.rhs(q)
        plan.set_element_scale(scale)
        res, qo, un = 0.5 * q, torch.empty_like(q), torch.empty_like(q)
        plan.rk_stage(q, qo, res, 0.3, 0.7, 1e-2, rhs_unscaled=un)
        plan.finish()
        assert (plan.info()["block"] == 128) == partner
        got.append((r, res, qo, un))
    for a, b in zip(*got):
        # two orders of summation of the same products: 1e-12 as the parity bound
        assert float(torch.linalg.norm(a - b)) <= 1e-12 * float(torch.linalg.norm(b))


@pytest.mark.gpu
@pytest.mark.parametrize("equation", ["wave", "euler"])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("extra", [0, 1, 31, 33])
def test_adjoint_tile_edges_match_the_dense_kernels(equation, order, extra):
    """Transposed Jacobian and fused reverse stage with element scale around the
    tile size, from the smallest mesh that takes the kernels, against the dense
    kernels: those run on operators moved off the symmetry by 1e-11, which moves
    results by no more than that."""
    import torch

    from actx_dgfem_suite_gb300.mesh import TetMesh
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    from tests._helpers import jittered_box_mesh, make_problem
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    nel = (48, 48, 32, 16)[order - 1] * nsm + extra
    mesh = jittered_box_mesh(11)
    mesh = TetMesh(vertices=mesh.vertices, elements=mesh.elements[:nel])
    prob = make_problem(equation, mesh, order, seed=nel)
    q = torch.from_numpy(prob.fields).cuda()
    g = torch.Generator(device="cuda").manual_seed(nel)
    x = torch.randn(q.shape, dtype=q.dtype, device=q.device, generator=g)
    lq = torch.randn(q.shape, dtype=q.dtype, device=q.device, generator=g)
    scale = torch.linspace(0.8, 1.2, nel, dtype=torch.float64, device="cuda")
    got = []
    for off in (0.0, 1e-11):
        dm = DeviceMesh(prob.disc, "cuda:0")
        dm._weak = dm._weak.copy()
        dm._weak.reshape(-1)[1] += off * abs(dm._weak).max()
        plan = DevicePlan(dm, equation, prob.params, "fp64")
        y = plan.vjp(q, x)
        plan.set_element_scale(scale)
        lam, rbar, scr = 0.3 * x, torch.empty_like(x), torch.empty_like(x)
        out = [y, lam, rbar]
        if equation == "wave":
            cbar = torch.ones(nel, dtype=torch.float64, device="cuda")
            plan.adjoint_stage(x, 0.7, lam, rbar, lq, cbar, 0.4, 0.9, 1e-2, scr)
            out.append(cbar)
        else:
            plan.vjp_stage(q, x, 0.7, lam, rbar, 0.4, 0.9, 1e-2, scr)
        plan.finish()
        got.append(out)
    for a, b in zip(*got):
        assert float(torch.linalg.norm(a - b)) <= 1e-10 * float(torch.linalg.norm(b))


@pytest.mark.parametrize("strong", [False, True])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_triangle_blocks_reproduce_the_dense_operators(order, strong):
    """``pack_sym_ops_2d``: even and odd blocks under the swap of vertices 1 and
    2; operators off the symmetry are refused."""
    from actx_dgfem_suite_gb300.refelem import reference_tri
    f = ctypes.CDLL(str(_lib.library_path()))._ZN2dg15pack_sym_ops_2dEiPKdS1_PKiPhi
    f.restype = ctypes.c_int

    def pack(diff, lift, fnodes):
        arrs = [np.ascontiguousarray(diff), np.ascontiguousarray(lift),
                np.ascontiguousarray(fnodes, dtype=np.int32)]
        args = [ctypes.c_int(order)] + [ctypes.c_void_p(x.ctypes.data) for x in arrs]
        buf = np.zeros(f(*args, None, 0), dtype=np.uint8)
        got = f(*args, ctypes.c_void_p(buf.ctypes.data), buf.size)
        return buf if got == buf.size else None

    ref = reference_tri(order)
    diff = ref.diff if strong else ref.weak_diff
    npn, nfpt = ref.np_, 3 * ref.nfp
    buf = pack(diff, ref.lift, ref.face_nodes)
    nfx, ffx = order // 2 + 1, int(order % 2 == 0)
    npr, fpr = (npn - nfx) // 2, (nfpt - ffx) // 2
    dim, fdim = (npr + nfx, npr), (fpr + ffx, fpr)
    pitch = [(d + 1) & ~1 for d in dim]
    x, pos = buf.view(np.float64), 0
    vol, lft = {}, {}
    for r in range(2):
        for k in range(2):
            n = dim[r ^ k] * pitch[r]
            vol[r, k] = x[pos:pos + n].reshape(-1, pitch[r])[:, :dim[r]].T
            pos += n
    for r in range(2):
        n = fdim[r] * pitch[r]
        lft[r] = x[pos:pos + n].reshape(-1, pitch[r])[:, :dim[r]].T
        pos += n
    tab, pos = buf.view(np.int32), 2 * pos
    tables = []
    for n in (npn, npn, nfpt, nfpt):
        tables.append(tab[pos:pos + n])
        pos += (n + 3) // 4 * 4
    node_slot, slot_node, edge_slot, edge_node = tables
    assert list(slot_node[node_slot]) == list(range(npn))
    assert sorted(edge_slot) == list(range(nfpt))
    assert np.array_equal(edge_node, ref.face_nodes.reshape(-1))

    def mirror(v, pairs, even):
        u, w = v[:, :pairs].copy(), v[:, even:even + pairs].copy()
        v[:, :pairs], v[:, even:even + pairs] = u + w, u - w
        return v

    rng = np.random.default_rng(order)
    q, e = rng.standard_normal((7, npn)), rng.standard_normal((7, nfpt))
    g = rng.standard_normal((2, 7, 1))
    part = [slice(0, dim[0]), slice(dim[0], npn)]
    fpart = [slice(0, fdim[0]), slice(fdim[0], nfpt)]
    qs, es = np.empty_like(q), np.empty_like(e)
    qs[:, node_slot], es[:, edge_slot] = q, e
    mirror(qs, npr, dim[0])
    mirror(es, fpr, fdim[0])
    h = [g[0] + g[1], g[0] - g[1]]
    y, z = np.zeros_like(qs), np.zeros_like(qs)
    for r in range(2):
        for k in range(2):
            y[:, part[r]] += h[k] * (qs[:, part[r ^ k]] @ vol[r, k].T)
        z[:, part[r]] = es[:, fpart[r]] @ lft[r].T
    y, z = (mirror(v, npr, dim[0])[:, node_slot] for v in (y, z))
    dense = g[0] * (q @ diff[0].T) + g[1] * (q @ diff[1].T)
    size = sum(np.abs(g[r]) * (np.abs(q) @ np.abs(diff[r]).T) for r in range(2)).max()
    assert np.all(np.abs(y - dense) <= 3 * npn * EPS * size)
    lift = ref.lift.reshape(npn, -1)
    assert np.all(np.abs(z - e @ lift.T) <= 4 * nfpt * EPS * (np.abs(e) @ np.abs(lift).T).max())
    for which in range(3):
        d, li, fn = diff.copy(), ref.lift.copy(), ref.face_nodes.copy()
        if which == 0:
            d[0, 0, 1] += 1e-9 * np.abs(d).max()
        elif which == 1:
            li.reshape(-1)[1] = np.nan
        else:
            fn[0] = fn[2][::-1] if order > 1 else fn[2]
        assert pack(d, li, fn) is None, which


@pytest.mark.gpu
@pytest.mark.parametrize("equation", ["wave", "euler", "maxwell"])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("nel", [0, 1, 31, 33, 146])
def test_triangle_tile_edges_match_the_dense_kernel(equation, order, nel):
    """Element counts around the 32-element tile on a mesh whose elements are
    shuffled (glued sides inside and outside the tiles), RHS and RK stage: the
    dense kernel runs on operators moved off the symmetry by 1e-11."""
    import torch

    from actx_dgfem_suite_gb300.mesh import TriMesh
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    from tests._helpers import jittered_square_mesh, make_problem_2d
    # the kernel serves meshes from 48 elements per SM on
    nel += 48 * torch.cuda.get_device_properties(0).multi_processor_count
    mesh = jittered_square_mesh(61)
    el = mesh.elements
    if nel % 2:
        el = np.roll(el, nel % 3, axis=1)[np.random.default_rng(nel).permutation(len(el))]
    assert nel <= len(el)
    prob = make_problem_2d(equation, TriMesh(vertices=mesh.vertices, elements=el[:nel]), order,
                           seed=nel)
    q = torch.from_numpy(prob.fields).cuda()
    scale = torch.linspace(0.8, 1.2, nel, dtype=torch.float64, device="cuda")
    got = []
    for off in (0.0, 1e-11):
        dm = DeviceMesh(prob.disc, "cuda:0")
        for name in ("_weak", "_strong"):
            ops = getattr(dm, name).copy()
            ops.reshape(-1)[1] += off * abs(ops).max()
            setattr(dm, name, ops)
        plan = DevicePlan(dm, equation, prob.params, "fp64")
        r = plan.rhs(q)
        plan.set_element_scale(scale)
        res, qo, un = 0.5 * q, torch.empty_like(q), torch.empty_like(q)
        plan.rk_stage(q, qo, res, 0.3, 0.7, 1e-2, rhs_unscaled=un)
        plan.finish()
        got.append((r, res, qo, un, plan.info()["block"]))
    assert got[0][4] != got[1][4]                # two different kernels
    for a, b in zip(got[0][:4], got[1][:4]):
        assert float(torch.linalg.norm(a - b)) <= 1e-10 * float(torch.linalg.norm(b))


@pytest.mark.gpu
def test_triangles_glued_with_a_turn_are_not_shared():
    """Sides glued by the gather index whose normals are not opposite (a periodic
    sector) keep one flux per side, inside a tile too."""
    import torch

    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    from tests._helpers import jittered_square_mesh, make_problem_2d
    prob = make_problem_2d("euler", jittered_square_mesh(61), 2, seed=1)
    q = torch.from_numpy(prob.fields).cuda()
    got, blocks = [], []
    for off in (0.0, 1e-11):
        dm = DeviceMesh(prob.disc, "cuda:0")
        gather = dm.gather.cpu().numpy().view(np.uint32).copy()
        nodes, npn = prob.disc.ref.face_nodes, prob.disc.np_
        free = [(e, f) for e in range(prob.disc.nelements) for f in range(3)
                if gather[e, f, 0] >> 31]
        turned = 0
        for (e, f), (e2, f2) in zip(free[::2], free[1::2]):
            if e != e2 and abs((prob.disc.normal[e, f] + prob.disc.normal[e2, f2])).max() > 0.1:
                gather[e, f] = e2 * npn + nodes[f2][::-1]
                gather[e2, f2] = e * npn + nodes[f][::-1]
                turned += 1
        assert turned > 0
        dm.gather = torch.from_numpy(gather.view(np.int32)).cuda()
        ops = dm._weak.copy()
        ops.reshape(-1)[1] += off * abs(ops).max()
        dm._weak = ops
        plan = DevicePlan(dm, "euler", prob.params, "fp64")
        got.append(plan.rhs(q))
        plan.finish()
        blocks.append(plan.info()["block"])
    assert blocks[0] != blocks[1]
    assert float(torch.linalg.norm(got[0] - got[1])) <= 1e-10 * float(torch.linalg.norm(got[1]))


@pytest.mark.gpu
@pytest.mark.parametrize("equation", ["wave", "euler", "maxwell"])
@pytest.mark.parametrize("order,tiles,extra", [(1, 0, 2), (1, 0, 32), (1, 0, 34), (1, 0, 62),
                                               (1, 0, 64), (1, 2, 0), (1, 2, 2), (1, 6, 0),
                                               (2, 2, 0), (2, 2, 2), (2, 3, 0)])
def test_triangle_size_rule(equation, order, tiles, extra):
    """Element counts on both sides of the lines between the dense and the symmetric
    kernel, in rounds of 32 elements per SM: the kernel that the rule names, and the
    dense kernel's result (as above on operators moved by 1e-11)."""
    import torch

    from actx_dgfem_suite_gb300.mesh import TriMesh, generate_box_tri_mesh
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    from tests._helpers import make_problem_2d
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    nel = 32 * tiles * nsm + extra
    full = generate_box_tri_mesh(0.0, 1.0, (8, nel // 16 + 1))
    prob = make_problem_2d(equation, TriMesh(vertices=full.vertices, elements=full.elements[:nel]),
                           order, seed=nel)
    dense = 256 // prob.disc.np_                 # elements per tile
    rounds, dense_rounds = -(-nel // (32 * nsm)), -(-nel // (dense * nsm))
    if order == 1:
        symmetric = nel > 32 if equation == "euler" else nel >= 64 and rounds < 3 * dense_rounds
    else:
        symmetric = equation == "euler" or (rounds, dense_rounds) != (3, 2)
    q = torch.from_numpy(prob.fields).cuda()
    got = []
    for off in (0.0, 1e-11):
        dm = DeviceMesh(prob.disc, "cuda:0")
        for name in ("_weak", "_strong"):
            ops = getattr(dm, name).copy()
            ops.reshape(-1)[1] += off * abs(ops).max()
            setattr(dm, name, ops)
        plan = DevicePlan(dm, equation, prob.params, "fp64")
        r = plan.rhs(q)
        res, qo = 0.5 * q, torch.empty_like(q)
        plan.rk_stage(q, qo, res, 0.3, 0.7, 1e-2)
        plan.finish()
        assert (plan.info()["block"] == 128) == (symmetric and off == 0.0)
        got.append((r, res, qo))
    for a, b in zip(*got):
        assert float(torch.linalg.norm(a - b)) <= 1e-10 * float(torch.linalg.norm(b))


@pytest.mark.gpu
@pytest.mark.parametrize("equation,order,per_sm", [("wave", 4, 14), ("euler", 4, 14),
                                                   ("euler", 2, 25)])
@pytest.mark.parametrize("extra", [0, 1, 33])
def test_stage_size_rule(equation, order, per_sm, extra):
    """RK stages around the size from which they take the symmetric kernel: as the
    fused general kernel, and the bits of the RHS only above the line."""
    import torch

    from actx_dgfem_suite_gb300.mesh import TetMesh
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    from tests._helpers import jittered_box_mesh, make_problem
    nel = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    mesh = jittered_box_mesh(9)
    mesh = TetMesh(vertices=mesh.vertices, elements=mesh.elements[:nel])
    prob = make_problem(equation, mesh, order, seed=nel)
    q = torch.from_numpy(prob.fields).cuda()
    got = []
    for partner in (True, False):
        plan = DevicePlan(DeviceMesh(prob.disc, "cuda:0", with_partner=partner), equation,
                          prob.params, "fp64")
        r = plan.rhs(q)
        res, qo, un = 0.5 * q, torch.empty_like(q), torch.empty_like(q)
        plan.rk_stage(q, qo, res, 0.3, 0.7, 1e-2, rhs_unscaled=un)
        plan.finish()
        if partner:
            assert torch.equal(un, r) == (extra > 0)
        got.append((res, qo, un))
    for a, b in zip(*got):
        assert float(torch.linalg.norm(a - b)) <= 1e-12 * float(torch.linalg.norm(b))


@pytest.mark.gpu
@pytest.mark.parametrize("order,per_sm", [(1, 64), (2, 50), (3, 36)])
@pytest.mark.parametrize("extra", [0, 1, 31, 33])
def test_wave_adjoint_size_rule(order, per_sm, extra):
    """The wave adjoint from the smallest mesh that takes the symmetric kernel,
    against the dense one (operators moved by 1e-11)."""
    import torch

    from actx_dgfem_suite_gb300.mesh import TetMesh
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan
    from tests._helpers import jittered_box_mesh, make_problem
    nel = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    mesh = jittered_box_mesh(12)
    mesh = TetMesh(vertices=mesh.vertices, elements=mesh.elements[:nel])
    prob = make_problem("wave", mesh, order, seed=nel)
    x = torch.from_numpy(prob.fields).cuda()
    lq = x.roll(1, dims=0).contiguous()
    got = []
    for off in (0.0, 1e-11):
        dm = DeviceMesh(prob.disc, "cuda:0")
        dm._weak = dm._weak.copy()
        dm._weak.reshape(-1)[1] += off * abs(dm._weak).max()
        plan = DevicePlan(dm, "wave", prob.params, "fp64")
        y = plan.vjp(x, x)
        lam, rbar, scr = 0.3 * x, torch.empty_like(x), torch.empty_like(x)
        cbar = torch.ones(nel, dtype=torch.float64, device="cuda")
        plan.adjoint_stage(x, 0.7, lam, rbar, lq, cbar, 0.4, 0.9, 1e-2, scr)
        plan.finish()
        got.append((y, lam, rbar, cbar))
    for a, b in zip(*got):
        assert float(torch.linalg.norm(a - b)) <= 1e-10 * float(torch.linalg.norm(b))
