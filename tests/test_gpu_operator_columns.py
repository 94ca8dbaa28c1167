"""The register-resident operator kernels where their work split has edges: cell rows shorter and
longer than a warp's group of cells, a last group that is partly empty, meshes of several rounds of
the persistent grid (the cells are walked with carries), one cell, and Dirichlet faces that
constrain some columns only; against the oracle, FP64 to 1e-12 and FP32 to 2e-5 (max norm)."""
import numpy as np
import pytest
import torch

from meltpooldg_b200 import heat as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL64, TOL32 = 1e-12, 2e-5
KT = dict(law=1, rho=1.0, cp=1.0, k=1.0, k1=0.5)
# several rounds of the grid: more cells than 148 SMs x resident warps x cells per warp
LONG = {1: (61, 47, 53), 2: (37, 41, 43), 3: (29, 31, 37), 4: (23, 29, 31)}


def rel(a, b):
    a = a.double().cpu().numpy()
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("degree", [1, 2, 3, 4])
@pytest.mark.parametrize("cells", [(1, 1, 1), (33, 1, 2), (2, 17, 3), "long"])
@pytest.mark.parametrize("perturb", [0.0, 0.2])
@pytest.mark.parametrize("mask", [0b111111, 0b010010])
def test_operator_verbs(degree, cells, perturb, mask):
    cells = LONG[degree] if cells == "long" else cells
    if degree == 1 and min(cells) == 1 and mask == 0b111111:
        mask = 0b000001  # otherwise every DoF is constrained
    dt = 1e-3
    o = O.Oracle(degree, cells, perturb=perturb, seed=5, dirichlet_mask=mask)
    o.set_material(O.material(**KT), dt)
    g = H.HeatDiffuseOperator(H.box_mesh(degree, cells, perturb=perturb, seed=5,
                                         dirichlet=[f for f in range(6) if mask >> f & 1]))
    g.set_material(H.material(**KT))
    g.reset_time_increment(dt)
    rng = np.random.default_rng(degree)
    n = o.n_dofs
    src, Tl, To, q = (rng.uniform(lo, 1.0, n) for lo in (-1.0, 0.0, 0.0, 0.0))
    d = {k: torch.tensor(v, device="cuda") for k, v in dict(src=src, Tl=Tl, To=To, q=q).items()}
    g.set_linearization(d["Tl"], d["To"])
    ref = o.vmult(src, Tl, To)
    assert rel(g.vmult(g.new_vector(), d["src"]), ref) <= TOL64
    s32 = d["src"].float()
    assert rel(g.vmult(g.new_vector(torch.float32), s32), ref) <= TOL32
    assert rel(g.vmult_picard_f32(g.new_vector(torch.float32), s32),
               o.vmult(src, Tl, To, form=2)) <= TOL32
    assert rel(1.0 / g.inverse_diagonal_picard_f32(g.new_vector(torch.float32)),
               1.0 / o.inverse_diagonal(Tl, To, form=2)) <= TOL32
    assert rel(g.create_rhs(g.new_vector(), d["To"], d["q"]), o.create_rhs(Tl, To, q)) <= TOL64


@pytest.mark.parametrize("degree,cells", [(4, (23, 29, 31)), (5, (1, 1, 1)), (5, (13, 17, 19)),
                                          (6, (1, 3, 1)), (6, (11, 13, 17))])
@pytest.mark.parametrize("perturb", [0.0, 0.2])
@pytest.mark.parametrize("law", ["constant", "linear_k"])
def test_high_degree_operator(degree, cells, perturb, law):
    """The line kernel (and at p = 4, 5 the register-resident one with the constant law on a uniform
    box) on one cell, on a batch that is partly empty and over several rounds of the grid."""
    m = KT if law == "linear_k" else dict(law=0, rho=1.0, cp=1.0, k=1.0)
    mask, dt = 0b010010, 1e-3
    o = O.Oracle(degree, cells, perturb=perturb, seed=5, dirichlet_mask=mask)
    o.set_material(O.material(**m), dt)
    g = H.HeatDiffuseOperator(H.box_mesh(degree, cells, perturb=perturb, seed=5, dirichlet=(1, 4)))
    g.set_material(H.material(**m))
    g.reset_time_increment(dt)
    rng = np.random.default_rng(degree)
    src, Tl = rng.uniform(-1.0, 1.0, o.n_dofs), rng.uniform(0.0, 1.0, o.n_dofs)
    Tld = torch.tensor(Tl, device="cuda")
    g.set_linearization(Tld, Tld)
    s, ref = torch.tensor(src, device="cuda"), o.vmult(src, Tl, Tl)
    assert rel(g.vmult(g.new_vector(), s), ref) <= TOL64
    assert rel(g.vmult(g.new_vector(torch.float32), s.float()), ref) <= TOL32 * 10


@pytest.mark.parametrize("degree,cells", [(2, (16, 16, 16)), (3, (1, 2, 1)), (4, (9, 9, 9))])
def test_application_in_a_cuda_graph(degree, cells):
    """op.vmult (a zero fill and a kernel launched as its dependent) recorded and replayed on new
    operands, and repeated without a wait in between."""
    op = H.HeatDiffuseOperator(H.box_mesh(degree, cells, dirichlet=("z-",)))
    op.set_material(H.material())
    op.reset_time_increment(1e-3)
    x, y, z = (op.new_vector() for _ in range(3))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        op.sync_stream()
        op.vmult(y, x.uniform_())
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            op.vmult(y, x)
            op.vmult(z, y)
        x.uniform_()
        graph.replay()
    side.synchronize()
    op.sync_stream()
    ry = op.vmult(op.new_vector(), x)
    rz = op.vmult(op.new_vector(), ry)
    assert (y - ry).abs().max() <= 1e-13 * ry.abs().max()
    assert (z - rz).abs().max() <= 1e-12 * rz.abs().max()
