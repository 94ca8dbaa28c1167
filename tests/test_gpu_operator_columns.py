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


FIELD_LAWS = {
    # material, heaviside, velocity: T_old in the tangent; coefficient fields; both with convection
    "liquid_solid": (dict(law=2, rho=1.0, cp=1.0, k=0.5, rho_s=1.2, cp_s=0.8, k_s=2.5,
                          T_solidus=0.3, T_liquidus=0.7), False, False),
    "gas_liquid_velocity": (dict(law=3, rho=2.0, cp=3.0, k=5.0, rho_g=0.5, cp_g=1.5, k_g=0.3),
                            True, True),
    "three_phase_velocity": (dict(law=4, rho=1.0, cp=1.0, k=0.5, rho_s=1.2, cp_s=0.8, k_s=2.5,
                                  T_solidus=0.3, T_liquidus=0.7, rho_g=0.4, cp_g=1.5, k_g=0.2),
                             True, True),
}


@pytest.mark.parametrize("degree,cells", [(3, (29, 31, 37)), (4, (23, 29, 31)), (5, (13, 17, 19)),
                                          (6, (11, 13, 17))])
@pytest.mark.parametrize("perturb", [0.0, 0.2])
@pytest.mark.parametrize("law", list(FIELD_LAWS))
def test_field_laws_over_several_rounds(degree, cells, perturb, law):
    """The laws that use the line kernel's shared arrays more than once a batch (T_old's values) or
    read per-point fields, where every block takes several batches. FP64: a phase change's branches
    are taken at the same points."""
    m, with_h, with_v = FIELD_LAWS[law]
    mask, dt = 0b010010, 1e-2
    o = O.Oracle(degree, cells, perturb=perturb, seed=5, dirichlet_mask=mask)
    o.set_material(O.material(**m), dt)
    g = H.HeatDiffuseOperator(H.box_mesh(degree, cells, perturb=perturb, seed=5, dirichlet=(1, 4)))
    g.set_material(H.material(**m))
    g.reset_time_increment(dt)
    x = o.support_points()
    hv = 0.5 + 0.5 * np.tanh((x[:, 0] - 0.45) / 0.1) if with_h else None
    v = np.stack([np.sin(3 * x[:, 1]), 0.5 + x[:, 2], -x[:, 0] * x[:, 1]]) if with_v else None
    o.set_fields(hv, v)
    g.set_fields(*(None if f is None else torch.tensor(f, device="cuda") for f in (hv, v)))
    rng = np.random.default_rng(degree)
    src, Tl, To = (rng.uniform(lo, 1.0, o.n_dofs) for lo in (-1.0, 0.0, 0.0))
    d = {k: torch.tensor(a, device="cuda") for k, a in dict(src=src, Tl=Tl, To=To).items()}
    g.set_linearization(d["Tl"], d["To"])
    assert rel(g.vmult(g.new_vector(), d["src"]), o.vmult(src, Tl, To)) <= TOL64


@pytest.mark.parametrize("cells", [(1, 1, 1), (7, 1, 2), (23, 29, 31)])
@pytest.mark.parametrize("law", ["gas_liquid_velocity", "three_phase_velocity"])
def test_fp32_field_laws_on_deformed_cells(cells, law):
    """FP32 p = 4 on deformed meshes runs the line kernel with the 5 fields of the gas-liquid law and
    the 8 tangent fields of the three-phase law (built in FP64), 2e-5 as everywhere."""
    m, _, _ = FIELD_LAWS[law]
    dt = 1e-2
    o = O.Oracle(4, cells, perturb=0.2, seed=5, dirichlet_mask=0b010010)
    o.set_material(O.material(**m), dt)
    g = H.HeatDiffuseOperator(H.box_mesh(4, cells, perturb=0.2, seed=5, dirichlet=(1, 4)))
    g.set_material(H.material(**m))
    g.reset_time_increment(dt)
    x = o.support_points()
    hv = 0.5 + 0.5 * np.tanh((x[:, 0] - 0.45) / 0.1)
    v = np.stack([np.sin(3 * x[:, 1]), 0.5 + x[:, 2], -x[:, 0] * x[:, 1]])
    o.set_fields(hv, v)
    g.set_fields(torch.tensor(hv, device="cuda"), torch.tensor(v, device="cuda"))
    rng = np.random.default_rng(4)
    src, Tl, To = (rng.uniform(lo, 1.0, o.n_dofs) for lo in (-1.0, 0.0, 0.0))
    d = {k: torch.tensor(a, device="cuda") for k, a in dict(src=src, Tl=Tl, To=To).items()}
    g.set_linearization(d["Tl"], d["To"])
    y = g.vmult(g.new_vector(torch.float32), d["src"].float())
    assert rel(y, o.vmult(src, Tl, To)) <= TOL32


@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("cells", [(1, 1, 1), (33, 1, 2), (2, 17, 3), "long"])
@pytest.mark.parametrize("perturb", [0.0, 0.2])
@pytest.mark.parametrize("law", ["constant", "linear_k"])
def test_inverse_diagonal(degree, cells, perturb, law):
    """The register-plane diagonal on one cell, on rows one cell wide and over several rounds."""
    cells = LONG[degree] if cells == "long" else cells
    m = KT if law == "linear_k" else dict(law=0, rho=1.0, cp=1.0, k=1.0)
    mask, dt = 0b000001, 1e-3
    o = O.Oracle(degree, cells, perturb=perturb, seed=5, dirichlet_mask=mask)
    o.set_material(O.material(**m), dt)
    g = H.HeatDiffuseOperator(H.box_mesh(degree, cells, perturb=perturb, seed=5, dirichlet=(0,)))
    g.set_material(H.material(**m))
    g.reset_time_increment(dt)
    Tl = np.random.default_rng(degree).uniform(0.0, 1.0, o.n_dofs)
    Td = torch.tensor(Tl, device="cuda")
    g.set_linearization(Td, Td)
    d = g.compute_inverse_diagonal_from_matrixfree(g.new_vector())
    assert rel(1.0 / d, 1.0 / o.inverse_diagonal(Tl, Tl)) <= TOL64
