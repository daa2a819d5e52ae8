"""Sizes and branches at which the stage, relaxation and training kernels change path, against the
oracle: last blocks of 4-slot (tets) and 6-slot meshes, a gas phase with its own p_inf in the Gibbs
Newton, training batches that do not fill a tile or a pass over the blocks."""
import math
from pathlib import Path

import numpy as np
import pytest

from fooskagpu_b200 import cases, meshgen
from fooskagpu_b200.api import Mesh, Solver, Surrogate
from oracle import mlp_oracle
from oracle.oracle_py import Oracle

pytestmark = pytest.mark.gpu
ALL_BC = {"x0": "inlet", "x1": "outlet", "y0": "wall", "y1": "slip", "z0": "symmetry", "z1": "slip"}
TOL = {"fp64": (1e-10, 1e-9), "mixed": (2e-6, 1e-4)}   # as tests/test_gpu_edge.py: state, HLLC tie


# 66 = 64 + 2 (FP64 gradient block), 126 / 132 around 128 (FP32 gradient and gather blocks); the
# mixed box has 4, 5 and 6 faces per cell in one mesh
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("kind,nx,cells", [("tets", 1, 6), ("tets", 11, 66), ("tets", 21, 126), ("tets", 22, 132),
                                           ("elements", 3, None)])
def test_stage_kernels_at_block_edges(kind, nx, cells, prec):
    if kind == "tets":
        nm = meshgen.box_tets(nx, 1, 1, L=(nx * 1e-3, 1e-3, 1e-3), side_bc=ALL_BC)
    else:
        nm = meshgen.box_mixed(nx, 3, 2, L=(nx * 1e-3, 3e-3, 2e-3), side_bc=ALL_BC)
    m = Mesh.build(nm.nodes, nm.elems, nm.bcs)
    assert cells is None or m.n_elem == cells
    c = cases.reference_case()
    c.rkSteps = 3
    tol, c.hllcTieTol = TOL[prec]
    U = cases.perturbed_two_phase_ic(c, m.arrays()["cellCenter"], seed=9, vel=25.0)
    o = Oracle(m.view(), c)
    Uo = U.copy()
    s = Solver(m, c, precision=prec)
    s.set_state(U)
    for _ in range(2):
        o.step(Uo)
        s.step()
    err = np.abs(s.get_state() - Uo).max(axis=0) / np.maximum(np.abs(Uo).max(axis=0), 1e-300)
    o.close()
    s.close()
    assert err.max() < tol, err


@pytest.mark.parametrize("pinf_gas", [0.0, 2e5])
def test_gibbs_newton_with_stiffened_gas(pinf_gas):
    """p_inf of the gas: zero takes log10 p from log10(p + p_inf), else a logarithm of its own."""
    nm = meshgen.box_hexes(9, 8, 7, L=(9e-3, 8e-3, 7e-3))
    m = Mesh.build(nm.nodes, nm.elems, nm.bcs)
    c = cases.reference_case()
    c.pInf[1] = pinf_gas
    U = cases.perturbed_two_phase_ic(c, m.arrays()["cellCenter"], seed=4, vel=25.0)
    o = Oracle(m.view(), c)
    Uo = U.copy()
    st = o.relaxation(Uo)
    o.close()
    s = Solver(m, c, precision="fp64")
    s.set_state(U)
    sg = s.relaxation()
    err = np.abs(s.get_state() - Uo).max(axis=0) / np.maximum(np.abs(Uo).max(axis=0), 1e-300)
    s.close()
    assert st["nChem"] > 50 and {k: sg[k] for k in st} == st
    assert err.max() < 1e-11, err   # as the relaxation parity: round-off of the same iterates


@pytest.mark.parametrize("box", [(5, 6, 7), (8, 8, 8)])
def test_fp64_vortex_keeps_its_stop_decisions(box):
    """Four FP64 vortex steps against stored states.  The thermal Newton stops at an absolute residual, so a change
    of rounding anywhere in a step lets some cells stop one iterate earlier or later, which moves the pressure by
    about (1 - thermUrf) 1e-2 / 70 = 3e-5 (a rearranged Newton: 1.1e-4 and 2.6e-5 here); states whose every
    cell stops where it did agree to rounding, 1e-12 with room."""
    L = 2 * math.pi
    nm = meshgen.box_hexes(*box, L=(L, L, L), side_bc={})
    m = Mesh.build(nm.nodes, nm.elems, nm.bcs, periodic=(L, L, L))
    c = cases.tgv_case()
    c.adaptDtItr = 2
    c.hllcTieTol = 1e-9
    s = Solver(m, c, precision="fp64")
    s.set_state(cases.tgv_ic(c, m.arrays()["cellCenter"] + np.array([0.3, 1.1, 2.0])))
    for _ in range(4):
        s.step()
    U = s.get_state()
    s.close()
    ref = np.load(Path(__file__).parent / "golden" / "tgv_fp64_steps.npz")["%d_%d_%d" % box]
    err = np.abs(U - ref).max(axis=0) / np.maximum(np.abs(ref).max(axis=0), 1e-300)
    assert err.max() < 1e-12, err


def test_relaxation_kernels_agree_bitwise():
    """57,798 cells take the relaxation kernel of many cells, the two parts of the mesh (28,899 each) that of
    few: the same states bit for bit."""
    nm = meshgen.box_hexes(39, 39, 38, L=(39e-3, 39e-3, 38e-3))
    m = Mesh.build(nm.nodes, nm.elems, nm.bcs)
    c = cases.reference_case()
    U = cases.perturbed_two_phase_ic(c, m.arrays()["cellCenter"], seed=4, vel=25.0)
    s = Solver(m, c, precision="mixed")
    s.set_state(U)
    assert s.relaxation()["nChem"] > 1000
    whole = s.get_state()
    s.close()
    for p in range(2):
        part = m.partition(2, p)
        own = part.partition_maps()["cell_global"][:part.n_owned]
        s = Solver(part, c, precision="mixed")
        s.set_state(U[own])
        s.relaxation()
        assert np.array_equal(s.get_state(), whole[own])
        s.close()


def _relaxed(mesh, c, prec, U, log=False):
    """State after one relaxation, and the residual of it, which shows the primitive records bit for bit."""
    s = Solver(mesh, c, precision=prec)
    s.set_state(U)
    if log:
        s.relax_log(1_000_000)
    n = s.relaxation()["nChem"]
    V = s.get_state()
    R = None
    if mesh.n_owned == mesh.n_elem:
        s.compute_rhs()
        R = s.get_rhs()
    s.close()
    return V, R, n


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("pinf_gas", [0.0, 2e5])
@pytest.mark.parametrize("vel", [0.0, 25.0])
def test_every_relaxation_kernel_gives_the_same_states(prec, pinf_gas, vel):
    """The kernels of few and of many cells, with and without the sample log, and (where no cell is chemical) the one
    without the chemical branch: the same states and primitive records bit for bit."""
    nm = meshgen.box_hexes(39, 39, 38, L=(39e-3, 39e-3, 38e-3))
    m = Mesh.build(nm.nodes, nm.elems, nm.bcs)
    c = cases.reference_case()
    c.pInf[1] = pinf_gas
    U = cases.perturbed_two_phase_ic(c, m.arrays()["cellCenter"], seed=4, vel=vel)
    whole, R, n = _relaxed(m, c, prec, U)
    assert n > 1000
    V, Q, _ = _relaxed(m, c, prec, U, log=True)
    assert np.array_equal(V, whole) and np.array_equal(Q, R)
    for p in range(2):
        part = m.partition(2, p)
        own = part.partition_maps()["cell_global"][:part.n_owned]
        V, _, _ = _relaxed(part, c, prec, U[own])
        assert np.array_equal(V, whole[own])
    c.chemLimit = 1.0   # no cell is above it
    whole, R, n = _relaxed(m, c, prec, U)
    assert n == 0
    c.chemFlag = 0
    V, Q, _ = _relaxed(m, c, prec, U)
    assert np.array_equal(V, whole) and np.array_equal(Q, R)


# up to 400,000 cells the CFL kernel leaves the signal maxima at zero, above a memset does
@pytest.mark.parametrize("nx", [5, 100, 101])
def test_signal_maxima_start_from_zero(nx):
    """A dt step after one with faster signals: the new dt is that of the residual path."""
    nm = meshgen.box_hexes(nx, 100, 40, L=(nx * 1e-2, 1.0, 0.4))
    m = Mesh.build(nm.nodes, nm.elems, nm.bcs, gpu=True)
    c = cases.sod_case()
    c.adaptDtItr = c.relaxFlag = 1
    x = m.arrays()["cellCenter"]
    z = np.zeros(len(x))
    a, b = Solver(m, c, precision="mixed"), Solver(m, c, precision="mixed")
    for speed in (3.0, 0.0):
        U = cases.prim_to_cons(c, 0.5, z + 1, z + 1, speed * np.sin(9 * x[:, 1]), z, z, z + 1)
        for s in (a, b):
            s.set_state(U)
        a.step()
        b.compute_rhs(want_signal=True)
        assert a.time()[0] == b.compute_time_step()
    a.close()
    b.close()


# a tile holds 32 samples, a pass over the blocks 296 tiles
@pytest.mark.parametrize("n", [1, 31, 33, 296 * 32 + 1])
def test_training_gradient_batch_sizes(n):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 3)).astype(np.float32)
    Y = rng.standard_normal((n, 4)).astype(np.float32)
    g = Surrogate(seed=5)
    loss, grad = g.loss_grad(X, Y)
    lo, go = mlp_oracle.loss_grad(g.params(), X, Y)
    assert abs(loss - lo) <= 1e-5 * abs(lo)
    assert np.abs(grad - go).max() <= 1e-5 * np.abs(go).max()   # as tests/test_surrogate.py
    if n >= 33:
        # the first Adam step moves every parameter by lr g / (|g| + eps), g over the whole batch; FP32
        # rounding of a parameter of order 1, and of g where it is not far above eps, bound the difference
        g.set_data(X, Y)
        p0 = g.params()
        mean, std = X.astype(np.float64).mean(0), X.astype(np.float64).std(0)
        ym, ys = Y.astype(np.float64).mean(0), Y.astype(np.float64).std(0)
        _, ge = mlp_oracle.loss_grad(p0, ((X - mean) / std).astype(np.float32), ((Y - ym) / ys).astype(np.float32))
        g.train(1, batch=n, lr=1e-3, seed=1)
        sure = np.abs(ge) > 1e-4 * np.abs(ge).max()
        step = -1e-3 * ge / (np.abs(ge) + 1e-8)
        assert np.abs(g.params() - p0 - step)[sure].max() < 1e-6
    g.close()
