"""The matrix products of the Poisson solve and the trials that run them.

Power-of-two grids are solved by the fast transforms in poisson_solve, the
transform modules, density operators and trials of small grids
(electric_potential.fast_solve), so the products are asked for by name here:
against fp64 at the bars of the module tests, and under the GP tests that use a
128 x 128 grid, whose trials then run what larger grids' trials run."""
import numpy as np
import pytest
import torch

import oracle
import test_gpu_batch
import test_gpu_checkpoint
import test_gpu_gp
import test_gpu_gp_reference
from dreamplace_b200 import synthetic
from test_gpu_gp_reference import design, ref  # noqa: F401  (fixtures)
from test_gpu_ops import FIELD_TOL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dreamplace_b200._native import C
    return C


@pytest.fixture
def trials_on_products(C, monkeypatch):
    """Engines made under it solve split_bf16 trials by the products on every grid."""
    from dreamplace_b200 import engine
    made = []

    class Workspace(engine.PoissonWorkspace):
        def __init__(self, *args, **kw):
            super().__init__(*args, **kw)
            made.append(self)
    monkeypatch.setattr(engine, "FAST_TRIAL_SIDE", 0)
    monkeypatch.setattr(engine, "PoissonWorkspace", Workspace)
    yield
    split = [w for w in made if w.key[2] == 3]
    assert split and all(w.fft_work is None for w in split)
    assert C.tc_status() == 0


def rel_max(got, ref):
    return np.max(np.abs(got.cpu().numpy() - ref)) / np.max(np.abs(ref))


def placement_map(M, N, seed):
    """A density as GP has it: clusters over a noisy floor."""
    rng = np.random.RandomState(seed)
    u, v = np.arange(M)[:, None] / M, np.arange(N)[None, :] / N
    rho = 0.6 + 0.3 * rng.uniform(size=(M, N))
    for a, b, s, h in rng.uniform(size=(12, 4)):
        rho += (0.5 + 2 * h) * np.exp(-((u - a) ** 2 + (v - b) ** 2) / (2 * (0.02 + 0.1 * s) ** 2))
    return rho.astype(np.float32)


# the tile sizes of both product kernels, ragged sides, and the largest grid that trials are run on
@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16", "split_bf16"])
@pytest.mark.parametrize("shape", [(64, 64), (128, 256), (136, 200), (360, 360), (1024, 1024)])
def test_product_transforms_against_fp64(C, precision, shape):
    from dreamplace_b200._native import precision_code
    from dreamplace_b200.dct2_fft2 import transform_2d, transform_matrices
    M, N = shape
    prec = precision_code(precision)
    x = np.random.RandomState(M + N).uniform(-1, 1, size=(M, N)).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    (cM, chM, shM), (cN, chN, shN) = (transform_matrices(n, prec, xt.device) for n in shape)
    for left, right, alpha, f in ((cM, cN, 4.0 / (M * N), oracle.dct2), (chM, chN, 4.0, oracle.idct2),
                                  (chM, shN, 4.0, oracle.idct_idxst), (shM, chN, 4.0, oracle.idxst_idct)):
        err = rel_max(transform_2d(xt, left, right, alpha, prec), f(x))
        assert err <= FIELD_TOL[precision], (f.__name__, err)
    assert C.tc_status() == 0


@pytest.mark.parametrize("precision", ["fp32", "tf32", "bf16", "split_bf16"])
@pytest.mark.parametrize("shape", [(64, 64), (128, 256), (136, 200), (360, 360), (1024, 1024)])
def test_product_solve_against_fp64(C, precision, shape):
    """poisson_solve by the products, allocated and through a workspace (a trial's
    form: the map's operand filled and the energy zeroed by the caller)."""
    from dreamplace_b200._native import precision_code
    from dreamplace_b200.electric_potential import PoissonWorkspace, poisson_energy, poisson_solve
    M, N = shape
    bsx, bsy = 12.0, 9.5
    rho = placement_map(M, N, M + N)
    rex, rey, renergy = oracle.poisson(rho * np.float64(bsx * bsy), bsx, bsy)
    rt = torch.from_numpy(rho).cuda()
    launches = C.launch_count()
    solves = [poisson_solve(rt, bsx, bsy, precision, fast=False)]
    prec = precision_code(precision)
    assert C.launch_count() - launches >= 4  # four products (the fast transforms launch three passes)
    ws = PoissonWorkspace(M, N, prec, rt.device, fast=False)
    if prec:
        ws.rho.fill(rt)
    solves.append(poisson_solve(rt, bsx, bsy, precision, ws=ws, fast=False, prepared=True))
    for ex, ey, energy in solves:
        assert rel_max(ex, rex) <= FIELD_TOL[precision] and rel_max(ey, rey) <= FIELD_TOL[precision]
        assert abs(float(energy) - renergy) <= FIELD_TOL[precision] * abs(renergy)
    assert torch.equal(solves[0][0], ws.ex) and torch.equal(solves[0][1], ws.ey)
    energy = poisson_energy(rt, bsx, bsy, precision, fast=False)
    assert abs(float(energy) - renergy) <= FIELD_TOL[precision] * abs(renergy)
    assert C.tc_status() == 0


@pytest.mark.parametrize("deterministic", [0, 1])
def test_fused_trial_equals_its_pieces(trials_on_products, design, deterministic):  # noqa: F811
    test_gpu_gp.test_fused_trial_equals_its_pieces(design, "split_bf16", deterministic)


@pytest.mark.parametrize("deterministic", [0, 1])
def test_fused_trial_of_a_larger_grid(C, deterministic):
    test_gpu_gp.test_fused_trial_equals_its_pieces(synthetic.scaled(20000, num_bins=256, seed=4), "split_bf16",
                                                   deterministic)


def test_recapture_keeps_the_trajectory(trials_on_products, design):  # noqa: F811
    test_gpu_gp.test_recapture_with_one_timed_piece_keeps_the_trajectory(design)


def test_gp_converges_and_matches_plain(trials_on_products, design):  # noqa: F811
    test_gpu_gp.test_gp_converges_and_split_bf16_matches_plain(design)


def test_early_trajectory_matches_reference_loop(trials_on_products, design, ref):  # noqa: F811
    test_gpu_gp_reference.test_early_trajectory_matches_reference_loop(design, ref, "graph", "split_bf16")


@pytest.mark.parametrize("noise", [0.0, 0.025])
def test_final_hpwl_matches_reference_loop(trials_on_products, design, ref, noise):  # noqa: F811
    test_gpu_gp_reference.test_final_hpwl_within_half_percent_of_reference_loop(design, ref, "graph", "split_bf16",
                                                                                noise)


def test_resume_follows_the_original_trajectory(trials_on_products):
    test_gpu_checkpoint.test_resume_follows_the_original_trajectory()


def test_batched_designs_match_single_runs(trials_on_products):
    test_gpu_batch.test_batched_designs_match_single_runs()


def test_waits_that_expire_with_copies_in_flight(C):
    """A wait budget shorter than the copies take: a block that gives up drains
    its copies and MMAs before it returns, the status says so, and the next solve
    is what it was."""
    from dreamplace_b200.electric_potential import poisson_solve
    for precision, side in (("split_bf16", 136), ("tf32", 1024), ("split_bf16", 1024)):
        x = torch.from_numpy(placement_map(side, side, 7)).cuda()
        before = [t.clone() for t in poisson_solve(x, 10.0, 10.0, precision, fast=False)]
        assert C.tc_status() == 0
        try:
            C.tc_set_wait_budget(1)
            for _ in range(3):
                poisson_solve(x, 10.0, 10.0, precision, fast=False)
            status = C.tc_status()
        finally:
            C.tc_set_wait_budget(4_000_000_000)
        assert status in (0, 1, 2, 3)  # the hardware's own wait may outlast the copies
        after = poisson_solve(x, 10.0, 10.0, precision, fast=False)
        assert torch.equal(after[0], before[0]) and torch.equal(after[1], before[1])
        assert C.tc_status() == 0
