"""The fast transforms of power-of-two grids (csrc/fft.cu) against fp64, and
their dispatch against the matrix products that serve every other map.

Tolerances: a radix-R pass rounds each value a few times and a twiddle factor
is at most four products deep, so a transform of N points carries about
8 log2(N) roundings of 2^-24 in the 2-norm; the solve adds the reference's
fp32 spectral weights (a handful of roundings each).
"""
import math

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.fixture(scope="module")
def C():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dreamplace_b200._native import C
    return C


def rel(a, b):
    return np.linalg.norm(a.double().cpu().numpy() - b) / np.linalg.norm(b)


def density(M, N, seed):
    rng = np.random.RandomState(seed)
    return (0.6 + 0.8 * rng.uniform(size=(M, N))).astype(np.float32)


# the smallest and largest sides, every remainder of the radix split (8 8 2,
# 8 8 4, 8 8 8, 16 16 4, 16 16 8, 16 16 16) on each axis, rectangular both ways
@pytest.mark.parametrize("shape", [(64, 64), (64, 4096), (4096, 64), (128, 256), (256, 128), (512, 1024),
                                   (1024, 512), (2048, 128), (64, 2048)])
def test_transforms_and_solve_against_fp64(C, shape):
    from dreamplace_b200 import dct2_fft2
    from dreamplace_b200.electric_potential import poisson_energy, poisson_solve
    M, N = shape
    x = density(M, N, M + N)
    xt = torch.from_numpy(x).cuda()
    assert dct2_fft2.fft_serves(xt, 0) and dct2_fft2.fft_serves(xt, 3) and not dct2_fft2.fft_serves(xt, 1)
    tol = 8 * math.log2(M * N) * EPS
    for cls, ref in ((dct2_fft2.DCT2, oracle.dct2), (dct2_fft2.IDCT2, oracle.idct2),
                     (dct2_fft2.IDCT_IDXST, oracle.idct_idxst), (dct2_fft2.IDXST_IDCT, oracle.idxst_idct)):
        for precision in ("fp32", "split_bf16"):
            assert rel(cls(precision=precision)(xt), ref(x)) <= tol, (cls.__name__, precision)
    bsx, bsy = 12.0, 9.5
    rex, rey, renergy = oracle.poisson(x * np.float64(bsx * bsy), bsx, bsy)
    ex, ey, energy = poisson_solve(xt, bsx, bsy, "split_bf16")
    assert rel(ex, rex) <= 4 * tol and rel(ey, rey) <= 4 * tol
    assert math.isclose(float(energy), renergy, rel_tol=4 * tol)
    assert math.isclose(float(poisson_energy(xt, bsx, bsy, "fp32")), float(energy), rel_tol=1e-12)
    assert C.tc_status() == 0


@pytest.mark.parametrize("shape", [(64, 64), (256, 512)])
def test_dispatch_agrees_with_the_products(C, shape):
    """Every form of the call that the fast transforms take, beside the products
    on the same values (a map whose rows start off a 16-byte boundary is theirs)."""
    from dreamplace_b200.dct2_fft2 import fft_serves
    from dreamplace_b200.electric_potential import PoissonWorkspace, poisson_solve
    M, N = shape
    x = torch.from_numpy(density(M, N, 3)).cuda()
    # a hi + lo operand carries its values to 2^-16 and four products follow one
    # another; the mean of the map, whose field is zero, brings its share of that
    # to the deviations that make the field, and as the mean is the same in every
    # row its errors add up along an axis: up to 8 times for these sides (2-norm)
    tol = 32 * 2.0 ** -16 * float(x.square().mean().sqrt() / x.std())
    near = lambda a, b: float((a - b).norm()) <= tol * float(b.norm())  # noqa: E731
    off = torch.empty(M * N + 1, device="cuda")[1:].view(M, N)
    off.copy_(x)
    assert not fft_serves(off, 3) and off.is_contiguous()
    for scale in (1.0, 0.125):
        for fast in (False, True):
            pex, pey, pen = poisson_solve(off, 3.0, 2.0, "split_bf16", fast, scale)
            for ws in (None, PoissonWorkspace(M, N, 3, x.device)):
                fex, fey, fen = poisson_solve(x, 3.0, 2.0, "split_bf16", fast, scale, ws)
                assert near(fex, pex) and near(fey, pey)
                assert math.isclose(float(fen), float(pen), rel_tol=2 * tol)
                assert fast == (float(fen) == 0.0)
                if ws is not None:  # a workspace also serves a map of the products
                    wex, _, wen = poisson_solve(off, 3.0, 2.0, "split_bf16", fast, scale, ws)
                    assert torch.equal(wex, pex) and math.isclose(float(wen), float(pen), rel_tol=1e-12)
    with pytest.raises(RuntimeError):  # fp32 products refuse such rows
        poisson_solve(off, 3.0, 2.0, "fp32")


def test_product_bounded_wait_on_a_ragged_grid(C):
    """The tensor-core product's bounded wait, on a grid that the fast transforms
    do not take: the launch reports the expired wait and the next solve is right."""
    from dreamplace_b200.electric_potential import poisson_solve
    x = torch.from_numpy(density(136, 136, 5)).cuda()
    before = poisson_solve(x, 10.0, 10.0, "split_bf16")[0].clone()
    assert C.tc_status() == 0
    try:
        C.tc_set_wait_budget(20_000_000)  # ~10 ms
        C.tc_set_skip_loads(1)
        poisson_solve(x, 10.0, 10.0, "split_bf16")
        status = C.tc_status()
    finally:
        C.tc_set_skip_loads(0)
        C.tc_set_wait_budget(4_000_000_000)
    assert status == 2
    assert torch.equal(poisson_solve(x, 10.0, 10.0, "split_bf16")[0], before)
    assert C.tc_status() == 0


def test_row_wait_that_expires_with_its_copies_in_flight(C):
    """A wait budget shorter than the copies take: blocks that give up wait for
    what they issued before they return, the status says so, and the next solve
    is what it was."""
    from dreamplace_b200.electric_potential import poisson_solve
    for side in (64, 1024, 4096):
        x = torch.from_numpy(density(side, side, 7)).cuda()
        before = [t.clone() for t in poisson_solve(x, 10.0, 10.0, "fp32")]
        assert C.tc_status() == 0
        try:
            C.tc_set_wait_budget(1)
            for _ in range(3):
                poisson_solve(x, 10.0, 10.0, "fp32")
            status = C.tc_status()
        finally:
            C.tc_set_wait_budget(4_000_000_000)
        assert status in (0, 2)  # the hardware's own wait may outlast the copies
        after = poisson_solve(x, 10.0, 10.0, "fp32")
        assert torch.equal(after[0], before[0]) and torch.equal(after[1], before[1])
        assert C.tc_status() == 0


@pytest.mark.parametrize("shape", [(64, 128), (1024, 64)])
def test_interleaved_field_of_the_c_abi(C, shape):
    """dp_poisson_fft's exy, the field as pairs for hosts that gather both
    components of a bin, beside its planar maps: the same bits."""
    import ctypes
    import os
    from dreamplace_b200.dct2_fft2 import fft_table
    from dreamplace_b200.electric_potential import poisson_solve
    M, N = shape
    lib = ctypes.CDLL(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dreamplace_b200",
                                   "lib", "libdreamplace_b200.so"))
    x = torch.from_numpy(density(M, N, 2)).cuda()
    ex, ey, energy = poisson_solve(x, 3.0, 2.0, "fp32")
    tw = [fft_table(n, x.device) for n in shape]
    work, exy = torch.empty(3 * M * N, device="cuda"), torch.empty(M, N, 2, device="cuda")
    e2 = torch.empty(1, dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    torch.cuda.synchronize()
    rc = lib.dp_poisson_fft(p(x), M, N, ctypes.c_float(1.0), ctypes.c_float(3.0 / 2.0), p(tw[0]), p(tw[1]), p(work),
                            None, None, p(exy), p(e2), 1, None)
    torch.cuda.synchronize()
    assert rc == 0
    assert torch.equal(exy[..., 0], ex) and torch.equal(exy[..., 1], ey)
    assert math.isclose(float(e2), float(energy), rel_tol=1e-12)
