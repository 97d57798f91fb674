"""The forward solver's three mappings (one block of warps per SM, two per SM, one warp per mode)
at the sizes where their tiles end (run on a B200 with -m gpu)."""
import numpy as np
import pytest

from conftest import background
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

# (lmaxg, lmaxgp, lmaxr, lmaxnu, nqmax): the smallest state; 32 and 33 hierarchy rows (one and two
# row warps); the default; 16 momentum bins (19 chains); 128 rows (the last size of 256 threads)
SIZES = [(3, 3, 3, 3, 1), (9, 7, 9, 9, 1), (9, 7, 9, 10, 1), (11, 11, 11, 8, 3), (3, 3, 3, 3, 16),
         (12, 12, 17, 17, 5)]
NAMES = ("lmaxg", "lmaxgp", "lmaxr", "lmaxnu", "nqmax")


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the -m gpu tests need a GPU")
    return torch


def _solve(bg, size, ks, full, max_steps):
    from discoeb_b200.perturbations import solve_modes
    tout = bg["tau_of_a_spline"].evaluate(np.array([0.02, 0.5, 1.0]))
    return solve_modes(param=bg, kmodes=ks, tau_out=tout, rtol=1e-4, atol=1e-6, pcoeff=0.25, icoeff=0.8, dcoeff=0.0,
                       factormax=20.0, factormin=0.3, max_steps=max_steps, return_full=full, return_stats=True,
                       on_failure="keep", **dict(zip(NAMES, size)))


# 70 steps: the largest modes stop at the step limit, between two outputs
@pytest.mark.parametrize("max_steps", [4096, 70])
@pytest.mark.parametrize("size", SIZES)
def test_gpu_block_and_one_warp_solves_are_the_same(torch_cuda, size, max_steps):
    bg = background("lcdm_mnu", 256)
    ks = np.geomspace(1e-4, 2.0, 12)
    y, status, nsteps = _solve(bg, size, ks, False, max_steps)  # one block per SM
    assert (status == 0).all() if max_steps == 4096 else (status != 0).any()
    for copies in (50, 256):  # 600 modes: two blocks per SM; 3072 modes: one warp per mode
        yt, st, ns = _solve(bg, size, np.tile(ks, copies), False, max_steps)
        # the same operations in the same order: equal bit for bit
        np.testing.assert_array_equal(st, np.tile(status, copies))
        np.testing.assert_array_equal(ns, np.tile(nsteps, copies))
        np.testing.assert_array_equal(yt, np.tile(y, (copies, 1, 1)))
    # whole states: the projection of the radiation rows runs in a kernel of its own, which may
    # round it differently (a few units in the last place of rows that sum a dozen terms)
    yf, sf, nf = _solve(bg, size, ks, True, max_steps)
    yw, sw, nw = _solve(bg, size, np.tile(ks, 256), True, max_steps)
    np.testing.assert_array_equal(nw[:12], nf)
    np.testing.assert_array_equal(np.isnan(yw[:12]), np.isnan(yf))
    scale = np.nanmax(np.abs(yf), axis=0, keepdims=True)
    assert np.nanmax(np.abs(yw[:12] - yf) / np.where(scale > 0, scale, 1.0)) < 1e-13


@pytest.mark.parametrize("size", [(13, 12, 17, 17, 5), (50, 50, 17, 17, 5)])  # above 256 threads
def test_gpu_wide_block_solve_matches_oracle(torch_cuda, size):
    bg = background("lcdm_mnu", 256)
    ks = np.geomspace(1e-4, 1.0, 4)
    y, status, _ = _solve(bg, size, ks, False, 4096)
    assert (status == 0).all()
    yo, _, st = O.evolve_perturbations(param=bg, aexp_out=np.array([0.02, 0.5, 1.0]), kmin=0, kmax=0, num_k=0,
                                       rtol=1e-4, atol=1e-6, max_steps=4096, kmodes=ks, mode="clip",
                                       de_guard_eps=1e-9, return_full=False, **dict(zip(NAMES, size)))
    for idx in (0, 2, 4, 6, 8, 10):  # the same step sequence: agreement far below the solver's tolerance
        np.testing.assert_allclose(y[:, :, idx], yo[:, :, idx], rtol=1e-6, atol=1e-12)


# the recording solve of the adjoint: 12 modes on a block each, the same modes in a batch of a warp each
@pytest.mark.parametrize("every", [1, 7])
@pytest.mark.parametrize("size", [(3, 3, 3, 3, 1), (11, 11, 11, 8, 3)])
def test_gpu_recorded_block_and_one_warp_solves_are_the_same(torch_cuda, size, every):
    import math
    from discoeb_b200.gradients import AdjointProblem
    theta = dict(omega_c=0.120, omega_b=0.0224, h=0.674, n_s=0.965, ln10As=math.log(21.0), w0=-0.9, wa=0.1, m_nu=0.06)
    ks = np.geomspace(1e-3, 0.5, 12)
    out = []
    for k in (ks, np.tile(ks, 160)):  # 1920 modes: above both sizes' line
        p = AdjointProblem(theta, aexp_out=np.array([0.5, 1.0]), kmodes=k, rtol=1e-4, atol=1e-6, checkpoint_every=every,
                           **dict(zip(NAMES, size)))
        p.launch_forward()
        P, status, _ = p.forward_power()
        assert (status == 0).all()
        out.append((P[0][:12], np.sort(p.d_nacc.cpu().numpy())[::len(k) // 12]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
