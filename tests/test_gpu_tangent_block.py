"""The block form of the forward-mode solve at the sizes where its tiles end, against the reverse sweep
(run on a B200 with -m gpu): both are the derivative of the same discrete solve."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THETA = dict(omega_c=0.120, omega_b=0.0224, h=0.674, n_s=0.965, ln10As=math.log(21.0), w0=-0.9, wa=0.1, m_nu=0.06)
NAMES = ("lmaxg", "lmaxgp", "lmaxr", "lmaxnu", "nqmax")


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the -m gpu tests need a GPU")
    return torch


# the smallest state; 32 and 33 hierarchy rows; 16 momentum bins (46 slots: two per lane); 128 rows,
# all six directions at the shared-memory limit
@pytest.mark.parametrize("size", [(3, 3, 3, 3, 1), (9, 7, 9, 9, 1), (9, 7, 9, 10, 1), (3, 3, 3, 3, 16),
                                  (12, 12, 17, 17, 5)])
def test_gpu_block_tangents_equal_the_reverse_sweep(torch_cuda, size):
    from discoeb_b200.gradients import AdjointProblem, JacobianProblem
    kw = dict(aexp_out=np.array([0.02, 0.5, 1.0]), kmin=1e-4, kmax=2.0, num_k=6, rtol=1e-4, atol=1e-6,
              **dict(zip(NAMES, size)))
    jp = JacobianProblem(THETA, **kw)
    jp.launch()
    P, J, status, _ = jp.result()
    w = np.random.default_rng(0).uniform(0.5, 2.0, P.shape) / P
    ap = AdjointProblem(THETA, **kw)
    ap.launch_forward()
    ap.launch_backward(w)
    g = ap.gradient(w)[0]
    # sums of some 10^2 steps x 8 stages in another order: 1e-8, as for the two modes elsewhere
    expect = np.einsum("dkn,kn->d", J, w)
    np.testing.assert_allclose(g, expect, rtol=1e-8, atol=1e-12 * np.abs(expect).max())


# whole states at many output times (their projection runs in a kernel of its own), six directions in
# one block and, at 219 rows, in six
@pytest.mark.parametrize("size", [(11, 11, 11, 8, 3), (50, 50, 17, 17, 5)])
def test_gpu_whole_state_tangents_equal_the_output_fields(torch_cuda, size):
    from discoeb_b200.gradients import JacobianProblem
    kw = dict(kmin=1e-3, kmax=0.5, num_k=5, rtol=1e-4, atol=1e-6, **dict(zip(NAMES, size)))
    a = np.geomspace(2e-3, 1.0, 12)
    full = JacobianProblem(THETA, aexp_out=a, full_state=True, **kw)
    full.launch()
    y, yd = [x.cpu().numpy() for x in full.states()]
    one = JacobianProblem(THETA, aexp_out=a, **kw)
    one.launch()
    one.result()
    y20, y20d = one.d_out.cpu().numpy()[one.inv], one.d_outd.cpu().numpy()[:, one.inv]
    assert np.isfinite(yd).all()
    # eta, which every row feeds, stands in both outputs; sums of a few terms, so 1e-12 of its range
    np.testing.assert_allclose(y20[..., 0], y[..., 2], rtol=1e-13, atol=0)
    scale = np.abs(yd[..., 2]).max(axis=(1, 2), keepdims=True)
    assert (np.abs(y20d[..., 0] - yd[..., 2]) <= 1e-12 * scale).all()
