"""A cosmology whose hierarchies differ from the first one's is reported and not solved, also where its
states have as many rows (run on a B200 with -m gpu)."""
import ctypes
import math

import numpy as np
import pytest

from conftest import background

pytestmark = pytest.mark.gpu

# 143 rows each: 17 multipoles of 5 momentum bins, 5 multipoles of 15
FIRST = dict(lmaxg=12, lmaxgp=12, lmaxr=17, lmaxnu=17, nqmax=5)
OTHER = dict(FIRST, lmaxnu=5, nqmax=15)
THETA = dict(omega_c=0.120, omega_b=0.0224, h=0.674, n_s=0.965, ln10As=math.log(21.0), w0=-0.9, wa=0.1, m_nu=0.06)
BAD_INDEX = 5


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the -m gpu tests need a GPU")
    return torch


def _relabel_second(torch, problem):
    """The second cosmology of the launch with the other hierarchies (its inputs are never read)."""
    host = type(problem.dcs[1].host).from_buffer_copy(problem.dcs[1].host)
    host.lmaxnu, host.nqmax = OTHER["lmaxnu"], OTHER["nqmax"]
    raw = bytes(ctypes.string_at(ctypes.addressof(host), ctypes.sizeof(host)))
    problem.d_cosmos[len(raw):2 * len(raw)] = torch.frombuffer(bytearray(raw), dtype=torch.uint8).cuda()


# a block per mode, one and two per SM, and a warp per mode; whole states and output fields
@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("copies", [1, 90, 400])
def test_gpu_forward_refuses_another_layout_of_the_same_size(torch_cuda, copies, full):
    from discoeb_b200.perturbations import CosmologyBatch
    bg = background("lcdm_mnu", 256)
    ks = np.tile(np.geomspace(1e-3, 0.05, 5), copies)
    batch = CosmologyBatch(params=[bg, bg], kmodes=ks, aexp_out=np.array([0.1]), rtol=1e-4, atol=1e-6,
                           return_full=full, **FIRST)
    batch.launch()
    y0 = batch.result()[0]
    _relabel_second(torch_cuda, batch)
    batch.launch()
    y, status, nsteps = batch.result(on_failure="ignore")
    assert (status[0] == 0).all() and (status[1] == BAD_INDEX).all() and (nsteps[1] == 0).all()
    np.testing.assert_array_equal(y[0], y0[0])
    assert np.isnan(y[1]).all()


@pytest.mark.parametrize("copies", [1, 400])
def test_gpu_adjoint_refuses_another_layout_of_the_same_size(torch_cuda, copies):
    torch = torch_cuda
    from discoeb_b200.gradients import AdjointBatch
    ks = np.tile(np.geomspace(1e-3, 0.05, 5), copies)
    batch = AdjointBatch([THETA, THETA], kmodes=ks, aexp_out=(0.1,), rtol=1e-4, atol=1e-6, step_capacity=512, **FIRST)
    _relabel_second(torch, batch)
    batch.launch_forward()
    P, status, _ = batch.forward_power(on_failure="ignore")
    assert (status[0] == 0).all() and (status[1] == BAD_INDEX).all()
    assert np.isfinite(P[0]).all() and np.isnan(P[1]).all()
    for forget in (False, True):  # the reverse sweep checks the layout itself
        if forget:
            batch.d_fstat[0].zero_()
        batch.launch_backward(np.ones((2, len(ks), 1)))
        torch.cuda.synchronize()
        status = batch.d_bstat.cpu().numpy()[batch.inv].reshape(2, -1)
        assert (status[0] == 0).all() and (status[1] == BAD_INDEX).all()


# 143 rows; 231 rows, above the block form's sizes
@pytest.mark.parametrize("size", [FIRST, dict(FIRST, lmaxg=100)])
def test_gpu_tangents_refuse_another_layout_of_the_same_size(torch_cuda, size):
    from discoeb_b200.gradients import JacobianBatch
    batch = JacobianBatch([THETA, THETA], kmodes=np.geomspace(1e-3, 0.05, 3), aexp_out=(0.1,), rtol=1e-4, atol=1e-6, **size)
    _relabel_second(torch_cuda, batch)
    batch.launch()
    P, J, status, _ = batch.result(on_failure="ignore")
    assert (status[0] == 0).all() and (status[1] == BAD_INDEX).all()
    assert np.isfinite(J[0]).all() and np.isnan(J[1]).all()
