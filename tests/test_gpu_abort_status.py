"""A mode whose tangents were given up reports it, also when its forward solve had already finished (run on
a B200 with -m gpu)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THETA = dict(omega_c=0.120, omega_b=0.0224, h=0.674, n_s=0.965, ln10As=math.log(21.0), w0=-0.9, wa=0.1, m_nu=0.06)
NAMES = ("lmaxg", "lmaxgp", "lmaxr", "lmaxnu", "nqmax")
ABORTED = 6


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the -m gpu tests need a GPU")
    return torch


# all directions in one block; a block for each of six; and above the block form's sizes, the step records
# in shared memory (three directions a block) and split
@pytest.mark.parametrize("size,records", [((11, 11, 11, 8, 3), True), ((50, 50, 17, 17, 5), True),
                                          ((60, 50, 17, 17, 5), False), ((60, 50, 17, 17, 5), True)])
@pytest.mark.parametrize("full", [False, True])
def test_gpu_tangents_given_up_after_the_forward_solve_abort_the_mode(torch_cuda, size, records, full):
    torch = torch_cuda
    from discoeb_b200.gradients import JacobianProblem
    prob = JacobianProblem(THETA, aexp_out=(1.0,), kmodes=np.full(4, 0.1), rtol=1e-4, atol=1e-6, full_state=full,
                           **dict(zip(NAMES, size)))
    # a solve of two accepted steps, which needs no slot of the hand-over twice
    prob.d_tout.copy_(1.001 * prob.d_ts[:1])
    for max_polls, expect in ((1, ABORTED), (0, 0), (1, ABORTED), (0, 0)):
        prob.ctrl.max_polls = max_polls
        prob.d_out.zero_()
        prob.d_outd.zero_()
        prob.launch(records=records)
        torch.cuda.synchronize()
        status, nsteps = prob.d_stat.cpu().numpy()
        assert (status == expect).all(), status
        assert (nsteps == 2).all()
        assert bool(torch.isfinite(prob.d_outd).all()) == (expect == 0)
