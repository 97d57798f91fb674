"""The gradient kernel of states above the block form's sizes: its two placements of the step records, and
the reverse sweep (run on a B200 with -m gpu)."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THETA = dict(omega_c=0.120, omega_b=0.0224, h=0.674, n_s=0.965, ln10As=math.log(21.0), w0=-0.9, wa=0.1, m_nu=0.06)
SIZE = dict(lmaxg=60, lmaxgp=50, lmaxr=17, lmaxnu=17, nqmax=5)  # 229 rows: no direction fits beside a block's forward


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the -m gpu tests need a GPU")
    return torch


@pytest.mark.parametrize("full", [False, True])
def test_gpu_split_records_equal_the_shared_form(torch_cuda, full):
    """Three directions a block with the step records in shared memory, five with the
    split record: the same code on the same steps, bit for bit"""
    torch = torch_cuda
    from discoeb_b200.gradients import JacobianProblem
    prob = JacobianProblem(THETA, aexp_out=np.array([0.2, 0.5, 1.0]), kmodes=np.geomspace(1e-3, 0.3, 5), rtol=1e-5,
                           atol=1e-8, full_state=full, **SIZE)
    assert prob.lib.discoeb_jvp_records_bytes(ctypes.byref(prob.dc.host), 6, prob.K) > 0
    out = []
    for records in (False, True):
        prob.d_out.fill_(7.0)
        prob.d_outd.fill_(7.0)
        prob.launch(records=records)
        assert (prob.d_stat[0].cpu().numpy() == 0).all()
        out.append((prob.d_out.clone(), prob.d_outd.clone()))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert bool(torch.isfinite(out[0][1]).all())


def test_gpu_tangents_above_the_block_form_equal_the_reverse_sweep(torch_cuda):
    from discoeb_b200.gradients import AdjointProblem, JacobianProblem
    kw = dict(aexp_out=np.array([0.02, 0.5, 1.0]), kmin=1e-4, kmax=1.0, num_k=5, rtol=1e-4, atol=1e-6, **SIZE)
    jp = JacobianProblem(THETA, **kw)
    jp.launch()
    P, J, status, _ = jp.result()
    assert (status == 0).all()
    w = np.random.default_rng(0).uniform(0.5, 2.0, P.shape) / P
    ap = AdjointProblem(THETA, **kw)
    ap.launch_forward()
    ap.launch_backward(w)
    # sums of some 10^2 steps x 8 stages in another order: 1e-8, as for the other sizes
    expect = np.einsum("dkn,kn->d", J, w)
    np.testing.assert_allclose(ap.gradient(w)[0], expect, rtol=1e-8, atol=1e-12 * np.abs(expect).max())
