"""Launches whose wavenumbers decide between the two forms of a solve: every mode is solved once, as in a
launch of few modes (run on a B200 with -m gpu)."""
import math

import numpy as np
import pytest

from conftest import background

pytestmark = pytest.mark.gpu

THETA = dict(omega_c=0.120, omega_b=0.0224, h=0.674, n_s=0.965, ln10As=math.log(21.0), w0=-0.9, wa=0.1, m_nu=0.06)
NAMES = ("lmaxg", "lmaxgp", "lmaxr", "lmaxnu", "nqmax")
SPREAD = np.geomspace(1e-4, 2.0, 14)  # modes of a third of the longest on the average: the short chain's
EQUAL = np.full(14, 0.02)             # the other form's


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the -m gpu tests need a GPU")
    return torch


# 700 modes: 25 rows; 143 rows of 15 bins; 144 rows (above 256 threads)
@pytest.mark.parametrize("size", [(3, 3, 3, 3, 1), (12, 12, 17, 5, 15), (13, 12, 17, 17, 5)])
@pytest.mark.parametrize("ks", [SPREAD, EQUAL], ids=["spread", "equal"])
@pytest.mark.parametrize("full", [False, True])
def test_gpu_forward_between_the_forms(torch_cuda, size, ks, full):
    from discoeb_b200.perturbations import CosmologyBatch
    kw = dict(params=[background("lcdm_mnu", 256)], aexp_out=np.array([0.02, 0.2]), rtol=1e-4, atol=1e-6,
              return_full=full, **dict(zip(NAMES, size)))
    few = CosmologyBatch(kmodes=ks, **kw)
    few.launch()
    y, _, n = few.result()
    many = CosmologyBatch(kmodes=np.tile(ks, 50), **kw)
    (many.d_full if full else many.d_out20).fill_(7.0)
    many.d_stat.fill_(7)
    many.launch()
    ym, status, nm = many.result()
    assert (status == 0).all()
    np.testing.assert_array_equal(nm[0], np.tile(n[0], 50))
    ref = np.tile(y[0], (50, 1, 1))
    if full:  # the projection of the radiation rows: a few units in the last place (a kernel of its own)
        assert (np.abs(ym[0] - ref) <= 1e-13 * np.abs(ref).max(axis=0, keepdims=True)).all()
    else:
        np.testing.assert_array_equal(ym[0], ref)


@pytest.mark.parametrize("ks", [SPREAD[:10], EQUAL[:10]], ids=["spread", "equal"])
def test_gpu_recording_between_the_forms(torch_cuda, ks):
    from discoeb_b200.gradients import AdjointProblem
    kw = dict(aexp_out=(0.2,), rtol=1e-4, atol=1e-6, step_capacity=1024, lmaxg=11, lmaxgp=11, lmaxr=11, lmaxnu=8, nqmax=3)
    out = []
    for copies in (1, 70):  # 700 modes
        p = AdjointProblem(THETA, kmodes=np.tile(ks, copies), **kw)
        p.d_out.fill_(7.0)
        p.d_nacc.fill_(-7)
        p.launch_forward()
        P, status, _ = p.forward_power()
        assert (status == 0).all()
        out.append((P[0][:10], np.sort(p.d_nacc.cpu().numpy())[::copies]))
        np.testing.assert_array_equal(P[0], np.tile(P[0][:10], (copies, 1)))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


# rows, directions asked for, modes, outputs, whole states: three groups a mode against one (161 rows); a
# direction each against three (219 rows), and against the split record, which wins with many outputs;
# one direction of a small state
@pytest.mark.parametrize("size,n_dir,copies,n_out,full", [((12, 12, 17, 17, 6), 6, 20, 1, False),
                                                          ((50, 50, 17, 17, 5), 6, 12, 3, False),
                                                          ((50, 50, 17, 17, 5), 6, 24, 130, True),
                                                          ((11, 11, 11, 8, 3), 1, 20, 2, True)])
@pytest.mark.parametrize("ks", [SPREAD[:10], EQUAL[:10]], ids=["spread", "equal"])
def test_gpu_tangents_between_the_forms(torch_cuda, size, n_dir, copies, n_out, full, ks):
    from discoeb_b200.gradients import JacobianProblem
    a = np.geomspace(0.01, 0.2, n_out) if n_out > 1 else (0.2,)
    kw = dict(aexp_out=a, rtol=1e-4, atol=1e-6, full_state=full, **dict(zip(NAMES, size)))
    out = []
    for m in (1, copies):
        p = JacobianProblem(THETA, kmodes=np.tile(ks, m), **kw)
        p.dirs = p.dirs[:n_dir]
        for t in (p.d_out, p.d_outd):
            t.fill_(7.0)
        p.d_stat.fill_(7)
        p.launch(records=full)
        assert (p.d_stat[0].cpu().numpy() == 0).all()
        out.append((p.d_out.cpu().numpy()[p.inv], p.d_outd.cpu().numpy()[:n_dir, p.inv], p.d_stat[1].cpu().numpy()[p.inv]))
    (y, yd, n), (ym, ydm, nm) = out
    np.testing.assert_array_equal(nm, np.tile(n, copies))
    # the same steps; sums of some 10^2 steps x 8 stages in another order: 1e-8 of each field's range
    # (whole states without row 0: the scale factor at an output is given, its tangent what is left of two
    # terms that cancel)
    if full:
        y, yd, ym, ydm = y[..., 1:], yd[..., 1:], ym[..., 1:], ydm[..., 1:]
    for one, many, axes in ((y, ym, (0, 1)), (yd, ydm, (1, 2))):
        rep = np.tile(one, (1,) * axes[0] + (copies, 1, 1))
        assert (np.abs(many - rep) <= 1e-8 * np.abs(rep).max(axis=axes, keepdims=True)).all()
