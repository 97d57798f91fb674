"""The block solver's chain substitutions at the lengths where they change (run on a B200 with -m gpu): 4 to 12
and 13 to 20 positions are rounded up to one of two register-resident lengths, longer chains and those of
more than five momentum bins walk by fours."""
import numpy as np
import pytest

from conftest import background

pytestmark = pytest.mark.gpu

NAMES = ("lmaxg", "lmaxgp", "lmaxr", "lmaxnu", "nqmax")


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the -m gpu tests need a GPU")
    return torch


# longest chain 4, 7, 12, 13, 16, 20, 21, 25 positions; photons, polarisation, neutrinos or bins the longest; one
# and six bins
@pytest.mark.parametrize("size", [(4, 3, 3, 3, 2), (5, 6, 4, 3, 3), (12, 5, 6, 3, 2), (5, 12, 6, 3, 2), (7, 6, 15, 4, 5),
                                  (6, 5, 7, 19, 3), (9, 20, 5, 3, 2), (25, 8, 7, 3, 2), (12, 11, 15, 3, 1),
                                  (9, 10, 13, 6, 6)])
def test_gpu_block_and_one_warp_solves_are_the_same_at_every_chain_length(torch_cuda, size):
    from discoeb_b200.perturbations import CosmologyBatch
    bg = background("lcdm_mnu", 256)
    ks = np.geomspace(0.3, 1.0, 12)
    kw = dict(params=[bg], aexp_out=np.array([0.02, 0.3]), rtol=1e-4, atol=1e-6, **dict(zip(NAMES, size)))
    out = []
    for copies in (1, 300):  # 3600 modes of similar length: a warp each
        batch = CosmologyBatch(kmodes=np.tile(ks, copies), **kw)
        batch.launch()
        y, _, n = batch.result()
        out.append((y[0][:12], n[0][:12]))
    # the same operations in the same order: equal bit for bit
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
