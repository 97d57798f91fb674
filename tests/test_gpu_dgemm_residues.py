"""The residue form of the FP64 product on the int8 tensor cores (large products with 6 or 7 slices) at the
edges of its range, against the FP64 product (run on a B200 with -m gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the -m gpu tests need a GPU")
    return torch


# m, n, k, slices, K ranges: ragged tiles in every dimension, 1 to 4 ranges; an odd row pitch (single
# loads); the longest range (16512) and one beyond it (digits); one tile row short of the residues
@pytest.mark.parametrize("m,n,k,slices,split", [(2049, 515, 12290, 7, 1), (2050, 513, 12291, 7, 2), (2304, 514, 12290, 6, 3),
                                                (2049, 1027, 8194, 7, 4), (1025, 770, 16512, 7, 1),
                                                (1025, 770, 16513, 7, 1), (2048, 516, 12290, 7, 1)])
@pytest.mark.parametrize("trans", [False, True])
def test_gpu_residue_products_within_the_splitting_bound(torch_cuda, m, n, k, slices, split, trans):
    torch = torch_cuda
    from discoeb_b200 import _abi
    lib = _abi.lib()
    g = torch.Generator(device="cuda").manual_seed(m + k)
    f64 = dict(dtype=torch.float64, device="cuda")

    def operand(rows):
        x = torch.randn((rows, k), generator=g, **f64) * torch.exp(14 * torch.rand((rows, 1), generator=g, **f64) - 7)
        x *= torch.exp(-torch.arange(k, **f64) / 900.0)
        x[0] = 0.0
        x[1, ::2] = -x[1, 0].abs()  # many equal extremes
        return x
    A, B = operand(m), operand(n)
    At, Bt = (A.t().contiguous(), B.t().contiguous()) if trans else (A, B)
    lda, ldb = (m, n) if trans else (k, k)
    C = torch.empty((m, n), **f64)
    nb = lib.discoeb_dgemm_i8_workspace_bytes(m, n, k, slices, split)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    rc = lib.discoeb_dgemm_i8(m, n, k, At.data_ptr(), lda, int(trans), Bt.data_ptr(), ldb, int(trans), C.data_ptr(), n,
                              slices, split, ws.data_ptr(), nb, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    aA, aB = A.abs(), B.abs()
    bound = 2 * 2.0 ** (1 - 7 * slices) * (aA.amax(1)[:, None] * aB.sum(1)[None, :] + aA.sum(1)[:, None] * aB.amax(1)[None, :])
    bound += 8 * 2.2e-16 * (aA @ aB.t())
    assert bool(((C - A @ B.t()).abs() <= bound).all())
