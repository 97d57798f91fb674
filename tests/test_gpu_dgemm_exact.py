"""The residue form of the FP64 product on the int8 tensor cores drops nothing: products of integers within
its digits come out correctly rounded, and real operands lose their own rounding to the digits only (run on
a B200 with -m gpu)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# ragged tiles, just above the line of the residues: 9 x 3 x 97 and 9 x 8 x 35 tiles
SHAPES = {7: (2049, 515, 12290), 6: (2049, 1795, 4354)}


def _entries(m, n):
    """checked entries: the tiles' edges"""
    return np.r_[0:3, 255:257, 1023, m - 2:m], np.r_[0:2, 127, 255:257, n - 3, n - 1]


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("no CUDA device: the -m gpu tests need a GPU")
    return torch


def _product(torch, A, B, slices, split, trans):
    from discoeb_b200 import _abi
    m, n, k = SHAPES[slices]
    lib = _abi.lib()
    At, Bt = (A.t().contiguous(), B.t().contiguous()) if trans else (A, B)
    lda, ldb = (m, n) if trans else (k, k)
    C = torch.empty((m, n), dtype=torch.float64, device="cuda")
    nb = lib.discoeb_dgemm_i8_workspace_bytes(m, n, k, slices, split)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    assert lib.discoeb_dgemm_i8(m, n, k, At.data_ptr(), lda, int(trans), Bt.data_ptr(), ldb, int(trans), C.data_ptr(), n,
                                slices, split, ws.data_ptr(), nb, torch.cuda.current_stream().cuda_stream) == 0
    return C.cpu().numpy()


@pytest.mark.parametrize("slices,split", [(7, 1), (7, 4), (6, 2), (6, 3)])
@pytest.mark.parametrize("trans", [False, True])
def test_gpu_residue_products_of_integers_are_exact(torch_cuda, slices, split, trans):
    torch = torch_cuda
    rng = np.random.default_rng(slices + split)
    m, n, k = SHAPES[slices]
    rows, cols = _entries(m, n)
    bits = 7 * slices  # a row's largest is just below 2^(bits - 1): the last digit's unit is 1

    def operand(count):
        hi = rng.integers(-(2**24), 2**24, (count, k))
        lo = rng.integers(0, 2 ** (bits - 25), (count, k))
        hi[:, 0], lo[:, 0] = 2**24 - 1, 1  # every row has its largest at the same exponent
        return hi, lo, 2.0 ** rng.integers(-60, 60, (count, 1))  # and a power of two of its own
    sh = bits - 25
    (ah, al, sa), (bh, bl, sb) = operand(m), operand(n)
    A = torch.from_numpy((ah * 2.0**sh + al) * sa).cuda()
    B = torch.from_numpy((bh * 2.0**sh + bl) * sb).cuda()
    C = _product(torch, A, B, slices, split, trans)
    whole = lambda hi, lo: [int(h) * 2**sh + int(x) for h, x in zip(hi, lo)]  # noqa: E731
    columns = {j: whole(bh[j], bl[j]) for j in cols}
    for i in rows:
        a = whole(ah[i], al[i])
        for j in cols:
            exact = sum(x * y for x, y in zip(a, columns[j]))
            got = C[i, j] / sa[i, 0] / sb[j, 0]
            # three limbs put together with two roundings
            assert abs(int(got) - exact) * 2**52 <= abs(exact) + 2**52, (i, j)


@pytest.mark.parametrize("slices,split", [(7, 2), (6, 1)])
@pytest.mark.parametrize("trans", [False, True])
def test_gpu_residue_products_lose_the_operands_rounding_only(torch_cuda, slices, split, trans):
    torch = torch_cuda
    rng = np.random.default_rng(10 * slices + split)
    m, n, k = SHAPES[slices]
    rows, cols = _entries(m, n)
    A = rng.standard_normal((m, k)) * np.exp(14 * rng.random((m, 1)) - 7)
    B = rng.standard_normal((n, k)) * np.exp(14 * rng.random((n, 1)) - 7)
    C = _product(torch, torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), slices, split, trans)
    for i in rows:
        for j in cols:
            a, b = A[i].astype(np.longdouble), B[j].astype(np.longdouble)
            exact, aa, ab = (a * b).sum(), np.abs(a), np.abs(b)
            # half a unit of the last digit, at most 2^(-7 slices) 128 / 127 of the row's largest, on each operand,
            # and the result's two roundings
            bound = 2.0 ** (-7 * slices) * 128 / 127 * (aa.max() * ab.sum() + aa.sum() * ab.max()) + 2.0**-52 * abs(exact)
            assert abs(C[i, j] - exact) <= bound * (1 + 1e-9), (i, j)
