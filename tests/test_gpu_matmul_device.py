"""Products of a resident matrix with many columns on device pointers (l2b_matrix_matmul_device): its workspace."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def resident(pkg, synth):
    """(type, in, out) -> matmul(x, y, columns) on the current stream."""
    import torch
    from llama2_jl_b200 import _lib as L
    handles = []

    def make(t, n_in, n_out):
        A = synth.matrix(t, n_in, n_out, seed=n_in + n_out)
        h = C.c_void_p()
        L.check(L.lib().l2b_matrix_create(t, L.ptr(A.data), n_in, n_out, 1, C.byref(h)))
        handles.append(h)
        return A, lambda x, y, n: L.check(L.lib().l2b_matrix_matmul_device(h, 0, x.data_ptr(), n, y.data_ptr(), torch.cuda.current_stream().cuda_stream))
    yield make
    torch.cuda.synchronize()
    for h in handles:
        L.lib().l2b_matrix_destroy(h)


# at both shapes the smaller count falls into more partial results than the larger one when the cuts hang on the columns
@pytest.mark.parametrize("n_in,n_out,most,fewer", [(4096, 14336, 513, (129, 16)), (4096, 4096, 257, (54, 128, 1)), (2048, 300, 130, (129, 17))])
def test_only_more_columns_allocate(resident, n_in, n_out, most, fewer):
    """Calls with fewer columns than an earlier one take no memory, and a graph that holds the earlier one stays good."""
    import torch
    A, matmul = resident(12, n_in, n_out)
    x = torch.randn((most, n_in), generator=torch.Generator(device="cuda").manual_seed(n_out), device="cuda")
    y, z = torch.zeros((most, n_out), device="cuda"), torch.zeros((most, n_out), device="cuda")
    matmul(x, y, most)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        matmul(x, z, most)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, z)
    free = torch.cuda.mem_get_info()[0]
    for n in fewer:
        matmul(x, y, n)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    for n in fewer:
        part = torch.cuda.CUDAGraph()
        with torch.cuda.graph(part):  # (a call that allocated would be refused here)
            matmul(x, y, n)
        y.zero_()
        part.replay()
        want = x[:n].double() @ torch.from_numpy(_dense(A)).cuda().double().T
        assert (y[:n] - want).abs().max() <= 4e-6 * want.abs().max()
        assert (y[n:] == 0).all()
    x.copy_(-x)
    z.zero_()
    graph.replay()
    matmul(x, y, most)
    assert torch.equal(y, z)


def test_more_columns_than_a_grid_holds(resident):
    """70 000 columns of a matrix whose products are added up from parts, in a workspace of a thousand; columns at the cuts and the ends."""
    import torch
    n_in, n_out, n = 2560, 130, 70000
    A, matmul = resident(13, n_in, n_out)
    x = torch.randn((n, n_in), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    y = torch.full((n, n_out), float("nan"), device="cuda")
    matmul(x, y, 16)  # (kernels are loaded by their first call)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    matmul(x, y, n)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 64 << 20
    assert torch.isfinite(y).all()
    some = torch.tensor([0, 127, 128, 1023, 1024, 1025, 65535, 65536, 69000, n - 1], device="cuda")
    want = x[some].double() @ torch.from_numpy(_dense(A)).cuda().double().T
    assert (y[some] - want).abs().max() <= 4e-6 * want.abs().max()


@pytest.mark.parametrize("t", [12, 13])
def test_long_rows_keep_their_precision(resident, t):
    """56 super-blocks in one sum.  2.05e-7 is the relative error (2-norms, against 64 bits) of such rows with exact integer sums inside each
    super-block and one f32 addition behind it; a chain over every 64 values (280 additions) is at 2.5e-7 to 3.1e-7."""
    import torch
    n_in, n_out, n = 14336, 133 * 128, 128
    A, matmul = resident(t, n_in, n_out)
    x = torch.randn((n, n_in), generator=torch.Generator(device="cuda").manual_seed(t), device="cuda")
    for cols in (16, 48, 128):
        y = torch.empty((cols, n_out), device="cuda")
        matmul(x, y, cols)
        for first in (0, n_out - 512):
            want = x[:cols].double() @ torch.from_numpy(_dense(A.rows(first, first + 512))).cuda().double().T
            assert (y[:, first:first + 512] - want).norm() < 2.05e-7 * want.norm(), cols


@pytest.mark.parametrize("t,n_in,n_out", [(12, 4096, 1030), (13, 1024, 384), (12, 512, 19000)])
def test_a_column_has_the_same_bits_in_any_company(resident, t, n_in, n_out):
    """Tiles of 32, 64 and 128 columns, full and partly filled, one and several of them."""
    import torch
    _, matmul = resident(t, n_in, n_out)
    x = torch.randn((1100, n_in), generator=torch.Generator(device="cuda").manual_seed(t), device="cuda")
    want = torch.empty((1100, n_out), device="cuda")
    matmul(x, want, 1100)
    for first, n in [(0, 1), (7, 4), (0, 16), (3, 17), (0, 33), (1, 64), (0, 65), (90, 128), (5, 129), (1000, 100)]:
        y = torch.empty((n, n_out), device="cuda")
        matmul(x[first:], y, n)
        assert torch.equal(y, want[first:first + n]), (first, n)


def _dense(A):
    from llama2_jl_b200 import _lib as L
    out = np.empty((A.out_dim, A.in_dim), np.float32)
    L.check(L.lib().l2b_dequantize(A.ggml_type, L.ptr(A.data), out.size, L.ptr(out)))
    return out
