"""The film export around its rule for one or four values a thread: every byte against double precision on both
sides of the rule and for exponents without an estimate, and one launch for a small film of any size."""
import ctypes as C

import numpy as np
import pytest

from rbr_b200 import abi
from test_film_bytes_gpu import expected, values

pytestmark = pytest.mark.gpu

RESIDENT = 148 * 2048  # values


@pytest.mark.parametrize("gamma,tonemap", [(2.2, True), (0.25, False), (0.2499, False), (0.1, True)])
@pytest.mark.parametrize("n", [3, 3 * 35, RESIDENT - 1, RESIDENT + 2, RESIDENT + 5])
def test_bytes_around_the_rule(ctx, gamma, tonemap, n):
    torch = pytest.importorskip("torch")
    n -= n % 3
    film = values(n, gamma, 12)
    buf = torch.from_numpy(film).cuda()
    out = torch.full((n + 8,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    st = ctx.lib.rbr_film_to_rgb8(ctx.h, C.c_void_p(buf.data_ptr()), n // 3, 1, 1.5, gamma, int(tonemap), C.c_void_p(out.data_ptr()),
                                  None)
    assert st == abi.RBR_OK, ctx.last_error()
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.array_equal(got[:n], expected(film, gamma, tonemap, 1.5)) and (got[n:] == 7).all()


@pytest.mark.parametrize("width,height", [(1, 1), (7, 5), (64, 48), (101, 99)])
def test_small_films_take_one_launch_of_one_value_a_thread(ctx, width, height):
    torch = pytest.importorskip("torch")
    driver = pytest.importorskip("cuda.bindings.driver")
    n = width * height * 3
    buf, out = torch.rand(n, device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        ctx.lib.rbr_film_to_rgb8(ctx.h, C.c_void_p(buf.data_ptr()), width, height, 1.0, 2.2, 1, C.c_void_p(out.data_ptr()),
                                 C.c_void_p(torch.cuda.current_stream().cuda_stream))
    _, _, count = driver.cuGraphGetNodes(driver.CUgraph(graph.raw_cuda_graph()))
    _, nodes, _ = driver.cuGraphGetNodes(driver.CUgraph(graph.raw_cuda_graph()), count)
    params = [driver.cuGraphKernelNodeGetParams(x)[1] for x in nodes]
    assert len(params) == 1 and params[0].gridDimX * params[0].blockDimX >= n
