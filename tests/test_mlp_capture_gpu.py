"""Training steps captured in a CUDA graph: the update kernel is launched
programmatically behind the gradient kernel, in a graph as on a stream.  Four
captured steps behind a copy give the parameters of four plain steps, bit for
bit (fixed-order sums)."""
import ctypes as C

import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 8192, 12000])
def test_captured_steps_equal_plain_steps(cuda, n):
    import torch
    from q_psdm_b200 import surrogate as S
    p = M.init_params(3, out_scale=1.0).astype(np.float32)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    x = torch.rand(n, 5, device="cuda", generator=gen)
    t = torch.rand(n, 2, device="cuda", generator=gen)
    a, b = S.Mlp(0, params=p), S.Mlp(0, params=p)
    x2 = torch.zeros_like(x)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        x2.copy_(x)
        for _ in range(4):
            assert a.L.qpsdm_mlp_train_step(a.h, x2.data_ptr(), t.data_ptr(), n, C.c_float(1e-3),
                                            None, C.c_void_p(stream.cuda_stream)) == 0
    graph.replay()
    torch.cuda.synchronize()
    for _ in range(4):
        b.train_step(x, t, 1e-3)
    b.status()
    assert np.array_equal(a.params(), b.params())
    del graph
