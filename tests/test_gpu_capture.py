"""kls_det_batch_device under stream capture, after a call of 16 omegas: more of them than
that call's are captured in launch sequences that its buffers hold."""
import ctypes as C

import numpy as np
import pytest
import torch

import kalnajs_log_spirals_b200 as K
from tests.test_gpu_parity import kconfig

pytestmark = pytest.mark.gpu

GRID = dict(m=2, G=1.0, L0=1.0, n_zang=4, q1=7, Ne=7, Rc_min=0.01, Rc_max=10.0, v_min=0.01,
            N_alpha=41, alpha_max=10.0, l_min=-4, l_max=4, nw=401, nwa=41)


@pytest.mark.parametrize("NR", [12, 40])           # over the table / self-similar
@pytest.mark.parametrize("n", [16, 17, 40, 64, 100])
def test_capture_after_sixteen(lib_path, NR, n):
    pc = K.precompute_all(kconfig(**GRID, NR=NR))
    om = np.linspace(0.6, 1.0, n) + 0.1j
    d_om = torch.tensor(om.view(np.float64), device="cuda")
    d_det = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    pc.ctx.call("kls_set_stream", C.c_void_p(stream.cuda_stream))

    def run(count):
        pc.ctx.call("kls_det_batch_device", C.c_void_p(d_om.data_ptr()), count, K.KLS_MODE_FP64,
                    C.c_void_p(d_det.data_ptr()), C.c_void_p(None))

    torch.cuda.synchronize()
    run(16)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        run(n)
    d_det.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    got = d_det.cpu().numpy().view(np.complex128)
    del graph
    pc.ctx.call("kls_set_stream", C.c_void_p(None))
    assert np.array_equal(got, K.compute_determinant_batched(om, pc))
    pc.close()
