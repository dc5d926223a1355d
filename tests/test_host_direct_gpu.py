"""Results in pinned host memory, stored by the matmul itself or by a copy behind it: the same bits as in the device buffer and as
the plain matmul's, call after call on one stream."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from relax_b200 import _lib, ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N,K", [(4096, 256), (4100, 2560), (4095, 512), (11008, 2048), (4096, 288)])
def test_host_results(cuda_lib, M, N, K):
    wq, s = (torch.from_numpy(a).cuda() for a in synth.make_weights(N, K, np.random.default_rng(N + K)))
    gen = torch.Generator().manual_seed(M)
    x_dev = torch.empty((M, K), dtype=torch.float16, device="cuda")
    y_dev = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    calls = [(torch.randn((M, K), generator=gen).half().pin_memory(), torch.full((M, N), float("nan"), dtype=torch.float16).pin_memory()) for _ in range(6)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for x_host, y_host in calls:               # (the staging buffers are shared: every call waits for the one in front)
        assert cuda_lib.b200_q4f16_matmul_host(x_host.data_ptr(), x_dev.data_ptr(), wq.data_ptr(), s.data_ptr(), y_dev.data_ptr(),
                                               y_host.data_ptr(), M, N, K, stream.cuda_stream) == 0, _lib.last_error()
    stream.synchronize()
    assert (y_dev.cpu().view(torch.int16) == calls[-1][1].view(torch.int16)).all()
    for x_host, y_host in calls:
        want = ops.q4f16_matmul(x_host.cuda(), wq, s).cpu()
        assert (y_host.view(torch.int16) == want.view(torch.int16)).all()


SIZES = [(4096, 256), (4100, 2560), (4095, 512), (11008, 2048), (4096, 288)]
# both sides of the lines between the two ways back
MORE = [(1, 256), (17, 1024), (8192, 1024), (8200, 1024), (16384, 1024), (16392, 1024), (12280, 4096), (12296, 4096), (4096, 4096), (6144, 768)]


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N,K,graph", [(*nk, True) for nk in SIZES] + [(*nk, graph) for nk in MORE for graph in (False, True)])
def test_host_results_launched_and_captured(cuda_lib, M, N, K, graph):
    wq, s = (torch.from_numpy(a).cuda() for a in synth.make_weights(N, K, np.random.default_rng(N + K)))
    gen = torch.Generator().manual_seed(M)
    x_dev = torch.empty((M, K), dtype=torch.float16, device="cuda")
    y_dev = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    calls = [(torch.randn((M, K), generator=gen).half().pin_memory(), torch.full((M, N), float("nan"), dtype=torch.float16).pin_memory()) for _ in range(6)]
    stream = torch.cuda.Stream()

    def launch():
        for x_host, y_host in calls:
            assert cuda_lib.b200_q4f16_matmul_host(x_host.data_ptr(), x_dev.data_ptr(), wq.data_ptr(), s.data_ptr(), y_dev.data_ptr(),
                                                   y_host.data_ptr(), M, N, K, stream.cuda_stream) == 0, _lib.last_error()

    torch.cuda.synchronize()
    if graph:                                  # (another choice of the way back; nothing runs before the replay)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            launch()
        assert torch.isnan(calls[0][1]).all()
        with torch.cuda.stream(stream):
            g.replay()
    else:
        launch()
    stream.synchronize()
    assert (y_dev.cpu().view(torch.int16) == calls[-1][1].view(torch.int16)).all()
    for x_host, y_host in calls:
        want = ops.q4f16_matmul(x_host.cuda(), wq, s).cpu()
        assert (y_host.view(torch.int16) == want.view(torch.int16)).all()
