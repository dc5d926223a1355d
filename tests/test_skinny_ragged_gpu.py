"""Two to eight rows with a K of whole scale groups only, or scales off 16 bytes: the skinny kernel's form for them against the oracle at
the ends of its chunks (256 k), stages and row tiles, both layouts; nothing past the ends may be used."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import q4f16
from relax_b200 import _lib, ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [2, 3, 4, 5, 8])
@pytest.mark.parametrize("N,K", [(1, 32), (16, 96), (17, 224), (33, 288), (2400, 480), (640, 2016), (257, 2080), (8640, 3200), (100, 4128),
                                 (2380, 4352), (48, 6176), (96, 8160)])
def test_ragged_rows(cuda_lib, M, N, K):
    rng = np.random.default_rng(M + N + K)
    wq, s = synth.make_weights(N, K, rng)
    w = q4f16.dequantize(wq, s).astype(np.float64)
    x = rng.standard_normal((M, K)).astype(np.float16)
    paired = (M + N) % 2 == 1
    # guard values behind every operand: NaN scales and activations, all-ones words
    fx, fs = np.full(M * K + 512, np.nan, np.float16), np.full(s.size + 513, np.nan, np.float16)
    fw = np.full(wq.size + 256, 0xffffffff, np.uint32)
    off = int(K % 256 == 0)                                 # scales off 16 bytes where K alone is not ragged
    fx[:M * K], fs[off:off + s.size], fw[:wq.size] = x.ravel(), s.ravel(), wq.ravel()
    tx, ts, tw = (torch.from_numpy(a).cuda() for a in (fx, fs, fw))
    twq = tw[:wq.size].view(N, K // 8)
    if paired:
        tw[:wq.size] = ops.q4f16_repack(twq.contiguous(), "paired").view(-1)
    y = torch.full((M + 1, N), float("nan"), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    before = cuda_lib.b200_launch_count()
    assert cuda_lib.b200_q4f16_matmul_layout(tx.data_ptr(), tw.data_ptr(), ts.data_ptr() + 2 * off, y.data_ptr(), M, N, K, int(paired), 0) == 0, _lib.last_error()
    torch.cuda.synchronize()
    assert cuda_lib.b200_launch_count() == before + 1 and cuda_lib.b200_device_error_flags() == 0
    got, xf = y.cpu().numpy()[:M].astype(np.float64), x.astype(np.float64)
    ref = xf @ w.T
    # the bound of the parity tests: fp32 sums and one fp16 rounding
    assert (np.abs(got - ref) <= 2.0 ** -10 * np.abs(ref) + 8e-6 * (np.abs(xf) @ np.abs(w).T)).all(), np.abs(got - ref).max()
    assert bool(torch.isnan(y[M]).all())


# (Of the small sizes above those of a K below 2048 go to the streaming kernel, large products of five and eight rows to the
# weight-stationary one: the same holds for them.)
@pytest.mark.parametrize("M,N,K", [
    # K within one stage, many tiles a CTA (smaller products of so short a K are the streaming kernel's)
    (4, 12289, 1056), (3, 13985, 1248), (4, 8001, 1568), (3, 9440, 1824), (4, 6353, 2016),
    # the ends of the dispatch's ranges: on the other side are the weight-stationary and the streaming kernel
    (4, 14000, 1056), (4, 13999, 1056), (3, 2384, 8224), (3, 2368, 8224), (2, 4752, 2592), (2, 4736, 2592), (3, 2384, 2080), (3, 3552, 2080)])
def test_short_k_and_dispatch(cuda_lib, M, N, K):
    test_ragged_rows(cuda_lib, M, N, K)
