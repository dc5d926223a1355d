"""SwiGLU in the epilogue of the weight-stationary kernel against the matmul and the SwiGLU kernel as two launches: ends of the row
tiles (64 gate rows and their up rows) and of the batch columns, every number of K slices, a ragged K, both layouts."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from relax_b200 import _lib, ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,I,K", [(1, 1, 32), (9, 64, 256), (9, 63, 256), (16, 65, 512), (17, 200, 1024), (33, 688, 2048), (64, 1408, 1056),
                                   (64, 96, 4096), (100, 130, 4128), (128, 11008, 512), (128, 72, 8192), (12, 6912, 2560)])
@pytest.mark.parametrize("ksplit", [0, 1, 2, 4, 8])
def test_gate_up_against_two_launches(cuda_lib, M, I, K, ksplit):
    paired = ksplit in (2, 8)
    rng = np.random.default_rng(M + I + K)
    wq, s = synth.make_weights(2 * I, K, rng)
    x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float16)).cuda()
    twq, ts = torch.from_numpy(wq).cuda(), torch.from_numpy(s * np.float16(0.2)).cuda()
    if paired:
        twq = ops.q4f16_repack(twq, "paired")
    gu = torch.empty((M, 2 * I), dtype=torch.float16, device="cuda")
    got = torch.full((M, I), float("nan"), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    try:
        _lib.set_option("gemm.ws_ksplit", ksplit)
        _lib.set_option("weights.layout", 1 if paired else 0)
        assert cuda_lib.b200_q4f16_gate_up(x.data_ptr(), twq.data_ptr(), ts.data_ptr(), got.data_ptr(), M, I, K, 0) == 0, _lib.last_error()
        torch.cuda.synchronize()
        assert cuda_lib.b200_q4f16_matmul(x.data_ptr(), twq.data_ptr(), ts.data_ptr(), gu.data_ptr(), M, 2 * I, K, 0) == 0
        torch.cuda.synchronize()
    finally:
        _lib.set_option("gemm.ws_ksplit", 0)
        _lib.set_option("weights.layout", 0)
    assert cuda_lib.b200_device_error_flags() == 0
    g, u = gu.float().chunk(2, dim=1)
    want = g / (1 + torch.exp(-g)) * u
    # The two launches may cut K differently.  That moves gate and up by fp32 sums in another order, 8e-6 of sum |x w| (about
    # 0.01 K here) as in the parity tests, and so by an fp16 step each; silu's slope is below 1.1; then the result's own rounding.
    order = 8e-6 * 0.01 * K
    tol = 2.0 ** -10 * (1.1 * (g * u).abs() + 2 * want.abs()) + order * (1.1 * u.abs() + g.abs()) + 1e-6
    assert bool(((got.float() - want).abs() <= tol).all()), float((got.float() - want).abs().max())


def test_gate_up_refuses_and_applies(cuda_lib):
    t = torch.zeros(1 << 16, dtype=torch.float16, device="cuda")
    p = t.data_ptr()
    assert cuda_lib.b200_q4f16_gate_up(p, p, p, p, 129, 8, 256, 0) == _lib.EINVAL
    assert cuda_lib.b200_q4f16_gate_up(p, p, p, p, 9, 0, 256, 0) == _lib.EINVAL
    assert cuda_lib.b200_q4f16_gate_up(p, None, p, p, 9, 8, 256, 0) == _lib.EINVAL
    assert cuda_lib.b200_q4f16_gate_up_applies(p, 9, 8, 256) == 1 and cuda_lib.b200_q4f16_gate_up_applies(p, 8, 8, 256) == 0
    assert cuda_lib.b200_q4f16_gate_up_applies(p, 129, 8, 256) == 0
    # above 96 rows with several slices, or one round of single ones that fills the SMs
    for M, I, K, one in ((96, 5632, 5120, 1), (97, 5632, 5120, 0), (128, 1024, 4096, 1), (128, 512, 512, 0), (128, 8192, 4096, 1), (128, 8192, 4352, 0),
                         (128, 11008, 1024, 0)):
        assert cuda_lib.b200_q4f16_gate_up_applies(p, M, I, K) == one, (M, I, K)
