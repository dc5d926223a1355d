"""The native way from torch tensors to the C ABI: takes plain tensors, leaves everything else to the general path."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from relax_b200 import _lib, ops, synth


def _native():
    native = ops._torch_call()
    assert native, "the extension has been built"
    return native


def test_cpu_tensors_and_wrong_calls_are_left_alone():
    native = _native()
    x = torch.zeros(1, 32, dtype=torch.float16)
    assert native.matmul(x, x, x, x, -1) is False and native.dequantize(x, x, x) is False
    assert native.matmul(1, None, "x", x, -1) is False
    with pytest.raises(TypeError):
        native.matmul(x, x)
    with pytest.raises(TypeError):
        native.matmul(x, x, x, x, None)


@pytest.mark.gpu
def test_plain_tensors_are_taken_and_others_are_not(cuda_lib):
    native = _native()
    x, wq, s = (torch.from_numpy(a).cuda() for a in synth.make_case(3, 96, 256, seed=4))
    out, ref = (torch.full((3, 96), float("nan"), dtype=torch.float16, device="cuda") for _ in "12")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        stream.wait_stream(torch.cuda.default_stream())
        assert native.matmul(x, wq, s, out, -1) is True
        assert cuda_lib.b200_get_stream() == stream.cuda_stream
        assert ops._matmul_by_pointer(cuda_lib, x, wq, s, ref, None)
    torch.cuda.synchronize()
    assert (out.view(torch.int16) == ref.view(torch.int16)).all() and torch.isfinite(out).all()
    paired = ops.q4f16_repack(wq, "paired")
    assert native.matmul(x, paired, s, out, 1) is True
    torch.cuda.synchronize()
    assert (out.view(torch.int16) == ref.view(torch.int16)).all()
    w = torch.empty((96, 256), dtype=torch.float16, device="cuda")
    assert native.dequantize(wq, s, w) is True

    class Sub(torch.Tensor):
        pass

    wide = torch.zeros((3, 512), dtype=torch.float16, device="cuda")
    flat = torch.zeros(3 * 256 + 1, dtype=torch.float16, device="cuda")
    before = cuda_lib.b200_launch_count()
    for bad in ((x.as_subclass(Sub), wq, s, out), (wide[:, :256], wq, s, out), (wide[:, ::2], wq, s, out), (x.t(), wq, s, out), (x.float(), wq, s, out),
                (x, wq.view(torch.int32), s, out), (x, wq, s[:, :4], out), (x, wq, s, out[:2]), (x[0], wq, s, out), (x.cpu(), wq, s, out),
                (flat[1:].view(3, 256), wq, s, out)):                # (the last one off 16 bytes: the library refuses it)
        assert native.matmul(*bad, -1) is False
    assert native.matmul(x, wq, s, out, 7) is False and native.dequantize(wq, s, w[:, :128]) is False
    assert torch.vmap(lambda v: torch.as_tensor(native.matmul(v, wq, s, out, -1)) + 0 * v.sum())(x.unsqueeze(0)).item() == 0
    with torch.overrides.TorchFunctionMode():
        assert native.matmul(x, wq, s, out, -1) is False
    assert cuda_lib.b200_launch_count() == before
    # what the general path says about them has not changed
    with pytest.raises(_lib.B200Error):
        ops.q4f16_matmul(wide[:, :256], wq, s)
    assert np.isfinite(ops.q4f16_matmul(x, wq, s).float().cpu().numpy()).all()


@pytest.mark.gpu
@pytest.mark.parametrize("layout", [-2, -3, -256, 2, 7, -2 ** 40])
def test_numbers_that_are_no_layout_are_refused(cuda_lib, layout):
    x, wq, s = (torch.from_numpy(a).cuda() for a in synth.make_case(2, 64, 256, seed=9))
    out = torch.full((2, 64), float("nan"), dtype=torch.float16, device="cuda")
    before = cuda_lib.b200_launch_count()
    assert _native().matmul(x, wq, s, out, layout) is False
    assert cuda_lib.b200_launch_count() == before and torch.isnan(out).all()
    if -2 ** 31 <= layout:                                  # (the general path hands the number on as 32 bits)
        with pytest.raises(_lib.B200Error):
            ops.q4f16_matmul(x, wq, s, layout=layout)
        assert cuda_lib.b200_launch_count() == before
