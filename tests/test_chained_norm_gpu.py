"""The residual stream with its statistics: the matmul that adds to it and the matmuls and the output projection that normalise it
on the way in, against the oracle; every form of the skinny kernel and the ends of its ranges."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import decoder as odec
from oracle import q4f16
from relax_b200 import _lib, decoder, synth

pytestmark = pytest.mark.gpu
EPS = 1e-5


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _close(got, x, w, extra=0.0):
    """The matmul bound of the parity tests with the fast form's term (the weights unrounded): fp32 sums and one fp16 rounding."""
    xf, wf = x.astype(np.float64), w.astype(np.float64)
    ref = xf @ wf.T
    noise = 12 * 2.0 ** -11 / 3 ** 0.5 * np.sqrt((xf * xf) @ (wf * wf).T) if len(x) == 1 else 0.0
    bound = 2.0 ** -10 * np.abs(ref) + 8e-6 * (np.abs(xf) @ np.abs(wf).T) + noise + extra
    assert (np.abs(got.astype(np.float64) - ref) <= bound).all(), np.abs(got - ref).max()


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("N,K", [(16, 256), (2048, 2048), (272, 2560), (256, 6144), (4096, 4096), (512, 9216)])
def test_add_and_norm(cuda_lib, M, N, K):
    rng = np.random.default_rng(M * 1000 + N + K)
    wq, s = synth.make_weights(N, K, rng)
    w = q4f16.dequantize(wq, s)
    twq, ts = _t(wq), _t(s)
    x = rng.standard_normal((M, K)).astype(np.float16)
    y = (4 * rng.standard_normal((M, N))).astype(np.float16)
    tx, ty, stats = _t(x), _t(y), torch.full((M, N // 16), float("nan"), dtype=torch.float32, device="cuda")
    plain = torch.empty((M, N), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    assert cuda_lib.b200_q4f16_gemv(tx.data_ptr(), twq.data_ptr(), ts.data_ptr(), plain.data_ptr(), M, N, K, 0) == 0
    assert cuda_lib.b200_q4f16_gemv_add(tx.data_ptr(), twq.data_ptr(), ts.data_ptr(), ty.data_ptr(), stats.data_ptr(), M, N, K, 0, 0) == 0, _lib.last_error()
    torch.cuda.synchronize()
    # the same kernel's product, rounded, then the sum, rounded: bit for bit
    want = (y.astype(np.float32) + plain.cpu().numpy().astype(np.float32)).astype(np.float16)
    got = ty.cpu().numpy()
    assert (got.view(np.uint16) == want.view(np.uint16)).all()
    squares = (got.astype(np.float64) ** 2).reshape(M, N // 16, 16).sum(axis=2)
    np.testing.assert_allclose(stats.cpu().numpy(), squares, rtol=3e-6)           # sixteen fp32 terms
    # SwiGLU on the way in
    gu = rng.standard_normal((M, 2 * K)).astype(np.float16)
    tg, ty2 = _t(gu), _t(y)
    torch.cuda.synchronize()
    assert cuda_lib.b200_q4f16_gemv_swiglu(tg.data_ptr(), twq.data_ptr(), ts.data_ptr(), plain.data_ptr(), M, N, K, 0) == 0
    assert cuda_lib.b200_q4f16_gemv_add(tg.data_ptr(), twq.data_ptr(), ts.data_ptr(), ty2.data_ptr(), stats.data_ptr(), M, N, K, 1, 0) == 0
    torch.cuda.synchronize()
    want = (y.astype(np.float32) + plain.cpu().numpy().astype(np.float32)).astype(np.float16)
    assert (ty2.cpu().numpy().view(np.uint16) == want.view(np.uint16)).all()
    # the norm on the way into a matmul
    norm = (1 + 0.1 * rng.standard_normal(K)).astype(np.float16)
    tn, xstats = _t(norm), _t((x.astype(np.float64) ** 2).reshape(M, K // 16, 16).sum(axis=2).astype(np.float32))
    out = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    rc = cuda_lib.b200_q4f16_gemv_norm(tx.data_ptr(), xstats.data_ptr(), tn.data_ptr(), EPS, twq.data_ptr(), ts.data_ptr(), out.data_ptr(), M, N, K, 0)
    torch.cuda.synchronize()
    if rc == _lib.ENOTREADY:
        assert M > 4 and K >= 8192          # x does not fit beside a stage
        return
    assert rc == 0, _lib.last_error()
    h = odec.rmsnorm(x, norm, EPS)
    # the normalised value may fall on the other side of an fp16 rounding: half an ulp of x in a few terms
    slack = 2.0 ** -10 * np.sqrt((h.astype(np.float64) ** 2) @ (w.astype(np.float64) ** 2).T)
    _close(out.cpu().numpy(), h, w, slack)


@pytest.mark.parametrize("M,I,K", [(1, 8, 256), (1, 5632, 2048), (1, 1000, 4096), (2, 688, 2048), (4, 11008, 4096), (5, 72, 2560), (8, 2752, 4096)])
def test_norm_gate_up(cuda_lib, M, I, K):
    rng = np.random.default_rng(M * 100 + I)
    wq, s = synth.make_weights(2 * I, K, rng)
    x = rng.standard_normal((M, K)).astype(np.float16)
    norm = (1 + 0.1 * rng.standard_normal(K)).astype(np.float16)
    xstats = _t((x.astype(np.float64) ** 2).reshape(M, K // 16, 16).sum(axis=2).astype(np.float32))
    tx, tn, twq, ts = _t(x), _t(norm), _t(wq), _t(s)
    h = torch.empty_like(tx)
    a, b = (torch.full((M, I), float("nan"), dtype=torch.float16, device="cuda") for _ in "ab")
    torch.cuda.synchronize()
    assert cuda_lib.b200_q4f16_gemv_norm_gate_up(tx.data_ptr(), xstats.data_ptr(), tn.data_ptr(), EPS, twq.data_ptr(), ts.data_ptr(),
                                                 a.data_ptr(), M, I, K, 0) == 0, _lib.last_error()
    assert cuda_lib.b200_rmsnorm(tx.data_ptr(), None, tn.data_ptr(), h.data_ptr(), M, K, EPS, 0) == 0
    assert cuda_lib.b200_q4f16_gemv_gate_up(h.data_ptr(), None, None, None, 0.0, twq.data_ptr(), ts.data_ptr(), b.data_ptr(), M, I, K, 0) == 0
    torch.cuda.synchronize()
    # the separate norm: the statistics differ in the order of their sum, which moves h by an fp16 step in a few places
    a, b = a.float(), b.float()
    assert float((a - b).norm() / b.norm()) < 1e-3


@pytest.mark.parametrize("B,H,V", [(1, 256, 33), (3, 2048, 1000), (8, 4096, 515), (5, 5120, 64)])
def test_lm_head_norm(cuda_lib, B, H, V):
    rng = np.random.default_rng(B + H)
    x = rng.standard_normal((B, H)).astype(np.float16)
    w = (0.02 * rng.standard_normal((V, H))).astype(np.float16)
    norm = (1 + 0.1 * rng.standard_normal(H)).astype(np.float16)
    xstats = _t((x.astype(np.float64) ** 2).reshape(B, H // 16, 16).sum(axis=2).astype(np.float32))
    tx, tw, tn = _t(x), _t(w), _t(norm)
    logits = torch.empty((B, V), dtype=torch.float16, device="cuda")
    hout = torch.empty_like(tx)
    toks = torch.full((B,), -1, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(cuda_lib.b200_lm_head_scratch_bytes() // 4, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert cuda_lib.b200_lm_head_norm(tx.data_ptr(), xstats.data_ptr(), tn.data_ptr(), EPS, hout.data_ptr(), tw.data_ptr(), logits.data_ptr(), toks.data_ptr(),
                                      scratch.data_ptr(), B, V, H, 0, 0) == 0, _lib.last_error()
    torch.cuda.synchronize()
    h = odec.rmsnorm(x, norm, EPS)
    np.testing.assert_allclose(hout.cpu().numpy().astype(np.float32), h.astype(np.float32), rtol=2.0 ** -10, atol=1e-7)
    got = logits.cpu().numpy()
    slack = 2.0 ** -10 * np.sqrt((h.astype(np.float64) ** 2) @ (w.astype(np.float64) ** 2).T)
    xf, wf = h.astype(np.float64), w.astype(np.float64)
    assert (np.abs(got - xf @ wf.T) <= 2.0 ** -10 * np.abs(xf @ wf.T) + 8e-6 * (np.abs(xf) @ np.abs(wf).T) + slack).all()
    assert (toks.cpu().numpy() == got.astype(np.float32).argmax(axis=1)).all()


def test_embed_rows_stats(cuda_lib):
    rng = np.random.default_rng(5)
    table = rng.standard_normal((40, 272)).astype(np.float16)
    ids = torch.tensor([0, 39, 7], dtype=torch.int32, device="cuda")
    tt, out, stats = _t(table), torch.empty((3, 272), dtype=torch.float16, device="cuda"), torch.full((3, 17), float("nan"), device="cuda")
    torch.cuda.synchronize()
    assert cuda_lib.b200_embed_rows_stats(tt.data_ptr(), ids.data_ptr(), out.data_ptr(), stats.data_ptr(), 3, 272, 40, 0) == 0
    torch.cuda.synchronize()
    assert (out.cpu().numpy() == table[[0, 39, 7]]).all()
    np.testing.assert_allclose(stats.sum(dim=1).cpu().numpy(), (table[[0, 39, 7]].astype(np.float64) ** 2).sum(axis=1), rtol=1e-5)


@pytest.mark.parametrize("B,V", [(1, 1), (3, 7), (17, 8), (2, 1000), (64, 32000), (5, 8191), (20, 8200)])
def test_argmax_rows(cuda_lib, B, V):
    rng = np.random.default_rng(V)
    a = rng.integers(-50, 50, (B, V)).astype(np.float16)               # many ties
    a[0, V // 2:] = np.inf
    if B > 2:
        a[1, V - 1] = np.nan
        a[2] = -np.inf
    t, toks = _t(a), torch.full((B,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert cuda_lib.b200_argmax_rows(t.data_ptr(), toks.data_ptr(), B, V, 0) == 0, _lib.last_error()
    torch.cuda.synchronize()
    assert (toks.cpu().numpy() == a.argmax(axis=1)).all()              # (numpy: the first of equal ones, the first NaN)


def test_refusals(cuda_lib):
    t = torch.zeros(1 << 16, dtype=torch.float16, device="cuda")
    p, q = t.data_ptr(), t.data_ptr() + 65536
    L = cuda_lib
    assert L.b200_q4f16_gemv_add(p, p, p, q, p, 9, 64, 256, 0, 0) == _lib.EINVAL
    assert L.b200_q4f16_gemv_add(p, p, p, q, p, 1, 24, 256, 0, 0) == _lib.EINVAL
    assert L.b200_q4f16_gemv_add(p, p, p, p, p, 1, 64, 256, 0, 0) == _lib.EINVAL          # y is x
    assert L.b200_q4f16_gemv_add(p, p, p + 2, q, p, 1, 64, 256, 0, 0) == _lib.EINVAL
    assert L.b200_q4f16_gemv_norm(p, None, p, EPS, p, p, q, 1, 64, 256, 0) == _lib.EINVAL
    assert L.b200_q4f16_gemv_norm(p, p, p, EPS, p, p, q, 9, 64, 256, 0) == _lib.EINVAL
    assert L.b200_q4f16_gemv_norm(p, p, p, EPS, p, p, q, 1, 64, 288, 0) == _lib.EINVAL
    assert L.b200_q4f16_gemv_norm_gate_up(p, p, p, EPS, p, p, q, 1, 12, 256, 0) == _lib.EINVAL
    assert L.b200_lm_head_norm(p, p, p, EPS, None, p, q, None, None, 9, 64, 256, 0, 0) == _lib.EINVAL
    assert L.b200_argmax_rows(p, None, 1, 8, 0) == _lib.EINVAL and L.b200_argmax_rows(p, p, 1, 0, 0) == _lib.EINVAL
    assert L.b200_embed_rows_stats(p, p, q, None, 1, 64, 4, 0) == _lib.EINVAL
    assert L.b200_q4f16_gemv_add_applies(p, 9, 64, 256) == 0 and L.b200_q4f16_gemv_add_applies(p, 1, 64, 288) == 0
    assert L.b200_q4f16_gemv_add_applies(p, 8, 4096, 8192) == 0 and L.b200_q4f16_gemv_add_applies(p, 8, 4096, 4096) == 1


@pytest.mark.parametrize("variant", [0, 1, 2])
def test_the_question_about_the_fit_is_answered_as_the_launch_answers(cuda_lib, variant):
    K = [256, 2304, 2560, 4096, 4352, 6144, 7936, 8192, 8448, 8704, 9216, 12288, 16384]
    t = torch.zeros(64 * 16384 // 8, dtype=torch.int32, device="cuda")
    h = torch.zeros(64 * 16384, dtype=torch.float16, device="cuda")
    y, stats = torch.empty((8, 64), dtype=torch.float16, device="cuda"), torch.zeros(8 * 1024, dtype=torch.float32, device="cuda")
    _lib.set_option("gemv.variant", variant)
    try:
        for M in range(1, 9):
            for k in K:
                rc = cuda_lib.b200_q4f16_gemv_norm(h.data_ptr(), stats.data_ptr(), h.data_ptr(), 1e-5, t.data_ptr(), h.data_ptr(), y.data_ptr(), M, 64, k, 0)
                fits = rc != _lib.ENOTREADY
                assert rc == 0 or not fits
                ours = variant == 2 or (variant == 0 and not (M >= 5 and k >= 8192))          # (the rest: weight-stationary, streaming)
                assert cuda_lib.b200_q4f16_gemv_norm_applies(h.data_ptr(), M, 64, k) == int(fits and ours), (M, k)
    finally:
        _lib.set_option("gemv.variant", 0)
    torch.cuda.synchronize()
    assert cuda_lib.b200_device_error_flags() == 0


@pytest.mark.parametrize("B,option", [(5, ("gemv.variant", 2)), (8, ("gemv.variant", 2)), (8, ("gemm.ws_max_m", 4))])
def test_step_of_a_model_too_wide_for_the_normalising_forms(cuda_lib, B, option):
    """Against the engine that has a launch for every norm: the appended keys and values have its bits."""
    cfg = decoder.DecoderConfig(hidden=9216, heads=72, inter=1024, layers=2, vocab=320)
    layers = []
    for i in range(cfg.layers):
        layer = decoder.synth_layer_torch(cfg, 31 + i, "cuda")
        layer |= {name: (layer[name][0], layer[name][1] * 0.1) for name in ("qkv", "o", "gu", "down")}
        layers.append(layer | {"inter_local": cfg.inter})
    embed = torch.randn((cfg.vocab, cfg.hidden), dtype=torch.float16, device="cuda") * 0.1
    norm = torch.ones(cfg.hidden, dtype=torch.float16, device="cuda")
    before = _lib.get_option(option[0])
    out = []
    try:
        _lib.set_option(*option)
        for kw in ({}, dict(fused=False)):
            eng = decoder.DecodeEngine(cfg, layers, embed, norm, embed, B, 16, "cuda", **kw)
            assert eng.chained == (not kw)
            for _ in range(2):
                eng.tokens.copy_(torch.arange(B, dtype=torch.int32))
                launches = cuda_lib.b200_launch_count()
                eng.step()
                torch.cuda.synchronize()
                assert cuda_lib.b200_launch_count() - launches == eng.kernels_per_step()
            out.append(eng)
    finally:
        _lib.set_option(option[0], before)
    a, b = out
    for i in range(cfg.layers):
        assert torch.equal(a.kc[i][:, :2], b.kc[i][:, :2]) and torch.equal(a.vc[i][:, :2], b.vc[i][:, :2])
    assert float(a.kc[-1][:, :2].abs().max()) > 0
    # (the statistics of the last norm are added up in another order)
    scale = float(b.logits.abs().max())
    assert torch.isfinite(a.logits).all() and float((a.logits - b.logits).abs().max()) <= 4e-3 * scale
    assert cuda_lib.b200_device_error_flags() == 0
