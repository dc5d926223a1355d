"""CPU tests of which entry points a decode step asks for: the engine on the host, with a library that only writes down the calls
(what it is asked about sizes and options, the real one answers)."""
import pytest

torch = pytest.importorskip("torch")

from relax_b200 import _lib, decoder


class Recorder:
    """The library with every launch replaced by a note of it; `refuse`: entry points that answer B200_ENOTREADY."""

    def __init__(self, refuse=()):
        self.real, self.calls, self.refuse = _lib.lib(), [], refuse

    def __getattr__(self, name):
        fn = getattr(self.real, name)
        if name.endswith(("_applies", "_bytes")):
            return fn

        def note(*args):
            self.calls.append((name, args))
            return _lib.ENOTREADY if name in self.refuse else _lib.OK

        return note

    def names(self):
        return [name.removeprefix("b200_") for name, _ in self.calls]


def engine(hidden, batch, inter=768, layers=2, **kw):
    cfg = decoder.DecoderConfig(hidden=hidden, heads=hidden // 128, inter=inter, layers=layers, vocab=64)
    # (nothing reads the weights here: sixteen aligned bytes of each will do)
    w = dict.fromkeys(("qkv", "o", "gu", "down"), (torch.zeros(8, dtype=torch.int32), torch.zeros(8, dtype=torch.float16)))
    w |= {"norm1": torch.zeros(8, dtype=torch.float16), "norm2": torch.zeros(8, dtype=torch.float16), "inter_local": inter}
    eng = decoder.DecodeEngine(cfg, [dict(w) for _ in range(layers)], torch.zeros((64, 8), dtype=torch.float16),
                               torch.zeros(8, dtype=torch.float16), torch.zeros((64, 8), dtype=torch.float16), batch, 16, "cpu", **kw)
    eng.L = Recorder()
    return eng


@pytest.fixture
def option():
    before = {name: _lib.get_option(name) for name in ("gemv.variant", "gemm.ws_max_m")}
    yield _lib.set_option
    for name, value in before.items():
        _lib.set_option(name, value)


def layers(eng):
    """The calls of all layers and what is left to add behind the last."""
    delta = None
    for i in range(len(eng.layers)):
        delta = eng._chained_layer(i, delta, 0)
    return eng.L.names(), delta


CHAINED = ["q4f16_gemv_norm", "attn_decode_step", "q4f16_gemv_add", "q4f16_gemv_norm_gate_up", "q4f16_gemv_add"]
APART = ["rmsnorm_early_release", "q4f16_matmul", "attn_decode_step", "q4f16_matmul", "rmsnorm_early_release", "q4f16_matmul",
         "silu_mul_early_release", "q4f16_matmul"]


@pytest.mark.parametrize("batch", [1, 2, 5, 8])
def test_matmuls_of_a_step_follow_the_option(option, batch):
    eng = engine(512, batch, rope_epilogue=False)
    assert eng.chained
    assert layers(eng) == (2 * CHAINED, None)
    option("gemv.variant", 1)                               # the register-streaming kernel: no prologue, no epilogue
    eng = engine(512, batch)
    names, delta = layers(eng)
    assert names == 2 * APART and delta is eng.down
    assert eng.kernels_per_step() == 1 + len(names) + 1 + 1 + 1


@pytest.mark.parametrize("batch", [5, 8])
@pytest.mark.parametrize("name,value", [("gemv.variant", 2), ("gemm.ws_max_m", 4)])
def test_a_row_that_does_not_fit_is_normalised_by_itself(option, batch, name, value):
    """5..8 rows of a wide model stay in the skinny kernel only where an option asks for it; all of x beside a stage ends between
    8192 and 9216 values a row.  The forms without a norm cut K and go on."""
    option(name, value)
    scales = 1 << 20                                        # (only its alignment is looked at)
    applies = [_lib.lib().b200_q4f16_gemv_norm_applies(scales, batch, 3 * k, k) for k in (256, 4096, 8192, 9216, 16384)]
    assert applies == [1, 1, 1, 0, 0]
    assert _lib.lib().b200_q4f16_gemv_add_applies(scales, batch, 9216, 9216) == 1
    eng = engine(9216, batch)
    assert eng.chained
    names, delta = layers(eng)
    assert names == 2 * ["rmsnorm_early_release", "q4f16_matmul", "attn_decode_step", "q4f16_gemv_add", "rmsnorm_early_release",
                         "q4f16_gemv_gate_up", "q4f16_gemv_add"] and delta is None
    assert eng.kernels_per_step() == 1 + len(names) + 1 + 1


def test_up_to_four_rows_of_every_width_fit():
    for batch in (1, 2, 3, 4):
        for hidden in range(256, 16384 + 1, 256):
            assert _lib.lib().b200_q4f16_gemv_norm_applies(1 << 20, batch, 3 * hidden, hidden) == 1


@pytest.mark.parametrize("batch,kw", [(1, dict(fused=True)), (1, dict(fused=False)), (3, dict(fused=True)), (3, dict(fused=False)), (12, {}), (1, {}), (3, {})])
def test_only_a_step_promises_the_attention_a_finished_cache(monkeypatch, batch, kw):
    """A layer by itself stands behind whatever the caller launched, which may have written the position and the caches."""
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: type("S", (), {"cuda_stream": 0}))
    eng = engine(2560, batch, **kw)

    def flags():
        out = [args[-2] & _lib.ATTN_EARLY_KV_LOADS for name, args in eng.L.calls if name.startswith("b200_attn_decode")]
        eng.L.calls.clear()
        return out

    eng.layer_step(1, None, 0)
    assert flags() == [0]
    eng.step()
    assert flags() == [_lib.ATTN_EARLY_KV_LOADS] * len(eng.layers)
