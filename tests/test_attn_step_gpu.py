"""The one-launch decode attention at the sizes where its split can go wrong: every cluster size and CTA width, contexts around
the 16-token unit, caches that are only 8-byte aligned, early loads."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import decoder as odec
from relax_b200 import _lib

pytestmark = pytest.mark.gpu
F16 = np.float16
D = 128


def _dev(a, offset):
    """`a` on the GPU, its first element `offset` fp16 values behind a 16-byte boundary."""
    flat = torch.empty((a.size + offset,), dtype=torch.float16, device="cuda")
    out = flat[offset:].view(a.shape)
    out.copy_(torch.from_numpy(a))
    return out


# (B, heads) by the warps that a pair gets: 64, 32, 16, 8, 4 (one wave), 8 (between one and two waves), 4 (more than two)
SPLITS = [(1, 4), (2, 20), (5, 16), (5, 32), (10, 30), (21, 32), (40, 30)]


@pytest.mark.parametrize("B,nh", SPLITS)
@pytest.mark.parametrize("ctx", [1, 2, 16, 17, 18, 33, 130, 515])
def test_step_attention_against_the_oracle(cuda_lib, B, nh, ctx):
    max_ctx = 1040 if B * nh < 200 else 528
    offset = 4 if ctx in (17, 130) else 0                # 8-byte aligned only
    flags = 3 if ctx in (2, 33, 515) else 0              # (nothing that they may read early is written by the launch in front)
    pos = ctx - 1
    rng = np.random.default_rng(ctx * 7 + B)
    kc = np.full((B, max_ctx, nh, D), np.nan, F16)       # nothing above the position may be used
    vc = np.full((B, max_ctx, nh, D), np.nan, F16)
    kc[:, :pos] = rng.standard_normal((B, pos, nh, D)).astype(F16)
    vc[:, :pos] = rng.standard_normal((B, pos, nh, D)).astype(F16)
    qkv = rng.standard_normal((B, 3 * nh * D)).astype(F16)
    cos, sin = odec.rope_tables(max_ctx, D)
    tk, tv, tq = _dev(kc, offset), _dev(vc, offset), _dev(qkv, offset)
    tcos, tsin = torch.from_numpy(np.ascontiguousarray(cos)).cuda(), torch.from_numpy(np.ascontiguousarray(sin)).cuda()
    tpos = torch.tensor([pos], dtype=torch.int32, device="cuda")
    out, again = (torch.full((B, nh * D), float("nan"), dtype=torch.float16, device="cuda") for _ in "12")
    torch.cuda.synchronize()
    assert cuda_lib.b200_attn_decode_step(tq.data_ptr(), tcos.data_ptr(), tsin.data_ptr(), tpos.data_ptr(), tk.data_ptr(), tv.data_ptr(),
                                          out.data_ptr(), B, nh, max_ctx, flags, 0) == 0, _lib.last_error()
    torch.cuda.synchronize()
    # the appended entries; the others are untouched
    k = odec.rope(qkv[:, nh * D:2 * nh * D].reshape(B, nh, D), cos[pos], sin[pos])
    got_k = tk.cpu().numpy()
    # (the rotation is two products and a sum in fp32: the compiler's fusing moves it by an fp16 step at most)
    assert np.abs(got_k[:, pos].astype(np.float32) - k.astype(np.float32)).max() <= 2.0 ** -10 * 8
    assert (tv.cpu().numpy()[:, pos].view(np.uint16) == qkv[:, 2 * nh * D:].reshape(B, nh, D).view(np.uint16)).all()
    assert (got_k[:, :pos].view(np.uint16) == kc[:, :pos].view(np.uint16)).all() and np.isnan(got_k[:, ctx:]).all()
    # the result: the bound of the other attention tests
    q = odec.rope(qkv[:, :nh * D].reshape(B, nh, D), cos[pos], sin[pos])
    rows = sorted({0, B // 2, B - 1})
    kc[:, pos], vc[:, pos] = got_k[:, pos], qkv[:, 2 * nh * D:].reshape(B, nh, D)
    ref = odec.attention_decode(q[rows], kc[rows], vc[rows], ctx).astype(np.float64)
    got = out.cpu().numpy()[rows].astype(np.float64)
    assert (np.abs(got - ref) <= 2e-3 + 4e-3 * np.abs(ref)).all(), np.abs(got - ref).max()
    # the form without the rotation, on the rotated q and the cache as it now stands
    tq2 = _dev(np.ascontiguousarray(q.astype(F16)), offset)
    scratch = torch.empty(4, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert cuda_lib.b200_attn_decode(tq2.data_ptr(), tk.data_ptr(), tv.data_ptr(), tpos.data_ptr(), again.data_ptr(), scratch.data_ptr(),
                                     B, nh, max_ctx, flags & 1, 0) == 0, _lib.last_error()
    torch.cuda.synchronize()
    got = again.cpu().numpy()[rows].astype(np.float64)
    assert (np.abs(got - ref) <= 2e-3 + 4e-3 * np.abs(ref)).all(), np.abs(got - ref).max()


# (B, heads, cache) by the warps: 8 (four would leave a third wave nearly empty); 5 from the first to the last pair (one wave); 4 (one wave);
# 2 x 5 from the first to the last pair
@pytest.mark.parametrize("B,nh,max_ctx", [(41, 29, 1296), (27, 11, 528), (37, 12, 80), (18, 28, 528), (593, 1, 656), (37, 18, 656)])
@pytest.mark.parametrize("ctx", [1, 17, 81, 515])
def test_splits_at_the_ends_of_a_wave(cuda_lib, B, nh, max_ctx, ctx):
    ctx = min(ctx, max_ctx)
    pos = ctx - 1
    rng = np.random.default_rng(ctx)
    kc, vc = (np.full((B, max_ctx, nh, D), np.nan, F16) for _ in "kv")
    kc[:, :pos], vc[:, :pos] = (rng.standard_normal((B, pos, nh, D)).astype(F16) for _ in "kv")
    qkv = rng.standard_normal((B, 3 * nh * D)).astype(F16)
    cos, sin = odec.rope_tables(max_ctx, D)
    tk, tv, tq = (_dev(a, 0) for a in (kc, vc, qkv))
    tcos, tsin = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (cos, sin))
    tpos = torch.tensor([pos], dtype=torch.int32, device="cuda")
    out = torch.full((B, nh * D), float("nan"), dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    assert cuda_lib.b200_attn_decode_step(tq.data_ptr(), tcos.data_ptr(), tsin.data_ptr(), tpos.data_ptr(), tk.data_ptr(), tv.data_ptr(),
                                          out.data_ptr(), B, nh, max_ctx, 3, 0) == 0, _lib.last_error()
    torch.cuda.synchronize()
    rows = [0, B // 2, B - 1]
    q = odec.rope(qkv[:, :nh * D].reshape(B, nh, D), cos[pos], sin[pos])
    kc[:, pos], vc[:, pos] = tk.cpu().numpy()[:, pos], qkv[:, 2 * nh * D:].reshape(B, nh, D)
    ref = odec.attention_decode(q[rows], kc[rows], vc[rows], ctx).astype(np.float64)
    got = out.cpu().numpy()[rows].astype(np.float64)
    assert (np.abs(got - ref) <= 2e-3 + 4e-3 * np.abs(ref)).all(), np.abs(got - ref).max()


def test_step_attention_refuses(cuda_lib):
    t = torch.zeros(4096, dtype=torch.float16, device="cuda")
    p = t.data_ptr()

    def call(qkv=p, cos=p, kc=p, B=1, nh=1, ctx=4, flags=0):
        return cuda_lib.b200_attn_decode_step(qkv, cos, p, p, kc, p, p, B, nh, ctx, flags, 0)

    assert call(flags=4) == _lib.EINVAL and call(qkv=p + 4) == _lib.EINVAL and call(cos=p + 8) == _lib.EINVAL
    assert call(kc=None) == _lib.EINVAL and call(B=0) == _lib.EINVAL and call(nh=70000) == _lib.EINVAL
