"""Decode-step harness for a Llama-style q4f16 decoder: the callers either side of the quantised
matmul (RMSNorm, RoPE + KV cache, attention, SwiGLU) wired to the C-ABI kernels, optionally
tensor-parallel with one NCCL all-reduce after each row-parallel matmul.

torch is used for device memory, streams, CUDA graphs and the NCCL process group; every kernel of a step is
this library's for batches of up to 16 (above that the fp16 output projection is a plain library GEMM).

Layout per rank (world size t, hidden H, heads nh, head dim 128, intermediate I):

    qkv   q4  [3*H/t, H]      rows = q heads | k heads | v heads of this rank
    o     q4  [H, H/t]        row-parallel   -> all-reduce
    gu    q4  [2*I_r, H]      rows = gate | up rows of this rank's slice of I
    down  q4  [H, I_r]        row-parallel   -> all-reduce
    KV    fp16 [B, max_ctx, nh/t, 128] per layer, K and V
"""
from __future__ import annotations

import ctypes
import dataclasses

import numpy as np
import torch

from . import _lib, tp


@dataclasses.dataclass
class DecoderConfig:
    hidden: int = 4096
    heads: int = 32
    inter: int = 11008
    layers: int = 32
    vocab: int = 32000
    eps: float = 1e-5
    theta: float = 10000.0
    head_dim: int = 128

    def __post_init__(self):
        if self.hidden != self.heads * self.head_dim or self.head_dim != 128:
            raise ValueError("the attention kernels take head_dim 128 and hidden = heads * 128")


def rope_tables(max_pos: int, head_dim: int, theta: float, device):
    half = head_dim // 2
    inv = theta ** (-np.arange(half, dtype=np.float64) * 2.0 / head_dim)
    ang = np.arange(max_pos, dtype=np.float64)[:, None] * inv[None, :]
    cos = torch.from_numpy(np.cos(ang).astype(np.float32)).to(device)
    sin = torch.from_numpy(np.sin(ang).astype(np.float32)).to(device)
    return cos.contiguous(), sin.contiguous()


def synth_layer_numpy(cfg: DecoderConfig, seed: int):
    """Full (unsharded) random layer on the host: nibbles uniform 0..15, scales U(0.005, 0.02),
    norm weights ~ N(1, 0.02).  Small configurations only (tests)."""
    from . import synth

    rng = np.random.default_rng(seed)
    H, I = cfg.hidden, cfg.inter
    w = {}
    for name, (n, k) in (("qkv", (3 * H, H)), ("o", (H, H)), ("gu", (2 * I, H)), ("down", (H, I))):
        w[name] = synth.make_weights(n, k, rng)
    w["norm1"] = (1.0 + 0.02 * rng.standard_normal(H)).astype(np.float16)
    w["norm2"] = (1.0 + 0.02 * rng.standard_normal(H)).astype(np.float16)
    return w


def synth_layer_torch(cfg: DecoderConfig, seed: int, device):
    """Same distributions generated on the device (model-sized tensors)."""
    from . import synth

    H, I = cfg.hidden, cfg.inter
    w = {}
    for j, (name, (n, k)) in enumerate((("qkv", (3 * H, H)), ("o", (H, H)), ("gu", (2 * I, H)), ("down", (H, I)))):
        w[name] = synth.make_weights_torch(n, k, seed * 16 + j, device)
    gen = torch.Generator(device=device)
    gen.manual_seed(seed * 16 + 9)
    w["norm1"] = (1.0 + 0.02 * torch.randn(H, device=device, generator=gen)).to(torch.float16)
    w["norm2"] = (1.0 + 0.02 * torch.randn(H, device=device, generator=gen)).to(torch.float16)
    return w


def to_device(layer: dict, device):
    out = {}
    for k, v in layer.items():
        if isinstance(v, tuple):
            out[k] = tuple(torch.from_numpy(np.ascontiguousarray(a)).to(device) if isinstance(a, np.ndarray) else a.to(device)
                           for a in v)
        elif isinstance(v, np.ndarray):
            out[k] = torch.from_numpy(v).to(device)
        else:
            out[k] = v
    return out


class DecodeEngine:
    """Buffers and kernel sequence of one decode step for `batch` sequences.

    `layers` is a list of per-rank layer shards (see tp.shard_layer) on `device`; `embed` the fp16
    embedding table [vocab, H]; `lm_head` fp16 [vocab_local, H] (rows of this rank's vocabulary
    slice) or None to stop at the final norm; `final_norm` fp16 [H].
    """

    def __init__(self, cfg: DecoderConfig, layers, embed, final_norm, lm_head, batch: int, max_ctx: int,
                 device, rank: int = 0, world: int = 1, group=None, fused=None, peer_reduce: bool = True,
                 fused_attention=False, guard=None, verify: bool = True, layer_kernel=None, rope_epilogue: bool = True):
        self.cfg, self.batch, self.max_ctx, self.device = cfg, batch, max_ctx, torch.device(device)
        self.rank, self.world, self.group = rank, world, group
        self.layers, self.embed, self.final_norm, self.lm_head = layers, embed, final_norm, lm_head
        self.L = _lib.lib()
        H, B = cfg.hidden, batch
        self.nh_local = cfg.heads // world
        if cfg.heads % world:
            raise ValueError("heads must divide by the tensor-parallel size")
        # host-side checks of the tensor-parallel set-up: shard shapes agree across ranks before anything is
        # launched; `guard` (tp.StepGuard on a CPU-capable group) is consulted before every eager step
        self.guard = guard
        if world > 1 and verify and layers:
            tp.verify_sharding(layers, rank, world, cfg.hidden, cfg.inter, group=group)
        f16 = dict(dtype=torch.float16, device=self.device)
        hl = H // world
        il_max = max(l["inter_local"] for l in layers) if layers else cfg.inter
        # fused: RMSNorm (+ residual add) runs inside the staging of the next skinny matmul, which forms the statistics itself; needs
        # batch <= 16, the skinny kernel's range.  Only on request, and at batch 1 where the chained form does not apply: every CTA
        # of a fused kernel recomputes the statistics of all the batch's rows, and from two rows on separate norms are faster
        # (when both forms had the same kernels besides, a layer at context 2000: 80 against 88 us at batch 2, 124 against 176 at batch 8).
        self.fused = (B == 1) if fused is None else (bool(fused) and B <= 16)
        # chained: up to 8 rows, o and down add their product to the residual stream themselves and leave the sums of squares of its
        # rows behind, from which qkv, gate|up and the output projection normalise it while they stage it: no launch for the norms.
        # The default where it applies; `fused` = True or False select the two forms that form the statistics afresh.
        self.chained = fused is None and world == 1 and not layer_kernel and B <= 8 and cfg.hidden % 256 == 0
        # rotary embedding, KV append and attention are one launch; True and "rope" take the entry points whose loads all wait for
        # the qkv matmul, False the one whose first loads of older cache entries run beside it
        self.fused_attention = "rope" if fused_attention == "rope" else bool(fused_attention)
        self.x = torch.zeros((B, H), **f16)            # residual stream
        self.x2 = torch.zeros((B, H), **f16)           # its second buffer (fused path ping-pongs)
        self.h = torch.zeros((B, H), **f16)            # normalised activations
        self.qkv = torch.zeros((B, 3 * hl), **f16)
        self.q = torch.zeros((B, self.nh_local, 128), **f16)
        self.attn = torch.zeros((B, hl), **f16)
        self.o = torch.zeros((B, H), **f16)
        self.gu = torch.zeros((B, 2 * il_max), **f16)   # (where SwiGLU is a launch of its own)
        self.act = torch.zeros((B, il_max), **f16)
        self.down = torch.zeros((B, H), **f16)
        self.kc = [torch.zeros((B, max_ctx, self.nh_local, 128), **f16) for _ in layers]
        self.vc = [torch.zeros((B, max_ctx, self.nh_local, 128), **f16) for _ in layers]
        self.scratch = torch.zeros((4,), dtype=torch.float32, device=self.device)     # (the attention entry points ask for one)
        self.stats = torch.zeros((B, max(H // 16, 1)), dtype=torch.float32, device=self.device)   # chained: sums of squares of x
        self.pos = torch.zeros((1,), dtype=torch.int32, device=self.device)
        self.tokens = torch.zeros((B,), dtype=torch.int32, device=self.device)
        self.cos, self.sin = rope_tables(max_ctx, 128, cfg.theta, self.device)
        vl = lm_head.shape[0] if lm_head is not None else 0
        self.logits_local = torch.zeros((B, vl), **f16) if vl else None
        self.logits = torch.zeros((B, vl * world), **f16) if vl and world > 1 else self.logits_local
        self.gathered = torch.zeros((world, B, vl), **f16) if vl and world > 1 else None
        self.lm_scratch = torch.zeros((max(int(self.L.b200_lm_head_scratch_bytes()), 16) // 4,), dtype=torch.float32, device=self.device)
        self.graph = None
        self.launches_per_step = 0
        # batch 1: one persistent kernel per layer (b200_decode_layer) instead of five launches.  Off by default:
        # measured on B200 at the 7B shape it is slower (2.00 against 1.53 ms per token), because every stage boundary
        # inside it costs what a dependent launch costs, and its attention stage has only eight warps per SM with loads in
        # flight
        self.layer_kernel = False if layer_kernel is None else bool(layer_kernel)
        # batch 1: rotary embedding + KV append run in the epilogue of the qkv matmul (b200_q4f16_gemv_norm_rope, with fused
        # prologues b200_q4f16_gemv_rmsnorm_rope)
        self.rope_epilogue = bool(rope_epilogue) and self.fused and B == 1 and not self.fused_attention and not self.layer_kernel
        if self.layer_kernel and B != 1:
            raise ValueError("the one-kernel-per-layer path is the batch-1 path")
        # tensor parallel: the sum over ranks after o and down runs over NVLink peer memory, inside those matmul
        # kernels (b200_q4f16_gemv_allreduce) for up to 8 rows, as a kernel of this library behind the mid-batch
        # matmul above that (b200_allreduce_peer); with peer_reduce=False it is an NCCL all-reduce
        self.peer = None
        self.epoch = torch.zeros((1,), dtype=torch.int32, device=self.device)
        if world > 1 and (peer_reduce or self.layer_kernel):
            self._setup_peer_reduce()
        if self.layer_kernel:
            self._setup_layer_kernel()

    def _setup_peer_reduce(self):
        import torch.distributed._symmetric_memory as symm_mem

        B, H, nl, world = self.batch, self.cfg.hidden, len(self.layers), self.world
        ybytes = B * H * 2
        ybytes = (ybytes + 255) // 256 * 256
        fbytes = 2 * nl * world * 4
        total = 2 * ybytes + fbytes
        buf = symm_mem.empty(total, dtype=torch.uint8, device=self.device)
        buf.zero_()
        torch.cuda.synchronize(self.device)
        hdl = symm_mem.rendezvous(buf, group=self.group if self.group is not None else torch.distributed.group.WORLD)
        torch.distributed.barrier(group=self.group)
        ptrs = [int(p) for p in hdl.buffer_ptrs]
        self.peer = {
            "buf": buf, "hdl": hdl,
            "y": [[p + k * ybytes for p in ptrs] for k in range(2)],          # [kind][rank]
            "flags": [p + 2 * ybytes for p in ptrs],
            "done": torch.zeros((1,), dtype=torch.int32, device=self.device),
        }

    def _setup_layer_kernel(self):
        """Buffers and one B200DecodeLayer descriptor per layer.  The residual stream rotates through three
        buffers (a layer reads x_in, writes x_mid = x_in + delta and x_out = x_mid + o; the next layer's x_in is this
        layer's x_out and it may overwrite the two others)."""
        cfg, L = self.cfg, self.L
        H, dev = cfg.hidden, self.device
        f16 = dict(dtype=torch.float16, device=dev)
        self.xr = [self.x, self.x2, torch.zeros((1, H), **f16)]
        nbytes = int(L.b200_decode_layer_scratch_bytes(self.nh_local, self.max_ctx))
        self.layer_scratch = [torch.zeros(((nbytes + 3) // 4,), dtype=torch.int32, device=dev) for _ in self.layers]
        self.layer_desc = []
        for i, w in enumerate(self.layers):
            d = _lib.DecodeLayer()
            d.world, d.rank = self.world, self.rank
            d.hidden, d.inter_local, d.max_ctx = H, w["inter_local"], self.max_ctx
            d.heads, d.eps = cfg.heads, cfg.eps
            xin, xmid, xout = self.xr[(2 * i) % 3], self.xr[(2 * i + 1) % 3], self.xr[(2 * i + 2) % 3]
            d.x_in, d.x_mid, d.x_out = xin.data_ptr(), xmid.data_ptr(), xout.data_ptr()
            d.delta_in = self.down.data_ptr() if i > 0 else None
            d.qkv, d.attn, d.o, d.act, d.down = (self.qkv.data_ptr(), self.attn.data_ptr(), self.o.data_ptr(), self.act.data_ptr(),
                                                 self.down.data_ptr())
            d.norm1, d.norm2 = w["norm1"].data_ptr(), w["norm2"].data_ptr()
            d.cos_t, d.sin_t, d.pos = self.cos.data_ptr(), self.sin.data_ptr(), self.pos.data_ptr()
            d.k_cache, d.v_cache = self.kc[i].data_ptr(), self.vc[i].data_ptr()
            d.scratch, d.step = self.layer_scratch[i].data_ptr(), self.epoch.data_ptr()
            d.wq_qkv, d.s_qkv = w["qkv"][0].data_ptr(), w["qkv"][1].data_ptr()
            d.wq_o, d.s_o = w["o"][0].data_ptr(), w["o"][1].data_ptr()
            d.wq_gu, d.s_gu = w["gu"][0].data_ptr(), w["gu"][1].data_ptr()
            d.wq_down, d.s_down = w["down"][0].data_ptr(), w["down"][1].data_ptr()
            if self.world > 1:
                d.reduce_o = self._reduce_desc(0, i, self.o)
                d.reduce_down = self._reduce_desc(1, i, self.down)
            self.layer_desc.append(d)
        self.x_last = self.xr[(2 * len(self.layers)) % 3]     # the residual stream after the last layer

    def _reduce_desc(self, kind: int, layer: int, out):
        d = _lib.PeerReduce()
        d.world, d.rank = self.world, self.rank
        for r in range(self.world):
            d.peer_y[r] = self.peer["y"][kind][r]
            d.peer_flags[r] = self.peer["flags"][r]
        d.flag_base = (kind * len(self.layers) + layer) * self.world
        d.epoch = self.epoch.data_ptr()
        d.done_counter = self.peer["done"].data_ptr()
        d.out = out.data_ptr()
        return d

    # ------------------------------------------------------------------ kernel calls
    def _check(self, rc):
        if rc:
            raise _lib.B200Error(rc, _lib.last_error())

    def _matmul(self, x, w, y, n, k, sp):
        self._check(self.L.b200_q4f16_matmul(x.data_ptr(), w[0].data_ptr(), w[1].data_ptr(), y.data_ptr(), self.batch, n, k, sp))

    # up to this many rows the sum over ranks runs inside the skinny matmul kernel; above, the matmul (mid-batch
    # or prefill kernel) writes its partial result into the peer-mapped buffer and b200_allreduce_peer adds up
    PEER_FUSED_MAX_ROWS = 8

    def _matmul_then_peer_sum(self, kind: int, layer: int, x, w, out, n, k, sp):
        d = self._reduce_desc(kind, layer, out)
        self._check(self.L.b200_q4f16_matmul(x.data_ptr(), w[0].data_ptr(), w[1].data_ptr(), self.peer["y"][kind][self.rank],
                                             self.batch, n, k, sp))
        self._check(self.L.b200_allreduce_peer(self.batch * n, ctypes.byref(d), sp))

    def _gate_up_in_one(self, w) -> bool:
        """Whether SwiGLU runs in the epilogue of the gate|up matmul: with fused prologues, else where the library would
        take that matmul through the kernel that has the epilogue (asked anew each time: options may change)."""
        return (self.fused and not self.chained) or bool(self.L.b200_q4f16_gemv_gate_up_applies(w["gu"][1].data_ptr(), self.batch, w["inter_local"], self.cfg.hidden))

    def _gate_up_wide(self, w) -> bool:
        """Whether the gate|up matmul goes to the kernel for more rows, which has SwiGLU in its epilogue too."""
        return bool(self.L.b200_q4f16_gate_up_applies(w["gu"][1].data_ptr(), self.batch, w["inter_local"], self.cfg.hidden))

    def _in_skinny(self, w, n, k) -> bool:
        """Whether the chained forms, which the skinny kernel has, are the ones for this matmul (asked anew each time, as below)."""
        return bool(self.L.b200_q4f16_gemv_add_applies(w[1].data_ptr(), self.batch, n, k))

    def _norm_in_skinny(self, w, n, k) -> bool:
        """The same for a matmul that normalises the residual stream on its way in, all of which has to fit beside it."""
        return bool(self.L.b200_q4f16_gemv_norm_applies(w[1].data_ptr(), self.batch, n, k))

    def _add(self, x, w, out, k, sp, swiglu=False):
        """The residual stream += x . W^T, statistics included: None.  Or, where the chained form does not apply, `out` with the
        product still to be added.  `swiglu`: x is gate | up, SwiGLU is applied first."""
        H = self.cfg.hidden
        if self._in_skinny(w, H, k):
            self._check(self.L.b200_q4f16_gemv_add(x.data_ptr(), w[0].data_ptr(), w[1].data_ptr(), self.x.data_ptr(),
                                                   self.stats.data_ptr(), self.batch, H, k, int(swiglu), sp))
            return None
        if swiglu:
            self._check(self.L.b200_silu_mul_early_release(x.data_ptr(), self.act.data_ptr(), self.batch, k, sp))
            x = self.act
        self._matmul(x, w, out, H, k, sp)
        return out

    def _norm(self, delta, norm, sp):
        """h = rmsnorm(x += delta) as a launch of its own."""
        self._check(self.L.b200_rmsnorm_early_release(self.x.data_ptr(), delta.data_ptr() if delta is not None else None, norm.data_ptr(),
                                                      self.h.data_ptr(), self.batch, self.cfg.hidden, self.cfg.eps, sp))

    def _chained_layer(self, i: int, delta, sp: int):
        """One layer in the chained form: qkv, attention, o, gate|up, down.  `delta` as in :meth:`layer_step`; None: the residual
        stream is complete and has its statistics."""
        cfg, L, B, w = self.cfg, self.L, self.batch, self.layers[i]
        H, il = cfg.hidden, w["inter_local"]
        roped = False
        skinny = delta is None and self._norm_in_skinny(w["qkv"], 3 * H, H)
        if skinny and self.rope_epilogue:
            rc = L.b200_q4f16_gemv_norm_rope(self.x.data_ptr(), self.stats.data_ptr(), w["norm1"].data_ptr(), cfg.eps,
                                             w["qkv"][0].data_ptr(), w["qkv"][1].data_ptr(), self.cos.data_ptr(), self.sin.data_ptr(),
                                             self.pos.data_ptr(), self.q.data_ptr(), self.kc[i].data_ptr(), self.vc[i].data_ptr(),
                                             self.nh_local, H, sp)
            if rc != _lib.ENOTREADY:        # (else the exact form is selected)
                self._check(rc)
                roped = True
        if skinny and not roped:
            self._check(L.b200_q4f16_gemv_norm(self.x.data_ptr(), self.stats.data_ptr(), w["norm1"].data_ptr(), cfg.eps,
                                               w["qkv"][0].data_ptr(), w["qkv"][1].data_ptr(), self.qkv.data_ptr(), B, 3 * H, H, sp))
        elif not roped:
            self._norm(delta, w["norm1"], sp)
            self._matmul(self.h, w["qkv"], self.qkv, 3 * H, H, sp)
        self._attention(i, roped, sp)
        delta = self._add(self.attn, w["o"], self.o, H, sp)
        if not self._gate_up_in_one(w):
            self._norm(delta, w["norm2"], sp)
            self._matmul(self.h, w["gu"], self.gu, 2 * il, H, sp)
            return self._add(self.gu, w["down"], self.down, il, sp, swiglu=True)
        if delta is None and self._norm_in_skinny(w["gu"], 2 * il, H):
            self._check(L.b200_q4f16_gemv_norm_gate_up(self.x.data_ptr(), self.stats.data_ptr(), w["norm2"].data_ptr(), cfg.eps,
                                                       w["gu"][0].data_ptr(), w["gu"][1].data_ptr(), self.act.data_ptr(), B, il, H, sp))
        else:
            self._norm(delta, w["norm2"], sp)
            self._check(L.b200_q4f16_gemv_gate_up(self.h.data_ptr(), None, None, None, 0.0, w["gu"][0].data_ptr(), w["gu"][1].data_ptr(),
                                                  self.act.data_ptr(), B, il, H, sp))
        return self._add(self.act, w["down"], self.down, il, sp)

    def _attention(self, i: int, roped: bool, sp: int, early: bool = True):
        """`roped`: the qkv matmul has rotated q and appended k and v, else all of that is done here.

        `early` (loads): the position and the older cache entries are final before any kernel of a step but its first can begin.
        A kernel begins only after the one in front of it has begun, embed_rows lets its successor begin only after it
        has waited for everything in front of it, and every kernel waits for its predecessor before it ends."""
        L, B = self.L, self.batch
        loads = _lib.ATTN_EARLY_KV_LOADS if early else 0
        if roped:
            self._check(L.b200_attn_decode_early_release(self.q.data_ptr(), self.kc[i].data_ptr(), self.vc[i].data_ptr(),
                                                         self.pos.data_ptr(), self.attn.data_ptr(), self.scratch.data_ptr(), B,
                                                         self.nh_local, self.max_ctx, loads, sp))
        elif self.fused_attention == "rope":
            self._check(L.b200_attn_decode_rope(self.qkv.data_ptr(), self.cos.data_ptr(), self.sin.data_ptr(), self.pos.data_ptr(),
                                                self.kc[i].data_ptr(), self.vc[i].data_ptr(), self.attn.data_ptr(),
                                                self.scratch.data_ptr(), B, self.nh_local, self.max_ctx, sp))
        elif self.fused_attention:
            self._check(L.b200_attn_decode_fused(self.qkv.data_ptr(), self.cos.data_ptr(), self.sin.data_ptr(), self.pos.data_ptr(),
                                                 self.kc[i].data_ptr(), self.vc[i].data_ptr(), self.attn.data_ptr(),
                                                 self.scratch.data_ptr(), B, self.nh_local, self.max_ctx, sp))
        else:
            self._check(L.b200_attn_decode_step(self.qkv.data_ptr(), self.cos.data_ptr(), self.sin.data_ptr(), self.pos.data_ptr(),
                                                self.kc[i].data_ptr(), self.vc[i].data_ptr(), self.attn.data_ptr(), B, self.nh_local,
                                                self.max_ctx, loads | _lib.ATTN_EARLY_RELEASE, sp))

    def _allreduce(self, t):
        if self.world > 1:
            torch.distributed.all_reduce(t, group=self.group)

    def layer_step(self, i: int, delta, sp: int, within_step: bool = False):
        """One layer; `delta` is the tensor still to be added to the residual stream (or None).
        Returns the layer's MLP output (to be added by whoever consumes the stream next).

        Outside a step (`within_step` False) whatever the caller launched in front may have written the position and the
        caches, and no kernel between it and the attention waits before it lets the next one begin: no early loads then.

        The early-release forms: behind every one of them is a matmul (or the output projection), which reads nothing
        but weights before it has waited for the kernel in front."""
        cfg, L, B, w = self.cfg, self.L, self.batch, self.layers[i]
        H, hl, il = cfg.hidden, cfg.hidden // self.world, w["inter_local"]
        dptr = delta.data_ptr() if delta is not None else None
        roped = False
        if self.fused and self.rope_epilogue:
            # residual stream: x --(+delta)--> x2 --(+o)--> x; rotary embedding and KV append in the matmul's epilogue
            rc = L.b200_q4f16_gemv_rmsnorm_rope(self.x.data_ptr(), dptr, w["norm1"].data_ptr(), self.x2.data_ptr(), cfg.eps,
                                                w["qkv"][0].data_ptr(), w["qkv"][1].data_ptr(), self.cos.data_ptr(),
                                                self.sin.data_ptr(), self.pos.data_ptr(), self.q.data_ptr(),
                                                self.kc[i].data_ptr(), self.vc[i].data_ptr(), self.nh_local, H, sp)
            if rc == _lib.ENOTREADY:
                self.rope_epilogue = False      # (the exact form is selected: two kernels from now on)
            else:
                self._check(rc)
                roped = True
        if roped:
            pass
        elif self.fused:
            # residual stream: x --(+delta)--> x2 --(+o)--> x
            self._check(L.b200_q4f16_gemv_rmsnorm(self.x.data_ptr(), dptr, w["norm1"].data_ptr(), self.x2.data_ptr(), cfg.eps,
                                                  w["qkv"][0].data_ptr(), w["qkv"][1].data_ptr(), self.qkv.data_ptr(),
                                                  B, 3 * hl, H, sp))
        else:
            self._check(L.b200_rmsnorm_early_release(self.x.data_ptr(), dptr, w["norm1"].data_ptr(), self.h.data_ptr(), B, H,
                                                     cfg.eps, sp))
            self._matmul(self.h, w["qkv"], self.qkv, 3 * hl, H, sp)
        self._attention(i, roped, sp, early=within_step)
        if self.peer is not None and B <= self.PEER_FUSED_MAX_ROWS:
            d = self._reduce_desc(0, i, self.o)
            self._check(L.b200_q4f16_gemv_allreduce(self.attn.data_ptr(), w["o"][0].data_ptr(), w["o"][1].data_ptr(),
                                                    self.peer["y"][0][self.rank], B, H, hl, 0, ctypes.byref(d), sp))
        elif self.peer is not None:
            self._matmul_then_peer_sum(0, i, self.attn, w["o"], self.o, H, hl, sp)
        else:
            self._matmul(self.attn, w["o"], self.o, H, hl, sp)
            self._allreduce(self.o)
        if self.fused:
            self._check(L.b200_q4f16_gemv_gate_up(self.x2.data_ptr(), self.o.data_ptr(), w["norm2"].data_ptr(), self.x.data_ptr(),
                                                  cfg.eps, w["gu"][0].data_ptr(), w["gu"][1].data_ptr(), self.act.data_ptr(),
                                                  B, il, H, sp))
        else:
            self._check(L.b200_rmsnorm_early_release(self.x.data_ptr(), self.o.data_ptr(), w["norm2"].data_ptr(), self.h.data_ptr(),
                                                     B, H, cfg.eps, sp))
            rc = _lib.ENOTREADY
            if self._gate_up_wide(w):
                rc = L.b200_q4f16_gate_up(self.h.data_ptr(), w["gu"][0].data_ptr(), w["gu"][1].data_ptr(), self.act.data_ptr(), B, il, H, sp)
            elif self._gate_up_in_one(w):
                rc = L.b200_q4f16_gemv_gate_up(self.h.data_ptr(), None, None, None, 0.0, w["gu"][0].data_ptr(),
                                               w["gu"][1].data_ptr(), self.act.data_ptr(), B, il, H, sp)
            if rc == _lib.ENOTREADY:
                self._matmul(self.h, w["gu"], self.gu, 2 * il, H, sp)
                rc = L.b200_silu_mul_early_release(self.gu.data_ptr(), self.act.data_ptr(), B, il, sp)
            self._check(rc)
        if self.peer is not None and B <= self.PEER_FUSED_MAX_ROWS:
            d = self._reduce_desc(1, i, self.down)
            self._check(L.b200_q4f16_gemv_allreduce(self.act.data_ptr(), w["down"][0].data_ptr(), w["down"][1].data_ptr(),
                                                    self.peer["y"][1][self.rank], B, H, il, 0, ctypes.byref(d), sp))
            return self.down
        if self.peer is not None:
            self._matmul_then_peer_sum(1, i, self.act, w["down"], self.down, H, il, sp)
            return self.down
        self._matmul(self.act, w["down"], self.down, H, il, sp)
        self._allreduce(self.down)
        return self.down

    def step(self):
        """One decode step on the current stream: embeds self.tokens, runs every layer at position
        self.pos, writes logits (when there is an lm_head), samples greedily into self.tokens and
        advances self.pos.  All inputs live on the device, so the step can be captured and replayed."""
        cfg, L, B = self.cfg, self.L, self.batch
        if self.guard is not None and not torch.cuda.is_current_stream_capturing():
            self.guard.check()
        sp = torch.cuda.current_stream(self.device).cuda_stream
        if self.chained:
            self._check(L.b200_embed_rows_stats(self.embed.data_ptr(), self.tokens.data_ptr(), self.x.data_ptr(), self.stats.data_ptr(), B,
                                                cfg.hidden, self.embed.shape[0], sp))
        else:
            self._check(L.b200_embed_rows(self.embed.data_ptr(), self.tokens.data_ptr(), self.x.data_ptr(), B, cfg.hidden,
                                          self.embed.shape[0], sp))
        delta = None
        xlast = self.x
        if self.layer_kernel:
            for i in range(len(self.layers)):
                self._check(L.b200_decode_layer(ctypes.byref(self.layer_desc[i]), sp))
            if self.layers:
                delta, xlast = self.down, self.x_last
        else:
            for i in range(len(self.layers)):
                delta = self._chained_layer(i, delta, sp) if self.chained else self.layer_step(i, delta, sp, within_step=True)
        normed = not (self.chained and delta is None and self.lm_head is not None)
        if normed:
            self._check(L.b200_rmsnorm_early_release(xlast.data_ptr(), delta.data_ptr() if delta is not None else None,
                                                     self.final_norm.data_ptr(), self.h.data_ptr(), B, cfg.hidden, cfg.eps, sp))
        if not normed:
            self._check(L.b200_lm_head_norm(self.x.data_ptr(), self.stats.data_ptr(), self.final_norm.data_ptr(), cfg.eps,
                                            self.h.data_ptr(), self.lm_head.data_ptr(), self.logits_local.data_ptr(), self.tokens.data_ptr(),
                                            self.lm_scratch.data_ptr(), B, self.lm_head.shape[0], cfg.hidden, 0, sp))
        elif self.lm_head is not None:
            own = B <= 16                       # the library's output projection takes up to 16 rows; above that a library GEMM
            if own:
                toks = self.tokens.data_ptr() if self.world == 1 else None
                self._check(L.b200_lm_head(self.h.data_ptr(), self.lm_head.data_ptr(), self.logits_local.data_ptr(), toks,
                                           self.lm_scratch.data_ptr(), B, self.lm_head.shape[0], cfg.hidden, 0, sp))
            else:
                torch.matmul(self.h, self.lm_head.t(), out=self.logits_local)
            if self.world > 1:
                # gather the vocabulary slices: [world, B, V_l] -> [B, world * V_l]
                torch.distributed.all_gather_into_tensor(self.gathered, self.logits_local, group=self.group)
                self.logits.view(B, self.world, -1).copy_(self.gathered.permute(1, 0, 2))
            if not own or self.world > 1:
                self._check(L.b200_argmax_rows(self.logits.data_ptr(), self.tokens.data_ptr(), B, self.logits.shape[1], sp))
        self._check(L.b200_advance_pos(self.pos.data_ptr(), 1, sp))
        if self._counts_steps():
            self._check(L.b200_advance_pos(self.epoch.data_ptr(), 1, sp))

    def _counts_steps(self) -> bool:
        """Whether something in a step reads the step counter (flags of the sums over ranks, arrival counters of the layer kernel)."""
        return self.peer is not None or self.layer_kernel

    def kernels_per_step(self) -> int:
        """Kernels of this library launched by one step: embed, 5 to 10 per layer, final norm, output projection for up to
        16 rows, sampling where it is not part of that, one or two counters."""
        head = int(self.lm_head is not None and self.batch <= 16)
        tail = 1 + int(self._counts_steps()) + int(self.lm_head is not None and (self.batch > 16 or self.world > 1))
        if self.layer_kernel:
            return 1 + len(self.layers) + 1 + head + tail
        if self.chained:
            ready, norms = True, 0          # the residual stream has its statistics; norms as launches of their own
            per_layer = 0
            for w in self.layers:
                per_layer += 5
                norms += not (ready and self._norm_in_skinny(w["qkv"], 3 * self.cfg.hidden, self.cfg.hidden))
                ready = self._in_skinny(w["o"], self.cfg.hidden, self.cfg.hidden)
                one = self._gate_up_in_one(w)
                norms += not (ready and one and self._norm_in_skinny(w["gu"], 2 * w["inter_local"], self.cfg.hidden))
                ready = self._in_skinny(w["down"], self.cfg.hidden, w["inter_local"])
                per_layer += 0 if one or ready else 1          # (SwiGLU as a launch of its own)
            return 1 + per_layer + norms + (0 if ready and head else 1) + head + tail
        peer_sums = 2 if self.peer is not None and self.batch > self.PEER_FUSED_MAX_ROWS else 0
        per_layer = 0
        for w in self.layers:
            mlp = 2 if self.fused else 3 if self._gate_up_in_one(w) or self._gate_up_wide(w) else 4        # (norm,) gate|up (, SwiGLU), down
            per_layer += (1 if self.fused else 2) + 2 + mlp + peer_sums           # (norm,) qkv, attention, o
        return 1 + per_layer + 1 + head + tail

    def capture(self, stream):
        """Captures one step into a CUDA graph on `stream` (after one eager warm-up step, which
        also lets NCCL set up its channels outside the capture)."""
        stream.wait_stream(torch.cuda.current_stream(self.device))   # buffers were filled on the caller's stream
        with torch.cuda.stream(stream):
            pos0 = int(self.pos.item())
            tok0 = self.tokens.clone()
            self.step()
            stream.synchronize()
            self.pos.fill_(pos0)
            self.tokens.copy_(tok0)
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph, stream=stream):
                self.step()
            self.pos.fill_(pos0)
            self.tokens.copy_(tok0)
            stream.synchronize()
        return self.graph

    def set_position(self, pos: int):
        self.pos.fill_(int(pos))
