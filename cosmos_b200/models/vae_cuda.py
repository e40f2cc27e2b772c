"""Tokenizer encoder and decoder on the sm_100a kernels: activations live in zero-bordered channels-last volumes
[frames, H + 2, W + 2, C] (bf16) and every 3x3x3 causal convolution is an implicit GEMM on the tensor cores
(csrc/conv_tcgen05.cu). A convolution's epilogue also does what follows it: the residual, the channel RMS-norm + SiLU, the
nearest upsampling, the layout that a strided convolution reads, or the conversion to pixels, so that a layer is one launch.
Clips run in temporal chunks; the causal context of every convolution (the last two frames of its input) is carried from
chunk to chunk, so the result equals one pass over the clip. These two frames are a tensor of their own (`Volume.tail`), which the
next chunk's convolution reads where it is.

Built from a `CausalVideoVAE` (same weights); requires channel widths that are multiples of 64.
"""
from __future__ import annotations

from typing import Dict, List, Optional, Tuple

import torch
import torch.nn.functional as F

from .. import ops
from .vae import CausalVideoVAE, ResBlock

TAIL = 2  # frames that a convolution needs of the chunk before (temporal kernel 3, stride 1)
SAME, S2D, UP, DOWN = 0, 1, 2, 3   # layouts that a convolution can write (csrc/kernels.h, ConvOut)
NORM_WIDTHS = (64, 128, 256)       # channels that the fused norm takes: a thread of the epilogue holds a whole row


def _pack_weight(w: torch.Tensor, cin_pad: int) -> torch.Tensor:
    """[Cout, Cin, 3, 3, 3] -> [Cout, 27 * cin_pad] bf16, tap-major (kt, kh, kw) then channel."""
    cout, cin = w.shape[:2]
    p = torch.zeros(cout, 3, 3, 3, cin_pad, dtype=torch.bfloat16, device=w.device)
    p[..., :cin] = w.permute(0, 2, 3, 4, 1).to(torch.bfloat16)
    return p.reshape(cout, 27 * cin_pad).contiguous()


def _bf16_terms(w: torch.Tensor, n: int = 3) -> torch.Tensor:
    """fp32 [rows, cols] -> [n * rows, cols] bf16 whose n blocks of rows add up to it (three terms hold all 24 bits)."""
    out, rest = [], w.float()
    for _ in range(n):
        out.append(rest.to(torch.bfloat16))
        rest = rest - out[-1].float()
    return torch.cat(out).contiguous()


class Volume:
    """Padded channels-last frames of one chunk: all but the last two in `body`, those in `tail` (a single frame is the tail's
    second). A tail outlives its chunk as the next one's context without keeping the body."""

    def __init__(self, frames: int, frame_shape, device, zero: bool = False):
        new = torch.zeros if zero else torch.empty
        self.frames = frames
        self.body = new(max(0, frames - TAIL), *frame_shape, dtype=torch.bfloat16, device=device)
        self.tail = new(TAIL, *frame_shape, dtype=torch.bfloat16, device=device)

    @property
    def parts(self) -> List[torch.Tensor]:
        return [self.body, self.tail]

    def pieces(self) -> List[Tuple[int, int, torch.Tensor]]:
        """(first frame, end, the tensor that holds them) of both parts."""
        n = self.body.shape[0]
        return [p for p in ((0, n, self.body), (n, self.frames, self.tail[n + TAIL - self.frames:])) if p[1] > p[0]]


class _CLConvs:
    """Packed weights and the launches that encoder and decoder share."""

    def __init__(self, vae: CausalVideoVAE, eps: float):
        self.device = next(vae.parameters()).device
        assert self.device.type == "cuda" and ops.load_extension(), "the channels-last tokenizer runs on CUDA, on the kernel library"
        self.latent_channels = vae.latent_channels
        self.eps = eps
        self.w: Dict[str, torch.Tensor] = {}
        self.b: Dict[str, torch.Tensor] = {}
        self.g: Dict[str, torch.Tensor] = {}

    def _add_conv(self, name: str, m, cin_pad: Optional[int] = None) -> None:
        assert m.k == (3, 3, 3)
        cp = cin_pad or m.weight.shape[1]
        assert cp % 64 == 0 and m.weight.shape[0] % 32 == 0, "channel widths must be multiples of 64"
        self.w[name] = _pack_weight(m.weight.data, cp)
        self.b[name] = m.bias.data.float().contiguous()

    def _add_res(self, name: str, blk: ResBlock) -> None:
        self.g[name + ".n1"] = blk.n1.gamma.data.to(torch.bfloat16).contiguous()
        self.g[name + ".n2"] = blk.n2.gamma.data.to(torch.bfloat16).contiguous()
        self._add_conv(name + ".c1", blk.c1)
        self._add_conv(name + ".c2", blk.c2)

    # ------------------------------------------------------------------ launches
    def _ctx(self, cache: Dict, key: str, vol: Volume) -> Optional[torch.Tensor]:
        """The context frames of `vol` (None: the clip starts here); its own tail takes their place for the next chunk."""
        ctx = cache.get(key)
        if vol.frames == 1:
            vol.tail[0].copy_(ctx[1]) if ctx is not None else vol.tail[0].zero_()
        cache[key] = vol.tail
        return ctx if ctx is not None or self.finite else torch.zeros_like(vol.tail)

    def _finish(self) -> None:
        """The kernel leaves out products with an absent context, which are zero as long as the weights are finite; otherwise zeros
        stand in for it."""
        self.finite = bool(torch.stack([w.isfinite().all() for w in self.w.values()]).all())

    def _volume(self, frames: int, *frame_shape, zero: bool = False) -> Volume:
        return Volume(frames, frame_shape, self.device, zero)

    def _conv(self, cache: Dict, name: str, x: Volume, resid: Optional[Volume] = None, skip: Optional[Volume] = None,
              norm: Optional[torch.Tensor] = None, raw: bool = True, mode: int = SAME, a: int = 0, b: int = 0,
              frames: Optional[int] = None) -> Tuple[Optional[Volume], Optional[Volume]]:
        """One convolution of `x`. Returns (result, silu(rmsnorm(result) * norm)); `raw` False: the first is not wanted. `mode`,
        `a`, `b`: the layout written (`ops.conv3d_chunk`); `frames`: its frame count, where it differs from x's."""
        ctx = self._ctx(cache, name, x)
        w = self.w[name]
        cout = w.shape[0]
        hp, wp = x.tail.shape[-3:-1]
        shape = {DOWN: (hp + 1, wp + 1, cout), S2D: (4, hp // 2, wp // 2, cout), UP: (2 * hp - 2, 2 * wp - 2, cout),
                 SAME: (hp, wp, cout)}[mode]
        fused = norm is not None and cout in NORM_WIDTHS
        n = frames or x.frames
        out = self._volume(n, *shape) if raw or not fused else None
        out_norm = self._volume(n, *shape) if fused else None
        parts = lambda v: [] if v is None else v.parts  # noqa: E731
        torch.ops.cosmos_b200.conv3d_chunk(x.parts, ctx, w, self.b[name], parts(resid), parts(skip), parts(out), parts(out_norm),
                                           norm if fused else None, self.eps, mode, x.frames, a, b)
        if norm is not None and not fused:
            out_norm = self._volume(n, *shape)
            for (_, _, src), (_, _, dst) in zip(out.pieces(), out_norm.pieces()):
                dst.copy_(torch.ops.cosmos_b200.rmsnorm_silu(src, norm, self.eps))
        return out, out_norm


class CLDecoder(_CLConvs):
    def __init__(self, vae: CausalVideoVAE):
        super().__init__(vae, vae.dec_norm.eps)
        self._add_conv("in", vae.dec_in, 64)
        self._add_res("mid", vae.dec_mid)
        self.ups: List[bool] = []
        for i, (blk, up) in enumerate(zip(vae.dec_blocks, vae.dec_up)):
            assert blk.skip is None
            self._add_res(f"b{i}", blk)
            self._add_conv(f"u{i}", up.conv)
            self.ups.append(up.temporal)
        self.g["out"] = vae.dec_norm.gamma.data.to(torch.bfloat16).contiguous()
        wo = vae.dec_out.weight.data  # [3, 64, 3, 3, 3]
        assert wo.shape[0] == 3 and wo.shape[1] == 64, "the RGB head expects 64 input channels"
        self.w_out = _bf16_terms(wo.permute(0, 2, 3, 4, 1).reshape(3, 27 * 64))
        self.b_out = vae.dec_out.bias.data.float().contiguous()
        self._finish()
        self.finite = self.finite and bool(wo.isfinite().all())

    # ------------------------------------------------------------------ public
    @torch.no_grad()
    def decode_chunk(self, z: torch.Tensor, cache: Dict, first: bool) -> torch.Tensor:
        """z [C, tc, h, w] -> uint8 frames [T, 8h, 8w, 3]."""
        c, tc, h, w = z.shape
        vol = self._volume(tc, h + 2, w + 2, 64, zero=True)
        for s, e, part in vol.pieces():
            part[:, 1:-1, 1:-1, :c] = z[:, s:e].permute(1, 2, 3, 0)
        x, n = self._conv(cache, "in", vol, norm=self.g["mid.n1"])
        _, n = self._conv(cache, "mid.c1", n, norm=self.g["mid.n2"], raw=False)
        x, n = self._conv(cache, "mid.c2", n, resid=x, norm=self.g["b0.n1"])
        last = len(self.ups) - 1
        for i, temporal in enumerate(self.ups):
            _, n = self._conv(cache, f"b{i}.c1", n, norm=self.g[f"b{i}.n2"], raw=False)
            if temporal:
                tc = 2 * tc - 1 if first else 2 * tc
            x, _ = self._conv(cache, f"b{i}.c2", n, resid=x, mode=UP, a=int(temporal), b=int(first), frames=tc)
            x, n = self._conv(cache, f"u{i}", x, norm=self.g["out" if i == last else f"b{i + 1}.n1"], raw=i < last)
        return torch.ops.cosmos_b200.conv3d_rgb_chunk(n.parts, self._ctx(cache, "out", n), self.w_out, self.b_out, n.frames)

    @torch.no_grad()
    def decode(self, z: torch.Tensor, chunk_latents: int = 2) -> torch.Tensor:
        """z [1, C, T, h, w] -> uint8 [1, T_pix, 8h, 8w, 3]."""
        assert z.shape[0] == 1
        cache: Dict = {}
        outs = []
        for s in range(0, z.shape[2], chunk_latents):
            outs.append(self.decode_chunk(z[0, :, s:s + chunk_latents], cache, s == 0))
        return torch.cat(outs, dim=0)[None]

    @torch.no_grad()
    def decode_to_host(self, z: torch.Tensor, chunk_latents: int = 2) -> torch.Tensor:
        """`decode` with the frames on the host: a chunk's frames go through one of two pinned buffers on a stream of their
        own and from there into the result while the next chunk is computed."""
        assert z.shape[0] == 1
        t = z.shape[2]
        out = torch.empty(1 + 4 * (t - 1), 8 * z.shape[3], 8 * z.shape[4], 3, dtype=torch.uint8)
        stage = [torch.empty(min(4 * chunk_latents, out.shape[0]), *out.shape[1:], dtype=torch.uint8, pin_memory=True)
                 for _ in range(2)]
        cur, side = torch.cuda.current_stream(self.device), torch.cuda.Stream(self.device)
        cache: Dict = {}
        done, waiting = 0, []

        def drain():
            nonlocal done
            ev, buf = waiting.pop(0)
            ev.synchronize()
            out[done:done + buf.shape[0]].copy_(buf)
            done += buf.shape[0]

        for i, s in enumerate(range(0, t, chunk_latents)):
            frames = self.decode_chunk(z[0, :, s:s + chunk_latents], cache, s == 0)
            buf = stage[i % 2][:frames.shape[0]]
            side.wait_stream(cur)
            with torch.cuda.stream(side):
                buf.copy_(frames, non_blocking=True)
                ev = torch.cuda.Event()
                ev.record(side)
            frames.record_stream(side)
            waiting.append((ev, buf))
            if len(waiting) == 2:   # the older buffer is free again before the next chunk asks for it
                drain()
        while waiting:
            drain()
        return out


def even_frames(t0: int, n: int):
    """Temporal stride 2 over a chunk of `n` frames whose first frame has index `t0` in its level's timeline: the
    causal strided convolution keeps the frames with an even index. Returns (offset of the first kept frame inside
    the chunk, number of kept frames, index of the first kept frame in the next level's timeline)."""
    first = t0 % 2
    return first, max(0, (n - first + 1) // 2), (t0 + 1) // 2


class CLEncoder(_CLConvs):
    """Tokenizer encoder on the same kernel as `CLDecoder`.

    * A strided convolution (the three down-sampling steps: stride 2 in space, the last two also in time) computes the kept
      positions and frames alone. It reads its input split by the parity of row and column, which the block before it writes;
      causal padding in time and `k // 2` padding in space make output (j, i) of the strided form the stride-1 form's
      (2j, 2i).
    * The 1x1x1 skip projections of the widening blocks are further columns of the block's second convolution: its sum runs
      over the 27 taps of its own input and then over the channels of the block's input.
    * The first layer's 9 spatial taps x 3 colours are packed into the 64 channels of an operand row. A tokenizer of another
      number of input channels (up to 64) has them zero-extended to 64 and takes all 27 taps.

    Frames are encoded in temporal chunks (the first frame alone, then `chunk_frames` at a time); each
    convolution's two context frames are carried over, so the result equals one pass over the clip.
    Reference behaviour: the tokenizer's causal encoder, cosmos_framework/inference (Wan2.2-style 4x8x8 VAE)."""

    def __init__(self, vae: CausalVideoVAE):
        super().__init__(vae, vae.enc_norm.eps)
        w = vae.enc_in.weight.data   # [C, in_channels, 3, 3, 3]
        self.in_channels = w.shape[1]
        if self.in_channels == 3:
            assert vae.enc_in.k == (3, 3, 3) and w.shape[0] % 64 == 0, "channel widths must be multiples of 64"
            p = torch.zeros(w.shape[0], 3, 64, dtype=torch.bfloat16, device=self.device)
            p[:, :, :27] = w.permute(0, 2, 3, 4, 1).reshape(w.shape[0], 3, 27).to(torch.bfloat16)
            self.w["in"] = p.reshape(w.shape[0], 192)
            self.b["in"] = vae.enc_in.bias.data.float().contiguous()
        else:
            self._add_conv("in", vae.enc_in, 64)
        self.downs: List[bool] = []
        self.skips: Dict[str, bool] = {}

        def res(name, blk: ResBlock):
            self._add_res(name, blk)
            self.skips[name] = blk.skip is not None
            if blk.skip is not None:
                sw = blk.skip.weight.data.reshape(blk.skip.weight.shape[0], -1).to(torch.bfloat16)
                self.w[name + ".c2"] = torch.cat([self.w[name + ".c2"], sw], dim=1).contiguous()
                self.b[name + ".c2"] = blk.c2.bias.data.float() + blk.skip.bias.data.float()

        for i, (blk, down) in enumerate(zip(vae.enc_blocks, vae.enc_down)):
            res(f"b{i}", blk)
            self._add_conv(f"d{i}", down.conv)
            assert down.conv.stride[1:] == (2, 2)
            self.downs.append(down.conv.stride[0] == 2)
        res("mid", vae.enc_mid)
        self.g["out"] = vae.enc_norm.gamma.data.to(torch.bfloat16).contiguous()
        self._add_conv("out", vae.enc_out)
        self._finish()

    def _res(self, cache, name, x, n, **kw):
        """One residual block; x: its input, n: silu(rmsnorm(x))."""
        _, n = self._conv(cache, name + ".c1", n, norm=self.g[name + ".n2"], raw=False)
        return self._conv(cache, name + ".c2", n, **({"skip": x} if self.skips[name] else {"resid": x}), **kw)

    @torch.no_grad()
    def encode_chunk(self, frames: torch.Tensor, cache: Dict, t0: int) -> torch.Tensor:
        """frames [C, n, H, W] in [-1, 1], on any device and of any dtype (global index of the first one: t0) -> moments
        [2C, n', H/8, W/8] fp32. Channels that the tokenizer does not have are ignored, missing ones are zero."""
        c, n, h, w = frames.shape
        assert c <= 64
        if self.in_channels == 3:
            frames = frames.to(self.device)
            if c != 3:
                frames = F.pad(frames[:3], (0, 0, 0, 0, 0, 0, 0, max(0, 3 - c)))
            if frames.dtype not in (torch.float32, torch.bfloat16):
                frames = frames.to(torch.bfloat16)
            if frames.stride(3) != 1 or frames.stride(2) != w or (n > 1 and frames.stride(1) != h * w):
                frames = frames.contiguous()
            vol = self._volume(n, h + 2, w + 2, 64)
            for s, e, part in vol.pieces():
                torch.ops.cosmos_b200.conv_pack_frames(frames[:, s:e], part)
        else:
            vol = self._volume(n, h + 2, w + 2, 64, zero=True)
            for s, e, part in vol.pieces():
                part[:, 1:-1, 1:-1, :c] = frames[:, s:e].permute(1, 2, 3, 0)
        x, y = self._conv(cache, "in", vol, norm=self.g["b0.n1"])
        last = len(self.downs) - 1
        for i, temporal in enumerate(self.downs):
            x, _ = self._res(cache, f"b{i}", x, y, mode=S2D)
            first, step, kept = 0, 1, n
            if temporal:
                first, kept, t0 = even_frames(t0, n)
                step = 2
            if kept == 0:   # an odd frame alone: nothing of it is kept, but the next chunk needs it as context
                self._ctx(cache, f"d{i}", x)
                return torch.empty(2 * self.latent_channels, 0, h // 8, w // 8, device=self.device)
            x, y = self._conv(cache, f"d{i}", x, norm=self.g["mid.n1" if i == last else f"b{i + 1}.n1"], mode=DOWN, a=first,
                              b=step, frames=kept)
            n = kept
        _, y = self._res(cache, "mid", x, y, norm=self.g["out"], raw=False)
        y, _ = self._conv(cache, "out", y)
        return torch.cat([part[:, 1:-1, 1:-1].permute(3, 0, 1, 2) for _, _, part in y.pieces()], dim=1).float()

    @torch.no_grad()
    def encode(self, video: torch.Tensor, chunk_frames: int = 8) -> torch.Tensor:
        """video [1, 3, 1 + 4k, H, W] in [-1, 1] (H, W multiples of 8) -> latent mean [1, C, 1 + k, H/8, W/8] fp32."""
        assert video.shape[0] == 1 and (video.shape[2] - 1) % 4 == 0 and chunk_frames % 4 == 0
        assert video.shape[3] % 8 == 0 and video.shape[4] % 8 == 0
        cache: Dict = {}
        t = video.shape[2]
        outs = [self.encode_chunk(video[0, :, :1], cache, 0)]
        for s in range(1, t, chunk_frames):
            outs.append(self.encode_chunk(video[0, :, s:s + chunk_frames], cache, s))
        moments = torch.cat(outs, dim=1)
        return moments[None, :self.latent_channels]
