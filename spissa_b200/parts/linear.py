"""y = x · Wᵀ with W stored [out, in] (crates/spissa-runtime/src/ops.rs:62-105).

``Linear`` holds one weight matrix and picks the kernel for a call by the operands'
storage types and sizes: bfloat16 activations on a bfloat16 weight go to the weight-streaming
kernel for a few tokens (decoding), to the tcgen05 kernel with the weight's rows as the instruction's M for some dozens
to some hundreds of tokens, and to the tcgen05 tile kernel otherwise, when the rows are multiples of 16 bytes;
32-bit products of more than ``GEMV_TOKENS`` rows go to the tcgen05 kernel that multiplies float32 in bfloat16 parts;
everything else goes to the FFMA kernels.
"""
from __future__ import annotations

import torch

from ..csrc import lib as K

_SM_COUNT: dict = {}


def sm_count(device=None) -> int:
    """Streaming multiprocessors of ``device`` (the current CUDA device when None), asked once per device."""
    index = torch.cuda.current_device() if device is None else (torch.device(device).index or 0)
    if index not in _SM_COUNT:
        _SM_COUNT[index] = int(torch.cuda.get_device_properties(index).multi_processor_count)
    return _SM_COUNT[index]
GEMV_TOKENS = 16          # up to this many tokens the weight-streaming kernel runs instead of 128-row tiles
GATED_GEMV_TOKENS = 16    # the same for the gate/up product
MID_TOKENS = 1023         # from there up to this many tokens the weight's rows are the instruction's M and the tokens its N
#                           (tc_mid.cu). Per layer of the 1B shape (QKV + output + gate/up + down, us) against what ran before
#                           (tc_stream.cu up to 64 tokens, tc_gemm.cu's tiles of 128 tokens beyond): 33 tokens 44 / 47, 64: 47 / 50,
#                           100: 53 / 92, 301: 67 / 122, 512: 83 / 108, 1,000: 138 / 201; of the 8B shape 100: 110 / 149,
#                           301: 171 / 254, 700: 321 / 416, 1,000: 430 / 435. Gated products, and from 1,024 tokens on all, go by the
#                           estimates of sp_tc_mid_or_pairs: tc_gemm.cu's pairs of CTAs read half as much per product where they have
#                           enough tiles
F32_PARTS_K = 128         # 32-bit products with sums at least so long go to tc_f32.cu. Relative error against 64 bits there / in order
#                           on FFMA: K = 8 1.0e-7 / 5e-8, 72: 1.2e-7 / 1.5e-7, 128: 1.3e-7 / 2.0e-7, 2,048: 1.6e-7 / 8.1e-7
STREAM_TOKENS = 64        # what tc_mid.cu does not take (gate and up rows in blocks of 64): tc_stream.cu up to this many tokens


PAIR_TOKENS = 1024        # from here on tc_gemm.cu computes all its tiles, of 256 rows, by pairs of CTAs
MOST_MID_TOKENS = 2048    # the most that tc_mid.cu is built for


def mid_takes(mode, x: torch.Tensor, w: torch.Tensor) -> bool:
    """Whether tc_mid.cu is the faster one for a product that tc_gemm.cu's tiles could take as well."""
    return (x.shape[0] <= MID_TOKENS and mode != K.TC_SILU_MUL) or not K.tc_mid_or_pairs(mode, x.shape[0], w.shape[0], w.shape[1], 1, x.device.index)


def tile_width(M: int, N: int, sms: int | None = None) -> int:
    """256-wide tiles (half the shared-memory traffic per FLOP) when they still occupy most SMs, else 128-wide;
    192-wide when that saves a round of tiles: 2,048 tokens x 3,072 outputs are 96 pair tiles of 256 columns, two
    rounds on 74 pairs of which the second is a third full, but 128 tiles of 192 columns, two rounds of shorter tiles.
    The rounds are counted as the kernel walks them, by pairs of row tiles from ``PAIR_TOKENS`` on: 6,000 tokens x 4,096 of
    the 8B shape are 6 rounds of 256 columns or 8 of 192, and a 192-wide tile costs an eighth more per column: the output
    product 213 us at 192, 160 at 256, the down product 675 and 566."""
    SM_COUNT = sms if sms else sm_count()
    paired = M >= PAIR_TOKENS
    m_tiles, walkers = ((M + 255) // 256, SM_COUNT // 2) if paired else ((M + 127) // 128, SM_COUNT)
    tiles_256 = m_tiles * ((N + 255) // 256)
    if tiles_256 < (walkers * 2) // 3:
        return 128
    if M > 128:
        cost_256 = -(-tiles_256 // walkers) * 256
        cost_192 = -(-(m_tiles * ((N + 191) // 192)) // walkers) * 192
        if cost_192 * (9 if paired else 10) <= cost_256 * (8 if paired else 9):
            return 192
    return 256


class Linear:
    def __init__(self, weight: torch.Tensor):
        if weight.dim() != 2:
            raise ValueError("a linear weight is a matrix [out, in]")
        self.weight = weight.contiguous()
        self.out_features, self.in_features = weight.shape

    def __call__(self, x: torch.Tensor, out: torch.Tensor | None = None, out_dtype=None,
                 accumulate: bool = False) -> torch.Tensor:
        """``accumulate`` adds the product into ``out`` (float32) instead of overwriting it."""
        if out is None:
            if accumulate:
                raise ValueError("accumulation needs the tensor to add into")
            out = torch.empty(x.shape[0], self.out_features, dtype=out_dtype or x.dtype, device=x.device)
        mode = K.TC_ACCUMULATE if accumulate else K.TC_STORE
        bf16 = x.dtype == torch.bfloat16                     # (a float32 model asks for no library of the bfloat16 kernels)
        if x.shape[0] <= GEMV_TOKENS and K.gemv_supported(x, self.weight):
            K.gemv(x, self.weight, out, mode)
        elif bf16 and x.shape[0] <= MOST_MID_TOKENS and mid_takes(mode, x, self.weight) and K.tc_mid_supported(x, self.weight, out, mode):
            K.tc_mid(x, self.weight, out, mode)
        elif x.shape[0] <= STREAM_TOKENS and K.tc_stream_supported(x, self.weight, mode):
            K.tc_stream(x, self.weight, out, mode)
        elif K.tc_gemm_supported(x, self.weight):
            width = x.shape[0] >= PAIR_TOKENS and K.tc_mid_or_pairs(mode, x.shape[0], self.out_features, self.in_features, 1, x.device.index)
            K.tc_gemm(x, self.weight, out, mode, width or tile_width(x.shape[0], self.out_features, sm_count(x.device)))
        elif x.shape[0] > GEMV_TOKENS and x.shape[1] >= F32_PARTS_K and K.tc_f32_supported(x, self.weight, out):
            K.tc_f32(x, self.weight, out, accumulate=accumulate)
        else:
            K.gemm_generic(x, self.weight, out, accumulate=accumulate)
        return out


class GatedLinear:
    """act(x·Wgᵀ) ⊙ (x·Wuᵀ) · mult as one product over the stacked weight (``act``: K.ACT_SILU or K.ACT_GELU; K.ACT_CLAMPED with
    its ``limit`` and ``slope``: g·sigmoid(slope·g)·(u + 1), g = min(x·Wgᵀ, limit), u = clamp(x·Wuᵀ, ±limit)).

    When the sizes allow, gate and up rows are interleaved in blocks (``block`` gate rows, then
    the ``block`` up rows of the same outputs) so that one tile of the tensor-core kernel holds
    both halves and applies act·up in its epilogue.
    """

    def __init__(self, gate: torch.Tensor, up: torch.Tensor, act: int = K.ACT_SILU, mult: float = 1.0, limit: float = 0.0,
                 slope: float = 0.0):
        I = gate.shape[0]
        self.act, self.mult = act, float(mult)
        self.limit, self.slope = float(limit), float(slope)
        if act == K.ACT_CLAMPED and self.mult != 1.0:
            raise ValueError("the clamped unit takes no factor")
        self.intermediate = I
        self.block = 128 if I % 128 == 0 else 64 if I % 64 == 0 else 0
        fused = self.block and gate.dtype == torch.bfloat16 and gate.shape[1] % 8 == 0
        if act == K.ACT_CLAMPED and not self.limit > 0:
            fused = 0                                    # the epilogues are built for positive limits
        if fused:
            h = self.block
            g = gate.reshape(I // h, h, -1)
            u = up.reshape(I // h, h, -1)
            self.weight = torch.stack([g, u], dim=1).reshape(2 * I, -1).contiguous()
        else:
            self.block = 0
            self.weight = torch.cat([gate, up], dim=0).contiguous()
        self.plain = Linear(self.weight)

    def __call__(self, x: torch.Tensor, act_dtype) -> torch.Tensor:
        out = torch.empty(x.shape[0], self.intermediate, dtype=act_dtype, device=x.device)
        kw = dict(act=self.act, mult=self.mult, limit=self.limit, slope=self.slope)
        if self.block and x.shape[0] <= GATED_GEMV_TOKENS and K.gemv_supported(x, self.weight):
            K.gemv(x, self.weight, out, K.TC_SILU_MUL, self.block, **kw)
        elif (self.block and x.shape[0] <= MOST_MID_TOKENS and mid_takes(K.TC_SILU_MUL, x, self.weight)
              and K.tc_mid_supported(x, self.weight, out, K.TC_SILU_MUL, self.block)):
            K.tc_mid(x, self.weight, out, K.TC_SILU_MUL, self.block, **kw)
        elif self.block and x.shape[0] <= STREAM_TOKENS and K.tc_stream_supported(x, self.weight, K.TC_SILU_MUL, self.block):
            K.tc_stream(x, self.weight, out, K.TC_SILU_MUL, self.block, **kw)
        elif self.block and K.tc_gemm_supported(x, self.weight):
            K.tc_gemm(x, self.weight, out, K.TC_SILU_MUL, 2 * self.block, **kw)
        elif self.act == K.ACT_CLAMPED:
            K.clamped_glu(self.plain(x, out_dtype=torch.float32), out, self.limit, self.slope)     # the clamps read unrounded products
        else:
            gu = self.plain(x, out_dtype=act_dtype)
            K.gated_mul(gu, out, self.act, self.mult)
        return out
