"""The layers of a pre-norm stack in one native call (``csrc/dense_layers.cu``): the kernels that the parts would launch, in the
same order with the same arguments, without the parts' host time between them.  Taken where every layer is an RMSNorm, grouped-query
attention, an RMSNorm and a gated feed-forward, all alike, in bfloat16, and the step runs on the tcgen05 attention kernels."""
from __future__ import annotations

import ctypes
import os
from typing import List, Optional

import torch

from .. import kernels, tracing
from ..config.plan import RopeSpec
from ..parts import LayerCache, StepContext, attention_backend, gemm_backend
from ..parts.attention import Attention
from ..parts.norm import RMSNorm
from ..parts.swiglu import SwiGLU

# tests switch it off to compare a step with the parts'
ENABLED = True

_PROGRAM = (("norm", "x", "h"), ("mixer", "h", "a"), ("add", "a", "x"), ("norm", "x", "h"), ("feed_forward", "h", "f"), ("add", "f", "x"))


def _library_product() -> Optional[int]:
    """The address of the library product that torch itself calls, in the library that torch has loaded; None if there is none."""
    try:
        lib = ctypes.CDLL(f"libcublas.so.{(torch.version.cuda or '').split('.')[0]}", mode=os.RTLD_NOLOAD)
        return ctypes.cast(lib.cublasGemmEx, ctypes.c_void_p).value
    except (OSError, AttributeError):
        return None


def _torch_calls_the_library() -> bool:
    """Whether torch's own product would be that call too: its switches choose another library, sums of another kind or an error."""
    return (torch.backends.cuda.preferred_blas_library().name in ("Default", "Cublas") and not torch.cuda.tunable.is_enabled()
            and torch._C._get_cublas_allow_bf16_reduced_precision_reduction() in (True, (True, True))
            and not torch.are_deterministic_algorithms_enabled())


class DenseLayers:
    def __init__(self, layers: List[tuple], gemm_ex: int):
        self.layers = layers        # (norm, attention, norm, feed-forward) of every run
        self.gemm_ex = gemm_ex      # address of the library product

    @staticmethod
    def of(plan, blocks, dtype, stream_dtype) -> Optional["DenseLayers"]:
        """None where the plan is another one."""
        if dtype != torch.bfloat16 or stream_dtype != torch.bfloat16 or plan.streams is not None or not plan.runs:
            return None
        layers = []
        for run in plan.runs:
            block = blocks[run.block]
            ops = block.spec.program
            if run.cache_from is not None or run.add_input or tuple((o.op, o.src, o.dst) for o in ops) != _PROGRAM:
                return None
            if any(o.mix is not None or (o.op == "add" and (o.scale != 1.0 or o.gain is not None)) for o in ops):
                return None
            n1, attn, n2, ff = (block.parts[(ops[i].op, ops[i].name)] for i in (0, 1, 3, 4))
            if type(attn) is not Attention or type(ff) is not SwiGLU or type(n1) is not RMSNorm or type(n2) is not RMSNorm:
                return None
            layers.append((n1, attn, n2, ff))
        n1, attn, n2, ff = layers[0]
        a, f, hidden = attn.spec, ff.spec, plan.hidden
        if any(x.spec != n1.spec or y.spec != a or z.spec != n2.spec or u.spec != f for x, y, z, u in layers):
            return None
        if a.rope is not None and not (type(a.rope) is RopeSpec and a.rope.kind == "rope" and a.rope.tables
                                       and (a.rope.layout == "interleaved" or a.rope.rotary_dim == a.head_dim)):
            return None
        if a.hidden != hidden or f.hidden != hidden or f.bias_suffix or hidden % 8 or not 64 <= hidden <= 32768:
            return None
        if f.intermediate % 8 or f.intermediate < 64 or a.head_dim % 16 or not 16 <= a.head_dim <= 128 or a.num_heads * a.head_dim < 64:
            return None
        gemm_ex = _library_product()
        return DenseLayers(layers, gemm_ex) if gemm_ex is not None else None

    def takes(self, ctx: StepContext, caches: List[Optional[LayerCache]]) -> bool:
        if not (ENABLED and kernels.vectorized and gemm_backend._enabled and attention_backend._enabled and attention_backend.PREFILL_TC
                and attention_backend.DECODE_TC) or gemm_backend.FUSE_EPILOGUES or tracing.ENABLED \
                or not _torch_calls_the_library():
            return False
        c0, s = caches[0], self.layers[0][1].spec
        if any(c is None or c.group != c0.group or c["k"].shape != c0["k"].shape for c in caches):
            return False
        plan = attention_backend._plan(ctx, s.head_dim)
        return ((not plan["tiles"] or attention_backend.prefill_tc_takes(s.head_dim, c0.page_size))
                and (not plan["small"] or self._decode_plan(ctx, c0, True) is not None))

    def _decode_plan(self, ctx, cache, early):
        s = self.layers[0][1].spec
        return attention_backend._decode_plan(ctx, s.num_heads, s.num_kv_heads, s.head_dim, cache.page_size, s.window,
                                              ctx.strides[cache.group], early=early)

    def forward(self, x: torch.Tensor, ctx: StepContext, caches: List[LayerCache]) -> torch.Tensor:
        """``x`` ``[T, hidden]`` goes through all layers in place; returns the last branch, which is still to be added to it.
        ``takes`` has been asked first, before the step's first kernel."""
        n1, attn, n2, ff = self.layers[0]
        s, f, ws, T, hidden = attn.spec, ff.spec, ctx.workspace, x.shape[0], x.shape[1]
        nh, nkv, d, bf = s.num_heads, s.num_kv_heads, s.head_dim, torch.bfloat16
        c0 = caches[0]
        num_pages, _, page_size, _ = c0["k"].shape
        rot = attn.position.rotary() if attn.position is not None else None
        plan = attention_backend._plan(ctx, d)
        # (the parts' own buffers)
        bufs = dict(x=x, h=ws.get("block.h", (T, hidden), bf), qkv=ws.get("attn.qkv", (T, (nh + 2 * nkv) * d), bf),
                    q=ws.get("attn.q", (T, nh, d), bf), o=ws.get("attn.o", (T, nh, d), bf), attn_out=ws.get("attn.out", (T, hidden), bf),
                    gate_up=ws.get(ff.scratch + ".gate_up", (T, 2 * f.intermediate), bf), act=ws.get(ff.scratch + ".act", (T, f.intermediate), bf),
                    ffn_out=ws.get(ff.scratch + ".out", (T, hidden), bf), positions=ctx.positions, req_of_token=ctx.req_of_token,
                    table=ctx.tables[c0.group], q_start=ctx.q_start, start_pos=ctx.start_pos, err=ctx.err)
        nums = dict(prefill_ctas=0, decode_ctas=0, splits_max=0, small=0, overlap=0)
        if rot is not None:
            bufs.update(cos_t=rot.cos, sin_t=rot.sin)
        if plan["tiles"]:
            bufs["work"], nums["prefill_ctas"], _ = attention_backend._prefill_work(ctx, nh, nkv, s.window)
        if plan["small"]:
            small = plan["small"]
            bufs["plan"], nums["decode_ctas"], splits, overlap = self._decode_plan(ctx, c0, False)
            nums.update(splits_max=splits, small=small, overlap=int(overlap))
            if splits > 1:
                bufs.update(part_o=ws.get("attn.part_o", (small * nh * splits * d,), torch.float32),
                            part_ml=ws.get("attn.part_ml", (small * nh * splits * 2,), torch.float32),
                            tickets=ws.get("attn.tickets", (small * nkv * ((nh // nkv + 15) // 16),), torch.int32))
        act, p0, p1 = kernels.activation_args(f.activation, f.act_params)
        nums.update(tokens=T, hidden=hidden, nh=nh, nkv=nkv, d=d, inter=f.intermediate, table_stride=ctx.strides[c0.group], page_size=page_size,
                    num_pages=num_pages, max_pos=rot.cos.shape[0] if rot else 0, rot=rot.rotary_dim if rot else 0,
                    interleaved=int(rot.interleaved) if rot else 0, window=int(s.window or 0), dec_max=attention_backend.DEC_MAX,
                    skinny=gemm_backend.SKINNY_MAX_TOKENS, many_rows=kernels.many_rows, activation=act)
        reals = dict(eps1=n1.spec.eps, offset1=n1.spec.weight_offset, eps2=n2.spec.eps, offset2=n2.spec.weight_offset, qk_eps=s.qk_norm_eps,
                     scale=s.scale, p0=p0, p1=p1)
        library = dict(gemm_ex=self.gemm_ex, blas=torch.cuda.current_blas_handle())
        table = [dict(w_qkv=a.w_qkv, w_o=a.w_o, w_gate_up=g.w_gate_up, w_down=g.w_down, norm1=p.weight, norm2=q.weight, q_norm=a.q_norm,
                      k_norm=a.k_norm, k_pages=c["k"], v_pages=c["v"]) for (p, a, q, g), c in zip(self.layers, caches)]
        kernels.dense_layers(bufs, nums, reals, library, table, lambda i: attention_backend.attend(
            bufs["o"], bufs["q"], caches[i], ctx, bufs["table"], nums["table_stride"], s.window, s.scale))
        return bufs["ffn_out"]
