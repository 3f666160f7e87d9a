"""Host side of the persistent token-step kernel (csrc/token_step.cu): the descriptors of a stack of layers and its
caches, built once and launched once per token."""
import ctypes
from typing import Optional, Sequence

import torch

from . import _lib, ops
from .modules import host_pos, uniform_pos


def layer_supported(layer) -> bool:
    """Whether a layer's token step is one the kernel computes: a plain approx STU layer or an attention layer."""
    if hasattr(layer, "stu"):
        return layer.stu.use_approx and not layer.stu.use_hankel_L and not layer.stu_mlp_enabled
    return hasattr(layer, "attn")


class TokenStep:
    """The step of `layers` on the cache entries `past` (one per layer, all at one position).  run() advances the caches
    by one token; the object keeps every tensor that the descriptors point to."""

    def __init__(self, layers: Sequence, past: Sequence, batch: int, x: torch.Tensor, model=None):
        self.dtype, self.device = x.dtype, x.device
        lib = _lib.load()
        table = (_lib.StepLayer * len(layers))()
        self.pos = [entry[-1] for entry in past]
        keep = [x, past]
        d = x.shape[-1]
        heads = window = 0
        softcap = 0.0
        for L, layer, entry in zip(table, layers, past):
            mlp = layer.mlp
            L.norm2, L.eps2 = layer.mlp_norm.weight.data_ptr(), layer.mlp_norm.eps
            L.wg, L.wu, L.wd = (m.weight.data_ptr() for m in (mlp.gate_proj, mlp.up_proj, mlp.down_proj))
            L.pos = entry[-1].data_ptr()
            if hasattr(layer, "stu"):
                MinT, taps, taps8 = layer.stu.prepared()
                keep += [MinT, taps, taps8]
                L.kind, L.Lh = 0, entry[0].shape[3]
                L.norm1, L.eps1 = layer.stu_norm.weight.data_ptr(), layer.stu_norm.eps
                L.w1, L.hist = MinT.data_ptr(), entry[0].data_ptr()
                L.taps = (taps8 if self.dtype == torch.bfloat16 else taps).data_ptr()
            else:
                attn = layer.attn
                heads, window, softcap = attn.n_heads, attn.window, float(attn.softcap or 0.0)
                L.kind, L.W = 1, entry[0].shape[1]
                L.norm1, L.eps1 = layer.attn_norm.weight.data_ptr(), layer.attn_norm.eps
                L.w1, L.wo = attn.c_attn.weight.data_ptr(), attn.c_proj.weight.data_ptr()
                L.k_ring, L.v_ring, L.slopes = entry[0].data_ptr(), entry[1].data_ptr(), attn.alibi_slopes.data_ptr()
        inter = layers[0].mlp.intermediate_size
        code = 1 if self.dtype == torch.bfloat16 else 0
        nbytes = lib.stu_token_step_workspace_bytes(d, inter, heads, code)
        ws = torch.zeros(nbytes, dtype=torch.uint8, device=self.device)
        a = self.args = _lib.StepArgs()
        a.n_layers, a.B, a.d, a.I, a.H, a.window, a.softcap = len(layers), batch, d, inter, heads, window, softcap
        a.x, a.workspace, a.workspace_bytes = x.data_ptr(), ws.data_ptr(), nbytes
        a.status = ops.status_word(self.device).data_ptr()
        if model is not None:
            a.V = model.lm_head.weight.shape[0]
            a.embedding, a.lm_head = model.tok_emb.weight.data_ptr(), model.lm_head.weight.data_ptr()
            a.norm_final, a.eps_final = model.norm.weight.data_ptr(), model.norm.eps
        blob = (ctypes.c_uint8 * lib.stu_token_step_plan_bytes(len(layers)))()
        self.n_stages = lib.stu_token_step_plan(ctypes.addressof(table), ctypes.addressof(a), code, ctypes.addressof(blob))
        _lib.check(min(self.n_stages, 0), "stu_token_step_plan")
        self.plan = torch.frombuffer(blob, dtype=torch.uint8).to(self.device)
        self._ws, self._keep = ws, keep

    @staticmethod
    def supported(layers: Sequence, past: Sequence, batch: int, d: int, dtype: torch.dtype) -> bool:
        if batch > 8 or len(layers) > _lib.STEP_MAX_LAYERS or dtype not in (torch.bfloat16, torch.float32):
            return False
        if any(e is None for e in past) or not all(layer_supported(layer) for layer in layers):
            return False
        t = host_pos(past[0][-1])
        if any(host_pos(e[-1]) != t or not uniform_pos(e[-1]) for e in past):
            return False
        inter = layers[0].mlp.intermediate_size
        heads = {layer.attn.n_heads for layer in layers if hasattr(layer, "attn")}
        if len(heads) > 1 or any(layer.mlp.intermediate_size != inter for layer in layers):
            return False
        params = [p for layer in layers for p in layer.parameters()]
        if any(p.dtype != dtype or not p.is_contiguous() for p in params):
            return False
        return bool(_lib.load().stu_token_step_supported(len(layers), batch, d, inter, max(heads, default=0),
                                                         1 if dtype == torch.bfloat16 else 0))

    def run(self, ids: Optional[torch.Tensor] = None, logits: Optional[torch.Tensor] = None):
        """One token per sequence: ids [B] int64 (any stride; None: the rows are in x), logits [B,V] rows."""
        a = self.args
        if ids is not None:
            a.ids, a.ids_stride = ids.data_ptr(), ids.stride(0)
        if logits is not None:
            a.logits, a.ld_logits = logits.data_ptr(), logits.stride(0)
        ops.token_step(self.plan, self.n_stages, a, self.dtype == torch.bfloat16)
        for p in self.pos:
            p._host_t += 1

    def check(self):
        """Raises when a step has given up on a wait (the steps after it then did nothing).  Waits for the steps so far."""
        if int(self._ws[4:8].view(torch.int32)):
            ops.check_status(self.device)
            raise RuntimeError(f"flash_stu_2_b200 device status 12: {ops.STATUS_TEXT[12]}")
