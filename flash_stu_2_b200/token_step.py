"""Host side of the persistent token-step kernel (csrc/token_step.cu): the descriptors of a stack of layers and its
caches, built once and launched once per token."""
import ctypes
from typing import Optional, Sequence

import torch

from . import _lib, ops
from .layers import AttentionLayer, STULayer
from .modules import host_pos, uniform_pos


def layer_supported(layer) -> bool:
    """Whether a layer's token step is one the kernel computes: a plain approx STU layer or an attention layer, whose
    forward() nobody overrides or listens to."""
    if type(layer) not in (STULayer, AttentionLayer) or "forward" in vars(layer) or layer._forward_hooks or layer._forward_pre_hooks:
        return False
    if hasattr(layer, "stu"):
        return layer.stu.use_approx and not layer.stu.use_hankel_L and not layer.stu_mlp_enabled
    return hasattr(layer, "attn")


def layer_weights(layer, d: int, inter: int):
    """(field of the descriptor, tensor, shape) of the weights that the kernel reads of a layer (an STU layer's M_inputs it
    reads as the derived transpose: no field)."""
    mlp = layer.mlp
    out = [("norm2", layer.mlp_norm.weight, (d,)), ("wg", mlp.gate_proj.weight, (inter, d)),
           ("wu", mlp.up_proj.weight, (inter, d)), ("wd", mlp.down_proj.weight, (d, inter))]
    if hasattr(layer, "stu"):
        return out + [("norm1", layer.stu_norm.weight, (d,)), (None, layer.stu.M_inputs, (d, d))]
    return out + [("norm1", layer.attn_norm.weight, (d,)), ("w1", layer.attn.c_attn.weight, (3 * d, d)),
                  ("wo", layer.attn.c_proj.weight, (d, d))]


def model_weights(model, d: int):
    """The same for the embedding, the final norm and the LM head."""
    head = model.lm_head.weight
    return [("embedding", model.tok_emb.weight, (head.shape[0], d)), ("norm_final", model.norm.weight, (d,)),
            ("lm_head", head, (head.shape[0], d))]


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
        inter = layers[0].mlp.intermediate_size
        for L, layer, entry in zip(table, layers, past):
            for field, w, _ in layer_weights(layer, d, inter):
                keep.append(w)   # (a parametrised weight is a new tensor at every look-up)
                if field:
                    setattr(L, field, w.data_ptr())
            L.eps2, L.pos = layer.mlp_norm.eps, entry[-1].data_ptr()
            if hasattr(layer, "stu"):
                MinT, taps, taps8 = layer.stu.prepared()
                keep += [MinT, taps, taps8]
                L.kind, L.Lh = 0, entry[0].shape[3]
                L.eps1, L.w1, L.hist = layer.stu_norm.eps, MinT.data_ptr(), entry[0].data_ptr()
                L.taps = (taps8 if self.dtype == torch.bfloat16 else taps).data_ptr()
            else:
                attn = layer.attn
                heads, window, softcap = attn.n_heads, attn.window, float(attn.softcap or 0.0)
                L.kind, L.W, L.eps1 = 1, entry[0].shape[1], layer.attn_norm.eps
                L.k_ring, L.v_ring, L.slopes = entry[0].data_ptr(), entry[1].data_ptr(), attn.alibi_slopes.data_ptr()
        code = 1 if self.dtype == torch.bfloat16 else 0
        nbytes = lib.stu_token_step_workspace_bytes(d, inter, heads, code)
        ws = torch.zeros(nbytes, dtype=torch.uint8, device=self.device)
        a = self.args = _lib.StepArgs()
        a.n_layers, a.B, a.d, a.I, a.H, a.window, a.softcap = len(layers), batch, d, inter, heads, window, softcap
        a.x, a.workspace, a.workspace_bytes = x.data_ptr(), ws.data_ptr(), nbytes
        a.status = ops.status_word(self.device).data_ptr()
        if model is not None:
            a.V = model.lm_head.weight.shape[0]
            for field, w, _ in model_weights(model, d):
                keep.append(w)
                setattr(a, field, w.data_ptr())
            a.eps_final = model.norm.eps
        blob = (ctypes.c_uint8 * lib.stu_token_step_plan_bytes(len(layers)))()
        self.n_stages = lib.stu_token_step_plan(ctypes.addressof(table), ctypes.addressof(a), code, ctypes.addressof(blob))
        _lib.check(min(self.n_stages, 0), "stu_token_step_plan")
        self.plan = torch.frombuffer(blob, dtype=torch.uint8).to(self.device)
        self._ws, self._keep = ws, keep

    @staticmethod
    def supported(layers: Sequence, past: Sequence, batch: int, d: int, dtype: torch.dtype, model=None) -> bool:
        """Whether the kernel takes these layers and caches (and the model's embedding and head) as they are: whatever it
        has no form of is the per-layer kernels' work."""
        if batch > 8 or len(layers) > _lib.STEP_MAX_LAYERS or dtype not in (torch.bfloat16, torch.float32):
            return False
        if any(e is None for e in past) or not all(layer_supported(layer) for layer in layers):
            return False
        t = host_pos(past[0][-1])
        if any(host_pos(e[-1]) != t or not uniform_pos(e[-1]) for e in past):
            return False
        inter = layers[0].mlp.intermediate_size
        attn = [layer.attn for layer in layers if hasattr(layer, "attn")]
        if any((a.n_heads, a.window, a.softcap) != (attn[0].n_heads, attn[0].window, attn[0].softcap) for a in attn):
            return False
        if model is not None and model.lm_head.weight.shape[0] >= 1 << 24:
            return False
        weights = [w for layer in layers for w in layer_weights(layer, d, inter)] + (model_weights(model, d) if model else [])
        if any(w.dtype != dtype or tuple(w.shape) != shape for _, w, shape in weights):
            return False
        if any(field and (not w.is_contiguous() or w.data_ptr() % 16) for field, w, _ in weights):
            return False
        return bool(_lib.load().stu_token_step_supported(len(layers), batch, d, inter, attn[0].n_heads if attn else 0,
                                                         1 if dtype == torch.bfloat16 else 0))

    @staticmethod
    def pays(layers: Sequence, batch: int, d: int, dtype: torch.dtype, t: int, steps: int) -> bool:
        """Whether `steps` steps from position t on take less time as persistent launches than replayed from a graph.

        A layer's part of the persistent step beyond (below zero: less than) its kernels', in microseconds, fitted to 257 pairs
        of models of 4 to 24 layers, 280 MB of weights and more, on one B200 (d 256 to 3072, 1 to 8 sequences, positions 100 to
        12000).  The tap sums over the history are what decides: the persistent
        kernel takes them at 2 TB/s (fp32: 1), the decode kernels at 5 and more.  us per step, persistent and graph: bf16, STU
        layers only, 10 of d = 1024, 1 sequence at 1100 183 and 189, 8 sequences at 3000 394 and 225; 6 of d = 1536, 1 sequence at
        100 148 and 206, 8 at 4000 397 and 319; with attention, 6 layers of d = 1536 at 400, 1 and 8 sequences 183 and 237, 296 and 311;
        fp32, 8 layers of d = 512 with 6144 hidden values, 2 and 8 sequences 207 and 247, 398 and 307.
        Below two units of 16 rows in the weight ring the stream stops between units: d = 3072, 1 sequence, 4 layers 359 and 348;
        fp32 d = 1536, 1 sequence 196 and 264, 4 sequences 297 and 286.
        Against that a graph's two eager steps, capture and instantiation cost 1.2 ms and 0.12 ms per layer on an idle
        host, but 20 to 170 ms in one call of ten on a busy one, where the persistent steps take what they always take
        (14 layers of d = 512, 54 steps: 21 to 173 ms against 20): four times the former is what it has to gain.  Counting that,
        the pairs lose 1.0 % against the better choice over 30 to 1500 steps (2.6 % with the lines fitted to the kernel before)."""
        bf16, inter = dtype == torch.bfloat16, layers[0].mlp.intermediate_size
        if _lib.load().stu_token_step_ring_slots(batch, d, inter, int(bf16)) < 31 and (bf16 or batch > 2):
            return False
        mid, many = t + steps // 2, batch > 4   # (more than four sequences: another instance of the kernel)
        beyond = 0.0
        for layer in layers:
            if hasattr(layer, "stu"):
                history = batch * d * (mid // 2) * (2e-6 if bf16 else 4e-6)   # MB
                if bf16:   # (the block step kernel is the hard one to beat)
                    beyond += 0.5 * history
                    beyond += 0.14 * batch + 1.4 * many if d <= 1024 and inter <= 4096 else \
                        -3 + 0.7 * batch + 2 * many - 0.021 * max(d - 1000, 0)
                else:
                    beyond += 4 - 0.022 * d + 0.5 * batch + 0.0008 * many * inter + 0.8 * (1 + 1 / batch) * history
            else:
                keys = min(mid, layer.attn.window + 1, 1025)
                if bf16:
                    beyond += 1.4 + 0.7 * batch + 6 * many - 0.023 * keys if d <= 1024 else -1.6 + 0.85 * batch + 3.5 * many - 0.01 * keys
                else:
                    beyond += 3.3 + 0.7 * batch + 0.0017 * many * inter - 0.0055 * d - 0.036 * keys + 2.6e-6 * batch * keys * d
        return beyond * steps < 4 * (1200 + 120 * len(layers))

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
