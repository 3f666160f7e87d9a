"""The history streams of a captured token step beside its chain (csrc/stu_stream_ahead.cu).

A model's token step is a chain of small dependent products, which leaves HBM idle most of the time, and of its STU layers' history
streams, which need nothing of the step that they run in: position t + 1 reads the other time parity than position t writes.  A
step that is captured for replay therefore computes the sums of ALL its STU layers for the position after it as one launch on a second
branch of the graph, on a few SMs, and in the chain adds the new token's own term to what the step before left."""
import torch

from . import ops
from .layers import STULayer
from .modules import STU, _sm_count, host_pos, own, uniform_pos

MAX_LAYERS = 64


class StreamAhead:
    """Buffers and size of one captured step; they belong to the graph that was captured with them."""

    enabled = True   # class switch used by tests to compare the two forms of the step

    def __init__(self, layers, past, B: int):
        self.entries = [(layer.stu, e) for layer, e in zip(layers, past) if hasattr(layer, "stu")]
        hist, pos = self.entries[0][1]
        self.t = host_pos(pos)
        self.part = torch.empty(len(self.entries), 2, B, hist.shape[1], dtype=torch.float32, device=hist.device)
        # (filled on the device: a copy from the host would wait for the prefill that is still running)
        self.ctl = torch.empty(4, dtype=torch.int32, device=hist.device)
        for i, v in enumerate((self.t, 0, self.t - 2 + self.t % 2, self.t - 1 - self.t % 2)):
            self.ctl[i].fill_(v)
        self.stream = torch.cuda.Stream(hist.device)

    @staticmethod
    def supported(layers, past, B: int) -> bool:
        """bf16 approx layers of one size at one position, where the token's projection is a GEMM of its own and nobody overrides the
        steps that this form of it takes the place of."""
        stus = [(layer, e) for layer, e in zip(layers, past) if hasattr(layer, "stu")]
        if not stus or len(stus) > MAX_LAYERS or B < STU.projected_decode_min_batch or not StreamAhead.enabled:
            return False
        if any(e is None for _, e in stus) or not (STU.pipelined_decode and STU.tensor_core_decode and STU.shared_tap_decode):
            return False
        shape, t = stus[0][1][0].shape, host_pos(stus[0][1][1])
        for layer, (hist, pos) in stus:
            stu = layer.stu
            if not (own(layer, STULayer, "forward", "_decode") and own(stu, STU, "decode_step")):
                return False
            if (layer.stu_mlp_enabled or not stu.use_approx or stu.use_hankel_L or hist.dtype != torch.bfloat16 or hist.shape != shape
                    or not hist.is_contiguous() or not uniform_pos(pos) or host_pos(pos) != t or hist.shape[1] % 8 or hist.shape[1] > 4096
                    or stu.prepared()[2] is None):
                return False
        return True

    @staticmethod
    def sms(layers: int, n_stu: int, B: int, d: int, t: int, weight_bytes: int, ring_bytes: int, sm_count: int, norm_apart: bool = True) -> int:
        """SMs for the streams of steps up to position t; 0 where the layers' own kernels are as good.
        Beside a chain an SM streams 45 to 60 GB/s (16, 20, 24, 28 and 32 of them, 12 layers of 32 x 1536 at 7000: 4788, 3818, 3265, 2809 and 2500 us
        a step), in slices of 256 positions with an eighth of taps beside them.  The rest of a step takes about 18 us a layer, its weights
        2.8 TB/s (from 1536 channels on more: 4.5 at 2400) and its keys and values 5.5.  The streams get the SMs that finish them well within that
        time: too few and the step waits for them (6 layers of 3072, 16 sequences at 3000, 8, 11, 14, 20 and 29 SMs: 1131, 737, 631, 679, 665 us, without
        712), too many and the chain misses them.  Up to 64 sequences its linears are clusters of up to 16 CTAs, which find no room between
        more than a fifth of the SMs (us, medians of 5 captures, without and with 16, 20, 24, 28, 32, 36, 40: 24 layers of 1536, 32 sequences at 2000 1794:
        1600, 1636, 1738, 1759, 1796, 1836, 2067; at 3000 1951: 2203, 1824, 1855, 1919, 1914, 2047, 2353; 64 at 3000 3096: 4498, 3519, 3040, 2819, 3039, 4073, 3860);
        from 65 on they are pairs, which leave a third (8 layers of 1536, 96 at 3000 1365: 32 1147, 40 1035, 49 1078).  Streams that these cannot
        finish ahead of the step's end are left to the layers (32 at 7000: 2452).
        Beside the chain a layer saves its stream at 4.5 TB/s and, where the norm behind it is a launch of its own, 2 us; the second branch costs
        about 8 (12 layers of 256, 16 sequences at 200: 215 us without, 219 with; at 1000 228 and 224)."""
        stream = n_stu * B * d * ((t // 2 + 255) // 256 * 256) * 2 * 1.125
        saved = stream / 4.5e12 + n_stu * (2e-6 if norm_apart else 0.5e-6)
        if saved <= 8e-6:
            return 0
        rest = 18e-6 * layers + weight_bytes / max(2.8e12, min(4.5e12, 1.9e9 * d)) + ring_bytes / 5.5e12
        n = max(8, min(sm_count // (5 if B <= 64 else 3), int(stream / (48e9 * rest)) + 1))
        return n if stream / (60e9 * n) < 0.97 * (rest + saved) else 0

    @classmethod
    def plan(cls, layers, past, B: int, last: int, weight_bytes: int):
        """The buffers for steps from here to position `last`, or None."""
        if not cls.supported(layers, past, B):
            return None
        ring = sum(2 * e[0].numel() * e[0].element_size() * min(last, e[0].shape[1]) // e[0].shape[1] for e in past if e is not None and len(e) == 3)
        stus = [(layer, e) for layer, e in zip(layers, past) if hasattr(layer, "stu")]
        hist, d = stus[0][1][0], stus[0][1][0].shape[1]
        apart = not all(ops.can_fuse_norm(B, layer.mlp.intermediate_size, d, ops.EPI_GELU_MUL, hist.dtype) for layer, _ in stus)
        n = cls.sms(len(layers), len(stus), B, d, last, weight_bytes, ring, _sm_count(hist.device), apart)
        if not n:
            return None
        self = cls(layers, past, B)
        self.n = n
        return self

    def launch(self, sms: int):
        ops.stream_ahead([e[0] for _, e in self.entries], [stu.prepared()[2] for stu, _ in self.entries], self.part, self.ctl, sms)

    def __enter__(self):
        """The sums of the first position, on the whole GPU; the layers then find theirs while the step is captured."""
        self.launch(_sm_count(self.part.device))
        for i, (_, (_, pos)) in enumerate(self.entries):
            pos._stream_ahead = (self.part[i], self.ctl)
        return self

    def __exit__(self, *exc):
        for _, (_, pos) in self.entries:
            del pos._stream_ahead

    def branch(self, stream):
        """In a capture on `stream`: the sums of the position after this step, on a branch that begins here."""
        self.stream.wait_stream(stream)
        with torch.cuda.stream(self.stream):
            self.launch(self.n)

    def join(self, stream):
        stream.wait_stream(self.stream)

    def note(self):
        """Behind the last step but one: the sums that the last one needs are there or will not be."""
        self.noted = torch.empty(4, dtype=torch.int32, pin_memory=True).copy_(self.ctl, non_blocking=True)
        self.at = torch.cuda.Event()
        self.at.record()

    def check(self):
        """Raises when a launch of the sums has given up on a wait: the steps from the position behind it on wrote nothing.  Waits for
        the steps up to note() (a call behind this one is prepared while the last one runs)."""
        self.at.synchronize()
        if min(self.noted[2:].tolist()) < 0:   # (a half that holds no position stays so)
            ops.check_status(self.part.device)
            raise RuntimeError(f"flash_stu_2_b200 device status 8: {ops.STATUS_TEXT[8]}")
