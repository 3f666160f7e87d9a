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
    def sms(layers: int, n_stu: int, B: int, d: int, t: int, weight_bytes: int, ring_bytes: int, sm_count: int) -> int:
        """SMs for the streams of steps up to position t; 0 where the layers' own kernels are as good.
        An SM streams about 80 GB/s (10 of them, 12 layers of 32 x 1536 at 2048, 4000 and 7900: 2183, 3379 and 6277 us), in slices of 256
        positions with an eighth of taps beside them.  The rest of a step takes about 18 us a layer, its weights 2.8 TB/s and its keys
        and values 5.5 (24 layers of 1536 and 32 sequences 1515 us, measured 1530; 24 of 512: 552, 632; 12 of 1024: 520, 580).  The streams
        get the SMs that finish them in 0.6 of that: fewer and the step waits for them (2048: 14 SMs 1671 us, 18 to 26 1534 to 1650, 32 and
        more 1539 to 1630; without 1708 to 1720), more and the chain misses them (64 sequences at 3000: 26 SMs 2336, 50 2556, without
        2774), a third of the GPU at most (32 at 7900: 40 1954, 50 2036, 32 2334, without 2278).
        Beside the chain a layer saves its stream at 4.5 TB/s and 2 us, the second branch costs about 8 (2 layers of 512, 16 sequences at 300:
        146 us without, 152 with)."""
        stream = n_stu * B * d * ((t // 2 + 255) // 256 * 256) * 2 * 1.125
        if stream / 4.5e12 + n_stu * 2e-6 <= 8e-6:
            return 0
        rest = 18e-6 * layers + weight_bytes / 2.8e12 + ring_bytes / 5.5e12
        return max(8, min(sm_count // 3, int(stream / (80e9 * 0.6 * rest)) + 1))

    @classmethod
    def plan(cls, layers, past, B: int, last: int, weight_bytes: int):
        """The buffers for steps from here to position `last`, or None."""
        if not cls.supported(layers, past, B):
            return None
        self = cls(layers, past, B)
        ring = sum(2 * e[0].numel() * e[0].element_size() * min(last, e[0].shape[1]) // e[0].shape[1] for e in past if e is not None and len(e) == 3)
        device = self.part.device
        self.n = cls.sms(len(layers), len(self.entries), B, self.part.shape[3], last, weight_bytes, ring, _sm_count(device))
        return self if self.n else None

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

    def check(self):
        """Raises when a launch of the sums has given up on a wait: the steps from the position behind it on wrote nothing.  Waits for
        the steps so far."""
        if int(self.ctl[2:].min()) < 0:   # (a half that holds no position stays so)
            ops.check_status(self.part.device)
            raise RuntimeError(f"flash_stu_2_b200 device status 8: {ops.STATUS_TEXT[8]}")
