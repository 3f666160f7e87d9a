"""Host side of the persistent token-step kernel: its plan and the walk of its weight stream, without a GPU."""
import ctypes

import pytest

from flash_stu_2_b200 import _lib

A = 1 << 20   # stands for an aligned device address: nothing here dereferences it


def _plan(d, inter, B, heads, bf16, V=50257, layers=4):
    """(args, plan in host memory, number of stages or the refusal) of a stack that alternates STU and attention layers."""
    lib, code = _lib.load(), int(bf16)
    table, a = (_lib.StepLayer * layers)(), _lib.StepArgs()
    for i, L in enumerate(table):
        for name in ("norm1", "w1", "wo", "norm2", "wg", "wu", "wd", "hist", "taps", "k_ring", "v_ring", "slopes", "pos"):
            setattr(L, name, A)
        L.kind, L.Lh, L.W = int(heads > 0 and i % 2 == 1), 64, 9
    a.n_layers, a.B, a.d, a.I, a.H, a.window, a.V = layers, B, d, inter, heads, 8, V
    a.x = a.embedding = a.norm_final = a.lm_head = a.logits = a.workspace = A
    blob = (ctypes.c_uint8 * lib.stu_token_step_plan_bytes(layers))()
    n = lib.stu_token_step_plan(ctypes.addressof(table), ctypes.addressof(a), code, ctypes.addressof(blob))
    return a, blob, n


def _stall(d, inter, B, heads, bf16):
    a, blob, n = _plan(d, inter, B, heads, bf16)
    assert n > 0
    return _lib.load().stu_token_step_walk(ctypes.addressof(blob), n, ctypes.addressof(a), int(bf16))


@pytest.mark.parametrize("bf16", [True, False])
@pytest.mark.parametrize("B", [1, 2, 3, 5, 8])
def test_weight_stream_never_waits_for_itself(bf16, B):
    """Every width and hidden size that the kernel accepts: the producer finds room for each unit of every CTA once what was
    issued before it is released (rings of few slots and units that skip to slot 0 are where it might not)."""
    lib, accepted = _lib.load(), 0
    step = 64 if B in (1, 8) else 192
    for d in range(step, 4097, step):
        for inter in [m * d for m in (1, 2, 3, 4, 6, 8, 12)] + [d // 2, d + 64, 3 * d + 16]:
            heads = d // 64
            if lib.stu_token_step_supported(4, B, d, inter, heads, int(bf16)):
                accepted += 1
                assert _stall(d, inter, B, heads, bf16) == 0, (d, inter)
    assert accepted > 20


@pytest.mark.parametrize("d,mlp,B,heads,bf16", [(3072, 4, 1, 24, True), (2560, 4, 3, 40, True), (2304, 4, 3, 36, True),
                                                (1536, 4, 1, 12, False), (1536, 12, 1, 12, False)])
def test_weight_stream_of_rings_of_24_to_30_slots(d, mlp, B, heads, bf16):
    if _lib.load().stu_token_step_supported(4, B, d, mlp * d, heads, int(bf16)):
        assert _stall(d, mlp * d, B, heads, bf16) == 0
