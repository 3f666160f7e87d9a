"""Host side of the persistent token-step kernel: its plan and the walk of its weight stream, without a GPU."""
import ctypes
import os
import re

import pytest
import torch

import flash_stu_2_b200 as F
from flash_stu_2_b200 import _lib
from flash_stu_2_b200.layers import STULayer
from flash_stu_2_b200.modules import STU
from flash_stu_2_b200.stream_ahead import StreamAhead
from flash_stu_2_b200.token_step import TokenStep

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


def test_descriptors_of_the_binding_have_the_layout_of_the_header():
    """What the binding fills in is what the library copies out of it: sizes, and one field from each end."""
    lib = _lib.load()
    stages = 5 * 32
    assert lib.stu_token_step_plan_bytes(2) - lib.stu_token_step_plan_bytes(1) - stages == ctypes.sizeof(_lib.StepLayer) == 128
    a, blob, n = _plan(512, 2048, 2, 8, True)
    table = (_lib.StepLayer * 4).from_buffer_copy(bytes(blob)[n * 32:n * 32 + 4 * 128])
    assert [L.kind for L in table] == [0, 1, 0, 1] and all(L.Lh == 64 and L.W == 9 and L.norm1 == L.pos == A for L in table)
    assert _lib.StepArgs.status.offset == ctypes.sizeof(_lib.StepArgs) - 8 == 120


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


def _model(dt=torch.float32, **kw):
    cfg = F.FlashSTUConfig(n_embd=64, n_layers=4, n_heads=2, seq_len=64, window_size=8, vocab_size=97, mlp_scale=4, num_eigh=8,
                           torch_dtype=dt, **kw)
    return F.FlashSTU(cfg).eval()


def _takes(m, batch=2):
    past = [(l.stu if hasattr(l, "stu") else l.attn).new_cache(batch, "cpu") for l in m.layers]
    return TokenStep.supported(m.layers, past, batch, 64, m.config.torch_dtype, m)


def _off_the_grid(w):
    return torch.nn.Parameter(torch.zeros(w.numel() + 1, dtype=w.dtype)[1:].view(w.shape))


def _narrow_mlp(m):
    m.layers[2].mlp.gate_proj = torch.nn.Linear(64, 200, bias=False)
    m.layers[2].mlp.up_proj = torch.nn.Linear(64, 200, bias=False)
    m.layers[2].mlp.down_proj = torch.nn.Linear(200, 64, bias=False)


@pytest.mark.parametrize("change", [
    lambda m: setattr(m.layers[1].attn.c_attn, "weight", _off_the_grid(m.layers[1].attn.c_attn.weight)),
    lambda m: setattr(m.layers[0].stu_norm, "weight", _off_the_grid(m.layers[0].stu_norm.weight)),
    lambda m: setattr(m.lm_head, "weight", _off_the_grid(m.lm_head.weight)),
    lambda m: setattr(m.tok_emb, "weight", _off_the_grid(m.tok_emb.weight)),
    lambda m: setattr(m.norm, "weight", _off_the_grid(m.norm.weight)),
    lambda m: setattr(m.lm_head, "weight", torch.nn.Parameter(m.lm_head.weight.bfloat16())),
    lambda m: setattr(m.tok_emb, "weight", torch.nn.Parameter(torch.zeros(90, 64))),
    lambda m: setattr(m.lm_head, "weight", torch.nn.Parameter(torch.zeros(64, 97).t())),
    lambda m: setattr(m.layers[3].attn, "softcap", 7.0), lambda m: setattr(m.layers[3].attn, "window", 5), _narrow_mlp])
def test_models_that_the_kernel_has_no_form_of_are_left_to_the_per_layer_kernels(change):
    """Weights off the 16-byte grid, of another dtype or shape than the configuration's, attention layers that differ."""
    m = _model()
    assert _takes(m)
    with torch.no_grad():
        change(m)
    assert not _takes(m)


def _own_forward(m):
    layer = m.layers[2]
    layer.forward = lambda *a, **kw: type(layer).forward(layer, *a, **kw)


def _subclass(m):
    m.layers[1].__class__ = type("Layer", (type(m.layers[1]),), {})


@pytest.mark.parametrize("change", [lambda m: m.layers[0].register_forward_hook(lambda *a: None), _own_forward, _subclass,
                                    lambda m: m.layers[3].register_forward_pre_hook(lambda *a: None)])
def test_layers_that_somebody_overrides_or_listens_to_are_called(change):
    m = _model()
    assert _takes(m)
    change(m)
    assert not _takes(m)


@pytest.mark.parametrize("d,layers,heads,mlp,dt,B,t,steps,attn,want", [
    (1024, 4, 16, 4, torch.bfloat16, 8, 12000, 64, False, False),    # a long history: the decode kernels stream it faster
    (1024, 4, 16, 4, torch.bfloat16, 8, 100, 1000, False, False),    # the block step kernel, the capture long paid for
    (1024, 4, 16, 4, torch.bfloat16, 8, 100, 12, False, True),       # ... and not
    (1536, 24, 12, 4, torch.bfloat16, 1, 333, 64, True, True), (1536, 4, 12, 4, torch.bfloat16, 8, 12000, 64, False, False),
    (512, 12, 8, 12, torch.float32, 2, 128, 127, True, True), (512, 4, 8, 4, torch.float32, 8, 4000, 64, False, False),
    (3072, 4, 24, 4, torch.bfloat16, 1, 100, 64, True, False), (1536, 4, 24, 4, torch.float32, 4, 100, 64, True, False)])
def test_form_of_the_step_follows_what_was_measured(d, layers, heads, mlp, dt, B, t, steps, attn, want):
    class Attn:
        n_heads, window = heads, 1024

    class Mlp:
        intermediate_size = mlp * d

    class StuLayer:
        mlp, stu = Mlp, None

    class AttnLayer:
        mlp, attn = Mlp, Attn

    stack = [AttnLayer if attn and i % 2 else StuLayer for i in range(layers)]
    assert TokenStep.pays(stack, B, d, dt, t, steps) is want


@pytest.mark.parametrize("d,layers,heads,mlp,dt,B,t,steps,attn,want", [
    (512, 8, 8, 12, torch.float32, 2, 200, 400, True, True), (512, 8, 8, 12, torch.float32, 8, 200, 400, True, False),       # 207/245, 397/309
    (768, 18, 12, 4, torch.bfloat16, 1, 400, 400, True, True), (768, 10, 12, 8, torch.bfloat16, 6, 4000, 400, False, False),   # 322/384, 436/286
    (1024, 10, 8, 4, torch.bfloat16, 1, 4000, 400, True, True), (1536, 6, 12, 4, torch.bfloat16, 8, 4000, 400, False, False),  # 239/295, 405/327
    (1536, 6, 12, 4, torch.bfloat16, 4, 400, 400, True, True)])                                                             # 233/271
def test_form_of_the_step_follows_pairs_of_the_kernel_as_it_is(d, layers, heads, mlp, dt, B, t, steps, attn, want):
    """us a step, persistent and graph, beside each case (up to the graph's capture, which 400 steps pay for)."""
    test_form_of_the_step_follows_what_was_measured(d, layers, heads, mlp, dt, B, t, steps, attn, want)


def test_tagged_words_are_read_in_elements_of_the_stores_width():
    """A word's value and tag come from one store only if they lie in one element of the reader's vector load (a vector access is
    as many accesses as it has elements): per type, every load of the words has elements as wide as the store."""
    text = open(os.path.join(os.path.dirname(_lib.LIB_PATH), "csrc", "token_step.cu")).read()
    for dt, bits in (("bf16", "32"), ("float", "64")):
        body = text[text.index(f"struct Tagged<{dt}> {{"):]
        body = body[:body.index("\n};")]
        stores = re.findall(r"st\.relaxed\.gpu\.global\.[ub](\d+)", body)
        loads = re.findall(r"ld\.relaxed\.gpu\.global\.v(\d)\.[ub](\d+)", body)
        assert stores == [bits] and loads == [(str(128 // int(bits)), bits)], (dt, stores, loads)
    assert len(re.findall(r"ld\.relaxed\.gpu\.global", text)) == 2   # nobody else reads them


def test_kernels_that_end_a_chain_of_early_launches():
    """The STU decode kernel reads positions and history ahead of its programmatic wait, which the layer's previous step wrote: a
    kernel between the two has to wait before it lets its successor start.  The tcgen05 GEMM always does, gate/up products and linears
    whose caller vouches for no weights do in every form."""
    csrc = os.path.join(os.path.dirname(_lib.LIB_PATH), "csrc")
    body = {}
    for name, kernel in (("gemm_tc", "gemm_tc_kernel"), ("gemm_tc", "skinny_umma_kernel"), ("skinny_stage", "skinny_stage_kernel"),
                         ("skinny_wide", "skinny_wide_kernel"), ("stream", "stream_bf16_kernel"), ("stream", "stream_f32_kernel")):
        text = open(os.path.join(csrc, name + ".cu")).read()
        body[kernel] = text[text.index("__global__", text.index(f"{kernel}(") - 400):]
        body[kernel] = body[kernel][:body[kernel].index("\n}\n")]
    for kernel, text in body.items():
        triggers = [text[:m.start()] for m in re.finditer(r"pdl_trigger\(\)", text)]
        early = [t for t in triggers if t.endswith("if (early_trigger) ")]
        if kernel in ("gemm_tc_kernel", "skinny_wide_kernel"):
            assert not early
        else:
            assert re.search(r"early_trigger = early(_weights)? && PdlTrigger<EPI>::ahead_of_wait", text), kernel
        late = [t for t in triggers if t not in early]
        assert len(late) == 1 and "pdl_wait()" in late[0], kernel
        assert not re.search(r"if \(early(_weights)?\) pdl_trigger", text)


def test_early_reads_of_the_finish_kernel_are_the_callers_choice(monkeypatch):
    """stream_finish starts beside the kernels in front, and reads what the step before wrote ahead of its wait, only where it is told
    to; the captured step is what tells it."""
    from types import SimpleNamespace

    from flash_stu_2_b200 import ops
    calls = []
    monkeypatch.setattr(ops, "_cuda", lambda *a: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "status_word", lambda dev: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(_lib, "native", lambda: SimpleNamespace(stu_stream_finish=lambda *a: calls.append(a[-2]) or 0))
    rows = lambda: torch.zeros(2, 8, dtype=torch.bfloat16)
    hist, taps8, part = torch.zeros(2, 8, 2, 8), torch.zeros(8, 8, 16), torch.zeros(2, 2, 8)
    pos, ctl = torch.zeros(2, 2, dtype=torch.int32), torch.zeros(4, dtype=torch.int32)
    pos._host_t = 0
    ops.stream_finish(rows(), rows(), hist, taps8, pos, part, ctl, torch.zeros(8), 1e-6, rows())
    monkeypatch.setattr(STU, "project_step", staticmethod(lambda x, *a: rows()))
    stu = SimpleNamespace(prepared=lambda: (None, None, taps8), project_step=STU.project_step)
    STU.stream_step(stu, rows(), None, 1e-6, (hist, pos), rows(), (part, ctl), torch.zeros(8), 1e-6)
    assert calls == [1, 1 | ops.FLAG_OVERLAP]


def _sub_stu(m):
    m.layers[2].stu.__class__ = type("Stu", (STU,), {"decode_step": lambda self, *a: STU.decode_step(self, *a)})


def _sub_layer(m):
    m.layers[2].__class__ = type("Layer", (STULayer,), {"_decode": lambda self, *a: STULayer._decode(self, *a)})


def _foreign_layer(m):
    m.layers[0] = torch.nn.Module()
    m.layers[0].stu, m.layers[0].stu_mlp_enabled = m.layers[2].stu, False


@pytest.mark.parametrize("change", [lambda m: setattr(m.layers[0].stu, "decode_step", lambda *a: None), _own_forward, _sub_stu, _sub_layer,
                                    _foreign_layer])
def test_overridden_steps_are_not_streamed_beside_the_chain(monkeypatch, change):
    m = _model().bfloat16()
    monkeypatch.setattr(STU, "prepared", lambda self: (None, None, True))
    pos = torch.zeros(16, 2, dtype=torch.int32)
    pos._host_t, pos._uniform = 3, True
    past = [(torch.zeros(16, 64, 2, 8, dtype=torch.bfloat16), pos) for _ in m.layers]
    assert StreamAhead.supported(m.layers, past, 16)
    change(m)
    assert not StreamAhead.supported(m.layers, past, 16)


@pytest.mark.parametrize("where,name", [("stu", "decode_step"), ("mlp", "apply_residual")])
def test_overridden_parts_of_an_fp32_step_are_called(monkeypatch, where, name):
    """The native call for a whole fp32 layer step takes the place of decode_step and apply_residual where they are the classes' own."""
    layer = _model().layers[0]
    taken, called = [], []
    monkeypatch.setattr(STU, "layer_step_f32", lambda self, *a: taken.append(1) or 3)
    entry, x = (torch.zeros(2, 64, 2, 8), torch.zeros(2, 2, dtype=torch.int32)), torch.zeros(2, 1, 64)
    assert layer._decode(x, entry) is entry and taken == [1]
    monkeypatch.setattr(STU, "decode_step", lambda self, *a: entry)
    monkeypatch.setattr(type(layer.mlp), "apply_residual", lambda self, *a, **k: None)
    part = getattr(layer, where)
    setattr(part, name, lambda *a, **k: called.append(name) or entry)
    assert layer._decode(x, entry) is entry and taken == [1] and called == [name]


def test_sms_for_the_streams_beside_a_step():
    """What decides whether and on how many SMs a captured step's history streams run beside it: none for a few short streams or for more than
    a fifth of the GPU (from 65 sequences on, a third) can finish, more for longer histories up to there."""
    big = lambda t, B=32: StreamAhead.sms(24, 12, B, 1536, t, 1_800_000_000, 75_000_000 * B, 148)
    assert StreamAhead.sms(4, 2, 16, 512, 300, 60_000_000, 10_000_000, 148) == 0
    assert 16 <= big(2176) <= 26 and big(500) == 8 and big(4000) == 29 and big(8000) == 0 and big(8000, 16) == 29
    assert all(0 < big(t) <= big(t + 512) for t in range(256, 4000, 256))
    assert 29 < big(4000, 65) <= 49 and big(4000, 64) in (0, 29)
    # narrow layers of 16 sequences, whose norm is fused either way: a launch less is saved
    small = lambda t, **kw: StreamAhead.sms(12, 6, 16, 256, t, 40_000_000, 50_000_000, 148, **kw)
    assert small(200, norm_apart=False) == 0 and small(1000, norm_apart=False) == 8 and small(200) == 8


def test_nothing_is_allocated_for_steps_that_are_not_streamed(monkeypatch):
    m = _model().bfloat16()
    monkeypatch.setattr(STU, "prepared", lambda self: (None, None, True))
    monkeypatch.setattr(StreamAhead, "__init__", lambda *a: pytest.fail("built"))
    monkeypatch.setattr("flash_stu_2_b200.stream_ahead._sm_count", lambda dev: 148)
    pos = torch.zeros(16, 2, dtype=torch.int32)
    pos._host_t, pos._uniform = 3, True
    past = [(torch.zeros(16, 64, 2, 8, dtype=torch.bfloat16), pos) for _ in m.layers]
    assert StreamAhead.plan(m.layers, past, 16, 10, 1_000_000) is None
