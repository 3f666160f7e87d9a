"""Host-side mirror of the reference API: construction, state-dict keys, filters, cache plumbing."""
import os

import pytest
import torch

import flash_stu_2_b200 as F
from oracle import stu_oracle as O


def _cfg(tmp_path, **kw):
    L, K = kw.pop("seq_len", 64), kw.pop("num_eigh", 8)
    phi = F.get_spectral_filters(L, K, dtype=torch.float32, device="cpu")
    fp = os.path.join(tmp_path, "phi.pt")
    F.save_spectral_filters(phi, fp, metadata={"seq_len": L, "K": K})
    base = dict(n_embd=32, n_layers=4, n_heads=4, seq_len=L, window_size=8, vocab_size=97, mlp_scale=4, num_eigh=K,
                torch_dtype=torch.float32, filter_path=fp)
    base.update(kw)
    return F.FlashSTUConfig(**base)


def test_filters_match_oracle_and_roundtrip(tmp_path):
    phi = F.get_spectral_filters(64, 8, dtype=torch.float32, device="cpu")
    ref = O.spectral_filters(64, 8)
    assert torch.allclose(phi, ref, rtol=0, atol=0)
    p = os.path.join(tmp_path, "sub", "f")
    F.save_spectral_filters(phi, p)
    back = F.load_spectral_filters(p + ".pt", device="cpu", dtype=torch.bfloat16, verify_shape=(64, 8))
    assert back.dtype == torch.bfloat16 and torch.equal(back, phi.bfloat16())
    with pytest.raises(ValueError):
        F.load_spectral_filters(p + ".pt", device="cpu", verify_shape=(64, 9))
    assert F.nearest_power_of_two(2 * 8192 - 1, round_up=True) == 16384


def test_state_dict_keys_match_reference(tmp_path, golden):
    g = golden("models")
    for name in ("stu_only_approx_fp32", "hybrid_approx_fp32", "stu_only_full_fp32"):
        r = g[name]
        m = F.FlashSTU(_cfg(str(tmp_path), use_attn=r["cfg"]["use_attn"], use_approx=r["cfg"]["use_approx"]))
        assert set(m.state_dict().keys()) == set(r["sd"].keys())
        m.load_state_dict(r["sd"])
        assert m.tok_emb.weight is m.lm_head.weight
    blk = F.FlashSTUBlock(d_model=64, sequence_length=128, num_filters=8, torch_dtype=torch.float32)
    assert set(blk.state_dict().keys()) == set(golden("blocks")["approx_float32"]["sd"].keys())
    assert not blk.is_attention_block and blk.get_num_params() > 0


def test_layer_alternation_and_alibi(tmp_path, golden):
    m = F.FlashSTU(_cfg(str(tmp_path)))
    kinds = [type(l).__name__ for l in m.layers]
    assert kinds == ["STULayer", "AttentionLayer", "STULayer", "AttentionLayer"]
    m2 = F.FlashSTU(_cfg(str(tmp_path), use_attn=False))
    assert all(type(l).__name__ == "STULayer" for l in m2.layers)
    for H, s in golden("alibi_slopes").items():
        cfg = _cfg(str(tmp_path), n_embd=8 * H, n_heads=H)
        assert torch.allclose(F.Attention(cfg).alibi_slopes.double(), s.double(), rtol=1e-6, atol=0)


def test_unsupported_switches_fail_loudly(tmp_path):
    for kw in (dict(bias=True), dict(stu_enable_mlp_sandwich=True, bias=True)):
        with pytest.raises(NotImplementedError):
            F.FlashSTU(_cfg(str(tmp_path), use_attn=False, **kw))
    # the sandwich itself constructs, with the reference's parameter names
    m = F.FlashSTU(_cfg(str(tmp_path), use_attn=False, stu_enable_mlp_sandwich=True, stu_mlp_hidden_size=24))
    keys = set(m.state_dict())
    assert {"layers.0.stu_mlp_in_proj.weight", "layers.0.stu_mlp_out_proj.weight"} <= keys
    assert m.layers[0].stu.M_inputs.shape == (24, 24)


def test_model_refuses_cpu(tmp_path):
    m = F.FlashSTU(_cfg(str(tmp_path)))
    with pytest.raises(RuntimeError, match="no CPU path"):
        m(torch.zeros(1, 4, dtype=torch.long))


def test_reorder_cache_keeps_structure():
    hist, pos = torch.arange(24.).view(3, 2, 2, 2), torch.tensor([[5, 0]] * 3, dtype=torch.int32)
    kv = (torch.arange(12.).view(3, 2, 2), torch.arange(12.).view(3, 2, 2), pos.clone())
    out = F.FlashSTU._reorder_cache(((hist, pos), kv, None), torch.tensor([2, 0, 0]))
    assert out[2] is None and torch.equal(out[0][0][0], hist[2]) and out[1][2].shape == (3, 2)


def test_checkpoint_round_trip_and_vocabulary_resize(tmp_path):
    """save_pretrained / from_pretrained (flash_stu/model.py:338-366) keep every tensor, the dtype and the
    tok_emb / lm_head tie; resize_token_embeddings keeps the tie and updates the config."""
    import os
    import torch
    import flash_stu_2_b200 as F
    from oracle import stu_oracle as O
    L, K = 64, 8
    fp = os.path.join(str(tmp_path), "phi.pt")
    F.save_spectral_filters(O.spectral_filters(L, K), fp)
    cfg = F.FlashSTUConfig(n_embd=32, n_layers=4, n_heads=4, seq_len=L, window_size=8, vocab_size=97, mlp_scale=4,
                           num_eigh=K, torch_dtype=torch.bfloat16, filter_path=fp, use_attn=True)
    torch.manual_seed(0)
    m = F.FlashSTU(cfg)
    ckpt = os.path.join(str(tmp_path), "ckpt")
    m.save_pretrained(ckpt)
    m2 = F.FlashSTU.from_pretrained(ckpt)
    assert m2.config.torch_dtype == torch.bfloat16 and next(m2.parameters()).dtype == torch.bfloat16
    # a float32 model comes back as float32 (not as the bfloat16 default of the config class), bit for bit
    m32 = F.FlashSTU(F.FlashSTUConfig(n_embd=32, n_layers=2, n_heads=4, seq_len=L, window_size=8, vocab_size=97,
                                      mlp_scale=4, num_eigh=K, torch_dtype=torch.float32, filter_path=fp))
    ck32 = os.path.join(str(tmp_path), "ckpt32")
    m32.save_pretrained(ck32)
    r32 = F.FlashSTU.from_pretrained(ck32)
    assert r32.config.torch_dtype == torch.float32
    assert all(v.dtype == torch.float32 and torch.equal(v, m32.state_dict()[k]) for k, v in r32.state_dict().items())
    # buffers that are not part of a checkpoint (the STU layers' filters, the ALiBi slopes) are re-derived on load
    assert all(torch.equal(l.stu.phi, r32.phi) for l in r32.layers if hasattr(l, "stu"))
    assert all(torch.equal(a.attn.alibi_slopes, b.attn.alibi_slopes)
               for a, b in zip(m2.layers, m.layers) if hasattr(a, "attn"))
    sd1, sd2 = m.state_dict(), m2.state_dict()
    assert set(sd1) == set(sd2) and all(torch.equal(sd1[k], sd2[k]) for k in sd1)
    assert m2.lm_head.weight.data_ptr() == m2.tok_emb.weight.data_ptr()
    m2.resize_token_embeddings(101)
    assert m2.tok_emb.weight.shape == (101, 32) and m2.lm_head.weight.shape == (101, 32)
    assert m2.config.vocab_size == 101 and m2.lm_head.weight.data_ptr() == m2.tok_emb.weight.data_ptr()
    assert torch.equal(m2.tok_emb.weight[:97], sd1["tok_emb.weight"])
    # beam reordering of a cache (flash_stu/model.py:404-426): every tensor of every layer entry, batch on dim 0
    hist = torch.arange(2 * 3 * 2 * 8, dtype=torch.float32).view(2, 3, 2, 8)
    pos = torch.tensor([[5, 0], [7, 0]], dtype=torch.int32)
    out = F.FlashSTU._reorder_cache(((hist, pos), None), torch.tensor([1, 0]))
    assert torch.equal(out[0][0], hist[[1, 0]]) and out[0][1][:, 0].tolist() == [7, 5] and out[1] is None


def test_block_power_iteration_reproduces_the_leading_hankel_eigenpairs():
    """top_eigenpairs_subspace (used for filters when the dense solver refuses the matrix) against numpy eigh."""
    import numpy as np
    import torch
    from flash_stu_2_b200.filters import get_hankel, top_eigenpairs_subspace
    L, K = 384, 16
    Zn = get_hankel(L)
    w, V = top_eigenpairs_subspace(torch.tensor(Zn), K)
    wr, Vr = np.linalg.eigh(Zn)
    assert np.allclose(w.numpy()[-10:], wr[-10:], rtol=1e-9, atol=1e-15)
    assert (V[:, -8:].abs() - torch.tensor(Vr[:, -8:]).abs()).abs().max() < 1e-9
    assert torch.allclose(V.T @ V, torch.eye(K, dtype=torch.float64), atol=1e-10)


def test_lds_feature_rows_shrink_to_the_memory_there_is(monkeypatch):
    """The prefill of the distilled form holds the features of several sequences at once only where they fit."""
    room, real = 5000, torch.empty

    def empty(*shape, **kw):
        if shape[0] > room:
            raise torch.cuda.OutOfMemoryError("no room")
        return real(*shape, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    x = torch.zeros(8, 1000, 4)
    for most, got in ((8, 4), (5, 3), (3, 3), (1, 1)):   # 8 -> 4, 5 -> 3
        G, U = F.MiniSTU._lds_features(most, 1000, 1024, 16, x)
        assert G == got and U.shape == ((G - 1) * 1000 + 1024, 16)
    room = 1000
    with pytest.raises(torch.cuda.OutOfMemoryError):
        F.MiniSTU._lds_features(8, 1000, 1024, 16, x)


@pytest.mark.parametrize("B,d,dt,early", [
    (16, 1024, torch.bfloat16, (True, True)), (9, 64, torch.bfloat16, (True, True)), (8, 1024, torch.bfloat16, (False, False)),
    (1, 2048, torch.bfloat16, (True, True)), (5, 256, torch.bfloat16, (True, True)), (6, 256, torch.bfloat16, (False, False)),
    (8, 128, torch.float32, (True, False)), (4, 1024, torch.float32, (False, False)), (1, 1024, torch.float32, (True, False))])
def test_which_lds_steps_start_beside_the_kernels_in_front(B, d, dt, early):
    assert F.MiniSTU._lds_early(B, d, dt) == early


@pytest.mark.parametrize("M,N,K,epi,fused", [
    (8, 50000, 4096, 0, True), (17, 512, 512, 0, False), (9, 2304, 768, 2, True), (16, 2048, 1024, 2, True), (12, 2440, 768, 2, False),
    (12, 1536, 1536, 2, False), (9, 2304, 1024, 0, True), (16, 2440, 512, 0, False), (9, 1024, 2048, 0, True), (9, 1536, 1536, 0, False),
    (16, 1024, 3072, 0, False), (12, 4608, 1536, 0, False)])
def test_which_linears_fuse_their_norm(M, N, K, epi, fused):
    from flash_stu_2_b200 import ops
    assert ops.can_fuse_norm(M, N, K, epi, torch.bfloat16) is fused


@pytest.mark.parametrize("B,T,out,group", [(16, 6000, 1024, 3), (8, 4700, 1024, 2), (4, 9000, 1024, 1), (16, 700, 1024, 13), (3, 100, 64, 3)])
def test_lds_contractions_are_grouped_by_the_gemms_own_tiles(monkeypatch, B, T, out, group):
    """As many sequences as leave the least time in all by the GEMM's plan (8 x 4700 to 1024 outputs: two sequences are two full waves of
    pairs' tiles, one alone is one of tiles half as high)."""
    from types import SimpleNamespace

    from flash_stu_2_b200 import ops
    x = torch.empty(0, dtype=torch.bfloat16)
    asked = []
    cost = ops.linear_tile_cost
    monkeypatch.setattr(ops, "linear_tile_cost", lambda *a: asked.append(a) or cost(*a))
    assert F.MiniSTU._lds_group(SimpleNamespace(output_dim=out), B, T, 48 * 1024, x) == group
    assert all(cols == out and rows % T == 0 for rows, cols in asked)


def test_captures_of_two_threads_hold_the_collector_until_the_last_is_done():
    import gc
    from flash_stu_2_b200.model import _CollectionHeld
    a, b = _CollectionHeld(), _CollectionHeld()
    assert gc.isenabled()
    a.__enter__(), b.__enter__()
    a.__exit__()
    assert not gc.isenabled()   # the other capture is still open
    b.__exit__()
    assert gc.isenabled()
    gc.disable()
    try:
        with _CollectionHeld():
            pass
        assert not gc.isenabled()
    finally:
        gc.enable()


@pytest.mark.parametrize("hd,B,H,T,window,t0,takes", [
    (128, 1, 1, 128, 16, 0, True), (128, 1, 1, 127, 16, 0, False), (128, 4, 8, 500, 500, 1, False),          # as heads of 128 were
    (64, 4, 16, 384, 500, 0, True), (64, 4, 16, 383, 500, 0, False), (64, 1, 12, 1024, 1024, 0, True), (64, 1, 12, 1023, 1024, 0, False),
    (64, 4, 16, 1999, 512, 0, True), (64, 4, 16, 800, 300, 0, False), (64, 4, 16, 896, 300, 0, True), (64, 4, 16, 4000, 200, 0, False),
    (64, 4, 16, 1999, 512, 7, False), (32, 4, 16, 1999, 512, 0, False), (96, 4, 16, 1999, 512, 0, False)])
def test_which_attention_kernel_takes_a_prefill(hd, B, H, T, window, t0, takes):
    from flash_stu_2_b200 import ops
    qkv = torch.empty(B, T, 3 * H * hd, dtype=torch.bfloat16, device="meta")
    assert ops.swa_prefill_tc5_supported(qkv, H, t0, window) is takes
    assert not ops.swa_prefill_tc5_supported(qkv.float(), H, t0, window)


@pytest.mark.parametrize("batch,d,K,t,pays", [(1, 512, 24, 7000, True), (8, 1024, 24, 3000, True), (8, 1024, 24, 7000, False), (16, 1024, 24, 1000, True),
                                             (16, 1024, 24, 2000, False), (16, 1024, 16, 4000, False), (16, 1024, 16, 2000, True), (32, 1536, 24, 0, False),
                                             (16, 1024, 32, 0, False), (12, 1024, 32, 0, True)])
def test_which_form_the_full_variants_step_takes(batch, d, K, t, pays):
    from flash_stu_2_b200 import ops
    assert ops.full_decode_step_pays(batch, d, K, t) is pays


@pytest.mark.parametrize("batch,d,K,t,pays", [(8, 1024, 24, 1499, False), (8, 1024, 24, 1500, True), (8, 1024, 8, 2999, False), (8, 1024, 32, 500, True),
                                             (5, 960, 24, 1500, True), (4, 1152, 24, 8000, False), (16, 1024, 24, 0, True), (16, 1024, 33, 4000, False),
                                             (19, 512, 1, 0, True), (40, 520, 24, 8000, False)])
def test_when_the_full_variants_step_goes_to_tcgen05(batch, d, K, t, pays):
    from flash_stu_2_b200 import ops
    assert ops.full_decode_step_tc5_pays(batch, d, K, t) is pays


def test_a_prefill_calls_another_modules_sub_layers(monkeypatch):
    """A layer whose STU is of another class, with no more of its interface than the prefill called: add_to_residual."""
    import flash_stu_2_b200 as F
    from flash_stu_2_b200 import ops

    class Other(torch.nn.Module):
        def add_to_residual(self, xn, x, entry=None, use_cache=False):
            x += 2 * xn
            return "entry" if use_cache else None

    cfg = F.FlashSTUConfig(n_embd=8, n_layers=1, n_heads=1, seq_len=16, vocab_size=1, mlp_scale=2, num_eigh=2, torch_dtype=torch.float32, use_attn=False)
    layer = F.FlashSTUBlock(config=cfg, phi=torch.zeros(16, 2)).layer
    layer.stu = Other()
    monkeypatch.setattr(ops, "rmsnorm", lambda x, *a: x.clone())
    layer.mlp.apply_residual = lambda xn, resid, out, **kw: out.add_(xn)
    x = torch.randn(2, 5, 8)
    y, entry = layer(x.clone(), use_cache=True)
    assert torch.equal(y, 2 * (x + 2 * x)) and entry == "entry"


@pytest.mark.parametrize("B,d,K,t0,t_end,pays", [(8, 64, 24, 0, 1000, True), (4, 512, 24, 0, 600, True), (8, 96, 16, 0, 2048, True), (4, 144, 1, 0, 219, False),
                                                 (8, 16, 1, 0, 415, False), (1, 988, 4, 265, 266, False), (3, 36, 4, 0, 867, False), (1, 16, 24, 0, 2000, True),
                                                 (2, 66, 24, 0, 2000, False), (8, 64, 24, 0, 199, False)])
def test_which_kernel_takes_the_full_variants_fp32_convolutions(B, d, K, t0, t_end, pays):
    from flash_stu_2_b200 import ops
    assert ops.full_conv_f32_tc5_pays(B, d, K, t0, t_end) is pays


def test_a_tile_form_that_is_asked_for_cuts_no_k():
    """The environment is read once, so each setting has a process of its own."""
    import os
    import subprocess
    import sys
    from flash_stu_2_b200 import _build
    code = ("import ctypes, sys; f = ctypes.CDLL(sys.argv[1]).stu_linear_workspace_elems; f.restype = ctypes.c_longlong; "
            "print(f(333, 1536, 6144, 0, 1))")
    env = {k: v for k, v in os.environ.items() if not k.startswith("STU_B200_TILE")}
    for asked in ({}, {"STU_B200_TILE_N": "128"}, {"STU_B200_TILE_N": "256"}, {"STU_B200_TILE_CTAS": "1"}, {"STU_B200_TILE_CTAS": "2"}):
        out = subprocess.run([sys.executable, "-c", code, _build.build_library()], env={**env, **asked}, capture_output=True, text=True, check=True).stdout
        assert (int(out) == 0) is bool(asked), asked


@pytest.mark.parametrize("sms,batch,t,pays", [(148, 9, 0, False), (132, 9, 0, True), (148, 4, 5000, False), (132, 4, 5000, False), (128, 4, 5000, True), (148, 5, 5000, True), (162, 5, 5000, False)])
def test_the_full_variants_step_asks_how_many_sms_there_are(monkeypatch, sms, batch, t, pays):
    """16 CTAs per sequence: more than there are SMs, or half of them and more from position 1500 on (24 filters)."""
    from flash_stu_2_b200 import ops
    monkeypatch.setattr(ops, "sm_count", lambda: sms)
    assert ops.full_decode_step_tc5_pays(batch, 1024, 24, t) is pays


@pytest.mark.parametrize("M,N,K", [(70, 30, 3072), (256, 512, 6144), (1000, 1536, 512), (65, 8, 256)])
@pytest.mark.parametrize("gate_up", [0, 1])
def test_an_fp32_product_is_not_split_over_clusters_that_the_gpu_does_not_hold(M, N, K, gate_up):
    import ctypes
    from flash_stu_2_b200 import _lib
    hook = _lib.load().stu_test_f32_tile
    for most in range(4):   # clusters of more than 2^most CTAs: none at a time
        room = (ctypes.c_int * 4)(*([148, 74, 33, 16][:most + 1] + [0] * (3 - most)))
        tile = hook(M, N, K, gate_up, room)
        assert tile // 16 in (32, 64, 128) and tile % 16 <= 2 ** most
    assert tile % 16 == 8 or K < 3072 or M > 256   # (with all of them long K over few tiles is split eightfold)
