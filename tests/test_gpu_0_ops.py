"""Kernel-level parity on a B200: every C-ABI op against the CPU oracle / an fp32 torch statement of the op.
Tolerances: fp32 1e-3 relative (observed far below), bf16 2e-2 relative, as the parity bar states."""
import math

import pytest
import torch

from oracle import stu_oracle as O
from parity import close

pytestmark = pytest.mark.gpu

TOL = {torch.float32: 1e-3, torch.bfloat16: 2e-2}


def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return torch.device("cuda:0")




@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(5, 32), (3, 7, 1024), (2, 50)])
def test_rmsnorm(dt, shape):
    from flash_stu_2_b200 import ops
    torch.manual_seed(0)
    x = (torch.randn(*shape) * 3).to(dt)
    w = torch.randn(shape[-1]).to(dt)
    y = ops.rmsnorm(x.to(dev()), w.to(dev()))
    ref = O.rmsnorm(x, w)
    close(y, ref, (1e-6 if dt == torch.float32 else 2 ** -7))


def _lin_ref(x, W, W2, resid, epi, dt):
    acc = x.double() @ W.double().t()
    if epi == 0:
        return acc.to(dt)
    if epi == 1:
        return (resid.float() + acc.to(dt).float()).to(dt)
    g = torch.nn.functional.gelu(acc.to(dt).float(), approximate="tanh").to(dt)
    return (g.float() * (x.double() @ W2.double().t()).to(dt).float()).to(dt)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,H,hd,window,t", [(1, 4, 32, 255, 900), (1, 3, 64, 511, 3), (2, 5, 64, 1024, 1024), (1, 2, 128, 1024, 5000),
                                             (3, 2, 128, 300, 301), (1, 1, 16, 2047, 1500), (40, 8, 64, 300, 120), (1, 2, 128, 1500, 127),
                                             (2, 3, 32, 20, 21), (1, 2, 64, 0, 7), (1, 2, 128, 1500, 128), (2, 2, 64, 1024, 0),
                                             (1, 4, 128, 1024, 320), (1, 1, 32, 2047, 190), (2, 1, 16, 1024, 5)])
def test_attention_decode_shares_keys(dt, B, H, hd, window, t):
    """One cached token: keys of a head shared by 1 to 8 CTAs, some of them without any, all of a cluster or its first ones; rings that have wrapped and rings that are
    not full; 64- to 512-byte rows.  Against the formula in float64 on the same rounded inputs; the output is rounded once (bf16: 2^-8
    of its row's largest, and the hardware tanh's 2^-11 on scores up to 6)."""
    from flash_stu_2_b200 import ops
    from flash_stu_2_b200.modules import new_pos
    if hd * torch.finfo(dt).bits // 128 not in (4, 8, 16, 32):
        pytest.skip("rows of 64 to 512 bytes")
    g = torch.Generator(device=dev()).manual_seed(B + hd + window + t)
    rand = lambda *s: torch.randn(*s, device=dev(), generator=g).to(dt)
    W, d, cap = window + 1, H * hd, 50.0
    k_ring, v_ring, qkv = rand(B, W, d), rand(B, W, d), rand(B, 1, 3 * d)
    slopes = torch.rand(H, device=dev(), generator=g) * 0.1
    pos = new_pos(B, dev())
    pos[:, 0] = t
    keys = list(range(max(0, t - window), t))
    slots = torch.tensor([j % W for j in keys], dtype=torch.long, device=dev())
    q, kn, vn = (p.double().view(B, 1, H, hd) for p in qkv.split(d, dim=2))
    k = torch.cat([k_ring[:, slots].double().view(B, -1, H, hd), kn], 1)
    v = torch.cat([v_ring[:, slots].double().view(B, -1, H, hd), vn], 1)
    s = cap * torch.tanh(torch.einsum("bqhc,bkhc->bhk", q, k) * hd ** -0.5 / cap)
    s = s - slopes.double()[None, :, None] * (t - torch.tensor(keys + [t], device=dev(), dtype=torch.float64))
    ref = torch.einsum("bhk,bkhc->bhc", s.softmax(-1), v).reshape(B, d)
    y = ops.swa_forward(qkv, k_ring, v_ring, pos, slopes, H, window, cap, update_cache=True)
    close(y.view(B, d), ref, 1e-5 if dt == torch.float32 else 1e-2)
    assert pos[:, 0].tolist() == [t + 1] * B and pos[0, 1].item() == 0
    assert torch.equal(k_ring[:, t % W], qkv[:, 0, d:2 * d]) and torch.equal(v_ring[:, t % W], qkv[:, 0, 2 * d:])


@pytest.mark.parametrize("hd", [64, 128])
def test_attention_decode_keeps_fp32s_precision(hd):
    """fp32 scores and weights of one token over 1025 keys: the mean relative error against float64 over 16 inputs.  Dot products in one chain per
    lane and weights relative to a reference that lags by up to 8 (whose exponents carry 8 times the rounding) had 2.1e-7 and 2.3e-7; one
    chain per vector and a reference that does not lag have 1.33e-7 and 1.43e-7, the kernel of 16 lanes per key had 1.35e-7."""
    from flash_stu_2_b200 import ops
    from flash_stu_2_b200.modules import new_pos
    B, H, W, t, errs = 4, 4, 1025, 1500, []
    d = H * hd
    for seed in range(16):
        g = torch.Generator(device=dev()).manual_seed(seed)
        rand = lambda *s: torch.randn(*s, device=dev(), generator=g)
        k_ring, v_ring, qkv, slopes = rand(B, W, d), rand(B, W, d), rand(B, 1, 3 * d), torch.rand(H, device=dev(), generator=g) * 0.1
        pos = new_pos(B, dev())
        pos[:, 0] = t
        at = torch.arange(t - W + 1, t, device=dev())
        q, kn, vn = (p.double().view(B, 1, H, hd) for p in qkv.split(d, dim=2))
        k, v = (torch.cat([r[:, at % W].double().view(B, -1, H, hd), n], 1) for r, n in ((k_ring, kn), (v_ring, vn)))
        s = torch.einsum("bqhc,bkhc->bhk", q, k) * hd ** -0.5 - slopes.double()[None, :, None] * torch.arange(W - 1, -1, -1, device=dev())
        ref = torch.einsum("bhk,bkhc->bhc", s.softmax(-1), v).reshape(B, d)
        y = ops.swa_forward(qkv, k_ring, v_ring, pos, slopes, H, W - 1, 0.0, update_cache=False).view(B, d).double()
        errs.append(float((y - ref).norm() / ref.norm()))
    assert sum(errs) / 16 < 1.7e-7, errs


@pytest.mark.parametrize("epi", [0, 1, 2])
@pytest.mark.parametrize("M,N,K", [(1, 128, 8), (128, 136, 64), (129, 256, 72), (255, 128, 136), (256, 264, 128), (257, 128, 192),
                                   (512, 2560, 200), (2600, 2048, 64), (19200, 264, 128)])
def test_linear_pair_tiles(M, N, K, epi):
    """Tiles that a pair of CTAs computes: rows that fill one CTA's half, both, or a row of the next tile; both tile widths; K of
    less than a block, of an odd number of blocks, of blocks and a piece; more tiles than pairs.  Sums in another order may round to
    the next value, 2^-7 of the output at most: once in a plain output, twice with a residual, four times in gate/up."""
    from flash_stu_2_b200 import ops
    g = torch.Generator(device=dev()).manual_seed(M + N + K)
    rand = lambda *s: torch.randn(*s, device=dev(), generator=g)
    x, W, W2 = rand(M, K).bfloat16(), (rand(N, K) / math.sqrt(K)).bfloat16(), (rand(N, K) / math.sqrt(K)).bfloat16()
    resid = rand(M, N).bfloat16()
    y = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device=dev())
    ops.linear(x, W, W2=W2 if epi == 2 else None, resid=resid if epi == 1 else None, out=y[:M], epilogue=epi, backend=ops.BACKEND_TCGEN05)
    ops.check_status()
    assert bool((y[M] == 7.0).all())
    close(y[:M], _lin_ref(x, W, W2, resid, epi, torch.bfloat16), (1, 2, 4)[epi] * 2 ** -7)


@pytest.mark.parametrize("M,N,K,epi,pad", [(300, 6144, 72, 2, 0), (257, 10240, 64, 2, 8), (100, 10248, 200, 2, 0), (1030, 2048, 512, 2, 0), (300, 12288, 72, 0, 0),
                                           (384, 12296, 136, 1, 8), (129, 18950, 64, 0, 3), (270, 12301, 776, 0, 0), (1030, 7680, 64, 1, 0), (128, 9480, 8, 2, 0)])
def test_linear_tiles_of_single_ctas(M, N, K, epi, pad):
    """Products whose tiles of 256 rows would fill their last wave badly are computed by single CTAs: the same bits as by pairs (rows that the
    pairs' tiles hold, in pieces of 256), whole and ragged tiles, gate/up, residuals, rows on and off the 16-byte grid."""
    from flash_stu_2_b200 import ops
    g = torch.Generator(device=dev()).manual_seed(M + N + K)
    rand = lambda *s: torch.randn(*s, device=dev(), generator=g)
    x, W, W2 = rand(M, K).bfloat16(), (rand(N, K) / math.sqrt(K)).bfloat16(), (rand(N, K) / math.sqrt(K)).bfloat16()
    resid = rand(M, N).bfloat16()
    kw = lambda r: dict(W2=W2 if epi == 2 else None, resid=resid[r] if epi == 1 else None, epilogue=epi, backend=ops.BACKEND_TCGEN05)
    y = torch.full((M + 1, N + pad), 7.0, dtype=torch.bfloat16, device=dev())
    ops.linear(x, W, out=y[:M, :N], **kw(slice(0, M)))
    few = ops.linear(x, W[:2048], W2=W2[:2048] if epi == 2 else None, resid=resid[:, :2048].contiguous() if epi == 1 else None, epilogue=epi,
                     backend=ops.BACKEND_TCGEN05)   # one wave of pairs
    ops.check_status()
    assert bool((y[M] == 7.0).all()) and bool((y[:, N:] == 7.0).all())
    close(y[:M, :N], _lin_ref(x, W, W2, resid, epi, torch.bfloat16), (1, 2, 4)[epi] * 2 ** -7)   # as of the pairs' tiles
    assert torch.equal(y[:M, :2048], few) or M > 1000   # (1030 rows: several waves either way)


@pytest.mark.parametrize("backend", [1, 2, 3])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("epi", [0, 1, 2])
def test_linear_backends(backend, dt, epi):
    from flash_stu_2_b200 import ops
    if backend == 2 and dt != torch.bfloat16:
        pytest.skip("tcgen05 path is bf16 only")
    torch.manual_seed(1)
    shapes = [(300, 200, 136), (128, 128, 64), (257, 520, 1032)] if backend != 3 else [(8, 200, 136), (33, 72, 1024), (2, 50, 64)]
    for (M, N, K) in shapes:
        x = torch.randn(M, K).to(dt)
        W = (torch.randn(N, K) / math.sqrt(K)).to(dt)
        W2 = (torch.randn(N, K) / math.sqrt(K)).to(dt)
        resid = torch.randn(M, N).to(dt)
        ref = _lin_ref(x, W, W2, resid, epi, dt)
        y = ops.linear(x.to(dev()), W.to(dev()), W2=W2.to(dev()) if epi == 2 else None,
                       resid=resid.to(dev()) if epi == 1 else None, epilogue=epi, backend=backend)
        ops.check_status()
        close(y, ref, TOL[dt] / 2)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_linear_narrow_output_long_rows(dt):
    """Decode linears whose output is narrow and whose rows are long (down projections of a wide MLP): bf16 splits K
    across a thread-block cluster and reduces through distributed shared memory, fp32 across the warps of a CTA."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(4)
    for (M, N, K, epi) in [(5, 512, 6144, 1), (20, 384, 4096, 0), (2, 512, 6144, 1), (8, 760, 8200, 0)]:
        x = torch.randn(M, K).to(dt)
        W = (torch.randn(N, K) / math.sqrt(K)).to(dt)
        resid = torch.randn(M, N).to(dt)
        ref = _lin_ref(x, W, None, resid, epi, dt)
        y = ops.linear(x.to(dev()), W.to(dev()), resid=resid.to(dev()) if epi == 1 else None, epilogue=epi, backend=3)
        ops.check_status()
        close(y, ref, TOL[dt] / 2)


@pytest.mark.parametrize("epi", [0, 1, 2])
def test_linear_17_to_64_rows(epi):
    """Decode linears of 17..64 token rows (bf16).  Store / residual: 32 output features per CTA, operands streamed
    through registers, K over a cluster of up to 4 CTAs.  Gate/up at up to 32 rows: the kernel that stages the
    activation rows in shared memory by bulk copies and has every weight load in flight at once (16 gate + 16 up rows
    per CTA, K over a cluster of up to 8 CTAs).  Ragged N, K and M included (K not a multiple of 32 falls back to the
    8-feature kernel)."""
    from flash_stu_2_b200 import ops
    dt = torch.bfloat16
    torch.manual_seed(8)
    for (M, N, K) in [(32, 1536, 6144), (32, 1536, 1536), (32, 4608, 1536), (17, 72, 1024), (48, 1000, 2056),
                      (64, 3072, 512), (33, 40, 264), (32, 6144, 1536), (25, 1000, 12288), (20, 40, 264),
                      (32, 104, 8192), (16, 1024, 49152), (11, 200, 8200), (20, 4750, 1504), (32, 9601, 544)]:
        if epi == 2 and M > 32 and N * K > 4e6:
            continue
        x = torch.randn(M, K).to(dt)
        W = (torch.randn(N, K) / math.sqrt(K)).to(dt)
        W2 = (torch.randn(N, K) / math.sqrt(K)).to(dt)
        resid = torch.randn(M, N).to(dt)
        ref = _lin_ref(x, W, W2, resid, epi, dt)
        y = ops.linear(x.to(dev()), W.to(dev()), W2=W2.to(dev()) if epi == 2 else None,
                       resid=resid.to(dev()) if epi == 1 else None, epilogue=epi, backend=3)
        ops.check_status()
        close(y, ref, TOL[dt] / 2, what=f"{M}x{N}x{K}")


@pytest.mark.parametrize("epi", [0, 1])
def test_linear_wide_tensor_core_tiles(epi):
    """Outputs with at least two waves of 128 x 256 tiles take the wide-tile tcgen05 kernel; ragged M, N and K."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(5)
    dt = torch.bfloat16
    for (M, N, K) in [(20000, 520, 136), (9000, 1024, 264), (38000, 776, 64)]:
        x = torch.randn(M, K).to(dt)
        W = (torch.randn(N, K) / math.sqrt(K)).to(dt)
        resid = torch.randn(M, N).to(dt)
        ref = _lin_ref(x, W, None, resid, epi, dt)
        y = ops.linear(x.to(dev()), W.to(dev()), resid=resid.to(dev()) if epi == 1 else None, epilogue=epi, backend=2)
        ops.check_status()
        close(y, ref, TOL[dt] / 2)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(65, 64, 24, 0), (200, 65, 70, 2), (256, 512, 6144, 1), (300, 130, 264, 2), (64, 700, 3000, 0),
                                   (2500, 2500, 40, 0), (100, 333, 1027, 1)])
def test_linear_cuda_core_tiles(dt, shape):
    """The CUDA-core GEMM at the edges of its 64 x 64 tiles, K split over clusters of 1 to 8 CTAs, ragged K and rows off
    the 16-byte grid; lower-triangular weights with and without the flag."""
    from flash_stu_2_b200 import ops
    M, N, K, epi = shape
    torch.manual_seed(7)
    x, W, W2 = torch.randn(M, K).to(dt), (torch.randn(N, K) / math.sqrt(K)).to(dt), (torch.randn(N, K) / math.sqrt(K)).to(dt)
    resid = torch.randn(M, N).to(dt)
    y = ops.linear(x.to(dev()), W.to(dev()), W2=W2.to(dev()) if epi == 2 else None,
                   resid=resid.to(dev()) if epi == 1 else None, epilogue=epi, backend=1)
    close(y, _lin_ref(x, W, W2, resid, epi, dt), TOL[dt] / 2)
    if epi == 0:
        Wl = torch.tril(W)
        y = ops.linear(x.to(dev()), Wl.to(dev()), epilogue=ops.EPI_STORE | ops.EPI_FLAG_CAUSAL, backend=1)
        close(y, _lin_ref(x, Wl, None, None, 0, dt), TOL[dt] / 2)
    ops.check_status()


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(70, 512, 512), (65, 200, 333), (4000, 2500, 2500)])
def test_linear_cuda_core_tiles_skip_what_a_triangular_weight_leaves_out(dt, shape):
    """The CUDA-core GEMM reads nothing of a lower-triangular weight past the last column of a tile (64 wide, K split or not): NaN
    from there on."""
    from flash_stu_2_b200 import ops
    M, N, K = shape
    torch.manual_seed(7)
    x, W = torch.randn(M, K).to(dt), torch.tril(torch.randn(N, K) / math.sqrt(K)).to(dt)
    hole = torch.arange(K)[None, :] >= (torch.arange(N)[:, None] // 64 + 1) * 64
    y = ops.linear(x.to(dev()), W.masked_fill(hole, float("nan")).to(dev()), epilogue=ops.EPI_STORE | ops.EPI_FLAG_CAUSAL, backend=1)
    close(y, _lin_ref(x, W, None, None, 0, dt), TOL[dt] / 2)
    ops.check_status()


@pytest.mark.parametrize("M,N,ld,at,K", [(300, 257, 259, 3, 768), (300, 640, 645, 7, 840), (300, 71, 77, 0, 776), (300, 320, 322, 1, 2048), (6000, 5121, 5121, 1, 832),
                                         (6000, 5121, 5121, 5, 840), (300, 12289, 12295, 2, 840)])
def test_linear_odd_rows_by_shifted_pieces_and_singly(M, N, ld, at, K):
    """Rows off the 16-byte grid on either side of the K and the number of tiles from which they are stored value by value (the last but
    one is; single CTAs' tiles): every phase of a row against the 16-byte pieces of memory, blocks of 64 columns and the columns behind the
    last; nothing is written between the rows."""
    from flash_stu_2_b200 import ops
    g = torch.Generator(device=dev()).manual_seed(N + K)
    x, W = torch.randn(M, K, device=dev(), generator=g).bfloat16(), (torch.randn(N, K, device=dev(), generator=g) / math.sqrt(K)).bfloat16()
    buf = torch.full((M * ld + at,), 7.0, dtype=torch.bfloat16, device=dev())
    y = buf[at:].view(M, ld)
    ops.linear(x, W, out=y[:, :N], backend=ops.BACKEND_TCGEN05)
    ops.check_status()
    close(y[:, :N], _lin_ref(x, W, None, None, 0, torch.bfloat16), 2 ** -7)   # the next value of an output at most
    assert bool((y[:, N:] == 7.0).all()) and bool((buf[:at] == 7.0).all())


@pytest.mark.parametrize("shape", [(129, 257, 64, 257), (300, 71, 72, 75), (65, 4097, 128, 4097), (2500, 5121, 64, 5121)])
def test_linear_output_rows_off_the_16_byte_grid(shape):
    """Plain stores of the tcgen05 GEMM to rows of any stride (an odd vocabulary), square and wide tiles; nothing is
    written between the rows."""
    from flash_stu_2_b200 import ops
    M, N, K, ld = shape
    torch.manual_seed(6)
    x, W = torch.randn(M, K).bfloat16(), (torch.randn(N, K) / math.sqrt(K)).bfloat16()
    buf = torch.full((M * ld + 1,), 7.0, dtype=torch.bfloat16, device=dev())
    y = buf[1:].view(M, ld)   # two bytes off the grid as well
    ops.linear(x.to(dev()), W.to(dev()), out=y[:, :N], backend=2)
    ops.check_status()
    close(y[:, :N], _lin_ref(x, W, None, None, 0, torch.bfloat16), 1e-2)
    assert bool((y[:, N:] == 7.0).all()) and float(buf[0]) == 7.0


@pytest.mark.parametrize("shape", [(3, 70, 37, 0, 40), (2, 300, 129, 5, 72), (1, 2000, 64, 16, 48), (4, 1024, 1999, 0, 1000),
                                   (2, 264, 96, 33, 67)])
def test_projection_into_history_off_the_block_grid(shape):
    """EPI_HIST of the tcgen05 GEMM for sequences, first positions and history pitches that are no multiple of its
    32-token blocks, square and wide tiles: every new position lands in its parity row, nothing else is written."""
    from flash_stu_2_b200 import ops
    B, d, T, t0, Lh = shape
    torch.manual_seed(8)
    x, W = torch.randn(B, T, 64).bfloat16(), (torch.randn(d, 64) / 8).bfloat16()
    hist = torch.full((B, d, 2, Lh), 7.0, dtype=torch.bfloat16, device=dev())
    ops.linear(x.view(B * T, 64).to(dev()), W.to(dev()), out=hist, epilogue=ops.EPI_HIST, hist_T=T, hist_t0=t0,
               hist_Lh=Lh, backend=2)
    ops.check_status()
    flat = hist.cpu().transpose(2, 3).reshape(B, d, 2 * Lh)
    close(flat[:, :, t0:t0 + T], _lin_ref(x.view(B * T, 64), W, None, None, 0, torch.bfloat16).view(B, T, d).transpose(1, 2),
          1e-2)
    assert bool((flat[:, :, :t0] == 7.0).all()) and bool((flat[:, :, t0 + T:] == 7.0).all())


def test_bounded_wait_expiry_is_reported_and_the_context_survives():
    """Failure detection inside the tcgen05 GEMM: with the copies of its first pipeline stage dropped (test hook) the
    consumer's bounded wait runs out after the shortened limit; the kernel reports status 3, frees its tensor memory
    and returns, the host raises, and the next GEMM on the same context is correct.  Nothing faults or hangs."""
    import time
    from flash_stu_2_b200 import _lib, ops
    lib = _lib.load()
    torch.manual_seed(21)
    dt = torch.bfloat16
    x = torch.randn(128, 64).to(dt)
    W = (torch.randn(128, 64) / 8).to(dt)
    xd, Wd = x.to(dev()), W.to(dev())
    ref = _lin_ref(x, W, None, None, 0, dt)
    close(ops.linear(xd, Wd, backend=2), ref, TOL[dt] / 2)      # the healthy kernel first
    ops.check_status()
    assert lib.stu_test_inject_wait_expiry(100) == 0
    try:
        t0 = time.monotonic()
        ops.linear(xd, Wd, backend=2)
        torch.cuda.synchronize()
        assert time.monotonic() - t0 < 5.0                           # returned by itself, within the shortened bound
        with pytest.raises(RuntimeError, match="status 3"):
            ops.check_status()
    finally:
        assert lib.stu_test_inject_wait_expiry(0) == 0
    close(ops.linear(xd, Wd, backend=2), ref, TOL[dt] / 2)      # same context, same kernel, healthy again
    big = torch.randn(300, 136).to(dt)
    Wb = (torch.randn(200, 136) / 12).to(dt)
    close(ops.linear(big.to(dev()), Wb.to(dev()), backend=2), _lin_ref(big, Wb, None, None, 0, dt), TOL[dt] / 2)
    ops.check_status()


def test_bounded_wait_expiry_of_single_ctas():
    """The same for the GEMM's form with a CTA in the place of a pair (300 x 12288 outputs), every CTA of which gives up."""
    from flash_stu_2_b200 import _lib, ops
    lib = _lib.load()
    g = torch.Generator(device=dev()).manual_seed(22)
    x, W = torch.randn(300, 136, device=dev(), generator=g).bfloat16(), (torch.randn(12288, 136, device=dev(), generator=g) / 12).bfloat16()
    want = ops.linear(x, W, backend=2)
    ops.check_status()
    close(want, _lin_ref(x, W, None, None, 0, torch.bfloat16), 2 ** -7)
    assert lib.stu_test_inject_wait_expiry(100) == 0
    try:
        ops.linear(x, W, backend=2)
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="status 3"):
            ops.check_status()
    finally:
        assert lib.stu_test_inject_wait_expiry(0) == 0
    assert torch.equal(ops.linear(x, W, backend=2), want)
    ops.check_status()


def _gives_up(call, status):
    """The next launch never has its first stage: it returns within its shortened bound and says so."""
    import time
    from flash_stu_2_b200 import _lib, ops
    lib = _lib.load()
    ops.check_status()
    assert lib.stu_test_inject_wait_expiry(100) == 0
    try:
        t0 = time.monotonic()
        call()
        torch.cuda.synchronize()
        assert time.monotonic() - t0 < 5.0
        with pytest.raises(RuntimeError, match=f"status {status}"):
            ops.check_status()
    finally:
        assert lib.stu_test_inject_wait_expiry(0) == 0


@pytest.mark.parametrize("shape", [(2500, 1000, 96), (100, 96, 4096), (300, 2000, 512)])
def test_bounded_wait_expiry_of_the_fp32_gemm(shape):
    """Two blocks of K, K split over a cluster of which one CTA gives up, eight blocks: nothing is stored by a cluster that lacks a part, and the next call is
    correct."""
    from flash_stu_2_b200 import ops
    M, N, K = shape
    g = torch.Generator(device=dev()).manual_seed(23)
    x, W = torch.randn(M, K, device=dev(), generator=g), torch.randn(N, K, device=dev(), generator=g)
    want, out = ops.linear(x, W), torch.full((M, N), 7.0, device=dev())
    _gives_up(lambda: ops.linear(x, W, out=out), 3)
    assert bool((out == 7.0).all())
    assert torch.equal(ops.linear(x, W, out=out), want)
    ops.check_status()


@pytest.mark.parametrize("shape", [(333, 1536, 6144), (5193, 1000, 4096)])   # parts alone; whole tiles of several accumulators ahead of them
def test_bounded_wait_expiry_of_a_linear_in_parts(shape):
    from flash_stu_2_b200 import ops
    M, N, K = shape
    g = torch.Generator(device=dev()).manual_seed(26)
    x, W = torch.randn(M, K, device=dev(), generator=g).bfloat16(), torch.randn(N, K, device=dev(), generator=g).bfloat16()
    want = _linear_in_parts(x, W)
    _gives_up(lambda: _linear_in_parts(x, W), 3)
    assert torch.equal(_linear_in_parts(x, W), want)
    ops.check_status()


def test_bounded_wait_expiry_of_the_fp32_convolutions():
    from flash_stu_2_b200 import ops
    torch.manual_seed(24)
    hist, phi = torch.randn(2, 8, 2, 256, device=dev()), torch.randn(500, 3, device=dev())
    U = [torch.empty(2 * 500, 2 * 3 * 8, device=dev()) for _ in range(3)]
    ops.full_conv_f32_tc5(hist, phi, U[0], True, 0, 500)
    _gives_up(lambda: ops.full_conv_f32_tc5(hist, phi, U[1], True, 0, 500), 9)
    ops.full_conv_f32_tc5(hist, phi, U[2], True, 0, 500)
    ops.check_status()
    assert torch.equal(U[0], U[2])


@pytest.mark.parametrize("t", [100, 1001])
def test_bounded_wait_expiry_of_the_full_variants_step(monkeypatch, t):
    """One stage (the position's) and more stages than the ring holds."""
    from flash_stu_2_b200 import ops
    monkeypatch.setattr(ops, "full_decode_step_tc5_pays", lambda *a: True)
    torch.manual_seed(25)
    B, d, K, Lh = 2, 64, 24, 512
    hist, x, w = (torch.randn(*s, device=dev()).bfloat16() for s in ((B, d, 2, Lh), (B, d), (d,)))
    phi = (torch.randn(2 * Lh, K, device=dev()) / 4).bfloat16()
    taps8 = ops.taps_rev8(torch.cat([ops.taps_even(phi, Lh), ops.taps_even(phi[1:], Lh)]))
    pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())

    def step():
        pos[:, 0] = t
        U = torch.full((B, 2 * K * d), 7.0, device=dev()).bfloat16()
        ops.full_decode_step(x, w, ops.RMS_EPS, hist, taps8, pos, U, 2 * Lh, True, t)
        return U

    want, given_up = step(), []
    _gives_up(lambda: given_up.append(step()), 9)
    assert bool((given_up[0] == 7.0).all()) and pos[:, 1].tolist() == [0] * B
    assert torch.equal(step(), want) and pos.tolist() == [[t + 1, 0]] * B
    ops.check_status()


def test_linear_fused_norm_decode():
    """RMSNorm fused into the mma.sync token-step linears (every row count up to 64; callers use it up to 16 rows)."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(2)
    for (M, N, K, epi) in [(8, 4096, 1024, 2), (32, 1536, 1536, 0), (5, 104, 64, 1), (48, 4608, 1536, 0),
                           (20, 1000, 520, 1), (64, 72, 2048, 0), (32, 6144, 1536, 2), (19, 200, 512, 2),
                           (16, 1536, 3072, 0), (12, 6144, 1504, 2), (32, 1536, 4104, 0), (64, 6144, 3072, 2)]:
        dt = torch.bfloat16
        x = torch.randn(M, K).to(dt)
        nw = torch.randn(K).to(dt)
        W = (torch.randn(N, K) / math.sqrt(K)).to(dt)
        W2 = (torch.randn(N, K) / math.sqrt(K)).to(dt)
        resid = torch.randn(M, N).to(dt)
        ref = _lin_ref(O.rmsnorm(x, nw), W, W2, resid, epi, dt)
        y = ops.linear(x.to(dev()), W.to(dev()), W2=W2.to(dev()) if epi == 2 else None,
                       resid=resid.to(dev()) if epi == 1 else None, epilogue=epi, norm_w=nw.to(dev()))
        ops.check_status()
        close(y, ref, 1e-2, what=f"{M}x{N}x{K}")


def test_linear_transposed_small_k():
    """phi @ M_filters: K = num_eigh = 24 inner dimension, weight given as [K, N]."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(3)
    for dt in (torch.float32, torch.bfloat16):
        phi = torch.randn(130, 24).to(dt)
        Mf = torch.randn(24, 72).to(dt)
        y = ops.linear(phi.to(dev()), Mf.to(dev()), transposed_weight=True, backend=1)
        close(y, (phi.double() @ Mf.double()).to(dt), TOL[dt] / 4)


def _hist_from(xp, Lh):
    B, T, d = xp.shape
    h = torch.zeros(B, d, 2, Lh, dtype=xp.dtype)
    for p in range(2):
        n = (T - p + 1) // 2
        h[:, :, p, :n] = xp[:, p::2].transpose(1, 2)
    return h


@pytest.mark.parametrize("dt,tc", [(torch.float32, False), (torch.bfloat16, False), (torch.bfloat16, True)])
@pytest.mark.parametrize("shape", [(2, 64, 16, 0), (3, 300, 40, 0), (9, 1100, 8, 0), (2, 1301, 8, 655)])
def test_conv_prefill_matches_fft_oracle(dt, tc, shape):
    """x += conv_plus + conv_minus of the reference (FFT, fp32) == 2 * even-tap direct sum."""
    from flash_stu_2_b200 import ops
    B, T, d, t0 = shape
    torch.manual_seed(4)
    L = T + 3
    Lh = ((L + 1) // 2 + 7) // 8 * 8
    xp = torch.randn(B, T, d).to(dt)
    fp = (torch.randn(L, d) / math.sqrt(L)).to(dt)
    x0 = torch.randn(B, T, d).to(dt)
    n = O.fft_length(L)
    plus, minus = O.convolve(xp, fp, n, True, True)
    ref = (x0.float() + (plus + minus).float()).to(dt)
    hist = _hist_from(xp, Lh).to(dev())
    taps = ops.taps_even(fp.to(dev()), Lh)
    yT = torch.full((B, d, 2, ((T + 1) // 2 + 7) // 8 * 8), float("nan"), dtype=dt, device=dev())
    x = x0[:, t0:].contiguous().to(dev())
    ops.conv_prefill_approx(hist, taps, yT, x, t0, T, use_tensor_cores=tc)
    # bf16: the reference rounds each branch before the add, the kernel rounds the folded sum once
    # bf16: the reference rounds each branch before adding them, the kernel rounds the folded sum once; on rows whose
    # largest value is small that is up to two bf16 ulps of the branch magnitude (observed 1.75e-2 per row)
    close(x, ref[:, t0:], (2e-5 if dt == torch.float32 else 1.5e-2), row_tol=(2e-5 if dt == torch.float32 else 2e-2))


@pytest.mark.parametrize("shape", [(2, 250, 16, 0), (3, 700, 24, 0), (9, 1100, 8, 0), (2, 1301, 8, 655),
                                   (1, 8800, 8, 0), (2, 9001, 8, 8300)])
def test_conv_prefill_tcgen05_matches_fft_oracle(shape):
    """The tcgen05 prefill convolution against the reference's FFT convolution (fp32): histories of one and of two
    accumulator-sized superblocks (more than 4096 positions per parity), more than 8 sequences, a resumed prefill
    (t0 > 0), and NaN in the cache past the valid positions, which must not reach any output."""
    from flash_stu_2_b200 import ops
    B, T, d, t0 = shape
    torch.manual_seed(4)
    L = T + 3
    Lh = ((L + 1) // 2 + 127) // 128 * 128
    xp = torch.randn(B, T, d).bfloat16()
    fp = (torch.randn(L, d) / math.sqrt(L)).bfloat16()
    x0 = torch.randn(B, T, d).bfloat16()
    plus, minus = O.convolve(xp, fp, O.fft_length(L), True, True)
    ref = (x0.float() + (plus + minus).float()).bfloat16()
    hist = _hist_from(xp, Lh)
    for p in range(2):
        hist[:, :, p, (T - p + 1) // 2:] = float("nan")
    hist = hist.to(dev())
    taps = ops.taps_even(fp.to(dev()), Lh)
    taps8 = ops.taps_rev8(taps)
    yT = torch.full((B, d, 2, ((T + 1) // 2 + 7) // 8 * 8), float("nan"), dtype=torch.bfloat16, device=dev())
    x = x0[:, t0:].contiguous().to(dev())
    assert ops.conv_prefill_tc5_supported(hist, x)
    ops.conv_prefill_approx_tc5(hist, taps8, yT, x, t0, T)
    ops.check_status()
    # the reference rounds each branch to bf16 before adding them; over thousands of positions the branches grow
    # against their sum, so a row of 8 channels sees up to three ulps of that rounding
    close(x, ref[:, t0:], 1.5e-2, row_tol=(2e-2 if T < 4096 else 3e-2))
    # and against the mma.sync kernel on the same operands: same products, fp32 sums in another order
    hist0 = torch.nan_to_num(hist, nan=0.0)
    x2 = x0[:, t0:].contiguous().to(dev())
    ops.conv_prefill_approx(hist0, taps, torch.zeros_like(yT), x2, t0, T, use_tensor_cores=True)
    close(x, x2, 8e-3, row_tol=1.6e-2)


@pytest.mark.parametrize("shape", [(65, 100, 1024), (127, 33, 1028), (129, 1, 2060), (300, 2049, 256), (1000, 700, 516), (8000, 96, 3072), (66, 512, 6144),
                                   (2000, 1030, 100)])
@pytest.mark.parametrize("epi", [0, 1, 2, 3])
def test_fp32_linear_on_tensor_cores(shape, epi):
    """fp32 products as six bf16 products: edges of tiles, of blocks of 64 of K and of its split over clusters, each epilogue.  Bar:
    against float64 no further off than the CUDA-core GEMM on the same operands, but for the rounding of the result itself (2^-24)."""
    from flash_stu_2_b200 import ops
    M, N, K = shape
    torch.manual_seed(5)
    x = torch.randn(M, K + 4, device=dev())[:, :K]          # rows that do not follow one another
    W, W2 = torch.randn(2, N, K, device=dev()) / math.sqrt(K)
    r = torch.randn(M, N, device=dev())
    full = x.double() @ W.double().t()
    Lh = (M // 16 + 1) * 8
    kw = {0: {}, 1: dict(resid=r), 2: dict(W2=W2), 3: dict(hist_T=M, hist_t0=1, hist_Lh=Lh)}[epi]
    err = []
    for backend in (0, 1):
        out = torch.zeros(1, N, 2, Lh, device=dev()) if epi == 3 else torch.full((M, N), float("nan"), device=dev())
        ops.linear(x, W, out=out, epilogue=epi, backend=backend, **kw)
        if epi == 3:
            t = torch.arange(1, M + 1, device=dev())
            assert int((out != 0).sum()) <= M * N
            out = out[0][:, t % 2, t // 2].t()
        want = {0: full, 1: r.double() + full, 2: torch.nn.functional.gelu(full, approximate="tanh") * (x.double() @ W2.double().t()), 3: full}[epi]
        err.append(float((out.double() - want).norm() / want.norm()))
    ops.check_status()
    assert err[0] <= max(err[1], 2.0 ** -24), err


@pytest.mark.parametrize("shape", [(4000, 2500, 2500), (70, 1100, 1100), (300, 2049, 1024), (66, 40, 3072)])
@pytest.mark.parametrize("epi", [0, 1, 2])
def test_fp32_linear_of_triangular_weights_stays_on_the_cuda_cores(shape, epi):
    """NaN past the blocks of 64 columns, of which that GEMM reads nothing; short rows are sums that it makes more exactly."""
    from flash_stu_2_b200 import ops
    M, N, K = shape
    torch.manual_seed(7)
    x, r = torch.randn(M, K, device=dev()), torch.randn(M, N, device=dev())
    hole = torch.arange(K, device=dev())[None, :] >= (torch.arange(N, device=dev())[:, None] // 64 + 1) * 64
    W, W2 = torch.tril(torch.randn(2, N, K, device=dev()) / math.sqrt(K)).masked_fill(hole, float("nan"))
    kw = {0: {}, 1: dict(resid=r), 2: dict(W2=W2)}[epi]
    y = [ops.linear(x, W, epilogue=epi | ops.EPI_FLAG_CAUSAL, backend=b, **kw) for b in (0, 1)]
    ops.check_status()
    assert bool(y[0].isfinite().all()) and torch.equal(*y)


@pytest.mark.parametrize("B,T,t0,N,K", [(3, 100, 5, 200, 1024), (7, 33, 0, 130, 2048), (2, 1000, 301, 72, 1028)])
def test_fp32_histories_of_several_sequences_on_tensor_cores(B, T, t0, N, K):
    """Tiles that end inside a sequence's positions and hold several, behind positions that are there and stay as they are."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(6)
    x, W = torch.randn(B * T, K, device=dev()), torch.randn(N, K, device=dev()) / math.sqrt(K)
    Lh = (t0 + T) // 2 + 9
    full = (x.double() @ W.double().t()).view(B, T, N)
    t, err = torch.arange(t0, t0 + T, device=dev()), []
    for backend in (0, 1):
        hist = torch.full((B, N, 2, Lh), 7.0, device=dev())
        ops.linear(x, W, out=hist, epilogue=ops.EPI_HIST, hist_T=T, hist_t0=t0, hist_Lh=Lh, backend=backend)
        got = hist[:, :, t % 2, t // 2].transpose(1, 2)
        assert int((hist != 7.0).sum()) == B * T * N
        err.append(float((got.double() - full).norm() / full.norm()))
    ops.check_status()
    assert err[0] <= max(err[1], 2.0 ** -24), err


# The largest second and third parts, of one sign: what the six products leave out of each is 2^-23.03 of it, and adds up
WORST = 1 + 2.0 ** -8 - 2.0 ** -23


@pytest.mark.parametrize("shape", [(640, 512, 256), (129, 96, 1024), (300, 640, 3072)])
@pytest.mark.parametrize("signs", [(1, 1), (-1, 1), (-1, -1)])
def test_fp32_linear_on_tensor_cores_largest_parts(shape, signs):
    """Bar: 2^-23 for what is left out, as much for either of the two instructions with an accumulator's largest products (their sums are cut off), and half an ulp
    for each of the K / 32 accumulators that are added up."""
    from flash_stu_2_b200 import ops
    M, N, K = shape
    x, W = torch.full((M, K), signs[0] * WORST, device=dev()), torch.full((N, K), signs[1] * WORST, device=dev())
    err = [float((ops.linear(x, W, backend=b).double() / (signs[0] * signs[1] * K * WORST ** 2) - 1).abs().max()) for b in (0, 1)]
    ops.check_status()
    assert err[0] <= (3 + K / 64) * 2.0 ** -23, err


@pytest.mark.parametrize("B,T,d,K", [(2, 900, 64, 3), (1, 513, 132, 2)])
def test_full_variant_fp32_convolutions_of_the_largest_parts(B, T, d, K):
    """As above with an accumulator for 64 positions of a parity, and one sum of the two parities' sums."""
    from flash_stu_2_b200 import ops
    Lh = (T // 2 + 8) // 8 * 8
    hist, phi = torch.full((B, d, 2, Lh), WORST, device=dev()), torch.full((T, K), WORST, device=dev())
    U = torch.full((B * T, K * d), float("nan"), device=dev())
    ops.full_conv_f32_tc5(hist, phi, U, False, 0, T)
    ops.check_status()
    terms = torch.arange(1, T + 1, device=dev(), dtype=torch.float64).view(1, T, 1)
    err = (U.double().view(B, T, K * d) / (terms * WORST ** 2) - 1).abs()
    assert bool((err <= (4 + 2 * math.ceil(T / 128)) * 2.0 ** -23).all()), float(err.max())


# (rows, outputs, K, distance of the outputs' rows): one tile in parts of unequal length, edges of tiles, odd row strides, whole tiles ahead of the split ones
@pytest.mark.parametrize("shape", [(65, 64, 24576, 64), (257, 513, 12296, 513), (333, 1536, 6144, 1540), (70, 1030, 49152, 1033), (140, 1001, 8200, 1002),
                                   (5193, 1000, 4096, 1000), (19851, 512, 3072, 512)])
@pytest.mark.parametrize("epi", [0, 1])
def test_linear_of_long_weights_in_parts(shape, epi):
    """bf16 products whose K is cut over the SMs.  Bars: a plain result is the float64 one rounded once, but for fp32 sums of K products; a
    residual is added to the rounded product; without the workspace the call is the product in one piece."""
    from flash_stu_2_b200 import _lib, ops
    M, N, K, ld = shape
    if epi and (N % 8 or ld % 8):
        ld = N = N // 8 * 8      # residual rows lie on the 16-byte grid
    assert _lib.load().stu_linear_workspace_elems(M, N, K, epi, 1) >= 2 * 65536
    torch.manual_seed(8)
    x = torch.randn(M, K + 8, device=dev()).bfloat16()[:, :K]
    W = (torch.randn(N, K + 16, device=dev()) / math.sqrt(K)).bfloat16()[:, :K]
    r = torch.randn(M, ld, device=dev()).bfloat16()[:, :N]
    buf = torch.full((M + 1, ld), 7.0, device=dev(), dtype=torch.bfloat16)
    out = buf[:M, :N]
    ops.linear(x, W, out=out, epilogue=epi, resid=r if epi else None)
    ops.check_status()
    assert bool((buf[M] == 7).all()) and bool((buf[:, N:] == 7).all())
    full = torch.cat([x[i:i + 2048].double() @ W.double().t() for i in range(0, M, 2048)])
    # sums of K products of order 1/sqrt(K): 2^-24 * sqrt(K) * a few, well below 1e-4 for every K here
    lo, hi = (full - 1e-4).bfloat16(), (full + 1e-4).bfloat16()
    if epi:
        lo, hi = (r.float() + lo.float()).bfloat16(), (r.float() + hi.float()).bfloat16()
    assert bool(((out >= lo) & (out <= hi)).all())
    if epi == 0:
        short = torch.empty(M, N, device=dev(), dtype=torch.bfloat16)
        work = torch.full((64,), float("nan"), device=dev())
        rc = _lib.load().stu_linear_split(x.data_ptr(), K + 8, W.data_ptr(), K + 16, 1, None, None, 0, short.data_ptr(), N, M, N, K, 0, 0, 0, 0, None, 0.0, 1, 0,
                                          work.data_ptr(), 64, torch.cuda.current_stream().cuda_stream)
        whole = torch.empty_like(short)
        rc2 = _lib.load().stu_linear(x.data_ptr(), K + 8, W.data_ptr(), K + 16, 1, None, None, 0, whole.data_ptr(), N, M, N, K, 0, 0, 0, 0, None, 0.0, 1, 0,
                                     torch.cuda.current_stream().cuda_stream)
        assert rc == rc2 == 0 and torch.equal(short, whole) and bool(work.isnan().all())


def _linear_in_parts(x, W, r=None):
    """stu_linear_split with the workspace that it wants: the op asks for one from 16384 of K on alone."""
    from flash_stu_2_b200 import _lib, ops
    (M, K), N = x.shape, W.shape[0]
    elems = _lib.load().stu_linear_workspace_elems(M, N, K, int(r is not None), 1)
    assert elems > 0
    work, y = torch.empty(elems, device=dev()), torch.empty(M, N, device=dev(), dtype=torch.bfloat16)
    ops.status_word(x.device)
    rc = _lib.load().stu_linear_split(x.data_ptr(), K, W.data_ptr(), K, 1, None, r.data_ptr() if r is not None else None, N, y.data_ptr(), N, M, N, K,
                                      int(r is not None), 0, 0, 0, None, 0.0, 1, 0, work.data_ptr(), elems, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and _lib.load().stu_linear_launches() == 2
    return y


@pytest.mark.parametrize("shape", [(5193, 1000, 4096), (19851, 512, 3072), (16384, 1536, 6144), (5193, 1001, 4104), (2100, 200, 24576)])
@pytest.mark.parametrize("epi", [0, 1])
def test_equal_rows_of_a_linear_in_parts_are_equal(shape, epi):
    """Tiles of which K is cut and, ahead of them, whole ones: an output is the same sum in either, so sequences of a batch do not differ by where they stand."""
    M, N, K = shape
    if epi:
        N = N // 8 * 8
    from flash_stu_2_b200 import ops
    torch.manual_seed(11)
    three = torch.randn(3, K, device=dev()).bfloat16()
    x, W = three.repeat(-(-M // 3), 1)[:M], (torch.randn(N, K, device=dev()) / math.sqrt(K)).bfloat16()
    r = torch.randn(3, N, device=dev()).bfloat16().repeat(-(-M // 3), 1)[:M] if epi else None
    y = _linear_in_parts(x, W, r)
    ops.check_status()
    assert torch.equal(y, y[:3].repeat(-(-M // 3), 1)[:M])
    full = three.double() @ W.double().t() + (r[:3].double() if epi else 0.0)
    assert float((y[:3].double() - full).abs().max()) <= 2.0 ** -7 * max(1.0, float(full.abs().max()))


@pytest.mark.parametrize("shape", [(333, 1536, 6144), (28924, 512, 2048), (16384, 1536, 6144), (900, 3072, 12288)])
def test_a_models_products_have_one_chain_whatever_the_batch(shape):
    """The rows of a prefill in one call and in calls of other sizes, through the tiles' forms and edges: the same results (an MLP's K)."""
    from flash_stu_2_b200 import _lib, ops
    M, N, K = shape
    assert _lib.load().stu_linear_workspace_elems(M, N, K, 1, 1) > 0   # (a cut would pay)
    torch.manual_seed(13)
    x, W, r = torch.randn(M, K, device=dev()).bfloat16(), (torch.randn(N, K, device=dev()) / math.sqrt(K)).bfloat16(), torch.randn(M, N, device=dev()).bfloat16()
    whole = ops.linear(x, W, resid=r, epilogue=1)
    for n in (72, M // 3, M - 72):   # (more rows than a token step's)
        assert torch.equal(ops.linear(x[:n], W, resid=r[:n], epilogue=1), whole[:n])
    ops.check_status()


@pytest.mark.parametrize("shape,launches", [((333, 1536, 24576), 2), ((65, 64, 24576), 2), ((333, 1536, 512), 1), ((64, 64, 24576), 1)])
def test_launches_of_a_linear_are_counted(shape, launches):
    """A product whose K is cut is added up in a launch of its own; on the CUDA cores (asked for, or rows that the tensor cores do not take) it is one launch."""
    from flash_stu_2_b200 import _lib, ops
    M, N, K = shape
    assert (_lib.load().stu_linear_workspace_elems(M, N, K, 0, 1) > 0) == (launches == 2)
    x, W = torch.ones(M, K, device=dev(), dtype=torch.bfloat16), torch.ones(N, K, device=dev(), dtype=torch.bfloat16)
    odd = torch.ones(M, K + 1, device=dev(), dtype=torch.bfloat16)[:, :K]   # rows off the 16-byte grid: not on the tensor cores
    for rows, backend, want in ((x, 0, launches), (x, 1, 1), (odd, 0, 1), (x, 0, launches)):
        before = ops.launch_count
        ops.linear(rows, W, backend=backend)
        assert ops.launch_count - before == want


@pytest.mark.parametrize("shape", [(128, 1024, 16384), (333, 1536, 24576), (65, 64, 24576)])
@pytest.mark.parametrize("given", [False, True])
def test_a_linear_in_parts_takes_its_workspace_from_the_arena(shape, given):
    """The buffer that a caller gives for a captured step holds the parts of K as well, for one product at a time; the sums are those of a call outside."""
    from flash_stu_2_b200 import _lib, ops
    M, N, K = shape
    torch.manual_seed(4)
    x, W = (torch.randn(r, K, device=dev()).bfloat16() for r in (M, N))
    parts = _lib.load().stu_linear_workspace_elems(M, N, K, 0, 1)
    assert parts > 0
    want = ops.linear(x, W)
    room = (2 * M * N + 255) // 256 * 256
    buffer = torch.empty(4 * parts + 3 * room, dtype=torch.uint8, device=dev())
    outs = [torch.empty_like(want) for _ in range(3)] if given else [None] * 3
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    with ops.arena(buffer):
        got = [ops.linear(x, W, out=out) for out in outs]
    assert torch.cuda.memory_stats()["allocation.all.allocated"] == before
    ops.check_status()
    assert all(torch.equal(g, want) for g in got)


@pytest.mark.parametrize("shape", [(8, 1024, 49152), (1, 640, 14720), (5, 768, 12296), (7, 1200, 4104), (8, 2049, 4096), (3, 4735, 8192)])
@pytest.mark.parametrize("epi", [0, 1])
@pytest.mark.parametrize("early", [False, True])
def test_linear_of_few_rows_over_long_weights(shape, epi, early):
    """Up to 8 rows: clusters of one, two and four CTAs, features and K that end inside a tile and a chunk, launched beside the kernel in
    front that writes its rows.  Bar: one rounding to bf16 of a sum of K products (and of its sum with the residual)."""
    from flash_stu_2_b200 import ops
    M, N, K = shape
    torch.manual_seed(9)
    x, W, r = torch.randn(M, K), torch.randn(N, K) / math.sqrt(K), torch.randn(M, N)
    x, W, r = (t.bfloat16().to(dev()) for t in (x, W, r))
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=dev())
    rows = ops.rmsnorm(x, torch.ones(K, dtype=torch.bfloat16, device=dev()), 1e-6)   # the kernel in front
    ops.linear(rows, W, resid=r if epi else None, out=out, epilogue=epi | (ops.FLAG_OVERLAP if early else 0))
    ops.check_status()
    full = rows.double() @ W.double().t()
    want = (r.double() + full.bfloat16().double()) if epi else full
    assert float((out.double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max()) + 1e-3


@pytest.mark.parametrize("shape", [(8, 1024, 49152), (1, 640, 14720), (5, 768, 12296), (7, 1200, 4104), (3, 4735, 8192)])
@pytest.mark.parametrize("epi", [0, 1])
def test_linear_of_few_rows_over_long_weights_output_by_output(shape, epi):
    """Each output by itself: the float64 sum rounded once, but for fp32 sums of K products of order 1 / sqrt(K) (2^-24 * sqrt(K) * a few, well below
    1e-4), and the residual added to that."""
    from flash_stu_2_b200 import ops
    M, N, K = shape
    torch.manual_seed(12)
    x, W, r = torch.randn(M, K, device=dev()), torch.randn(N, K, device=dev()) / math.sqrt(K), torch.randn(M, N, device=dev())
    x, W, r = (t.bfloat16() for t in (x, W, r))
    out = ops.linear(x, W, resid=r if epi else None, epilogue=epi)
    ops.check_status()
    full = x.double() @ W.double().t()
    lo, hi = (full - 1e-4).bfloat16(), (full + 1e-4).bfloat16()
    if epi:
        lo, hi = (r.float() + lo.float()).bfloat16(), (r.float() + hi.float()).bfloat16()
    assert bool(((out >= lo) & (out <= hi)).all())


@pytest.mark.parametrize("case", [(1, 8, 3, 0, 17, True), (3, 20, 5, 5, 257, True), (2, 64, 4, 0, 256, False), (1, 132, 7, 250, 515, True),
                                  (5, 64, 24, 0, 1000, True)])
def test_full_variant_fp32_convolutions_on_tensor_cores(case):
    """Edges of blocks of 128 positions of a parity and of tiles of 64 and 128 channels, a resumed prefill, one sign; NaN in the cache behind
    the last position.  Bar: against float64 no further off than the CUDA-core kernel, but for the rounding of E and of Q (2^-23)."""
    from flash_stu_2_b200 import ops
    B, d, K, t0, T, both = case
    torch.manual_seed(3)
    x, phi = torch.randn(B, T, d), torch.randn(T - 2, K) / 8
    hist = _hist_from(x, (T + 31) // 16 * 8)
    for p in range(2):
        hist[:, :, p, (T - p + 1) // 2:] = float("nan")
    hist, phi = hist.to(dev()), phi.to(dev())
    U = [torch.full((B * (T - t0), (1 + both) * K * d), float("nan"), device=dev()) for _ in range(2)]
    ops.full_conv_f32_tc5(hist, phi, U[0], both, t0, T)
    ops.full_conv(torch.nan_to_num(hist), phi, U[1], both, t0, T)
    ops.check_status()
    n = 1 << (2 * T).bit_length()
    X, sign = torch.fft.rfft(x.double().to(dev()), n=n, dim=1), torch.ones(T - 2, 1, device=dev(), dtype=torch.float64)
    sign[1::2] = -1
    want = torch.cat([torch.einsum("bfi,fk->bfki", X, torch.fft.rfft(f, n=n, dim=0)) for f in (phi.double(), phi.double() * sign)[:1 + both]], 2)
    want = torch.fft.irfft(want, n=n, dim=1)[:, t0:T].reshape(B * (T - t0), -1)
    err = [float((u.double() - want).norm() / want.norm()) for u in U]
    assert err[0] <= max(err[1], 2.0 ** -23), err
    again = torch.full_like(U[0], float("nan"))   # operands past 2^87: every sum made again on the CUDA cores, the other kernel's chains
    ops.full_conv_f32_tc5(hist * 2.0 ** 90, phi * 2.0 ** -90, again, both, t0, T)
    ops.check_status()
    assert torch.equal(again, U[1])


def test_full_variant_fp32_convolutions_of_values_without_a_split():
    """An infinity, a NaN and a value whose parts overflow reach the results that they reach in fp32 arithmetic, and no others."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(4)
    B, T, d, K = 1, 300, 8, 3
    x, phi = torch.randn(B, T, d), torch.rand(T, K) + 0.5
    x[0, 100, 1], x[0, 200, 2], x[0, 250, 3] = float("inf"), float("nan"), 1e36
    hist = _hist_from(x, 152).to(dev())
    U = torch.empty(T, 2 * K * d, device=dev())
    ops.full_conv_f32_tc5(hist, phi.to(dev()), U, True, 0, T)
    ops.check_status()
    lag = torch.arange(T)[:, None] - torch.arange(T)[None]
    for s in range(2):
        taps = phi.double() * torch.where(torch.arange(T)[:, None] % 2 == 0, 1.0, 1.0 - 2 * s)
        got = U.view(T, 2, K, d)[:, s].cpu()
        for i in (0, 1, 2, 3):
            start = {1: 100, 2: 200}.get(i, T)
            assert bool(got[:start, :, i].isfinite().all()) and not bool(got[start:, :, i].isfinite().any())
            m = torch.where(lag[:start, :start, None] >= 0, taps[lag[:start, :start].clamp_min(0)], torch.zeros((), dtype=torch.float64))
            want = torch.einsum("tsk,s->tk", m, x[0, :start, i].double())
            assert float(((got[:start, :, i].double() - want).abs() / want.abs().clamp_min(1)).max()) < 1e-4   # (300 products in one chain)


def test_fp32_linear_on_tensor_cores_values_without_a_split():
    """Infinities, NaN and values whose parts overflow come out as fp32 arithmetic has them."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(6)
    x, W = torch.randn(200, 1024), torch.randn(70, 1024) / 32
    x[3, 5], x[7, 9], x[9, 1], x[11, :] = float("inf"), float("nan"), 3e38, 0.0
    x[11, 4], W[8, 2], W[:, 9] = 1e36, float("-inf"), 0.0
    got = ops.linear(x.to(dev()), W.to(dev()))
    want = ops.linear(x.to(dev()), W.to(dev()), backend=1)
    ops.check_status()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()], want[want.isinf()])
    fin = want.isfinite()
    assert float(((got - want)[fin].abs() / want[fin].abs().clamp_min(1)).max()) < 2e-5   # (1024 products of order 1/32: rounding of the partial sums)


@pytest.mark.parametrize("shape", [(65, 100, 1024), (129, 1, 2060), (300, 2049, 256), (1000, 700, 516), (66, 512, 6144)])
@pytest.mark.parametrize("epi", [0, 1, 2, 3])
def test_fp32_sums_on_tensor_cores_made_again(shape, epi):
    """Operands past 2^87 have no split: every sum is made on the CUDA cores behind the instructions.  Edges of tiles, of K and of its split, each
    epilogue, several sequences of a history that begin at an odd position.  Bar: against float64 no further off than the CUDA-core GEMM."""
    from flash_stu_2_b200 import ops
    M, N, K = shape
    torch.manual_seed(7)
    x = 3e26 * torch.randn(M, K + 4, device=dev())[:, :K]
    W, W2 = 1e-26 * torch.randn(2, N, K, device=dev()) / math.sqrt(K)
    x[M // 2, K - 1], r = float("inf"), torch.randn(M, N, device=dev())
    full, T = x.double() @ W.double().t(), M // 3 if M % 3 == 0 else M // 5 if M % 5 == 0 else M
    Lh = (T + 20) // 16 * 8
    kw = {0: {}, 1: dict(resid=r), 2: dict(W2=W2), 3: dict(hist_T=T, hist_t0=3, hist_Lh=Lh)}[epi]
    want = {0: full, 1: r.double() + full, 2: torch.nn.functional.gelu(full, approximate="tanh") * (x.double() @ W2.double().t()), 3: full}[epi]
    err, fin = [], want.isfinite()
    for backend in (0, 1):
        out = torch.full((M // T, N, 2, Lh) if epi == 3 else (M, N), float("nan"), device=dev())
        ops.linear(x, W, out=out, epilogue=epi, backend=backend, **kw)
        if epi == 3:
            t = torch.arange(3, T + 3, device=dev())
            assert int((~out.isnan()).sum()) == M * N
            out = out[:, :, t % 2, t // 2].permute(0, 2, 1).reshape(M, N)
        assert torch.equal(out.isfinite(), fin) and torch.equal(out.isnan(), want.isnan())
        err.append(float((out.double() - want)[fin].norm() / want[fin].norm()))
    ops.check_status()
    assert err[0] <= max(err[1], 2.0 ** -24), err


@pytest.mark.parametrize("rows,weights", [(1e-36, 1.0), (1.0, 1e-36), (1e-35, 1e30), (3e-19, 3e-19), (1e-42, 1e6), (1e20, 1e4)])
def test_fp32_products_on_tensor_cores_of_small_and_large_operands(rows, weights):
    """Operands whose third parts bf16 would hold only as subnormals, or not at all, and products near the end of fp32's range.  Bars: against
    float64 no further off than the CUDA-core kernels on the same operands, but for the rounding of the result (E and Q: 2^-23)."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(12)
    x, W = rows * torch.randn(300, 512, device=dev()), weights * torch.randn(2000, 512, device=dev())
    want = x.double() @ W.double().t()
    err = [float((ops.linear(x, W, backend=b).double() - want).norm() / want.norm()) for b in (0, 1)]
    assert err[0] <= max(err[1], 2.0 ** -24), err
    B, T, d, K = 2, 500, 8, 3
    x, phi = rows * torch.randn(B, T, d), weights * torch.randn(T, K)
    hist = _hist_from(x, 256).to(dev())
    U = [torch.empty(B * T, 2 * K * d, device=dev()) for _ in range(2)]
    ops.full_conv_f32_tc5(hist, phi.to(dev()), U[0], True, 0, T)
    ops.full_conv(hist, phi.to(dev()), U[1], True, 0, T)
    ops.check_status()
    lag = torch.arange(T)[:, None] - torch.arange(T)[None]
    m = torch.where(lag[:, :, None] >= 0, phi.double()[lag.clamp_min(0)], torch.zeros((), dtype=torch.float64))
    want = [torch.einsum("tsk,bsi->btki", m * s, x.double()) for s in (torch.ones(()), (1.0 - 2 * (lag.abs() % 2))[:, :, None])]
    want = torch.stack(want, 2).reshape(B * T, -1)
    err = [float((u.cpu().double() - want).norm() / want.norm()) for u in U]
    assert err[0] <= max(err[1], 2.0 ** -23), err


@pytest.mark.parametrize("shape", [(1, 256, 1000, 0), (2, 1279, 900, 1270), (3, 1500, 760, 700), (2, 2049, 480, 1800), (9, 2817, 160, 2815),
                                   (1, 4095, 320, 0)])
def test_conv_prefill_tcgen05_stages_of_every_depth(shape):
    """Six to two operand stages (1 to 16 blocks of 128 positions of a parity), each gone round by more channels than it holds, blocks in
    front of the call's first position left out, NaN in the cache past the valid positions: against the mma.sync kernel on the same
    operands (the same products, fp32 sums in another order: two roundings to bf16)."""
    from flash_stu_2_b200 import ops
    B, T, d, t0 = shape
    torch.manual_seed(11)
    L = T + 3
    Lh = ((L + 1) // 2 + 127) // 128 * 128
    hist = _hist_from(torch.randn(B, T, d).bfloat16(), Lh)
    taps = ops.taps_even((torch.randn(L, d) / math.sqrt(L)).bfloat16().to(dev()), Lh)
    x0 = torch.randn(B, T - t0, d).bfloat16().to(dev())
    x1, x2 = x0.clone(), x0.clone()
    y_Lh = ((T + 1) // 2 + 7) // 8 * 8
    ops.conv_prefill_approx(hist.to(dev()), taps, torch.zeros(B, d, 2, y_Lh, dtype=torch.bfloat16, device=dev()), x2, t0, T, use_tensor_cores=True)
    for p in range(2):
        hist[:, :, p, (T - p + 1) // 2:] = float("nan")
    hist = hist.to(dev())
    assert ops.conv_prefill_tc5_supported(hist, x1)
    ops.conv_prefill_approx_tc5(hist, ops.taps_rev8(taps), torch.full((B, d, 2, y_Lh), float("nan"), dtype=torch.bfloat16, device=dev()), x1, t0, T)
    ops.check_status()
    close(x1, x2, 8e-3, row_tol=1.6e-2)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_history_scatter_epilogue(dt):
    from flash_stu_2_b200 import ops
    torch.manual_seed(5)
    for backend, (B, T, d, t0) in [(1, (2, 37, 24, 5)), (0, (2, 256, 128, 32)), (0, (3, 100, 64, 7))]:
        Lh = ((t0 + T + 1) // 2 + 7) // 8 * 8
        x = torch.randn(B, T, d).to(dt)
        Mi = (torch.randn(d, d) / math.sqrt(d)).to(dt)
        xp = (x.double() @ Mi.double()).to(dt)
        hist = torch.zeros(B, d, 2, Lh, dtype=dt, device=dev())
        ops.linear(x.reshape(B * T, d).to(dev()), Mi.t().contiguous().to(dev()), out=hist, epilogue=3, hist_T=T,
                   hist_t0=t0, hist_Lh=Lh, backend=backend)
        ops.check_status()
        full = torch.zeros(B, t0 + T, d, dtype=dt)
        full[:, t0:] = xp
        close(hist, _hist_from(full, Lh), TOL[dt] / 2)


def _decode_fixture(dt, B, T, d, L, seed=6):
    import math as _m
    torch.manual_seed(seed)
    x = torch.randn(B, T, d).to(dt)
    nw = (1 + 0.1 * torch.randn(d)).to(dt)
    Mi = (torch.randn(d, d) / _m.sqrt(d)).to(dt)
    fp = (torch.randn(L, d) / 8).to(dt)
    xn = O.rmsnorm(x, nw)
    xp = xn @ Mi
    plus, minus = O.convolve(xp, fp, O.fft_length(L), True, True)
    return x, nw, Mi, fp, xp, x + (plus + minus)


@pytest.mark.parametrize("dt,tc", [(torch.float32, False), (torch.bfloat16, False), (torch.bfloat16, True)])
@pytest.mark.parametrize("shape", [(3, 45, 64, 64), (9, 70, 40, 160), (10, 300, 256, 600)])
def test_decode_step_equals_prefill_row(dt, tc, shape):
    """S3: the fused decode kernel at time t reproduces row t of the full-prefix layer half
    (CUDA-core kernel and, for bf16, the tensor-core kernel fed by the reversed tap table)."""
    from flash_stu_2_b200 import ops
    B, T, d, L = shape
    Lh = ((L + 1) // 2 + 7) // 8 * 8
    x, nw, Mi, fp, xp, ref = _decode_fixture(dt, B, T, d, L)
    hist = torch.zeros(B, d, 2, Lh, dtype=dt, device=dev())
    pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
    taps = ops.taps_even(fp.to(dev()), Lh)
    taps8 = ops.taps_rev8(taps) if tc else None
    MinT = Mi.t().contiguous().to(dev())
    outs = []
    for t in range(T):
        out = torch.empty(B, d, dtype=dt, device=dev())
        ops.decode_approx(x[:, t].contiguous().to(dev()), nw.to(dev()), MinT, hist, taps, pos, out, taps8=taps8)
        outs.append(out.cpu())
    ops.check_status()
    got = torch.stack(outs, 1)
    assert pos[:, 0].tolist() == [T] * B and int(pos[0, 1]) == 0
    close(got, ref, (1e-5 if dt == torch.float32 else 1.5e-2))
    close(hist, _hist_from(xp, Lh), (1e-5 if dt == torch.float32 else 1e-2))


@pytest.mark.parametrize("shape", [(3, 45, 64, 64), (9, 70, 40, 160), (8, 300, 256, 600), (17, 140, 1024, 300)])
def test_decode_step_shared_tap_kernel(shape):
    """Batches at one common position: the kernel that owns 8 channels x 8 sequences per CTA (taps staged once
    in shared memory, projection and tap contraction as MMAs with the sequences as rows) reproduces the
    full-prefix rows; a ragged batch under the same flag is refused with status 6 and leaves the cache alone."""
    from flash_stu_2_b200 import ops
    dt = torch.bfloat16
    B, T, d, L = shape
    Lh = ((L + 1) // 2 + 7) // 8 * 8
    x, nw, Mi, fp, xp, ref = _decode_fixture(dt, B, T, d, L)
    hist = torch.zeros(B, d, 2, Lh, dtype=dt, device=dev())
    pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
    taps = ops.taps_even(fp.to(dev()), Lh)
    taps8 = ops.taps_rev8(taps)
    MinT = Mi.t().contiguous().to(dev())
    xd, nwd = x.to(dev()), nw.to(dev())
    outs = []
    for t in range(T):
        out = torch.empty(B, d, dtype=dt, device=dev())
        ops.decode_approx(xd[:, t].contiguous(), nwd, MinT, hist, taps, pos, out, taps8=taps8,
                          flags=ops.FLAG_UNIFORM_POS)
        outs.append(out)
    ops.check_status()
    got = torch.stack(outs, 1).cpu()
    assert pos[:, 0].tolist() == [T] * B and int(pos[0, 1]) == 0
    close(got, ref, 1.5e-2)
    close(hist, _hist_from(xp, Lh), 1e-2)
    if B > 1:
        pos[:, 0] = 5
        pos[1, 0] = 4          # ragged inside the first group of eight sequences
        before = hist.clone()
        ops.decode_approx(xd[:, 5].contiguous(), nwd, MinT, hist, taps, pos, out, taps8=taps8,
                          flags=ops.FLAG_UNIFORM_POS)
        with pytest.raises(RuntimeError, match="status 6"):
            ops.check_status()
        assert torch.equal(before[:2], hist[:2])


@pytest.mark.parametrize("shape", [(3, 45, 64, 64), (9, 70, 40, 160), (8, 300, 256, 600), (17, 140, 1024, 300),
                                   (5, 1300, 64, 2700)])
def test_decode_step_pipelined_kernel(shape):
    """The persistent bulk-copy pipeline form of the fused decode step (one CTA per SM, history and taps through a
    shared-memory ring, a row of 8 sequences x 8 channels summed inside one CTA in slice order): every step's row
    equals the full-prefix row; positions advance; a ragged batch is refused with status 6; channel shards of the same
    kernel concatenate to exactly the whole layer's output (the sum order does not depend on the grid)."""
    from flash_stu_2_b200 import ops
    dt = torch.bfloat16
    B, T, d, L = shape
    Lh = ((L + 1) // 2 + 7) // 8 * 8
    x, nw, Mi, fp, xp, ref = _decode_fixture(dt, B, T, d, L)
    hist = torch.zeros(B, d, 2, Lh, dtype=dt, device=dev())
    pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
    taps = ops.taps_even(fp.to(dev()), Lh)
    taps8 = ops.taps_rev8(taps)
    MinT = Mi.t().contiguous().to(dev())
    xd, nwd = x.to(dev()), nw.to(dev())
    # two channel shards fed the same inputs (stale values beyond the position must not matter: poison the tails)
    half = d // 2
    shards = []
    for r in range(2):
        sl = slice(r * half, (r + 1) * half)
        shards.append((MinT[sl].contiguous(), torch.full((B, half, 2, Lh), 3.0, dtype=dt, device=dev()),
                       ops.taps_rev8(taps[sl].contiguous()), torch.zeros(B, 2, dtype=torch.int32, device=dev())))
    outs = []
    for t in range(T):
        xt = xd[:, t].contiguous()
        out = torch.empty(B, d, dtype=dt, device=dev())
        ops.decode_approx_pipelined(xt, nwd, MinT, hist, taps8, pos, out)
        outs.append(out)
        if half % 8 == 0 and t % 7 == 0:
            ys = []
            for (Ms, hs, t8s, ps) in shards:
                ps[:, 0] = t
                if t:   # the shard caches follow the whole layer's (only steps t % 7 == 0 run through the shards)
                    sl = slice(0, half) if Ms is shards[0][0] else slice(half, d)
                    for par in range(2):
                        n = (t - par + 1) // 2
                        hs[:, :, par, :n] = hist[:, sl, par, :n]
                y = torch.empty(B, half, dtype=dt, device=dev())
                ops.decode_approx_pipelined(xt, nwd, Ms, hs, t8s, ps, y, add_residual=False)
                ys.append(y)
            sharded = (xt.float() + torch.cat(ys, 1).float()).to(dt)
            assert torch.equal(sharded, out), t
    ops.check_status()
    got = torch.stack(outs, 1).cpu()
    assert pos[:, 0].tolist() == [T] * B and int(pos[0, 1]) == 0
    close(got, ref, 1.5e-2)
    close(hist, _hist_from(xp, Lh), 1e-2)
    if B > 1:
        pos[:, 0] = 5
        pos[1, 0] = 4
        before = hist.clone()
        ops.decode_approx_pipelined(xd[:, 5].contiguous(), nwd, MinT, hist, taps8, pos, out)
        with pytest.raises(RuntimeError, match="status 6"):
            ops.check_status()
        assert torch.equal(before, hist)


@pytest.mark.parametrize("world", [2, 4])
def test_peer_exchange_of_the_token_step_with_all_ranks_emulated_on_one_gpu(world):
    """The fused exchanges of a tensor-parallel token step with every rank's buffers on this GPU: the channel-shard
    decode kernel stores its outputs straight into all inboxes (all-gather), the down projection stores its partial
    rows into all inboxes (all-reduce), and the combine kernel of every rank ends with the residual stream (and the
    next RMSNorm) the unfused path computes.  All producing kernels are launched before the first combine, so no
    kernel ever waits for one that has not run.  Repeated steps reuse the same inboxes and counters."""
    from flash_stu_2_b200 import ops
    from flash_stu_2_b200.peer import GATHER, REDUCE, PeerExchange
    dt = torch.bfloat16
    B, d, L, inter = 8, 64 * world, 40, 128 * world
    dl, il = d // world, inter // world
    Lh = ((L + 1) // 2 + 7) // 8 * 8
    torch.manual_seed(11)
    x, nw, Mi, fp, xp, ref = _decode_fixture(dt, B, 6, d, L)
    taps = ops.taps_even(fp.to(dev()), Lh)
    MinT = Mi.t().contiguous().to(dev())
    nwd = nw.to(dev())
    Wd = (torch.randn(d, inter) / math.sqrt(inter)).to(dt).to(dev())
    norm2 = (1 + 0.1 * torch.randn(d)).to(dt).to(dev())
    exs = PeerExchange.emulate([GATHER, REDUCE], B, d, world)
    try:
        ranks = []
        for r in range(world):
            sl = slice(r * dl, (r + 1) * dl)
            ranks.append(dict(MinT=MinT[sl].contiguous(), taps8=ops.taps_rev8(taps[sl].contiguous()),
                              hist=torch.zeros(B, dl, 2, Lh, dtype=dt, device=dev()),
                              pos=torch.zeros(B, 2, dtype=torch.int32, device=dev()),
                              hist_ref=torch.zeros(B, dl, 2, Lh, dtype=dt, device=dev()),
                              pos_ref=torch.zeros(B, 2, dtype=torch.int32, device=dev()),
                              Wd=Wd[:, r * il:(r + 1) * il].contiguous()))
        for t in range(6):
            xt = x[:, t].contiguous().to(dev())
            h = (torch.randn(B, inter) / 2).to(dt).to(dev())
            # ---- unfused: shard outputs gathered, partial products reduced (bf16 sums as a collective would form them)
            ys = []
            for rk in ranks:
                y = torch.empty(B, dl, dtype=dt, device=dev())
                ops.decode_approx_pipelined(xt, nwd, rk["MinT"], rk["hist_ref"], rk["taps8"], rk["pos_ref"], y,
                                            add_residual=False)
                ys.append(y)
            x1 = (xt.float() + torch.cat(ys, 1).float()).to(dt)
            n1 = ops.rmsnorm(x1, norm2)
            parts = [ops.linear(h[:, r * il:(r + 1) * il].contiguous(), rk["Wd"]) for r, rk in enumerate(ranks)]
            x2 = (x1.float() + torch.stack(parts).float().sum(0).to(dt).float()).to(dt)
            # ---- fused: every rank's producers first, then every rank's combine
            xs = [xt.clone() for _ in range(world)]
            xn = [torch.empty_like(xt) for _ in range(world)]
            for r, rk in enumerate(ranks):
                ops.decode_approx_push(xs[r], nwd, rk["MinT"], rk["hist"], rk["taps8"], rk["pos"], exs[r].dest(0), d)
            for r in range(world):
                exs[r].combine(0, xs[r], norm_w=norm2, xn=xn[r])
            for r, rk in enumerate(ranks):
                ops.linear_push(h[:, r * il:(r + 1) * il].contiguous(), rk["Wd"], exs[r].dest(1), d)
            for r in range(world):
                x_mid = xs[r].clone()
                exs[r].combine(1, xs[r])
                assert torch.equal(x_mid, x1), (t, r)
                close(xn[r], n1, 8e-3, what="next RMSNorm")   # the row sums are formed in another order
                if world == 2:
                    assert torch.equal(xs[r], x2), (t, r)    # two bf16 partials: one rounding either way
                else:
                    close(xs[r], x2, 8e-3)
            ops.check_status()
            for r in range(world):
                for e in range(2):
                    flags, epoch = exs[r].counters(e)
                    assert flags == [t + 1] * world and epoch == t + 1
        # a sender that never arrives: the bounded wait runs out, status 10, x untouched, the context stays usable
        before = xs[0].clone()
        ops.decode_approx_push(xs[0], nwd, ranks[0]["MinT"], ranks[0]["hist"], ranks[0]["taps8"], ranks[0]["pos"],
                               exs[0].dest(0), d)
        exs[0].combine(0, xs[0], wait_ms=50)
        with pytest.raises(RuntimeError, match="status 10"):
            ops.check_status()
        assert torch.equal(xs[0], before)
    finally:
        for ex in exs:
            ex.close()


@pytest.mark.parametrize("world", [2, 4])
def test_single_launch_exchange_kernel_with_the_other_ranks_stood_in_by_host_copies(world):
    """The exchange kernel (push + wait + combine + RMSNorm, one CTA per row) for every rank of a group on one GPU.
    What the other ranks would have delivered is copied into the rank's inbox from the host before its kernel runs,
    so the kernel never waits for another launch; its own rows must land in every other rank's inbox all the same."""
    from flash_stu_2_b200 import ops
    from flash_stu_2_b200.peer import GATHER, REDUCE, PeerExchange
    dt = torch.bfloat16
    B, d = 5, 128 * world
    dl = d // world
    torch.manual_seed(12)
    exs = PeerExchange.emulate([GATHER, REDUCE], B, d, world)
    norm = (1 + 0.1 * torch.randn(d)).to(dt).to(dev())
    try:
        for t in range(3):
            x0 = torch.randn(B, d).to(dt).to(dev())
            slices = [torch.randn(B, dl).to(dt).to(dev()) for _ in range(world)]
            parts = [(torch.randn(B, d) / 2).to(dt).to(dev()) for _ in range(world)]
            x1 = (x0.float() + torch.cat(slices, 1).float()).to(dt)
            x2 = (x1.float() + torch.stack(parts).float().sum(0).to(dt).float()).to(dt)
            for r in range(world):
                for s_ in range(world):
                    if s_ != r:
                        exs[r].fake_arrival(0, s_, slices[s_], t + 1)
                        exs[r].fake_arrival(1, s_, parts[s_], t + 1)
            for r in range(world):
                x = x0.clone()
                xn = torch.empty_like(x)
                exs[r].exchange(0, x, slices[r], norm_w=norm, xn=xn)
                assert torch.equal(x, x1), (t, r)
                close(xn, ops.rmsnorm(x1, norm), 8e-3)
                exs[r].exchange(1, x, parts[r])
                if world == 2:
                    assert torch.equal(x, x2), (t, r)
                else:
                    close(x, x2, 8e-3)
            ops.check_status()
        # nobody else arrives for a further step (counters put back below the row's epoch): bounded wait, status 10,
        # x untouched
        for s_ in range(1, world):
            exs[0].fake_arrival(0, s_, slices[s_], 0)
        x = x0.clone()
        exs[0].exchange(0, x, slices[0], wait_ms=50)
        with pytest.raises(RuntimeError, match="status 10"):
            ops.check_status()
        assert torch.equal(x, x0)
    finally:
        for ex in exs:
            ex.close()


@pytest.mark.parametrize("B,d,L,t,layers,sms", [(17, 64, 1100, 510, 3, 5), (16, 128, 600, 0, 1, 200), (8, 8, 2000, 1023, 2, 1), (33, 256, 1100, 1090, 2, 7),
                                                (16, 1032, 300, 297, 1, 148)])
def test_history_sums_ahead_of_the_step(B, d, L, t, layers, sms):
    """stream_ahead + stream_finish against the pipeline kernel and the norm kernel, bit for bit, over four steps: sequences that
    fill no group of eight, one to several slices, an odd number of rows per SM, positions up to the end of the capacity (where there
    is no next one).  The history past the position holds NaN."""
    from flash_stu_2_b200 import ops
    from flash_stu_2_b200.modules import new_pos
    g = torch.Generator(device=dev()).manual_seed(B + d + t)
    rand = lambda *s: torch.randn(*s, device=dev(), generator=g).bfloat16()
    Lh = (L // 2 + 7) // 8 * 8
    cap = 2 * Lh
    t = min(t, cap - 4) if t > 1024 else t
    hists, taps8s = [], []
    for _ in range(layers):
        h = rand(B, d, 2, Lh)
        h[:, :, 0, (t + 1) // 2:] = float("nan")
        h[:, :, 1, t // 2:] = float("nan")
        hists.append(h)
        taps8s.append(ops.taps_rev8(rand(d, Lh)))
    twins = [h.clone() for h in hists]
    pos = [new_pos(B, dev()) for _ in range(2 * layers)]
    for p in pos:
        p[:, 0] = t
    norm_w = rand(d)
    part = torch.full((layers, 2, B, d), float("nan"), device=dev())
    ctl = torch.tensor([t, 0] + ([t - 2, t - 1] if t % 2 == 0 else [t - 1, t - 2]), dtype=torch.int32, device=dev())
    ops.stream_ahead(hists, taps8s, part, ctl, sms)
    for step in range(4):
        ops.stream_ahead(hists, taps8s, part, ctl, sms)      # of position t + step + 1: ahead of this step's appends
        for i in range(layers):
            x, xp = rand(B, d), rand(B, d)
            want, out = torch.empty_like(x), torch.empty_like(x)
            ops.decode_approx_projected(x, xp, twins[i], taps8s[i], pos[2 * i], want)
            xn = ops.stream_finish(x, xp, hists[i], taps8s[i], pos[2 * i + 1], part[i], ctl, norm_w, 1e-6, out)
            ops.check_status()
            assert torch.equal(out, want) and torch.equal(xn, ops.rmsnorm(want, norm_w, 1e-6)), (step, i)
            assert torch.equal(pos[2 * i], pos[2 * i + 1]) and pos[2 * i + 1][0].tolist() == [t + step + 1, 0]
    for a, b in zip(hists, twins):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    # sums of another position are refused, nothing is appended
    ctl[2:] = -1
    if t + 4 < cap:
        before = hists[0].clone()
        ops.stream_finish(x, xp, hists[0], taps8s[0], pos[1], part[0], ctl, norm_w, 1e-6, out)
        with pytest.raises(RuntimeError, match="status 8"):
            ops.check_status()
        assert torch.equal(hists[0].view(torch.int16), before.view(torch.int16)) and pos[1][0, 0].item() == t + 4


@pytest.mark.parametrize("shape", [(17, 60, 256, 300), (32, 40, 128, 700), (9, 530, 64, 1100)])
def test_decode_step_with_the_projection_done_by_the_caller(shape):
    """Larger batches: rmsnorm + one GEMM give the projected input of the whole batch, the pipeline kernel only appends
    it, streams the history and adds the residual.  Every step's row equals the full-prefix row, the cache equals the
    projected inputs, positions advance."""
    from flash_stu_2_b200 import ops
    dt = torch.bfloat16
    B, T, d, L = shape
    Lh = ((L + 1) // 2 + 7) // 8 * 8
    x, nw, Mi, fp, xp_ref, ref = _decode_fixture(dt, B, T, d, L)
    hist = torch.full((B, d, 2, Lh), 3.0, dtype=dt, device=dev())   # stale values beyond the position must not matter
    pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
    taps8 = ops.taps_rev8(ops.taps_even(fp.to(dev()), Lh))
    MinT = Mi.t().contiguous().to(dev())
    xd, nwd = x.to(dev()), nw.to(dev())
    outs = []
    for t in range(T):
        xt = xd[:, t].contiguous()
        xp = ops.linear(ops.rmsnorm(xt, nwd), MinT)
        out = torch.empty(B, d, dtype=dt, device=dev())
        ops.decode_approx_projected(xt, xp, hist, taps8, pos, out)
        outs.append(out)
    ops.check_status()
    assert pos[:, 0].tolist() == [T] * B and int(pos[0, 1]) == 0
    close(torch.stack(outs, 1).cpu(), ref, 1.5e-2)
    want = _hist_from(xp_ref, Lh)
    for p_ in range(2):
        n = (T - p_ + 1) // 2
        close(hist[:, :, p_, :n], want[:, :, p_, :n], 1e-2)


def test_decode_step_channel_shards_tile_the_layer():
    """Tensor-parallel form of the fused decode step: two ranks' channel shards (own history, own rows of
    M_inputs^T, own taps) give, concatenated and added to the input, exactly the whole-layer kernel's output."""
    from flash_stu_2_b200 import ops
    dt = torch.bfloat16
    B, T, d, L = 5, 40, 64, 96
    Lh = ((L + 1) // 2 + 7) // 8 * 8
    x, nw, Mi, fp, xp, ref = _decode_fixture(dt, B, T, d, L)
    taps = ops.taps_even(fp.to(dev()), Lh)
    MinT = Mi.t().contiguous().to(dev())
    xd, nwd = x.to(dev()), nw.to(dev())
    hist = torch.zeros(B, d, 2, Lh, dtype=dt, device=dev())
    pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
    taps8 = ops.taps_rev8(taps)
    halves = []
    for r in range(2):
        sl = slice(r * d // 2, (r + 1) * d // 2)
        halves.append((MinT[sl].contiguous(), torch.zeros(B, d // 2, 2, Lh, dtype=dt, device=dev()),
                       ops.taps_rev8(taps[sl].contiguous()), torch.zeros(B, 2, dtype=torch.int32, device=dev())))
    for t in range(T):
        xt = xd[:, t].contiguous()
        whole = torch.empty(B, d, dtype=dt, device=dev())
        ops.decode_approx(xt, nwd, MinT, hist, taps, pos, whole, taps8=taps8, flags=ops.FLAG_UNIFORM_POS)
        ys = []
        for (Ms, hs, t8s, ps) in halves:
            y = torch.empty(B, d // 2, dtype=dt, device=dev())
            ops.decode_approx_shard(xt, nwd, Ms, hs, t8s, ps, y)
            ys.append(y)
        sharded = (xt.float() + torch.cat(ys, 1).float()).to(dt)
        assert torch.equal(sharded, whole), t
    ops.check_status()
    assert torch.equal(torch.cat([h[1] for h in halves], 1), hist)
    assert halves[0][3][:, 0].tolist() == [T] * B


@pytest.mark.parametrize("tc", [False, True])
def test_decode_step_with_ragged_positions(tc):
    """Sequences of one batch at different positions (what _reorder_cache / ragged prompts produce)."""
    from flash_stu_2_b200 import ops
    dt = torch.bfloat16
    B, T, d, L = 5, 50, 32, 64
    Lh = 32
    x, nw, Mi, fp, xp, ref = _decode_fixture(dt, B, T, d, L, seed=9)
    where = [7, 30, 30, 1, 49]
    hist_full = _hist_from(xp, Lh)
    hist = torch.zeros_like(hist_full)
    for b, t in enumerate(where):  # rows hold only the first t projected inputs
        for p in range(2):
            n = (t - p + 1) // 2
            hist[b, :, p, :n] = hist_full[b, :, p, :n]
    hist = hist.to(dev())
    pos = torch.zeros(B, 2, dtype=torch.int32)
    pos[:, 0] = torch.tensor(where, dtype=torch.int32)
    pos = pos.to(dev())
    taps = ops.taps_even(fp.to(dev()), Lh)
    taps8 = ops.taps_rev8(taps) if tc else None
    xin = torch.stack([x[b, t] for b, t in enumerate(where)]).to(dev())
    out = torch.empty(B, d, dtype=dt, device=dev())
    ops.decode_approx(xin, nw.to(dev()), Mi.t().contiguous().to(dev()), hist, taps, pos, out, taps8=taps8)
    ops.check_status()
    want = torch.stack([ref[b, t] for b, t in enumerate(where)])
    assert pos[:, 0].tolist() == [t + 1 for t in where]
    close(out, want, 1.5e-2)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cfg", [(2, 40, 4, 8, 8), (1, 70, 2, 64, 16), (2, 33, 3, 128, 100)])
def test_attention_prefill_and_cached_decode(dt, cfg):
    from flash_stu_2_b200 import ops
    B, T, H, hd, w = cfg
    d = H * hd
    torch.manual_seed(7)
    x = torch.randn(B, T, d).to(dt)
    p = {"attn.c_attn.weight": (torch.randn(3 * d, d) / math.sqrt(d)).to(dt),
         "attn.c_proj.weight": torch.eye(d).to(dt)}
    ref, _ = O.attention(x, p, H, w, 50.0)
    qkv = (x @ p["attn.c_attn.weight"].t()).to(dev())
    slopes = O.alibi_slopes(H).float().to(dev())
    W = w + 1
    kr = torch.zeros(B, W, d, dtype=dt, device=dev())
    vr = torch.zeros_like(kr)
    pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
    T1 = T - 5
    y1 = ops.swa_forward(qkv[:, :T1].contiguous(), kr, vr, pos, slopes, H, w, 50.0, update_cache=True)
    ys = [y1]
    for t in range(T1, T):
        ys.append(ops.swa_forward(qkv[:, t:t + 1].contiguous(), kr, vr, pos, slopes, H, w, 50.0, update_cache=True))
    got = torch.cat(ys, 1)
    assert pos[:, 0].tolist() == [T] * B
    close(got, ref, (1e-4 if dt == torch.float32 else 1.5e-2))
    # uncached call over the whole sequence
    dummy = torch.zeros(1, 1, 1, dtype=dt, device=dev())
    y = ops.swa_forward(qkv, dummy, dummy, torch.zeros(B, 2, dtype=torch.int32, device=dev()), slopes, H, w, 50.0,
                        update_cache=False)
    close(y, ref, (1e-4 if dt == torch.float32 else 1.5e-2))


@pytest.mark.parametrize("cfg", [(2, 300, 2, 100), (1, 700, 3, 256), (3, 260, 2, 1024), (2, 1031, 2, 77), (1, 128, 1, 16)])
def test_attention_prefill_on_tcgen05_matches_oracle(cfg):
    """Prefill from position 0, bf16, head dimension 128: the tcgen05 kernel (S and O in tensor memory, lazy row
    maximum) against the fp32 oracle and against the mma.sync kernel; ragged last query tile, windows shorter and
    longer than a key tile, the ring and the positions afterwards, then cached steps on top of it."""
    from flash_stu_2_b200 import ops
    B, T, H, w = cfg
    hd, dt = 128, torch.bfloat16
    d = H * hd
    torch.manual_seed(13)
    x = torch.randn(B, T, d).to(dt)
    p = {"attn.c_attn.weight": (torch.randn(3 * d, d) / math.sqrt(d)).to(dt),
         "attn.c_proj.weight": torch.eye(d).to(dt)}
    ref, _ = O.attention(x, p, H, w, 50.0)
    qkv = (x @ p["attn.c_attn.weight"].t()).to(dev())
    slopes = O.alibi_slopes(H).float().to(dev())
    W = w + 1
    T1 = T - 3
    q1 = qkv[:, :T1].contiguous()
    assert ops.swa_prefill_tc5_supported(q1, H, 0) or T1 < 128
    kr, vr = torch.zeros(B, W, d, dtype=dt, device=dev()), torch.zeros(B, W, d, dtype=dt, device=dev())
    pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
    kr2, vr2, pos2 = torch.zeros_like(kr), torch.zeros_like(vr), torch.zeros_like(pos)
    y1 = ops.swa_prefill_tc5(q1, kr, vr, pos, slopes, H, w, 50.0, update_cache=True)
    y2 = ops.swa_forward(q1, kr2, vr2, pos2, slopes, H, w, 50.0, update_cache=True)
    ops.check_status()
    close(y1, ref[:, :T1], 1.5e-2, what="tcgen05 vs oracle")
    close(y1, y2, 1.5e-2, what="tcgen05 vs mma.sync")
    assert torch.equal(kr, kr2) and torch.equal(vr, vr2) and torch.equal(pos, pos2)
    ys = [y1]
    for t in range(T1, T):
        ys.append(ops.swa_forward(qkv[:, t:t + 1].contiguous(), kr, vr, pos, slopes, H, w, 50.0, update_cache=True))
    close(torch.cat(ys, 1), ref, 1.5e-2)
    # a sequence that is not at position 0 is refused on the device
    ops.swa_prefill_tc5(q1, kr, vr, pos, slopes, H, w, 50.0, update_cache=False)
    with pytest.raises(RuntimeError, match="status 11"):
        ops.check_status()


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cfg", [(2, 300, 2, 64, 100), (1, 700, 3, 128, 256), (3, 260, 2, 128, 1024)])
def test_attention_chunked_prefill_across_many_key_tiles(dt, cfg):
    """Windows spanning several 64-key tiles, a second prefill chunk whose older keys come from the ring, then
    cached single-token steps (tensor-core prefill kernel and memory-bound decode kernel for bf16)."""
    from flash_stu_2_b200 import ops
    B, T, H, hd, w = cfg
    d = H * hd
    torch.manual_seed(11)
    x = torch.randn(B, T, d).to(dt)
    p = {"attn.c_attn.weight": (torch.randn(3 * d, d) / math.sqrt(d)).to(dt),
         "attn.c_proj.weight": torch.eye(d).to(dt)}
    ref, _ = O.attention(x, p, H, w, 50.0)
    qkv = (x @ p["attn.c_attn.weight"].t()).to(dev())
    slopes = O.alibi_slopes(H).float().to(dev())
    W = w + 1
    kr = torch.zeros(B, W, d, dtype=dt, device=dev())
    vr = torch.zeros_like(kr)
    pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
    cuts = [0, 131, T - 6]
    ys = [ops.swa_forward(qkv[:, a:b].contiguous(), kr, vr, pos, slopes, H, w, 50.0, update_cache=True)
          for a, b in zip(cuts[:-1], cuts[1:])]
    for t in range(T - 6, T):
        ys.append(ops.swa_forward(qkv[:, t:t + 1].contiguous(), kr, vr, pos, slopes, H, w, 50.0, update_cache=True))
    got = torch.cat(ys, 1)
    assert pos[:, 0].tolist() == [T] * B and int(pos[0, 1]) == 0
    close(got, ref, (1e-4 if dt == torch.float32 else 1.5e-2))


def test_sampling_matches_oracle():
    from flash_stu_2_b200 import ops
    torch.manual_seed(8)
    B, V = 6, 50257
    for dt in (torch.float32, torch.bfloat16):
        logits = (torch.randn(B, V) * 3).to(dt)
        out = torch.zeros(B, dtype=torch.int64, device=dev())
        ops.sample(logits.to(dev()), 1.0, None, None, False, None, out)
        assert torch.equal(out.cpu(), logits.float().argmax(-1))
        # (temperature, top_k, top_p): candidate-list path (top_k <= 1024), and the full-vocabulary filters: nucleus
        # without top-k, a top-k wider than the candidate list, and a nucleus inside such a top-k
        for (temp, k, p) in [(0.8, 40, None), (0.8, 5, 0.9), (1.3, 1, None), (1.0, None, None), (0.9, None, 0.9),
                             (1.0, None, 0.35), (0.7, 3000, None), (1.1, 5000, 0.8), (1.0, 1024, 0.95)]:
            u = torch.rand(B)
            z = O.filter_logits(logits, temp, k, p)
            want = O.pick_token(z, True, u).view(-1)
            ops.sample(logits.to(dev()), temp, k, p, True, u.to(dev()), out)
            ops.check_status()
            got = out.cpu()
            # the draw may differ only where u lands within rounding of a CDF boundary; require the
            # chosen token to be inside the filtered support and almost all draws identical
            assert all(torch.isfinite(z[b, got[b]]) for b in range(B)), (temp, k, p, got.tolist())
            if dt == torch.float32:
                frac = float((got == want).float().mean())
                assert frac >= 0.8, f"{frac:.2f} of the fp32 draws equal the oracle's ({got.tolist()} vs {want.tolist()})"


def test_sampling_row_with_a_nan_logit_draws_uniformly():
    """The reference replaces the distribution of a row whose softmax is not finite by a uniform one
    (flash_stu/model.py:293-296); the kernel takes the row's uniform for it and leaves the other rows alone."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(9)
    B, V = 4, 1000
    logits = torch.randn(B, V)
    logits[2, 17] = float("nan")
    u = torch.tensor([0.3, 0.9, 0.25, 0.5])
    out = torch.zeros(B, dtype=torch.int64, device=dev())
    ops.sample(logits.to(dev()), 1.0, 50, None, True, u.to(dev()), out)
    ops.check_status()
    got = out.cpu()
    assert int(got[2]) == int(0.25 * V)
    z = O.filter_logits(logits[[0, 1, 3]], 1.0, 50, None)
    assert all(torch.isfinite(z[i, got[b]]) for i, b in enumerate((0, 1, 3)))


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V", [4096, 4099, 50257, 65536])
def test_sampling_by_a_cluster_equals_one_cta_per_row(dt, V):
    """33 long rows run a top-k of at most 256 on a cluster of CTAs per row, 65 rows on one CTA per row: the same tokens, with
    infinities, NaN, ties across the k-th place and more ties than the candidate list holds."""
    _cluster_against_one_cta(dt, V, 33)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,V", [(9, 8447), (9, 8448), (9, 31487), (9, 31488), (32, 14336), (32, 49152), (32, 65536), (10, 10007)])
def test_sampling_by_a_cluster_of_few_rows(dt, rows, V):
    """The same on both sides of the lines from which on a cluster takes a row, the greedy pick among them."""
    _cluster_against_one_cta(dt, V, rows)


def _cluster_against_one_cta(dt, V, rows):
    from flash_stu_2_b200 import ops
    torch.manual_seed(10)
    B = 65
    z = torch.randn(B, V + 3) * 3
    z[1, 5], z[2, 7], z[3, :] = float("nan"), float("inf"), -float("inf")
    z[3, ::100] = torch.randn(z[3, ::100].shape)
    z[4, 100:160] = 20.0
    if V <= 51712:   # (a wider row with more ties than the list holds is refused with a status)
        z[5, :] = 1.5
        z[6, ::2] = 30.0
    z = z.to(dt).to(dev())[:, :V]
    u = torch.rand(B, device=dev())
    u[7], u[8] = 0.0, 1.0 - 2 ** -24
    for temp, k, p in [(1.0, None, None), (0.8, 40, None), (0.9, 100, 0.9), (1.0, 256, 0.5), (1.0, 1, None), (1.3, 50, 1.0)]:
        one, many = (torch.full((n,), -1, dtype=torch.int64, device=dev()) for n in (B, rows))
        ops.sample(z, temp, k, p, k is not None, u, one)
        ops.sample(z[:rows], temp, k, p, k is not None, u[:rows], many)
        ops.check_status()
        assert torch.equal(one[:rows], many), (temp, k, p)
        assert bool((many >= 0).all()) and bool((many < V).all())


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_full_variant_building_blocks(dt):
    """to_history, the three Toeplitz matrices, the causal GEMM flag and the combine step against plain torch."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(12)
    B, T, d, K, L, t0 = 2, 301, 40, 5, 320, 0
    S = ((T + 1) // 2 + 7) // 8 * 8
    x = torch.randn(B, T, d).to(dt)
    phi = (torch.randn(L, K) / 4).to(dt)
    hist = torch.zeros(B, d, 2, S, dtype=dt, device=dev())
    ops.to_history(x.to(dev()), hist, t0)
    assert torch.equal(hist.cpu(), _hist_from(x, S))
    Tz = torch.empty(3, S, S, dtype=dt, device=dev())
    ops.toeplitz(phi.to(dev()), 3, Tz)
    m = torch.arange(S)[:, None]
    s_ = torch.arange(S)[None, :]
    for kind, off in ((0, 0), (1, 1), (2, -1)):
        j = 2 * (m - s_) + off
        ok = (m >= s_) & (j >= 0) & (j < L)
        want = torch.where(ok, phi[:, 3][j.clamp(0, L - 1)], torch.zeros((), dtype=dt))
        assert torch.equal(Tz[kind].cpu(), want), kind
    rows = hist.view(B * d * 2, S)
    dense = ops.linear(rows, Tz[0], backend=0)
    causal = ops.linear(rows, Tz[0], epilogue=ops.EPI_STORE | ops.EPI_FLAG_CAUSAL, backend=0)
    ops.check_status()
    close(causal, dense, 1e-6)
    ref = (rows.cpu().double() @ Tz[0].cpu().double().t()).to(dt)
    close(causal, ref, TOL[dt] / 2)
    # E, Q -> U for one filter
    E = torch.randn(B * d * 2, S).to(dt)
    Q = torch.randn(B * d * 2, S).to(dt)
    U = torch.zeros(B * T, 2 * K * d, dtype=dt, device=dev())
    ops.full_combine(E.to(dev()), Q.to(dev()), U, B, d, K, 3, True, t0, T)
    Ev = E.view(B, d, 2, S)
    Qv = Q.view(B, d, 2, S)
    want = torch.zeros(B, T, 2, K, d, dtype=dt)
    for p in range(2):
        n = (T - p + 1) // 2
        want[:, p::2, 0, 3] = (Ev[:, :, p, :n].float() + Qv[:, :, p, :n].float()).to(dt).transpose(1, 2)
        want[:, p::2, 1, 3] = (Ev[:, :, p, :n].float() - Qv[:, :, p, :n].float()).to(dt).transpose(1, 2)
    assert torch.equal(U.cpu().view(B, T, 2, K, d), want)


@pytest.mark.parametrize("shape", [(1, 7, 16, 5, 300, 0, 90), (1, 5, 27, 3, 97, 0, 97), (3, 24, 33, 4, 200, 61, 200),
                                   (5, 1, 64, 2, 400, 128, 321), (2, 24, 96, 2, 130, 129, 130)])
@pytest.mark.parametrize("both", [True, False])
def test_full_convolution_of_all_filters(shape, both):
    """The one-launch fp32 operand U against float64 sums: 4, 8 and 16 threads across the channels, tiles that hold several
    sequences, odd channel counts, ranges that start inside the history, one position.  Bar: at most 200 fp32 roundings
    of 2^-24 per sum."""
    from flash_stu_2_b200 import ops
    B, K, d, pad, L, t0, t_end = shape
    torch.manual_seed(14)
    Lh = ((t_end + 1) // 2 + pad + 7) // 8 * 8
    x, phi = torch.randn(B, t_end, d), torch.randn(L, K) / 4
    hist = torch.full((B, d, 2, Lh), float("nan"), device=dev())   # what lies past the last input is not read
    ops.to_history(x.to(dev()), hist, 0)
    U = torch.full((B * (t_end - t0), (2 if both else 1) * K * d + 4), 7.0, device=dev())
    ops.full_conv(hist, phi.to(dev()), U, both, t0, t_end)
    ops.check_status()
    f = torch.zeros(max(L, t_end), K, dtype=torch.float64)
    f[:L] = phi
    lag = torch.arange(t_end)[:, None] - torch.arange(t_end)[None, :]
    want = []
    for sign in (1.0, -1.0)[: 2 if both else 1]:
        taps = f * torch.where(torch.arange(f.shape[0]) % 2 == 1, sign, 1.0)[:, None]
        T = torch.where((lag >= 0)[:, :, None], taps[lag.clamp_min(0)], torch.zeros((), dtype=torch.float64))
        want.append(torch.einsum("tsk,bsi->btki", T, x.double())[:, t0:].reshape(B * (t_end - t0), K * d))
    close(U[:, :-4], torch.cat(want, 1), 1e-5)
    assert bool((U[:, -4:] == 7.0).all())


@pytest.mark.parametrize("shape", [(1, 5, 40, 300, 0, 90), (3, 24, 72, 200, 61, 200), (2, 3, 136, 1400, 258, 1301),
                                   (5, 2, 64, 700, 640, 641), (2, 24, 264, 900, 0, 777), (1, 24, 512, 512, 0, 512)])
@pytest.mark.parametrize("both", [True, False])
def test_full_convolution_on_tensor_cores(shape, both):
    """The bf16 operand U against float64 sums: tiles of 64, 128 and 256 channels, fewer channels than a tile, tiles that hold
    several sequences, one and several blocks of positions, ranges that start inside the history, one position.  Bar: E, Q
    and their sum are each rounded to bf16 (2^-9 of each), and neither E nor Q exceeds 1.5 times the largest U of its row."""
    from flash_stu_2_b200 import ops
    B, K, d, L, t0, t_end = shape
    torch.manual_seed(15)
    Lh = ((t_end + 1) // 2 + 8 + 7) // 8 * 8
    x, phi = torch.randn(B, t_end, d).bfloat16(), (torch.randn(L, K) / 4).bfloat16()
    hist = torch.full((B, d, 2, Lh), 3.0, dtype=torch.bfloat16, device=dev())   # what lies past the last input has no effect
    ops.to_history(x.to(dev()), hist, 0)
    U = torch.full((B * (t_end - t0), (2 if both else 1) * K * d + 8), 7.0, dtype=torch.bfloat16, device=dev())
    assert ops.full_conv_tc5_supported(hist)
    ops.full_conv_tc5(hist, phi.to(dev()), U, both, t0, t_end)
    ops.check_status()
    f = torch.zeros(max(L, t_end), K, dtype=torch.float64)
    f[:L] = phi
    lag = torch.arange(t0, t_end)[:, None] - torch.arange(t_end)[None, :]
    want = []
    for sign in (1.0, -1.0)[: 2 if both else 1]:
        taps = f * torch.where(torch.arange(f.shape[0]) % 2 == 1, sign, 1.0)[:, None]
        T = torch.where((lag >= 0)[:, :, None], taps[lag.clamp_min(0)], torch.zeros((), dtype=torch.float64))
        want.append(torch.einsum("tsk,bsi->btki", T, x.double()).reshape(B * (t_end - t0), K * d))
    close(U[:, :-8], torch.cat(want, 1), 4 * 2 ** -9)
    assert bool((U[:, -8:] == 7.0).all())


@pytest.mark.parametrize("name,tol", [("std_full_float32", 1e-3), ("std_full_bfloat16", 2e-2),
                                       ("hankelL_full_float32", 1e-3), ("std_approx_float32", 1e-3),
                                       ("std_approx_bfloat16", 2e-2), ("hankelL_approx_float32", 1e-3),
                                       ("hankelL_approx_bfloat16", 2e-2), ("hankelL_full_bfloat16", 2e-2)])
def test_stu_operator_matches_reference_golden(golden, name, tol):
    """STU.forward (operator output, no residual) against the reference module's own outputs."""
    import flash_stu_2_b200 as F
    from flash_stu_2_b200 import ops
    r = golden("stu_modules")[name]
    dt = r["x"].dtype
    L, K = r["phi"].shape
    d = r["x"].shape[2]
    cfg = F.FlashSTUConfig(n_embd=d, seq_len=L, num_eigh=K, use_approx="_approx_" in name,
                           use_hankel_L=name.startswith("hankelL"), torch_dtype=dt, n_layers=1, vocab_size=1)
    m = F.STU(cfg, r["phi"].clone(), r["n"])
    with torch.no_grad():
        for k, v in r["params"].items():
            getattr(m, k).copy_(v)
    m = m.to(dev())
    with torch.no_grad():
        y = m(r["x"].to(dev()))
        T = r["T_short"]
        ys = m(r["x"][:, :T].contiguous().to(dev()))
    ops.check_status()
    close(y, r["y_full"], tol)
    close(ys, r["y_short"], tol)


@pytest.mark.parametrize("name,tol", [("tiled16_approx_float32", 1e-3), ("tiled20_approx_float32", 1e-3),
                                       ("tiled16_approx_bfloat16", 2e-2), ("tiled20_approx_bfloat16", 2e-2)])
def test_stu_operator_with_block_diagonal_tiling_matches_reference_golden(golden, name, tol):
    """d_in_tile / d_out_tile (flash_stu/modules/stu.py:123-191): only the diagonal blocks of M_inputs take part
    (tile 16 divides the width, tile 20 leaves a ragged last block)."""
    import flash_stu_2_b200 as F
    from flash_stu_2_b200 import ops
    r = golden("variants")[name]
    dt = r["x"].dtype
    L, K = r["phi"].shape
    d = r["x"].shape[2]
    cfg = F.FlashSTUConfig(n_embd=d, seq_len=L, num_eigh=K, use_approx=True, torch_dtype=dt, n_layers=1, vocab_size=1,
                           d_in_tile=r["tile"][0], d_out_tile=r["tile"][1])
    m = F.STU(cfg, r["phi"].clone(), r["n"])
    with torch.no_grad():
        for k, v in r["params"].items():
            getattr(m, k).copy_(v)
    m = m.to(dev())
    with torch.no_grad():
        y = m(r["x"].to(dev()))
    ops.check_status()
    close(y, r["y"], tol)


def test_mini_stu_spectral_matches_reference_golden(golden):
    import flash_stu_2_b200 as F
    from flash_stu_2_b200 import ops
    r = golden("mini_stu")["spectral_fp32"]
    L, K = r["phi"].shape
    m = F.MiniSTU(seq_len=L, num_filters=K, input_dim=r["x"].shape[2], output_dim=r["y"].shape[2],
                  precomputed_filters=r["phi"])
    m.load_state_dict(r["params"])
    m = m.to(dev())
    with torch.no_grad():
        y = m(r["x"].to(dev()))
    ops.check_status()
    close(y, r["y"], 1e-3)


@pytest.mark.parametrize("dt,tol", [(torch.float32, 1e-3), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("shape", [(2, 48, 6, 10), (3, 200, 64, 32)])
def test_mini_stu_lds_prefill_and_recurrent_decode(golden, dt, tol, shape):
    """MiniSTU(backend='lds'): prefill (convolution with the LDS impulse responses) and the recurrent decode
    steps against the float64 recurrence of the reference (mini_stu/stu_lds.py) on the same rounded inputs."""
    import flash_stu_2_b200 as F
    from flash_stu_2_b200 import ops
    B, T, din, dout = shape
    g = golden("mini_stu")["lds_fp64"]
    torch.manual_seed(13)
    m = F.MiniSTU(seq_len=T, num_filters=24, input_dim=din, output_dim=dout, backend="lds", dtype=dt)
    x = torch.randn(B, T, din).to(dt)
    Mr = m.distill_stu.M.detach().clone()
    Cr = m.lds_module.C.detach().clone()
    assert torch.equal(m.lds_module.A, g["A"]) and torch.equal(Cr, g["C"].to(dt))
    want = O.lds_forward(x.double(), g["A"], g["B_vec"], Cr.double(), g["h0"], Mr.double())
    m = m.to(dev())
    T1 = T - 9
    with torch.no_grad():
        y_all = m(x.to(dev()))
        y1, cache = m(x[:, :T1].to(dev()), use_cache=True)
        state_scan = cache[0].clone()
        rows = [y1]
        for t in range(T1, T):
            yt, cache = m(x[:, t:t + 1].to(dev()), past_key_value=cache, use_cache=True)
            rows.append(yt)
        # the convolution form of the same prefill (full-length impulse responses): same rows within tolerance, and
        # its final-state kernel gives bit for bit the state the chunked scan hands to the recurrent decode
        F.MiniSTU.chunked_scan_prefill = False
        try:
            y_conv, cache_conv = m(x[:, :T1].to(dev()), use_cache=True)
        finally:
            F.MiniSTU.chunked_scan_prefill = True
    ops.check_status()
    assert torch.equal(cache_conv[0], state_scan)
    close(y_conv, want[:, :T1], tol)
    close(y_all, want, tol)
    got = torch.cat(rows, 1)
    close(got, want, tol)
    if shape == (2, 48, 6, 10) and dt == torch.float32:
        # the reference module's own output (float64 run of MiniSTU(backend='lds')) with its M
        m2 = F.MiniSTU(seq_len=T, num_filters=24, input_dim=din, output_dim=dout, backend="lds", dtype=dt)
        with torch.no_grad():
            m2.distill_stu.M.copy_(g["M"].to(dt))
        m2 = m2.to(dev())
        with torch.no_grad():
            y2 = m2(g["x"].to(dt).to(dev()))
        close(y2, g["y"], 1e-3)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,d,D,F", [(1, 7, 160, 48), (2, 64, 161, 64), (3, 65, 3, 1), (1, 200, 256, 9), (5, 24, 64, 33), (2, 96, 100, 50)])
def test_lds_state_step_of_any_size(dt, B, d, D, F):
    """The recurrent step's state and features against float64, over its limits of modes and features: constants of sizes that divide
    neither the block nor its staging rounds, channels that fill no CTA; two steps, plain and beside the kernels in front."""
    from flash_stu_2_b200 import ops
    from flash_stu_2_b200.modules import new_pos
    g = torch.Generator(device=dev()).manual_seed(D + F)
    rand = lambda *s: torch.randn(*s, device=dev(), generator=g, dtype=torch.float64)
    A, Bv, C, h = rand(D).tanh(), rand(D), rand(D, F).to(dt), rand(B, d, D)
    want = h.clone()
    pos = new_pos(B, dev())
    torch.cuda.synchronize()
    for overlap in (False, True):
        x, U = rand(B, d).to(dt), torch.full((B, F * d), 7.0, dtype=dt, device=dev())
        ops.lds_decode_features(x, h, A, Bv, C, U, pos, overlap)
        want = torch.addcmul(A * want, Bv, x.double()[..., None])
        assert (h - want).abs().max() <= 1e-14 * want.abs().max()   # fma against product and sum
        close(U.view(B, F, d), (h @ C.double()).transpose(1, 2), 1e-6 if dt == torch.float32 else 2 ** -8)
    ops.check_status()
    assert pos[:, 0].tolist() == [2] * B


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("S,ld,L", [(1, 1, 3), (7, 8, 40), (8, 8, 16), (9, 16, 9), (33, 35, 60), (264, 264, 700), (1024, 1024, 4096),
                                    (1025, 1032, 900), (2056, 2060, 5000)])
def test_toeplitz_matrices_of_any_size(dt, S, ld, L):
    """The three matrices of a filter on both sides of the change from 8 to 32 rows per CTA, over several column tiles, with
    rows on and off the 16-byte grid, filters shorter than the matrices; nothing is written between the rows."""
    from flash_stu_2_b200 import _lib
    torch.manual_seed(3)
    phi = torch.randn(L, 3).to(dt)
    out = torch.full((3, S, ld), 7.0, dtype=dt, device=dev())
    col = phi.to(dev())[:, 1]
    rc = _lib.load().stu_toeplitz(col.data_ptr(), 3, L, out.data_ptr(), S, ld, int(dt == torch.bfloat16),
                                  torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    lag = torch.arange(S)[:, None] - torch.arange(S)[None, :]
    for kind, tap in enumerate((2 * lag, 2 * lag + 1, 2 * lag - 1)):
        f = phi[:, 1][tap.clamp(0, L - 1)]
        want = torch.where((lag >= 0) & (tap >= 0) & (tap < L), f, torch.zeros((), dtype=dt))
        assert torch.equal(out[kind, :, :S].cpu(), want), kind
    assert bool((out[:, :, S:] == 7.0).all())


@pytest.mark.parametrize("shape", [(8, 200, 768, 0), (5, 40001, 132, 0), (8, 19000, 772, 1), (1, 300, 1540, 0), (7, 4736, 260, 2), (7, 4737, 260, 2),
                                   (3, 97, 1284, 1), (6, 64, 4, 0), (8, 1, 640, 0), (6, 18945, 768, 0), (6, 18944, 768, 0)])
def test_fp32_linears_of_up_to_8_rows_at_the_edges_of_their_split(shape):
    """1 to 13 chunks of K over 1 to 8 warps, one and several rounds of CTAs, the widths around which a product of 5 to 8 rows
    changes kernels, with the norm fused and apart."""
    from flash_stu_2_b200 import ops
    M, N, K, epi = shape
    torch.manual_seed(15)
    x, nw = torch.randn(M, K), 1.0 + 0.1 * torch.randn(K)
    W, W2, resid = torch.randn(N, K) / math.sqrt(K), torch.randn(N, K) / math.sqrt(K), torch.randn(M, N)
    kw = dict(W2=W2.to(dev()) if epi == 2 else None, resid=resid.to(dev()) if epi == 1 else None, epilogue=epi)
    y = ops.linear(x.to(dev()), W.to(dev()), **kw)
    close(y, _lin_ref(x, W, W2, resid, epi, torch.float32), TOL[torch.float32] / 2)
    xn = x * torch.rsqrt(x.pow(2).mean(1, keepdim=True) + ops.RMS_EPS) * nw
    y = ops.linear(x.to(dev()), W.to(dev()), norm_w=nw.to(dev()), **kw)
    close(y, _lin_ref(xn, W, W2, resid, epi, torch.float32), TOL[torch.float32] / 2)
    ops.check_status()


@pytest.mark.parametrize("B,d,K,L,signs", [(1, 40, 5, 64, 2), (3, 72, 24, 200, 2), (2, 264, 32, 96, 1), (8, 1024, 24, 520, 2), (9, 528, 16, 90, 2)])
def test_full_variant_step_kernel(B, d, K, L, signs):
    """The one-kernel step of the full variant against float64 sums at the first positions, around whole 8s and 32s of a parity
    and at the last one: U, the appended input, the position; 16 and 32 channels per CTA, channels and filters that fill no
    tile; what the cache holds past the position has no effect.  Bar: as for the prefill's U (E, Q and their sum rounded to bf16)."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(16)
    Lh = ((L + 1) // 2 + 7) // 8 * 8
    x, phi = (3 * torch.randn(B, L, d)).bfloat16(), (torch.randn(L, K) / 4).bfloat16()
    w = (1 + 0.1 * torch.randn(d)).bfloat16()
    xn = O.rmsnorm(x, w)
    f = phi.to(dev())
    taps8 = ops.taps_rev8(torch.cat([ops.taps_even(f, Lh), ops.taps_even(f[1:], Lh)]))
    for t in sorted({0, 1, 2, 15, 16, 17, 31, 33, 62, 63, L - 2, L - 1}):
        hist = torch.full((B, d, 2, Lh), float("nan"), dtype=torch.bfloat16, device=dev())
        if t:
            ops.to_history(xn[:, :t].to(dev()), hist, 0)
        pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
        pos[:, 0] = t
        U = torch.full((B, signs * K * d), 7.0, dtype=torch.bfloat16, device=dev())
        row = x[:, t].to(dev())
        assert ops.full_decode_step_supported(row, hist, K)
        ops.full_decode_step(row, w.to(dev()), ops.RMS_EPS, hist, taps8, pos, U, L, signs == 2)
        ops.check_status()
        assert pos.tolist() == [[t + 1, 0]] * B
        close(hist[:, :, t & 1, t >> 1], xn[:, t], 2 ** -7)
        past = xn[:, :t + 1].double().flip(1)
        past[:, 0] = hist[:, :, t & 1, t >> 1].cpu().double()   # (its rounding may differ by one unit)
        taps = phi[:t + 1].double()
        want = [torch.einsum("tk,bti->bki", taps * (s ** torch.arange(t + 1))[:, None], past).reshape(B, K * d) for s in (1.0, -1.0)]
        close(U, torch.cat(want[:signs], 1), 4 * 2 ** -9)
    pos[:, 0] = L
    ops.full_decode_step(row, w.to(dev()), ops.RMS_EPS, hist, taps8, pos, U, L, signs == 2)
    with pytest.raises(RuntimeError, match="status 2"):
        ops.check_status()
    assert int(pos[0, 0]) == L


@pytest.mark.parametrize("B,d,K,L,signs", [(1, 64, 5, 64, 2), (3, 128, 24, 260, 2), (2, 192, 32, 96, 1), (1, 128, 9, 1100, 2), (3, 3200, 8, 40, 2)])
def test_full_variant_step_kernel_on_tensor_cores(monkeypatch, B, d, K, L, signs):
    """The same on tcgen05: filters that fill no 8, positions around whole stages of 128 and past the ring's depth, both depths of the ring."""
    from flash_stu_2_b200 import ops
    monkeypatch.setattr(ops, "full_decode_step_tc5_pays", lambda *a: True)
    torch.manual_seed(17)
    Lh = ((L + 1) // 2 + 7) // 8 * 8
    x, phi = (3 * torch.randn(B, L, d)).bfloat16(), (torch.randn(L, K) / 4).bfloat16()
    w = (1 + 0.1 * torch.randn(d)).bfloat16()
    xn = O.rmsnorm(x, w)
    f = phi.to(dev())
    taps8 = ops.taps_rev8(torch.cat([ops.taps_even(f, Lh), ops.taps_even(f[1:], Lh)]))
    for t in sorted({t for t in (0, 1, 2, 15, 16, 33, 126, 127, 128, 129, 130, 255, 256, 257, 767, 768, 769, 900, L - 2, L - 1) if t < L}):
        hist = torch.full((B, d, 2, Lh), float("nan"), dtype=torch.bfloat16, device=dev())
        if t:
            ops.to_history(xn[:, :t].to(dev()), hist, 0)
        pos = torch.zeros(B, 2, dtype=torch.int32, device=dev())
        pos[:, 0] = t
        U = torch.full((B, signs * K * d), 7.0, dtype=torch.bfloat16, device=dev())
        ops.full_decode_step(x[:, t].to(dev()), w.to(dev()), ops.RMS_EPS, hist, taps8, pos, U, L, signs == 2, t)
        ops.check_status()
        assert pos.tolist() == [[t + 1, 0]] * B
        close(hist[:, :, t & 1, t >> 1], xn[:, t], 2 ** -7)
        past = xn[:, :t + 1].double().flip(1)
        past[:, 0] = hist[:, :, t & 1, t >> 1].cpu().double()   # (its rounding may differ by one unit)
        taps = phi[:t + 1].double()
        want = [torch.einsum("tk,bti->bki", taps * (s ** torch.arange(t + 1))[:, None], past).reshape(B, K * d) for s in (1.0, -1.0)]
        close(U, torch.cat(want[:signs], 1), 4 * 2 ** -9)
    # the row as it was appended, without a norm: the same bits
    new, again = hist[:, :, t & 1, t >> 1].clone(), torch.empty_like(U)
    hist[:, :, t & 1, t >> 1], pos[:, 0] = float("inf"), t
    ops.full_decode_step(new, None, 0.0, hist, taps8, pos, again, L, signs == 2, t)
    ops.check_status()
    assert torch.equal(again, U) and torch.equal(hist[:, :, t & 1, t >> 1], new)
    pos[:, 0] = L
    ops.full_decode_step(x[:, 0].to(dev()), w.to(dev()), ops.RMS_EPS, hist, taps8, pos, U, L, signs == 2, L)
    with pytest.raises(RuntimeError, match="status 2"):
        ops.check_status()
    assert int(pos[0, 0]) == L


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,d", [(2368, 64), (2401, 264), (5000, 1024), (2500, 1536), (2400, 3072), (2999, 1000)])
def test_rmsnorm_of_many_rows(dt, rows, d):
    """A warp per row: widths that fill no round of the lanes, more rows than a multiple of the CTAs' warps."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(21)
    x, w = (torch.randn(rows, d) * 3).to(dt), torch.randn(d).to(dt)
    close(ops.rmsnorm(x.to(dev()), w.to(dev())), O.rmsnorm(x, w), 1e-6 if dt == torch.float32 else 2 ** -7)


@pytest.mark.parametrize("epi", [0, 2])
@pytest.mark.parametrize("shape", [(33, 70, 64, 72), (129, 8, 72, 16), (300, 1000, 136, 1000), (2500, 5121, 64, 5128), (257, 64, 200, 64)])
def test_linear_outputs_by_tensor_copies(shape, epi):
    """Plain and gate/up outputs of the tcgen05 GEMM on rows of the 16-byte grid: last rows and columns that fill no block of 32 x
    64, rows wider than the output; nothing beside it is written."""
    from flash_stu_2_b200 import ops
    M, N, K, ld = shape
    torch.manual_seed(19)
    x, W, W2 = torch.randn(M, K).bfloat16(), (torch.randn(N, K) / math.sqrt(K)).bfloat16(), (torch.randn(N, K) / math.sqrt(K)).bfloat16()
    buf = torch.full((M + 64, ld), 7.0, dtype=torch.bfloat16, device=dev())
    ops.linear(x.to(dev()), W.to(dev()), W2=W2.to(dev()) if epi else None, out=buf[:M, :N], epilogue=epi, backend=2)
    ops.check_status()
    close(buf[:M, :N], _lin_ref(x, W, W2, None, epi, torch.bfloat16), 1e-2)
    assert bool((buf[:M, N:] == 7.0).all()) and bool((buf[M:] == 7.0).all())


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,nch,Ck,F,K", [(64, 3, 128, 48, 320), (128, 2, 64, 40, 200), (64, 1, 32, 8, 32), (72, 2, 128, 5, 136)])
def test_lds_features_skip_what_a_toeplitz_operand_leaves_out(dt, d, nch, Ck, F, K):
    """Features whose operand is zero behind its diagonal: the blocks that are skipped take nothing from the sums (the same bits as with
    them), wherever the last row of a tile lies."""
    from flash_stu_2_b200 import ops
    g = torch.Generator(device=dev()).manual_seed(K)
    W = torch.randn(Ck * F, K, device=dev(), generator=g) / math.sqrt(K)
    tau, col = torch.arange(Ck * F, device=dev()) // F, torch.arange(K, device=dev())
    W = W.masked_fill(col[None, :] > (K - Ck + tau)[:, None], 0.0).to(dt).contiguous()
    Z = torch.randn(nch * d, K, device=dev(), generator=g).to(dt)
    a, b = (torch.full((nch * Ck, F * d), 7.0, dtype=dt, device=dev()) for _ in range(2))
    ops.lds_chunk_features(W, Z, a, d, Ck, F, causal=True)
    ops.lds_chunk_features(W, Z, b, d, Ck, F)   # (says nothing of W: its hist_t0 and hist_Lh are not looked at)
    ops.check_status()
    assert torch.equal(a, b)
    full = torch.randn(Ck * F, K, device=dev(), generator=g).to(dt)
    ops.lds_chunk_features(full, Z, b, d, Ck, F)
    close(b, (full.double() @ Z.double().t()).view(Ck, F, nch, d).permute(2, 0, 1, 3).reshape(nch * Ck, F * d), 1e-5 if dt == torch.float32 else 2 ** -8)
    want = (W.double() @ Z.double().t()).view(Ck, F, nch, d).permute(2, 0, 1, 3).reshape(nch * Ck, F * d)
    close(a, want, 1e-5 if dt == torch.float32 else 2 ** -8)


@pytest.mark.parametrize("d,chunks,rows,K", [(64, 3, 96, 72), (192, 2, 130, 320), (40, 5, 96, 64), (1024, 2, 6144, 320)])
def test_lds_features_in_column_blocks(d, chunks, rows, K):
    """The blocked output of the LDS features: blocks of whole 64s leave by tensor copies, others by the lanes."""
    from flash_stu_2_b200 import ops
    F = 6 if rows % 6 == 0 else 5
    Ck = rows // F
    torch.manual_seed(20)
    W, Z = (torch.randn(Ck * F, K) / math.sqrt(K)).bfloat16(), torch.randn(chunks * d, K).bfloat16()
    U = torch.full((chunks * Ck + 1, F * d), 7.0, dtype=torch.bfloat16, device=dev())
    ops.lds_chunk_features(W.to(dev()), Z.to(dev()), U[:chunks * Ck], d, Ck, F)
    ops.check_status()
    want = (W.double() @ Z.double().t()).view(Ck, F, chunks, d).permute(2, 0, 1, 3).reshape(chunks * Ck, F * d)
    close(U[:-1], want, 1e-2)
    assert bool((U[-1] == 7.0).all())


@pytest.mark.parametrize("gain", [0.2, 3.0, 12.0])
@pytest.mark.parametrize("cap", [50.0, 4.0, 0.0])
@pytest.mark.parametrize("hd", [64, 128])
def test_attention_prefill_soft_cap_small_and_large(hd, cap, gain):
    """Scores far below the cap (polynomial), beyond it (hardware tanh) and mixed within a tile; no cap; both head dimensions.  Bar:
    P and the output are rounded to bf16 (2^-9 each), the hardware tanh is off by 2^-11 of a score of at most cap."""
    from flash_stu_2_b200 import ops
    B, T, H, w = 2, 333, 3, 150
    d = H * hd
    torch.manual_seed(18)
    qkv = torch.randn(B, T, 3 * d)
    qkv[:, :, :2 * d] *= gain ** 0.5
    qkv[:, 100:200, :d] *= 0.1
    qkv = qkv.bfloat16().to(dev())
    slopes = O.alibi_slopes(H).float().to(dev())
    dummy = torch.zeros(1, 1, 1, dtype=torch.bfloat16, device=dev())
    y = ops.swa_prefill_tc5(qkv, dummy, dummy, torch.zeros(B, 2, dtype=torch.int32, device=dev()), slopes, H, w, cap, update_cache=False)
    ops.check_status()
    q, k, v = [a.double().view(B, T, H, hd).transpose(1, 2) for a in qkv.split(d, dim=2)]
    s = q @ k.transpose(2, 3) / math.sqrt(hd)
    s = cap * torch.tanh(s / cap) if cap else s
    lag = torch.arange(T, device=dev())[:, None] - torch.arange(T, device=dev())[None, :]
    s = s - slopes.double()[None, :, None, None] * lag
    s = s.masked_fill((lag < 0) | (lag > w), float("-inf"))
    want = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B, T, d)
    close(y, want, 1.5e-2 if cap != 50.0 or gain < 12 else 3e-2)


def test_linear_through_the_extension_module_checks_what_the_interpreter_checks():
    """Shapes, strides and dtypes that the fast call does not take get the general path's answer."""
    from flash_stu_2_b200 import ops
    x, W = torch.randn(5, 64, device=dev()), torch.randn(32, 64, device=dev())
    want = x @ W.t()
    close(ops.linear(x, W), want, 1e-5)
    close(ops.linear(x, W.t().contiguous(), transposed_weight=True), want, 1e-5)
    close(ops.linear(torch.randn(7, 128, device=dev())[:5].copy_(torch.cat([x, x], 1))[:, 64:], W), want, 1e-5)   # rows of a wider tensor
    buf = torch.full((5, 40), 7.0, device=dev())
    assert ops.linear(x, W, out=buf[:, :32]).data_ptr() == buf.data_ptr() and bool((buf[:, 32:] == 7).all())
    for bad in (lambda: ops.linear(x[:, :60], W), lambda: ops.linear(x, W, out=buf), lambda: ops.linear(x, W, W2=W[:16]),
                lambda: ops.linear(x, W, resid=x, epilogue=ops.EPI_RESID), lambda: ops.linear(x.t(), W)):
        with pytest.raises(AssertionError):
            bad()
    with pytest.raises(TypeError):
        ops.linear(x.double(), W.double())
    with pytest.raises(RuntimeError, match="no CPU path"):
        ops.linear(x, W.cpu())
    close(ops.rmsnorm(x.t(), torch.ones(5, device=dev())), O.rmsnorm(x.t().cpu(), torch.ones(5)), 1e-5)
    with torch.inference_mode():
        assert ops.linear(x, W).is_inference()


@pytest.mark.parametrize("epi", [0, 1, 2])
@pytest.mark.parametrize("shape", [(130, 96, 72), (64, 16, 1000), (300, 33, 40), (70, 160, 3072), (1000, 32, 17)])
def test_cuda_core_gemm_of_few_columns(shape, epi):
    """fp32 tiles of 32 and 64 columns, ragged in every direction, K split over a cluster and not, against float64.  Bar: sums of K
    products in fp32, each rounding at most 2^-24 of the sum of magnitudes (below 4 sqrt(K) of a result's size here)."""
    from flash_stu_2_b200 import ops
    M, N, K = shape
    torch.manual_seed(17)
    x, W, W2, r = torch.randn(M, K), torch.randn(N, K) / math.sqrt(K), torch.randn(N, K) / math.sqrt(K), torch.randn(M, N)
    y = ops.linear(x.to(dev()), W.to(dev()), W2=W2.to(dev()) if epi == 2 else None, resid=r.to(dev()) if epi == 1 else None,
                   epilogue=epi, backend=1)
    acc = x.double() @ W.double().t()
    want = acc if epi == 0 else r.double() + acc if epi == 1 else \
        torch.nn.functional.gelu(acc, approximate="tanh") * (x.double() @ W2.double().t())
    close(y, want, 4 * math.sqrt(K) * 2 ** -22, row_tol=1e-4)
    ops.check_status()


def _leave_an_error_behind():
    """A launch that the host refuses (more blocks along y than a grid has), nothing reaches the device: the error stays noted."""
    from flash_stu_2_b200 import _lib, ops
    t = torch.zeros(64, 8, dtype=torch.bfloat16, device=dev())
    a = t.data_ptr()
    assert _lib.load().stu_decode_approx(a, 8, a, a, a, a, a, a, a, 8, 1 << 20, 8, 8, 1e-6, a, 1, ops._stream()) > 0


def test_an_error_left_behind_raises_and_a_product_in_place_is_made_at_most_once():
    """A launch after which the library sees an error raises, even where the product itself went out; it is not made again, which
    would add the branch to the residual twice.  The error is gone with that."""
    from flash_stu_2_b200 import ops
    x, W, w = torch.randn(5, 64, device=dev()), torch.randn(64, 64, device=dev()), torch.ones(64, device=dev())
    y, branch = torch.randn(5, 64, device=dev()), x @ W.t()
    before = y.clone()
    for _ in range(2):   # (the first call registers the status word, the first native one loads the kernel, which clears errors)
        ops.linear(x, W, resid=y, out=torch.empty_like(y), epilogue=ops.EPI_RESID)
    _leave_an_error_behind()
    with pytest.raises(RuntimeError, match="CUDA error"):
        ops.linear(x, W, resid=y, out=y, epilogue=ops.EPI_RESID)
    if not torch.equal(y, before):
        close(y, before + branch, 1e-5)
    y.copy_(before)
    close(ops.linear(x, W, resid=y, out=y, epilogue=ops.EPI_RESID), before + branch, 1e-5)
    ops.rmsnorm(x, w)
    _leave_an_error_behind()
    with pytest.raises(RuntimeError, match="CUDA error"):
        ops.rmsnorm(x, w)
    close(ops.rmsnorm(x, w), O.rmsnorm(x.cpu(), w.cpu()), 1e-5)
    ops.check_status()


def test_full_variant_step_right_behind_its_tap_table():
    """The step is launched with the programmatic attribute: on a stream where the kernel directly in front writes the tap table,
    what it takes of that table is the new one.  Other taps in the same buffer each time; the first position (U = x f[0]: E alone,
    which is Q's zero added and subtracted), so that everything hangs on the tap at distance 0.  Bar: products rounded to bf16 once."""
    from flash_stu_2_b200 import _lib, ops
    B, d, K, Lh = 4, 256, 24, 512
    torch.manual_seed(22)
    x = torch.randn(B, d).bfloat16().to(dev())
    taps = [torch.randn(2 * K, Lh).bfloat16().to(dev()) for _ in range(8)]
    taps8 = ops.taps_rev8(taps[0])
    hists = [torch.zeros(B, d, 2, Lh, dtype=torch.bfloat16, device=dev()) for _ in taps]
    pos = [torch.zeros(B, 2, dtype=torch.int32, device=dev()) for _ in taps]
    U = [torch.empty(B, 2 * K * d, dtype=torch.bfloat16, device=dev()) for _ in taps]
    torch.cuda.synchronize()
    for tp, h, p, u in zip(taps, hists, pos, U):
        _lib.check(_lib.native().stu_taps_rev8(tp, taps8, 2 * K, Lh, 1, ops._stream()), "stu_taps_rev8")
        ops.full_decode_step(x, None, 0.0, h, taps8, p, u, 2 * Lh, True)
    ops.check_status()
    for tp, u in zip(taps, U):
        want = (tp[:K, 0].double()[None, :, None] * x.double()[:, None, :]).reshape(B, K * d)
        close(u, torch.cat([want, want], 1), 2 ** -8)


@pytest.mark.parametrize("hd", [64, 128])
def test_attention_prefill_rows_do_not_depend_on_later_tokens(hd):
    """What follows a position changes no bit of its output, also where the later keys' scores lie beyond the soft cap (which takes
    another tanh) in the tile that the position's own keys are in.  (Rows of one warp share a reference maximum: whole warps
    of 32 positions in front of the change are compared.)"""
    from flash_stu_2_b200 import ops
    B, T, H, w = 1, 200, 2, 300
    torch.manual_seed(23)
    qkv = torch.randn(B, T, 3 * H * hd)
    loud = qkv.clone()
    loud[:, 97:] *= 40.0
    slopes = O.alibi_slopes(H).float().to(dev())
    dummy = torch.zeros(1, 1, 1, dtype=torch.bfloat16, device=dev())
    a, b = [ops.swa_prefill_tc5(x.bfloat16().to(dev()), dummy, dummy, torch.zeros(B, 2, dtype=torch.int32, device=dev()), slopes, H, w,
                                50.0, update_cache=False) for x in (qkv, loud)]
    ops.check_status()
    assert torch.equal(a[:, :96], b[:, :96]) and not torch.equal(a[:, 97:], b[:, 97:])


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,d", [(2367, 256), (2368, 256), (2369, 512), (3551, 1000), (3552, 1000), (3555, 1024), (3552, 776), (5919, 1536),
                                    (5920, 1536), (5921, 2048), (11839, 2056), (11840, 2056), (11841, 3072)])
def test_rmsnorm_of_many_rows_on_both_sides_of_its_lines(dt, rows, d):
    """Rows per warp and rows per CTA, in front of and behind the line of each width: a row's bits are those of a call of few rows."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(24)
    x, w = (torch.randn(rows, d, device=dev()) * 3).to(dt), torch.randn(d, device=dev()).to(dt)
    y = ops.rmsnorm(x, w)
    assert torch.equal(y[-300:], ops.rmsnorm(x[-300:].contiguous(), w)) and torch.equal(y[:300], ops.rmsnorm(x[:300].contiguous(), w))
    close(y[::97].cpu(), O.rmsnorm(x[::97].cpu(), w.cpu()), 1e-6 if dt == torch.float32 else 2 ** -7)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k", [3, 255, 256, 257, 511, 512, 513, 700, 1000, 1024])
@pytest.mark.parametrize("nucleus", [None, 0.3, 0.97])
def test_draws_among_few_and_many_survivors(dt, k, nucleus):
    """Top-k of up to 1024 entries, ties among them in bf16, with and without a nucleus: both sorts of the survivors.  Uniforms in the
    middle of an entry's share of the running sum, a nucleus that ends in the middle of one: the entry itself is drawn
    (shares of 10^-4 and more, fp32 sums of at most 1024 terms are off by less than 10^-5)."""
    from flash_stu_2_b200 import ops
    torch.manual_seed(k)
    z = (0.7 * torch.randn(3001)).to(dt)
    if dt == torch.bfloat16:   # ties at the k-th place would add survivors: push what ties with it from outside below
        first = torch.argsort(z.float(), descending=True, stable=True)
        z[first[k:]] -= 1.0
    w = z.double()
    kept = (w >= torch.topk(w, k)[0][-1]).nonzero()[:, 0]
    assert len(kept) == k
    top_p = None
    if nucleus is not None:
        order = kept[torch.argsort(w[kept], descending=True, stable=True)]
        share = torch.softmax(w[order], 0)
        last = min(int((share.cumsum(0) < nucleus).sum()), k - 2)
        top_p = float(share[:last].sum() + share[last] / 2)       # the mass in front of entry last + 1 is beyond it
        kept = order[:last + 1].sort()[0]
    share = torch.softmax(w[kept], 0)
    picks = torch.randint(0, len(kept), (16,))
    u = (share.cumsum(0) - share / 2)[picks].float()
    out = torch.full((16,), -1, dtype=torch.int64, device=dev())
    ops.sample(z.to(dev()).repeat(16, 1), 1.0, k, top_p, True, u.to(dev()), out)
    ops.check_status()
    assert torch.equal(out.cpu(), kept[picks])


@pytest.mark.parametrize("T", [128, 129, 383, 384, 385])
@pytest.mark.parametrize("w", [100, 300, 700])
def test_heads_of_64_on_both_attention_kernels(T, w):
    """Around the line between the two prefill kernels for heads of 64: outputs, rings and positions of either agree.  Bar: P and the
    output are rounded to bf16 in both, the hardware tanh and the polynomial are within 2^-11 of the function."""
    from flash_stu_2_b200 import ops
    B, H = 2, 3
    torch.manual_seed(25)
    qkv = torch.randn(B, T, 3 * H * 64).bfloat16().to(dev())
    slopes = O.alibi_slopes(H).float().to(dev())
    rings = [torch.zeros(2, B, w + 1, H * 64, dtype=torch.bfloat16, device=dev()) for _ in range(2)]
    pos = [torch.zeros(B, 2, dtype=torch.int32, device=dev()) for _ in range(2)]
    a, b = [f(qkv, r[0], r[1], p, slopes, H, w, 50.0, update_cache=True)
            for f, r, p in zip((ops.swa_prefill_tc5, ops.swa_forward), rings, pos)]
    ops.check_status()
    close(a, b, 1.5e-2)
    assert torch.equal(rings[0], rings[1]) and torch.equal(pos[0], pos[1]) and pos[0][:, 0].tolist() == [T] * B


@pytest.mark.parametrize("shape", [(1, 3, 64, 300, 0, 300), (1, 3, 72, 300, 10, 299), (1, 2, 128, 130, 0, 129), (1, 2, 136, 90, 0, 90), (3, 2, 88, 700, 300, 700)])
def test_full_convolution_tiles_of_64_128_and_256_channels(shape):
    """Rows on both sides of half a tile (64, 72; 128, 136), and a last tile of 8 rows, few tiles for the SMs: the bars of the test of
    the operand."""
    test_full_convolution_on_tensor_cores(shape, True)


@pytest.mark.parametrize("gain", [1.0, 8.0, 30.0])
def test_attention_prefill_of_heads_of_64_is_as_exact_as_the_running_maximum(gain):
    """Error against float64 of the tcgen05 kernel, whose reference maximum lags, and of the mma.sync kernel, whose does not: on the same
    inputs the former is no larger (by 1.01 at most: the two differ by which of 2 million roundings go which way)."""
    from flash_stu_2_b200 import ops
    T, H, w = 1024, 16, 512
    torch.manual_seed(26)
    qkv = torch.randn(1, T, 3 * H * 64, device=dev())
    qkv[:, :, :2 * H * 64] *= gain ** 0.5
    qkv = qkv.bfloat16()
    slopes = O.alibi_slopes(H).float().to(dev())
    dummy = torch.zeros(1, 1, 1, dtype=torch.bfloat16, device=dev())
    q, k, v = [a.double().view(1, T, H, 64).transpose(1, 2) for a in qkv.split(H * 64, dim=2)]
    s = 50 * torch.tanh(q @ k.transpose(2, 3) / 8 / 50)
    lag = torch.arange(T, device=dev())[:, None] - torch.arange(T, device=dev())[None, :]
    s = (s - slopes.double()[None, :, None, None] * lag).masked_fill((lag < 0) | (lag > w), float("-inf"))
    want = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(1, T, H * 64)
    err = [float((f(qkv, dummy, dummy, torch.zeros(1, 2, dtype=torch.int32, device=dev()), slopes, H, w, 50.0, update_cache=False).double()
                  - want).norm()) for f in (ops.swa_prefill_tc5, ops.swa_forward)]
    ops.check_status()
    assert err[0] <= 1.01 * err[1], err
