"""The layer's forward on more than 32 rows against the float64 value of the same packed operands: edges of the 128-row and
64/128/256-column tiles, ranks that do not fill a 64-rank stage, shapes that split K over a cluster and that do not."""
import ctypes

import pytest
import torch

from biloco_b200 import _lib, fp4, kernel
from biloco_b200.layer import BiLoCoLinear

pytestmark = pytest.mark.gpu


def exact(layer, x):
    """float64 value: NVFP4 activation (one scale for all rows) and weight as their codes say, exact low-rank term."""
    xs = (x / layer.smooth_scale) if layer.smoothed else x
    p, sf, gs = fp4.quantize_nvfp4(xs.float(), fp4.CONFIG_X)
    a = fp4.dequantize_nvfp4(p, sf, gs).double()
    w = fp4.dequantize_nvfp4(layer.W_codes, layer.W_sf.view(torch.float8_e4m3fn), layer.w_gscale).double()
    y = a @ w.T
    if layer.rank:
        z = (xs.double() @ kernel.unpack_signs(layer.V_packed).double().T) * layer.S.double()
        y = y + z @ kernel.unpack_signs(layer.U_packed).double()
    return y + layer.bias.double() if layer.bias is not None else y


@pytest.mark.parametrize("rows,K,N,R,smooth,bias", [
    (33, 256, 8, 1, False, False),           # the smallest of everything
    (127, 512, 72, 40, True, True),
    (128, 768, 136, 64, False, True),
    (129, 1024, 264, 65, True, False),
    (300, 2560, 1000, 200, False, False),    # 64-column tiles
    (2000, 4096, 136, 512, False, False),    # z: rings that wrap, no K split
    (640, 1024, 4104, 512, False, True),     # more tiles than SMs, last tile one piece wide
    (1000, 512, 9728, 128, True, False),
    (2048, 1280, 5120, 129, False, False),   # 256-column tiles, several per CTA
    (257, 512, 384, 0, True, True),          # NVFP4 alone
])
def test_prompt_matches_exact_value(rows, K, N, R, smooth, bias):
    g = torch.Generator(device="cuda").manual_seed(rows + N)
    ops = BiLoCoLinear.synthetic(K, N, max(R, 1), "cuda", seed=rows).export_operands()
    if R == 0:
        ops["V_packed"], ops["U_packed"], ops["S"] = ops["V_packed"][:0], ops["U_packed"][:0], ops["S"][:0]
    else:       # (random codes give large FP4 sums: coefficients of a size that makes the low-rank term as large)
        ops["S"] = (torch.randn(R, device="cuda", generator=g) * 0.2).to(torch.bfloat16)
    if smooth:
        ops["smooth_scale"] = (torch.rand(K, device="cuda", generator=g) * 2 + 0.5).to(torch.bfloat16)
    if bias:
        ops["bias"] = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    layer = BiLoCoLinear.from_operands(ops)
    x = torch.randn(rows, K, device="cuda", generator=g)
    x[:, torch.randperm(K, device="cuda", generator=g)[: K // 100 + 1]] *= 20
    x[rows // 2, :32] = 0.0
    x = x.to(torch.bfloat16)
    want = exact(layer, x)
    first = None
    for _ in range(3):
        y = layer(x)
        first = y if first is None else first
        assert torch.equal(y, first)                                   # fixed order of every sum
    # bf16 rounding is 2^-9; fp32 accumulation and the two-part z add a few 2^-17 of the largest partial sums
    den = torch.maximum(want.abs(), 1e-3 * want.abs().max())
    assert float(((y.double() - want).abs() / den).max()) <= 1e-2
    assert float(torch.linalg.norm(y.double() - want) / torch.linalg.norm(want)) <= 2e-3
    st = (ctypes.c_int32 * 16)()
    _lib.check(_lib.load().biloco_b200_prompt_status(st, torch.cuda.current_stream().cuda_stream), "prompt_status")
    assert st[0] == 0


@pytest.mark.parametrize("rows,N,R", [(33, 136, 2), (40, 136, 96), (261, 1024, 66), (2049, 5120, 64)])      # (64-, 128- and 256-column tiles)
def test_prompt_rows_behind_the_last_32_keep_fp32_z(rows, N, R):
    """Ranks in pairs of opposite U signs whose z are large and equal but for one element of one pair: the output is twice that element. One
    to eight rows behind the last whole 32 have z in full (a decode launch of as many rows has), so the output is right to a bf16
    rounding and fp32 roundings of the large terms; of z as two bf16 parts 2^-17 could be missing, 1 % of these outputs."""
    K = 4096
    ops = BiLoCoLinear.synthetic(K, N, R, "cuda", seed=1).export_operands()
    ops["W_codes"] = torch.zeros_like(ops["W_codes"])
    g = torch.Generator(device="cuda").manual_seed(rows)
    V, U = torch.ones(R, K, device="cuda"), torch.ones(R, N, device="cuda")
    V[R - 1, 1234] = -1.0
    U[1::2] = -1.0
    ops["V_packed"], ops["U_packed"] = kernel.pack_signs(V), kernel.pack_signs(U)
    ops["S"] = torch.ones(R, device="cuda", dtype=torch.bfloat16)
    x = (torch.rand(rows, K, device="cuda", generator=g) + 0.5).to(torch.bfloat16)
    y = BiLoCoLinear.from_operands(ops)(x).double()
    want = ((x.double() @ V.double().T) @ U.double())
    last = slice(rows - rows % 32, rows)
    err = (y - want)[last].abs()
    assert bool((err <= want[last].abs() * 2.0 ** -9 + 4 * 4096 * 1.5 * 2.0 ** -24).all()), float((err / want[last].abs()).max())


@pytest.mark.parametrize("wscale,xscale", [(1e-38, 1e-6), (0.0, 1.0), (1e-30, 1e-6), (1e-3, 1e-36)])
def test_prompt_with_a_vanishing_alpha(wscale, xscale):
    """alpha = w_gscale * activation scale underflows to zero, or is subnormal, or small with small activations: the low-rank term stays
    (z is kept divided by alpha inside)."""
    rows, K, N, R = 50, 512, 136, 96
    ops = BiLoCoLinear.synthetic(K, N, R, "cuda", seed=4).export_operands()
    ops["w_gscale"] = torch.full((1,), wscale, device="cuda")
    ops["S"] = torch.ones_like(ops["S"])
    g = torch.Generator(device="cuda").manual_seed(4)
    x = (torch.randn(rows, K, device="cuda", generator=g) * xscale).to(torch.bfloat16)
    y = BiLoCoLinear.from_operands(ops)(x).double()
    want = (x.double() @ kernel.unpack_signs(ops["V_packed"]).double().T) @ kernel.unpack_signs(ops["U_packed"]).double()
    if wscale == 1e-3:                       # (here the NVFP4 part is not negligible)
        p, sf, gs = fp4.quantize_nvfp4(x.float(), fp4.CONFIG_X)
        alpha = ops["w_gscale"] * gs
        one = torch.ones(1, device="cuda")
        want = want + (fp4.dequantize_nvfp4(p, sf, one).double() @ fp4.dequantize_nvfp4(ops["W_codes"], ops["W_sf"], one).double().T) * alpha.double()
    assert float(torch.linalg.norm(y - want) / torch.linalg.norm(want)) <= 2e-3       # (bf16 rounding)


@pytest.mark.parametrize("R", [0, 32])
def test_prompt_with_a_nan(R):
    """One NaN element: the tensor scale is what fp4.activation_scale_from_amax makes of a NaN maximum (1); rows without a NaN have the
    value of that quantisation, the row with it is NaN where its low-rank term is."""
    rows, K, N = 70, 512, 136
    ops = BiLoCoLinear.synthetic(K, N, max(R, 1), "cuda", seed=4).export_operands()
    if R == 0:
        ops["V_packed"], ops["U_packed"], ops["S"] = ops["V_packed"][:0], ops["U_packed"][:0], ops["S"][:0]
    layer = BiLoCoLinear.from_operands(ops)
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(rows, K, device="cuda", generator=g).to(torch.bfloat16)
    x[41, 100] = float("nan")
    y = layer(x)
    gs = fp4.activation_scale_from_amax(x.float().abs().max().reshape(1))
    ok = torch.arange(rows, device="cuda") != 41
    p, sf, _ = fp4.quantize_nvfp4(x[ok].float(), fp4.CONFIG_X, gs)
    want = fp4.dequantize_nvfp4(p, sf, gs).double() @ fp4.dequantize_nvfp4(layer.W_codes, layer.W_sf.view(torch.float8_e4m3fn), layer.w_gscale).double().T
    if R:
        want = want + ((x[ok].double() @ kernel.unpack_signs(layer.V_packed).double().T) * layer.S.double()) @ kernel.unpack_signs(layer.U_packed).double()
    assert float(torch.linalg.norm(y[ok].double() - want) / torch.linalg.norm(want)) <= 2e-3       # (bf16 rounding; the derived scale gives 0.1)
    assert bool(y[41].isnan().all()) == bool(R)


@pytest.mark.parametrize("rule", ["mse", "static_6", "static_4"])
@pytest.mark.parametrize("rows,K", [(1, 16), (127, 48), (129, 336), (300, 1024)])
def test_weight_quantiser_bytes_equal_the_cpu_restatement(rows, K, rule):
    """Codes, scale atoms (zero padding included) and tensor scale, bit for bit; elements on rounding boundaries among them (few
    distinct magnitudes: quotients that are ties) and all-zero blocks; a given tensor scale."""
    g = torch.Generator().manual_seed(rows + K)
    x = torch.randn(rows, K, generator=g) * 0.02
    half = rows // 2
    x[half:] = torch.tensor([0.25, 0.375, 0.5, 0.75, 1.0, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0])[torch.randint(0, 11, (rows - half, K), generator=g)] * 0.01
    x[-1, :16] = 0.0
    for gscale in (None, 3e-4):
        want = fp4.quantize_nvfp4(x, rule, gscale)
        got = fp4.quantize_nvfp4(x.cuda(), rule, gscale)
        assert torch.equal(got[0].cpu(), want[0])
        assert torch.equal(got[1].view(torch.uint8).cpu(), want[1].view(torch.uint8))
        assert torch.equal(got[2].cpu(), want[2])


@pytest.mark.parametrize("rule", ["mse", "static_6", "static_4"])
@pytest.mark.parametrize("special", [(float("nan"),), (float("inf"),), (-float("inf"), float("nan")), ()])
def test_weight_quantiser_keeps_what_is_not_finite(special, rule):
    """NaN and infinities, and given tensor scales that are not positive: the bytes of the torch operations on the same device (a
    NaN's block decodes to NaN, it is not lost in a maximum)."""
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(130, 80, device="cuda", generator=g) * 0.02
    x[3, :16] = 0.0
    for i, v in enumerate(special):
        x[7 + 60 * i, 37] = v                # one element of a block
        x[9, 0] = v                          # (both in one block)
    for gscale in (None, 3e-4, 0.0, -3e-4, float("nan")):
        want = fp4._quantize_nvfp4_torch(x, rule, gscale)
        got = fp4.quantize_nvfp4(x, rule, gscale)
        for a, b in zip(got, want):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8)), gscale
    if special and special[-1] != special[-1]:
        q = fp4.fake_quantize_fp4(x, rule)
        assert bool(q[7 + 60 * (len(special) - 1), 32:48].isnan().all())


@pytest.mark.parametrize("M,K,smooth,norm,swiglu", [
    (1, 64, False, False, False), (1, 28672, False, True, False), (3, 576, True, True, False), (7, 2560, False, False, True),
    (17, 8192, True, False, False),          # sixteen CTAs, two rows per group
    (32, 9728, False, False, True), (128, 12288, True, False, False), (128, 320, False, True, False),      # shares beyond shared memory; four rows per group
])
def test_activation_quantiser_splits(M, K, smooth, norm, swiglu):
    """Every way the quantiser splits rows over its groups: codes, scales and tensor scale bit for bit what the CPU restatement makes
    of the activation it formed (which is the plain composition's to a bf16 unit, exactly so without a norm or exp)."""
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn(M, K * (2 if swiglu else 1), device="cuda", generator=g).to(torch.bfloat16)
    s = (torch.rand(K, device="cuda", generator=g) * 2 + 0.5).to(torch.bfloat16) if smooth else None
    w = (torch.rand(K, device="cuda", generator=g) + 0.5).to(torch.bfloat16) if norm else None
    ref = x
    if norm:
        ref = (x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-6)).to(torch.bfloat16) * w
    if swiglu:
        ref = torch.nn.functional.silu(x[:, :K]) * x[:, K:]
    if smooth:
        ref = ref / s
    q = None
    for _ in range(2):                       # (the second call reuses the buffers)
        q = fp4.quantize_activation(x, "mse", smooth=s, norm_weight=w, swiglu=swiglu, out=q)
        X = q["X"].float()
        assert float(((X - ref.float()).abs() / ref.float().abs().clamp(min=1e-30)).max()) <= (2.0 ** -6 if norm or swiglu else 0.0)
        p, sf, gs = fp4.quantize_nvfp4(q["X"].float().cpu(), "mse")
        assert torch.equal(q["A"][0].cpu(), p) and torch.equal(q["gscale"].cpu(), gs)
        assert torch.equal(q["A_sf"].view(torch.uint8).cpu(), sf.view(torch.uint8))


@pytest.mark.parametrize("rule", ["mse", "static_6", "static_4"])
@pytest.mark.parametrize("M,K", [(1, 64), (5, 512), (32, 2560)])
def test_activation_quantiser_leaves_nan_elements_out(M, K, rule):
    """A NaN element gets the code of a zero with its sign and counts for no maximum; a block that holds one keeps the divisor 6 under
    the mse rule (both errors are NaN, and the comparison takes 4 only where its error is smaller)."""
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    bits = x.view(torch.int16)
    spots = [(0, 3, 0x7FC0), (M - 1, K - 1, -0x40), (M // 2, K // 2, 0x7F81), (M // 2, K // 2 + 8, -0x7F)]      # (either sign, both halves of a block)
    for r, c, v in spots:
        bits[r, c] = v
    if K > 64:
        x[0, 32:48] = float("nan")           # a block of nothing else
    nan = x.isnan()
    q = fp4.quantize_activation(x, rule)
    clean = torch.where(nan, torch.zeros_like(x), x).float()
    gs = q["gscale"]
    p, sf, want_gs = fp4.quantize_nvfp4(clean, rule)
    p6, sf6, _ = fp4.quantize_nvfp4(clean, "static_6", want_gs) if rule == "mse" else (p, sf, None)
    assert torch.equal(gs, want_gs)
    blk = nan.view(M, K // 16, 16).any(-1)
    s = torch.where(blk, fp4.unswizzle_scales(sf6, M, K), fp4.unswizzle_scales(sf, M, K))
    assert torch.equal(fp4.unswizzle_scales(q["A_sf"], M, K), s)
    codes = lambda t: torch.stack([t & 15, t >> 4], -1).view(M, K)
    want = torch.where(blk.repeat_interleave(16, 1), codes(p6), codes(p))
    live = s.view(torch.float8_e4m3fn).float().repeat_interleave(16, 1) * gs > 0
    want = torch.where(nan, torch.where((bits < 0) & live, 8, 0).to(torch.uint8), want)
    assert torch.equal(codes(q["A"][0]), want)


@pytest.mark.parametrize("K,rows", [(512, 8), (2560, 32), (64, 128), (320, 40)])
def test_activation_buffers_are_padded_again(K, rows):
    """Buffers of an earlier call with more rows, or with anything in them: everything beyond the rows of this call is zero, in the codes, the
    scale atoms and the record (which equals that of fresh buffers)."""
    g = torch.Generator(device="cuda").manual_seed(K)
    big = torch.randn(min(rows, 32), K, device="cuda", generator=g).to(torch.bfloat16)
    q = fp4.quantize_activation(big, "mse", rows=rows)
    for M in (big.shape[0] - 3, 1, big.shape[0]):
        x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
        if M == 1:
            q["A"].random_(0, 256, generator=g)
            q["A_sf"].view(torch.uint8).random_(0, 256, generator=g)
            if q["A_rec"] is not None:
                q["A_rec"].random_(0, 256, generator=g)
        if q["A_rec"] is not None and _lib.load().biloco_b200_act_rec_bytes(M, K) != q["A_rec"].numel():
            q["A_rec"] = None                # (another record form)
        q = fp4.quantize_activation(x, "mse", rows=rows, out=q)
        p, sf, _ = fp4.quantize_nvfp4(x.float(), "mse")
        assert torch.equal(q["A"][0, :M], p) and not bool(q["A"][0, M:].any())
        assert torch.equal(q["A_sf"].view(torch.uint8), sf.view(torch.uint8))
        fresh = fp4.quantize_activation(x, "mse", rows=rows)
        if q["A_rec"] is not None:
            assert torch.equal(q["A_rec"], fresh["A_rec"])


def test_operands_that_start_anywhere():
    """Views that do not start on 16 bytes: a weight given to the quantiser, a prompt's bias and signs."""
    g = torch.Generator(device="cuda").manual_seed(2)
    flat = torch.randn(48 * 64 + 3, device="cuda", generator=g)
    for off in (1, 2, 3):
        W = flat[off:off + 48 * 64].view(48, 64)
        for a, b in zip(fp4.quantize_nvfp4(W, "mse"), fp4.quantize_nvfp4(W.clone(), "mse")):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    K, N, R, rows = 512, 136, 40, 50
    ops = BiLoCoLinear.synthetic(K, N, R, "cuda", seed=4).export_operands()
    ops["bias"] = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    x = torch.randn(rows, K, device="cuda", generator=g).to(torch.bfloat16)
    want = BiLoCoLinear.from_operands(ops)(x)
    odd = dict(ops)
    odd["bias"] = torch.empty(N + 1, device="cuda", dtype=torch.bfloat16)[1:].copy_(ops["bias"])
    odd["V_packed"] = torch.empty(R * K // 8 + 4, device="cuda", dtype=torch.uint8)[4:].view(R, K // 8).copy_(ops["V_packed"])
    layer = BiLoCoLinear.from_operands(odd)
    assert layer.bias.data_ptr() % 16 and layer.V_packed.data_ptr() % 8
    assert torch.equal(layer(x), want)
