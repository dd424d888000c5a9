"""BiLoCoLinear backed by the fused kernel: y = (x/s) V diag(alpha) U^T + FP4(x/s) FP4(R)^T + b.

Same constructor, ``quantize`` and ``forward`` signatures as the reference module (``biloco/layer.py:16-64``), but
``quantize`` keeps what the fused kernel streams — packed NVFP4 codes and block scales of the residual, bit-packed
signs, bf16 coefficients — instead of dequantised bf16 copies, and ``forward`` enqueues two launches up to 32 rows (the
NVFP4 activation quantiser with the SmoothQuant division folded in, then the fused linear) and four above (maximum,
quantiser, low-rank coefficients, GEMM), with no host synchronisation. ``forward_fake_quant`` restates the reference's unfused bf16 forward on the same operands with
plain torch ops; the tests use it as the device-side comparator.
"""
import ctypes

import torch
import torch.nn as nn

from . import _lib, fp4
from .peel import decompose

METHODS = ("biloco", "fp4")
MAX_ROWS = 32     # activation rows per fused launch


class _DecodePlan:
    """One layer's decode forward at a fixed number of rows, bound in the library (biloco_b200_layer_plan_run: quantiser and
    fused launch): a call checks what can differ from call to call and hands over three addresses. Keeps the launcher and the
    activation buffers alive; not copied or pickled with the layer (the copy builds its own)."""

    def __init__(self, layer, q, g):
        lib = _lib.load()
        self.keep = (layer.W_codes, layer.W_sf, layer.w_gscale, layer.smooth_scale, layer.V_packed, layer.S, q, g)
        self.g, self.smoothed, self.dev, self.N = g, layer.smoothed, q["A"].get_device(), layer.out_features
        self._padded = 0
        self._gs, self._sm = layer.w_gscale.data_ptr(), layer.smooth_scale.data_ptr()
        self.residual = g.residual if layer.bias is not None else None
        self._c = self.residual.data_ptr() if self.residual is not None else None
        R = layer.rank
        h = ctypes.c_void_p()
        wt = g.W_tiled if g.W_tiled is not None and g.W_tiled.numel() else None
        rec = q.get("A_rec") if g.mode != _lib.MODE_SLAB else None
        with torch.cuda.device(self.dev):
            _lib.check(lib.biloco_b200_layer_plan_create(
                layer.W_codes.data_ptr(), layer.W_sf.data_ptr(), wt.data_ptr() if wt is not None else None, layer.w_gscale.data_ptr(),
                layer.smooth_scale.data_ptr() if self.smoothed else None, q["X"].data_ptr() if self.smoothed else None,
                q["A"].data_ptr(), q["A_sf"].data_ptr(), rec.data_ptr() if rec is not None else None, q["gscale"].data_ptr(),
                q["alpha"].data_ptr(), g.V.data_ptr() if R else None, g.U_col32.data_ptr() if R else None, g.S.data_ptr() if R else None,
                g.z.data_ptr(), g.z.numel() * 4, g.M, g.N, g.K, R, g.mode, ctypes.byref(h)), "layer_plan_create")
        self._h, self._run, self._destroy = h.value, lib.biloco_b200_layer_plan_run, lib.biloco_b200_layer_plan_destroy

    def bound_to(self, layer):
        """Whether the layer's scale and smoothing vector are still where the plan has them (a caller may replace these buffers)."""
        b = layer._buffers
        return self.smoothed is layer._smoothed and b["w_gscale"].data_ptr() == self._gs and b["smooth_scale"].data_ptr() == self._sm

    def __call__(self, x, y, residual=None):
        self.g.epoch += 1
        rc = self._run(self._h, x.data_ptr(), self._c if residual is None else residual.data_ptr(), y.data_ptr(),
                       _lib.RULES[fp4.CONFIG_X] | self._padded, _raw_stream(self.dev))
        self._padded = 0x200           # (BILOCO_RULE_PADDED: the first run has written the buffers' zero padding)
        if rc:
            _lib.check(rc, f"biloco linear (mode {self.g.mode}, M={self.g.M}, N={self.N}, K={self.g.K})")
        return y

    def __del__(self):
        if getattr(self, "_h", None):
            self._destroy(self._h)
            self._h = None

    def __deepcopy__(self, memo):
        return None

    def __reduce__(self):
        return (type(None), ())


def _raw_stream(dev):
    return torch._C._cuda_getCurrentRawStream(dev)


def _aligned(t, n):
    """t, or a copy of it where its memory does not start on n bytes."""
    return t if t.data_ptr() % n == 0 else t.detach().clone()


class BiLoCoLinear(nn.Module):
    def __init__(self, linear: nn.Linear, rank: int, method: str = "biloco", smooth_factor: float = 0.5):
        super().__init__()
        assert method in METHODS, method
        self.in_features, self.out_features = linear.in_features, linear.out_features
        self.method = method
        self.rank = rank if method != "fp4" else 0
        self.smooth_factor = smooth_factor
        dev = linear.weight.device
        K, N, r = self.in_features, self.out_features, self.rank
        # The original weight is consumed by quantize() and then freed.
        self.weight = nn.Parameter(linear.weight.data.to(torch.bfloat16), requires_grad=False)
        self.bias = None if linear.bias is None else nn.Parameter(linear.bias.data.to(torch.bfloat16), requires_grad=False)
        self.register_buffer("smooth_scale", torch.ones(K, device=dev, dtype=torch.bfloat16))
        self.register_buffer("V_packed", torch.zeros(r, K // 8, device=dev, dtype=torch.uint8))
        self.register_buffer("U_packed", torch.zeros(r, N // 8, device=dev, dtype=torch.uint8))
        self.register_buffer("S", torch.zeros(r, device=dev, dtype=torch.bfloat16))
        self.register_buffer("W_codes", torch.zeros(N, K // 2, device=dev, dtype=torch.uint8))
        self.register_buffer("W_sf", torch.zeros(fp4.nvfp4_sf_bytes(N, K), device=dev, dtype=torch.uint8))
        self.register_buffer("w_gscale", torch.ones(1, device=dev, dtype=torch.float32))
        self._smoothed = None        # (decided from smooth_scale on first use, see `smoothed`)
        self._gemms = {}      # decode batch M -> BiLoCoGemm
        self._acts = {}       # (decode batch M, SwiGLU input?) -> reusable activation-quantiser outputs
        self._plans = {}      # decode batch M -> _DecodePlan
        self._ucol = None     # U signs by column, for more than MAX_ROWS rows (built on first use)
        self._status = None   # status words of launches for more than MAX_ROWS rows

    @classmethod
    def synthetic(cls, in_features: int, out_features: int, rank: int, device, seed: int = 0):
        """A quantised layer with random operands (random codes, block scales in [0.25, 2], random signs, coefficients
        ~ N(0, 0.01^2)), in the construction of the reference's timing scripts (scripts/problem.py:7-27): the same
        bytes and arithmetic as a decomposed layer without the decomposition. For throughput measurements."""
        self = cls.__new__(cls)
        nn.Module.__init__(self)
        K, N, r = in_features, out_features, rank
        self.in_features, self.out_features, self.method, self.rank, self.smooth_factor = K, N, "biloco", r, 0.5
        g = torch.Generator(device=device).manual_seed(seed)
        self.weight, self.bias = None, None
        self.register_buffer("smooth_scale", torch.ones(K, device=device, dtype=torch.bfloat16))
        self.register_buffer("V_packed", torch.randint(0, 256, (r, K // 8), device=device, dtype=torch.uint8, generator=g))
        self.register_buffer("U_packed", torch.randint(0, 256, (r, N // 8), device=device, dtype=torch.uint8, generator=g))
        self.register_buffer("S", (torch.randn(r, device=device, generator=g) * 0.01).to(torch.bfloat16))
        self.register_buffer("W_codes", torch.randint(0, 256, (N, K // 2), device=device, dtype=torch.uint8, generator=g))
        sf = (torch.rand(fp4.nvfp4_sf_bytes(N, K), device=device, generator=g) * 1.75 + 0.25).to(torch.float8_e4m3fn)
        self.register_buffer("W_sf", sf.view(torch.uint8))
        self.register_buffer("w_gscale", torch.full((1,), 1e-3, device=device, dtype=torch.float32))
        self._smoothed = False
        self._gemms, self._acts, self._plans, self._ucol, self._status = {}, {}, {}, None, None
        return self

    @classmethod
    def from_operands(cls, ops: dict):
        """A quantised layer around given packed operands (the dict of export_operands, e.g. one rank's shard of a layer
        made by biloco_b200.parallel.shard_column_parallel / shard_row_parallel)."""
        self = cls.__new__(cls)
        nn.Module.__init__(self)
        N, K = ops["W_codes"].shape[0], ops["W_codes"].shape[1] * 2
        self.in_features, self.out_features, self.method, self.smooth_factor = K, N, "biloco", 0.5
        self.rank = ops["V_packed"].shape[0]
        self.weight = None
        self.bias = None if ops.get("bias") is None else nn.Parameter(ops["bias"].to(torch.bfloat16), requires_grad=False)
        for name in ("smooth_scale", "V_packed", "U_packed", "S", "W_codes", "w_gscale"):
            self.register_buffer(name, ops[name].contiguous())
        self.register_buffer("W_sf", ops["W_sf"].view(torch.uint8).contiguous())
        self._smoothed = None
        self._gemms, self._acts, self._plans, self._ucol, self._status = {}, {}, {}, None, None
        return self

    # ------------------------------------------------------------------------------------------------------
    @torch.no_grad()
    def quantize(self, act_col_max: torch.Tensor = None, T: int = 5, device=None):
        """Smooth, split off the binary low-rank component, and pack the residual as NVFP4 (biloco/layer.py:34-52)."""
        from .kernel import pack_signs
        device = device or self.weight.device
        W = self.weight.data.to(device=device, dtype=torch.float32)          # (out, in)
        if act_col_max is not None:
            a = act_col_max.to(device=device, dtype=torch.float32).clamp(min=1e-6)
            w_col_max = W.abs().max(dim=0).values.clamp(min=1e-6)
            s = (a ** self.smooth_factor) / (w_col_max ** (1 - self.smooth_factor))
            self.smooth_scale.copy_(s.to(torch.bfloat16))
            self._smoothed = True
            W = W * s
        if self.rank > 0:
            U, V, alpha, R = decompose(W, r=self.rank, T=T)
            self.V_packed.copy_(pack_signs(V.T.contiguous()))
            self.U_packed.copy_(pack_signs(U.T.contiguous()))
            self.S.copy_(alpha.to(torch.bfloat16))
        else:
            R = W
        codes, sf, gs = fp4.quantize_nvfp4(R.to(torch.bfloat16).float(), fp4.CONFIG_W)
        self.W_codes.copy_(codes)
        self.W_sf.copy_(sf.view(torch.uint8))
        self.w_gscale.copy_(gs)
        self.weight = None
        self._forget()

    def _forget(self):
        """Drop what was derived from the operands or from where they are (launchers with their re-laid copies, quantiser buffers, plans). A
        CUDA graph captured over the layer holds addresses of these and has to be captured again."""
        self._gemms.clear()
        self._acts.clear()
        self._plans.clear()
        self._ucol = None

    @property
    def smoothed(self) -> bool:
        """Whether the activation has to be divided by smooth_scale (any entry different from 1). Derived from the buffer
        itself, once, so that a layer restored with load_state_dict or filled by copying buffers behaves like the one
        that was saved."""
        if self._smoothed is None:
            self._smoothed = bool((self.smooth_scale.float() != 1).any())
        return self._smoothed

    @smoothed.setter
    def smoothed(self, value):
        self._smoothed = None if value is None else bool(value)

    def _load_from_state_dict(self, *args, **kwargs):
        super()._load_from_state_dict(*args, **kwargs)
        self._smoothed = None
        self._forget()

    def _apply(self, fn, *args, **kwargs):
        """(.to, .cuda, ...) Launchers and plans go where an operand has moved; a call that changes nothing leaves them."""
        def where():
            return [(t.data_ptr(), t.dtype) for t in (*self._buffers.values(), *self._parameters.values()) if t is not None]
        before = where()
        super()._apply(fn, *args, **kwargs)
        if where() != before:
            self._forget()
        return self

    def status(self):
        """The first non-zero status words (synchronises; word 0: a device-side wait ran out, the output of that call is not whole) among the
        layer's launches at every row count, or sixteen zeros."""
        words = [g.status() for g in self._gemms.values()] + ([self._status.tolist()] if self._status is not None else [])
        return next((w for w in words if w[0]), [0] * 16)

    def reset_status(self):
        """Clear the status words (and with a launcher's its scratch), after status() reported a wait."""
        for g in self._gemms.values():
            g.reset()
        if self._status is not None:
            self._status.zero_()

    def export_operands(self):
        """What the fused kernel consumes, as a dict of tensors (the packed counterpart of the reference's state dict)."""
        return dict(W_codes=self.W_codes, W_sf=self.W_sf.view(torch.float8_e4m3fn), w_gscale=self.w_gscale,
                    V_packed=self.V_packed, U_packed=self.U_packed, S=self.S, smooth_scale=self.smooth_scale,
                    bias=self.bias)

    # ------------------------------------------------------------------------------------------------------
    def _gemm_for(self, M, alpha):
        from .kernel import BiLoCoGemm, _FP4Only
        g = self._gemms.get(M)
        if g is None:
            if self.rank > 0:
                g = BiLoCoGemm(self.W_codes, self.W_sf.view(torch.float8_e4m3fn), alpha, self.V_packed, self.U_packed, self.S, M=M,
                               back_to_back=False)      # (a quantiser launch sits between the linears)
            else:
                g = _FP4Only(self.W_codes, self.W_sf.view(torch.float8_e4m3fn), alpha, M=M)
            if self.bias is not None:     # added inside the kernel, before its single bf16 rounding
                g.residual = self.bias.detach().to(torch.bfloat16).unsqueeze(0).expand(M, self.out_features).contiguous()
            self._gemms[M] = g
        return g

    def _rows(self, x2, residual=None, swiglu=False):
        M, smoothed, dev = x2.shape[0], self.smoothed, x2.device
        if not swiglu:
            assert x2.is_cuda, "the kernel forward needs CUDA tensors"
            plan = self._plans.get(M)
            if plan is None or plan.dev != x2.get_device() or not plan.bound_to(self):
                q = self._acts.get((M, False))
                if q is None or q["A"].device != dev or (smoothed and q["X"] is None):
                    q = fp4._activation_buffers(M, M, self.in_features, dev, 1)
                    q["X"] = torch.empty((M, self.in_features), device=dev, dtype=torch.bfloat16) if smoothed else None
                    self._acts[(M, False)] = q
                plan = self._plans[M] = _DecodePlan(self, q, self._gemm_for(M, q["alpha"]))
            return plan(x2, torch.empty((M, self.out_features), device=dev, dtype=torch.bfloat16), residual)
        q = fp4.quantize_activation(x2, fp4.CONFIG_X, smooth=self.smooth_scale if smoothed else None,
                                    w_gscale=self.w_gscale, rows=M, out=self._acts.get((M, True)), swiglu=True, _padded=True)
        self._acts[(M, True)] = q
        g = self._gemm_for(M, q["alpha"])
        if self.bias is None:          # (with a bias, residual holds the broadcast bias)
            g.residual = residual
        return g(q["A"], q["A_sf"], q["X"], A_rec=q.get("A_rec")).view(-1, self.out_features)[:M]

    def forward_fused(self, x, residual=None, swiglu=False):
        """The kernel forward for at most 32 rows with the steps either side of the linear folded into its launches
        (not in the reference's interface): ``swiglu`` — x is [M, 2 * in_features] = [gate | up] and the layer's input is
        silu(gate) * up, formed inside the quantiser launch; ``residual`` (bf16 [M, out_features], layers without bias) is
        added inside the fused kernel before its single rounding to bf16."""
        assert self.weight is None and x.dim() == 2 and x.shape[0] <= MAX_ROWS and x.dtype == torch.bfloat16
        assert x.shape[1] == self.in_features * (2 if swiglu else 1)
        assert residual is None or (self.bias is None and residual.dtype == torch.bfloat16 and residual.is_contiguous()
                                    and residual.shape == (x.shape[0], self.out_features))
        return self._rows(x.contiguous(), residual=residual, swiglu=swiglu)

    def forward_quantized(self, q: dict, alpha: torch.Tensor):
        """The fused linear on an activation that has been quantised already (fp4.quantize_activation with this layer's
        rules and smoothing): q["A"], q["A_sf"], q["X"] for M <= 32 rows; alpha fp32 [1] = w_gscale * q["gscale"] on the
        device. Lets several layers that read the same activation (q/k/v, gate/up) share one quantiser launch."""
        M = q["X"].shape[0]
        g = self._gemm_for(M, alpha)
        if g.alpha.data_ptr() != alpha.data_ptr():       # (the launcher keeps the pointer it was built with)
            g.alpha = alpha
        return g(q["A"], q["A_sf"], q["X"], A_rec=q.get("A_rec")).view(-1, self.out_features)[:M]

    def _prompt(self, x2):
        """More rows than a fused launch takes (prefill, evaluation): ONE tensor scale over the whole smoothed activation, as
        the reference quantises it (biloco/fp4.py:3-4, biloco/layer.py:60), and the rows as the MMA's 128-row operand."""
        rows, K, N, R = x2.shape[0], self.in_features, self.out_features, self.rank
        assert x2.is_cuda, "the kernel forward needs CUDA tensors"
        lib = _lib.load()
        smooth = self.smooth_scale if self.smoothed else None
        if R and self._ucol is None:
            from .kernel import pack_u_col32
            self._ucol = pack_u_col32(self.U_packed, N, R)
        if self._status is None or self._status.device != x2.device:
            self._status = torch.zeros(16, device=x2.device, dtype=torch.int32)
        nbytes = lib.biloco_b200_prompt_ws_bytes(rows, N, K, R, 0 if smooth is None else 1)
        if nbytes == 0:
            raise RuntimeError(f"fused linear does not support M={rows} N={N} K={K} R={R}")
        ws = torch.empty(nbytes, device=x2.device, dtype=torch.uint8)
        y = torch.empty((rows, N), device=x2.device, dtype=torch.bfloat16)
        V = _aligned(self.V_packed, 8) if R else None         # (operands that are views into a larger buffer may start anywhere)
        bias = _aligned(self.bias, 16) if self.bias is not None else None
        with torch.cuda.device(x2.device):
            rc = lib.biloco_b200_prompt_linear(
                self.W_codes.data_ptr(), self.W_sf.data_ptr(), self.w_gscale.data_ptr(), x2.data_ptr(),
                smooth.data_ptr() if smooth is not None else None, V.data_ptr() if R else None,
                self._ucol.data_ptr() if R else None, self.S.data_ptr() if R else None,
                bias.data_ptr() if bias is not None else None, y.data_ptr(), ws.data_ptr(), nbytes, self._status.data_ptr(), rows, N, K, R,
                _lib.RULES[fp4.CONFIG_X], torch.cuda.current_stream().cuda_stream)
        _lib.check(rc, f"linear of {rows} rows (N={N}, K={K}, R={R})")
        return y

    def forward(self, x):
        shape = x.shape
        K = self.in_features
        plan = self._plans.get(x.numel() // K)       # (a plan exists only for a quantised layer that has run at this batch)
        if (plan is not None and x.dtype is torch.bfloat16 and shape[-1] == K and plan.dev == x.get_device() and x.is_contiguous()
                and plan.bound_to(self)):
            return plan(x, x.new_empty(shape[:-1] + (self.out_features,)))
        assert self.weight is None, "call quantize() first"
        x2 = x.to(torch.bfloat16).reshape(-1, K).contiguous()
        if x2.shape[0] <= MAX_ROWS:
            y = self._rows(x2)
        else:
            y = self._prompt(x2)
        return y.reshape(*shape[:-1], self.out_features).to(torch.bfloat16)

    # ------------------------------------------------------------------------------------------------------
    @torch.no_grad()
    def forward_fake_quant(self, x):
        """The reference's unfused forward (biloco/layer.py:54-64) on this module's operands, plain torch ops."""
        from .kernel import unpack_signs
        x_s = x.to(torch.bfloat16) / self.smooth_scale
        y = torch.zeros((*x_s.shape[:-1], self.out_features), dtype=torch.bfloat16, device=x_s.device)
        if self.rank > 0:
            V_scaled = (unpack_signs(self.V_packed) * self.S.float().unsqueeze(1)).to(torch.bfloat16)    # [r, K]
            U_T = unpack_signs(self.U_packed).to(torch.bfloat16)                                          # [r, N]
            y = y + (x_s @ V_scaled.T) @ U_T
        x_fq = fp4.fake_quantize_fp4(x_s.reshape(-1, self.in_features), fp4.CONFIG_X).reshape(x_s.shape)
        weight_fp4 = fp4.dequantize_nvfp4(self.W_codes, self.W_sf.view(torch.float8_e4m3fn), self.w_gscale).to(torch.bfloat16)
        y = y + x_fq @ weight_fp4.T
        if self.bias is not None:
            y = y + self.bias
        return y.to(torch.bfloat16)

    def extra_repr(self):
        return f"in={self.in_features}, out={self.out_features}, method={self.method}, rank={self.rank}"
