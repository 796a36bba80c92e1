"""A linear layer over the vector-wise N:M sparse multiply: ``y = x @ W.T + b`` with the
weight pruned to ``n_keep``:32 (per-vector L2 magnitude), compressed and packed on the GPU
once, and every forward one call of the multiply.

The forward is registered with ``torch.library`` as the operator
``nmspmm_b200::sparse_linear`` (with a fake kernel for tracing and an autograd formula), so
the layer can be traced, compiled around and differentiated.  Activations are taken
row-major as they come (``nmspmm_gemm_row_major``: the tensor-core path reads them so, the exact
path transposes on the GPU ahead of the multiply); nothing is padded or transposed in eager
PyTorch.  float16 / bfloat16 activations give a result of the same dtype
(``nmspmm_gemm_row_major_16``: widened exactly, summed in FP32, rounded once at the end); the
compressed weights are FP32.

The backward pass runs on the compressed weight too (``nmspmm_linear_grad``: both gradients in
FP32, n_keep / 32 of the work of the dense products); an unpruned weight (32 of 32), a
backward that is itself to be differentiated and large calls of a program that allows torch TF32
products take torch's own.

The reference has no framework binding (its only caller is its test driver,
tests/test_nmspmm.cu:8-160).
"""
import ctypes
from typing import Optional

_registered = None
_library = None         # the torch.library.Library that holds the operator (it lives as long as this object)
_scratch = None         # the operator's workspaces (pkg.Scratch)


_torch_module = None


def _torch():
    global _torch_module
    if _torch_module is None:
        import torch
        _torch_module = torch
    return _torch_module


def _dense_rows(raw_indices, n_keep: int):
    """(W, N) global k of every compressed value, from the raw window-local indices (W, N/32)."""
    torch = _torch()
    win = torch.arange(raw_indices.shape[0], device=raw_indices.device) // n_keep
    return (raw_indices.to(torch.int64) + (win * 32)[:, None]).repeat_interleave(32, dim=1)


def _dense_tf32_pays(M: int, N: int, K: int, n_keep: int) -> bool:
    """Whether the backward takes torch's dense products: only where the caller has allowed torch TF32
    matrix products, which are 32 / n_keep times the work at some twenty times the FP32 rate, and where
    the call is large enough for the expansion of B to pay.  Both gradients, B200, us: 4096 x 4096 x 4096 at
    4 / 8 / 16:32 815 / 1332 / 2607 by the kernels, 436 / 457 / 509 dense in TF32; 1024 rows 239 / 375 / 730
    against 219 / 222 / 258; 256 rows 91 / 127 / 223 against 128 / 148 / 204; 1024 x 1024 x 1024 at 8:32 56 against 97.
    (Dense in FP32 loses everywhere.)"""
    return (_torch().backends.cuda.matmul.fp32_precision == "tf32"        # whichever of torch's switches set it
            and M * n_keep >= 3000 and M * N * K * n_keep >= 3.4e10)


def _sparse_grads(pkg, x, values, raw_indices, n_keep: int, grad_y, want_x: bool, want_values: bool):
    """(grad_x, grad_values) by nmspmm_linear_grad, None where not wanted."""
    torch = _torch()
    lib = pkg.load_library()
    x, values, grad_y = x.contiguous(), values.contiguous(), grad_y.to(x.dtype).contiguous()
    raw_indices = raw_indices.to(torch.int32).contiguous()                # the kernels read (W, N/32) int32 as it lies
    if grad_y.data_ptr() % 16 != 0:
        grad_y = grad_y.clone()                                           # a view into the middle of a buffer: TMA wants 16 bytes
    dtype = pkg.dtype_id(x.dtype)
    d = pkg.make_desc(x.shape[0], values.shape[1], x.shape[1], n_keep, pkg.FORMAT_LOW, 32)
    grad_x = torch.empty_like(x) if want_x else None
    grad_values = torch.empty_like(values) if want_values else None
    need = int(lib.nmspmm_linear_grad_workspace_bytes(ctypes.byref(d), dtype, int(want_x), int(want_values)))
    ws = torch.empty(need, dtype=torch.uint8, device=x.device)
    ptr = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())  # noqa: E731
    rc = lib.nmspmm_linear_grad(ctypes.byref(d), dtype, ptr(x), ptr(grad_y), ptr(values), ptr(raw_indices), ptr(grad_x), ptr(grad_values),
                                ptr(ws), need, ctypes.c_void_p(torch.cuda.current_stream(x.device).cuda_stream))
    if rc != pkg.OK:
        raise pkg.NMSpMMError("nmspmm_linear_grad", rc)
    return grad_x, grad_values


def register_ops(pkg):
    """Defines ``torch.ops.nmspmm_b200.sparse_linear`` once per process and returns it."""
    global _registered, _scratch
    if _registered is not None:
        return _registered
    torch = _torch()
    scratch = _scratch = pkg.Scratch()

    # Defined through torch.library.Library rather than the custom_op decorator: the decorator's wrapper
    # around the body cost 7 us of host time a call, as much as the multiply of one token.
    global _library
    if torch._C._dispatch_has_kernel("nmspmm_b200::sparse_linear"):
        # Another copy of this package in the process (loaded under a second name) holds the operators: they
        # take everything they need as arguments.
        _registered = torch.ops.nmspmm_b200.sparse_linear.default
        return _registered
    _library = torch.library.Library("nmspmm_b200", "FRAGMENT")
    name = "nmspmm_b200::sparse_linear"
    _library.define("sparse_linear(Tensor x, Tensor values, Tensor packed, Tensor? column_info, Tensor raw_indices, SymInt n_keep, "
                    "SymInt fmt, SymInt layout_ns, SymInt vec_len, SymInt path) -> Tensor", tags=(torch.Tag.pt2_compliant_tag,))

    def sparse_linear(x, values, packed, column_info, raw_indices, n_keep, fmt, layout_ns, vec_len, path):
        """x (M, K) row-major float32 / float16 / bfloat16 . B (K, N) in N:M form -> (M, N) of x's dtype.  ``values`` (W, N) are the
        compressed weights, ``packed`` / ``column_info`` the packed indices the kernels read,
        ``raw_indices`` (W, N/32) the unpacked ones (used by the backward formula only)."""
        lib = pkg.load_library()
        if x.device != values.device:                                     # (a host x beside CUDA weights is dispatched here too)
            raise TypeError(f"x: expected a tensor on {values.device}, got one on {x.device}")
        x = x.contiguous()
        M, K = x.shape
        N = values.shape[1]
        dtype = pkg.dtype_id(x.dtype)
        d = ctypes.byref(pkg.GemmDesc(M, N, K, n_keep, fmt, layout_ns, path, 0, 0, vec_len))
        wide = dtype == pkg.DTYPE_F32
        y = x.new_empty((M, N))
        need = lib.nmspmm_gemm_row_major_call_bytes(d, dtype, x.data_ptr(), y.data_ptr())
        if need == 0:
            raise pkg.NMSpMMError("nmspmm_gemm_row_major_call_bytes", pkg.UNSUPPORTED)
        stream = pkg._raw_stream()
        ws, ws_bytes, _held = scratch.get(need, d, x, stream)
        ptrs = (x.data_ptr(), values.data_ptr(), packed.data_ptr(), None if column_info is None else column_info.data_ptr(),
                y.data_ptr(), ws, ws_bytes, stream)
        if wide:
            rc, where = lib.nmspmm_gemm_row_major(d, *ptrs), "nmspmm_gemm_row_major"
        else:
            rc, where = lib.nmspmm_gemm_row_major_16(d, dtype, *ptrs), "nmspmm_gemm_row_major_16"
        if rc != pkg.OK:
            raise pkg.NMSpMMError(where, rc)
        return y

    _library.impl("sparse_linear", sparse_linear, "CUDA")

    @torch.library.register_fake(name, lib=_library)
    def _(x, values, packed, column_info, raw_indices, n_keep, fmt, layout_ns, vec_len, path):
        return x.new_empty((x.shape[0], values.shape[1]))

    # The backward's kernels behind an operator of their own: whatever traces, batches or compiles a backward pass sees
    # one opaque call with a fake kernel.  A gradient that is not wanted comes back with no elements.
    _library.define("sparse_linear_grad(Tensor x, Tensor values, Tensor raw_indices, Tensor grad_y, SymInt n_keep, bool want_x, "
                    "bool want_values) -> (Tensor, Tensor)", tags=(torch.Tag.pt2_compliant_tag,))

    def sparse_linear_grad(x, values, raw_indices, grad_y, n_keep, want_x, want_values):
        grad_x, grad_values = _sparse_grads(pkg, x, values, raw_indices, n_keep, grad_y, want_x, want_values)
        return x.new_empty(0) if grad_x is None else grad_x, values.new_empty(0) if grad_values is None else grad_values

    _library.impl("sparse_linear_grad", sparse_linear_grad, "CUDA")

    @torch.library.register_fake("nmspmm_b200::sparse_linear_grad", lib=_library)
    def _(x, values, raw_indices, grad_y, n_keep, want_x, want_values):
        return x.new_empty(x.shape if want_x else (0,)), values.new_empty(values.shape if want_values else (0,))

    def setup_context(ctx, inputs, output):
        x, values, _packed, _ci, raw_indices, n_keep = inputs[:6]
        ctx.n_keep = n_keep
        ctx.save_for_backward(x, values, raw_indices)

    def backward(ctx, grad_y):
        x, values, raw_indices = ctx.saved_tensors
        want_x, want_values = ctx.needs_input_grad[0], ctx.needs_input_grad[1]
        # (with create_graph the formula has to be differentiable itself: the dense products below)
        if (ctx.n_keep in (16, 12, 8, 4) and not torch.is_grad_enabled()
                and not _dense_tf32_pays(x.shape[0], values.shape[1], x.shape[1], ctx.n_keep)):
            grad_x, grad_values = torch.ops.nmspmm_b200.sparse_linear_grad(x, values, raw_indices, grad_y, ctx.n_keep, want_x, want_values)
            return (grad_x if want_x else None, grad_values if want_values else None, *[None] * 8)
        rows = _dense_rows(raw_indices, ctx.n_keep)                       # (W, N) global k of every kept value
        grad_x = grad_values = None
        g32 = grad_y.to(torch.float32)
        if want_x:
            dense = torch.zeros((x.shape[1], values.shape[1]), dtype=torch.float32, device=values.device)
            dense.scatter_(0, rows, values)                               # B with explicit zeros, (K, N)
            grad_x = (g32 @ dense.t()).to(x.dtype)
        if want_values:
            grad_values = (x.to(torch.float32).t() @ g32).gather(0, rows)  # d/dB restricted to the kept positions
        return grad_x, grad_values, None, None, None, None, None, None, None, None

    torch.library.register_autograd(name, backward, setup_context=setup_context, lib=_library)
    _registered = torch.ops.nmspmm_b200.sparse_linear.default
    return _registered


class NMSparseLinear:
    """``weight`` is the usual (out_features, in_features) dense float32 CUDA tensor;
    in_features must be a multiple of 32 (64 for the 75 % / 87.5 % formats) and
    out_features a multiple of 128.  ``vec_len`` is the number of adjacent outputs that
    share their kept inputs (32 or 64).  ``values`` (the kept weights, a leaf tensor) and
    ``bias`` may be given ``requires_grad_()``; the sparsity pattern is fixed at construction."""

    def __init__(self, pkg, weight, n_keep: int, bias=None, vec_len: int = 32, path: Optional[int] = None):
        torch = _torch()
        self._pkg = pkg
        self._op = register_ops(pkg)
        self.out_features, self.in_features = weight.shape
        self.n_keep, self.vec_len = n_keep, vec_len
        self.path = pkg.PATH_FP32 if path is None else path
        w = weight.detach()
        if w.dtype in (torch.float16, torch.bfloat16) and w.is_cuda and w.numel() % 4 == 0:
            w = pkg.widen_device(w.contiguous())                          # exact; the compressed weights stay FP32
        dense = w.to(torch.float32).t().contiguous()                      # (K, N) row-major, as the pruning kernel reads it
        BT, self.raw_indices = pkg.prune_device(dense, n_keep, vec_len)   # (W, N) values, (W, N/32) window-local k
        self.op = pkg.NMSpMM(BT, self.raw_indices, self.in_features, n_keep, device=weight.device, vec_len=vec_len)
        self.values = self.op.B                                           # the layer's trainable tensor
        self.bias = None if bias is None else bias.detach().to(torch.float32)

    def __call__(self, x):
        torch = _torch()
        flat = x.dim() == 2 and x.shape[1] == self.in_features
        lead = x.shape[:-1]
        x2 = x if flat else x.reshape(-1, self.in_features)
        if x2.dtype not in (torch.float32, torch.float16, torch.bfloat16):
            x2 = x2.to(torch.float32)
        op = self.op
        args = (x2, self.values, op.D, op.column_info, self.raw_indices, self.n_keep, op.format, op.layout_ns, self.vec_len, self.path)
        if torch.is_grad_enabled() or torch.compiler.is_compiling():
            y = self._op(*args)
        else:
            # Nothing to record: straight to the operator's kernel, past the Python function behind its
            # autograd key, which would call it again just so (4 us).  Everything above that key --
            # tracing, functorch, dispatch modes, tensor subclasses -- still sees the call.
            with torch._C._AutoDispatchBelowAutograd():
                y = self._op(*args)
        if self.bias is not None:
            y = y + self.bias.to(y.dtype)
        return y if flat else y.reshape(*lead, self.out_features)

    def dense_weight(self):
        """The pruned weight as a dense (out_features, in_features) tensor (zeros where pruned),
        rebuilt from the compressed operand: what the layer multiplies by."""
        torch = _torch()
        dense = torch.zeros((self.in_features, self.out_features), dtype=torch.float32, device=self.values.device)
        dense.scatter_(0, _dense_rows(self.raw_indices, self.n_keep), self.values.detach())
        return dense.t().contiguous()
