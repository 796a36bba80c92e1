"""The work whose speed this repository is measured on: the calls a user of the vector-wise
N:M sparse multiply makes, over the sizes they are made at.

Sizes are those of the repository's own configurations (the 4096-cubed square, the
16 / 64 / 256 x 11008 x 4096 linear layer, 128 x 1024 x 131072 deep K, 8192 x 28672 x 8192 with
64-wide vectors) and of the layer shapes of its benchmark sweep.  A case is a dict:

    kind     "matmul"   NMSpMM.matmul: col-major A, float32 result
             "rows"     NMSpMM.matmul_rows: row-major A of any row count
             "linear"   NMSparseLinear forward, as in inference
             "train"    NMSparseLinear forward and backward, gradients of input and kept weights
             "weights"  NMSpMM.from_dense: prune, compress and pack a dense weight
             "host"     gemm_host: every operand and the result in pinned host memory
    path     "fp32" (exact) or "tf32" (tensor cores)
    M, N, K, n_keep (kept rows per 32), vec_len (columns per index list), dtype (activations)
"""
import torch

from __graft_entry__ import load_package

_DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _case(kind, path, M, N, K, n_keep, vec_len=32, dtype="f32"):
    return {"kind": kind, "path": path, "M": M, "N": N, "K": K, "n_keep": n_keep, "vec_len": vec_len, "dtype": dtype}


def listed():
    cases = {
        # one token through one attention projection of a half-precision model: the smallest call, all latency
        "decode_1_bf16": _case("linear", "tf32", 1, 4096, 4096, 8, dtype="bf16"),
        # a small decode batch through the up projection of a 7B layer: streaming the weights once
        "decode_16_tf32": _case("matmul", "tf32", 16, 11008, 4096, 8),
        # a larger decode batch on the exact path
        "batch_64_fp32": _case("matmul", "fp32", 64, 11008, 4096, 8),
        # a short prompt through the same layer in a half-precision model
        "prefill_256_bf16": _case("linear", "tf32", 256, 11008, 4096, 8, dtype="bf16"),
        # a batch whose sizes fit no tile: odd row count, ragged columns, K of an odd number of windows
        "ragged_777_fp32": _case("rows", "fp32", 777, 5760, 2080, 12),
        # the headline: the exact square multiply at 75 %
        "square_fp32": _case("matmul", "fp32", 4096, 4096, 4096, 8),
        # the same size on the tensor cores, at the mildest pruning
        "square_tf32_half": _case("matmul", "tf32", 4096, 4096, 4096, 16),
        # contraction far longer than the output is large, at the hardest pruning
        "deep_k_fp32": _case("matmul", "fp32", 128, 1024, 131072, 4),
        # the largest layer, 64-wide vectors
        "large_tf32": _case("matmul", "tf32", 8192, 28672, 8192, 8, vec_len=64),
        # fine-tuning the kept weights of a layer: forward, input gradient, weight gradient
        "train_2048_fp32": _case("train", "fp32", 2048, 4096, 4096, 8),
        # turning a trained dense weight into the packed operand
        "weights_eighth": _case("weights", "fp32", 1, 11008, 4096, 4),
        # the drop-in use: host buffers in, host buffer out
        "host_square_fp32": _case("host", "fp32", 4096, 4096, 4096, 8),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log_uniform(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def _flops(c):
    return 2.0 * c["M"] * c["N"] * (c["K"] // 32 * c["n_keep"])


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "matmul", "rows", "rows", "linear", "linear", "train", "weights", "host"])
    while True:
        path = "fp32" if kind in ("train", "weights", "host") else rng.choice(["fp32", "tf32"])
        n_keep = rng.choice([4, 8, 8, 12, 16])
        vec_len = rng.choice([32, 32, 64])
        dtype = rng.choice(["bf16", "f16", "f32"]) if kind in ("rows", "linear") else "f32"
        M = _log_uniform(rng, 1, 8192)
        N = max(1, _log_uniform(rng, 512, 28672) // 128) * 128
        K = max(8, _log_uniform(rng, 512, 22016) // 64) * 64
        if kind == "matmul" and rng.random() < 0.2:                       # deep K over few columns
            M, N, K = min(M, 256), min(N, 2048), _log_uniform(rng, 16384, 131072) // 64 * 64
        if kind in ("matmul", "host"):
            M = (M + 3) // 4 * 4                                          # a col-major A starts every k row on 16 bytes
        if kind == "rows" and n_keep >= 12 and rng.random() < 0.5:
            K += 32                                                       # an odd number of windows
        if kind == "weights":
            M = 1
        if kind in ("train", "host"):
            M = max(M, 64)
        c = _case(kind, path, M, N, K, n_keep, vec_len, dtype)
        # no more work than the largest listed case's time allows
        limit = {"matmul": 1.2e11, "rows": 1.2e11, "linear": 1.2e11, "train": 1.7e10, "weights": 1e18, "host": 3.5e10}[kind]
        if path == "tf32":
            limit = 6e11
        if _flops(c) <= limit and (kind != "weights" or K * N <= 8192 * 16384):
            return c


def _random_operand(pkg, c, gen):
    """Uniform kept values, random ascending indices per window and vector: the synthetic operand of the square workloads."""
    windows, vectors = c["K"] // 32, c["N"] // c["vec_len"]
    order = torch.rand((windows, 32, vectors), device="cuda", generator=gen).argsort(dim=1)[:, :c["n_keep"]]
    local = order.sort(dim=1).values.to(torch.int32).reshape(windows * c["n_keep"], vectors)
    index = local.repeat_interleave(c["vec_len"] // 32, dim=1).contiguous()
    values = torch.rand((windows * c["n_keep"], c["N"]), device="cuda", generator=gen) * 2 - 1
    return values, index


def prepare(case, seed):
    pkg = load_package()
    c = case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    path = pkg.PATH_TF32 if c["path"] == "tf32" else pkg.PATH_FP32
    state = {"pkg": pkg, "case": c, "path": path}
    M, N, K, n_keep, vec_len, dtype = c["M"], c["N"], c["K"], c["n_keep"], c["vec_len"], _DTYPES[c["dtype"]]
    kind = c["kind"]
    if kind == "matmul":
        values, index = _random_operand(pkg, c, gen)
        state["op"] = pkg.NMSpMM(values, index, K, n_keep, vec_len=vec_len)
        state["A"] = torch.rand((K, M), device="cuda", generator=gen) * 2 - 1
    elif kind == "host":
        values, index = _random_operand(pkg, c, gen)
        A = torch.rand((K, M), device="cuda", generator=gen) * 2 - 1
        state["desc"] = pkg.make_desc(M, N, K, n_keep, pkg.format_of(n_keep), 128, path, vec_len=vec_len)
        state["host"] = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in (A, values, index)]
        state["out"] = torch.zeros((M, N), pin_memory=True)
    elif kind == "weights":
        state["dense"] = torch.randn((K, N), device="cuda", generator=gen) * 0.02
    else:
        weight = torch.randn((N, K), device="cuda", generator=gen) * 0.02
        x = torch.randn((M, K), device="cuda", generator=gen).to(dtype)
        if kind == "rows":
            state["op"] = pkg.NMSpMM.from_dense(weight.t().contiguous(), n_keep, vec_len)
        else:
            state["layer"] = pkg.linear.NMSparseLinear(pkg, weight.to(dtype), n_keep, vec_len=vec_len, path=path)
        if kind == "train":
            state["layer"].values.requires_grad_(True)
            x.requires_grad_(True)
            state["grad_y"] = torch.randn((M, N), device="cuda", generator=gen)
        state["x"] = x
    return state


def run(state):
    c, pkg = state["case"], state["pkg"]
    kind = c["kind"]
    if kind == "matmul":
        return state["op"].matmul(state["A"], path=state["path"])
    if kind == "rows":
        return state["op"].matmul_rows(state["x"], path=state["path"])
    if kind == "linear":
        with torch.no_grad():
            return state["layer"](state["x"])
    if kind == "train":
        y = state["layer"](state["x"])
        grad_x, grad_values = torch.autograd.grad(y, (state["x"], state["layer"].values), state["grad_y"])
        return y.detach(), grad_x, grad_values
    if kind == "weights":
        op = pkg.NMSpMM.from_dense(state["dense"], c["n_keep"], c["vec_len"])
        packed = [op.B, op.D]
        if op.column_info is not None:
            packed.append(op.column_info)
        return packed
    pkg.gemm_host(state["desc"], *state["host"], state["out"], on_current_stream=True)
    return state["out"]


def work(case):
    c = case
    M, N, K, W = c["M"], c["N"], c["K"], c["K"] // 32 * c["n_keep"]
    index = 4 * W * (N // c["vec_len"])
    width = 2 if c["dtype"] != "f32" else 4
    if c["kind"] == "weights":
        lists = 4 * (N // 128) * (K // 64) * 64 if c["n_keep"] in (4, 8) else 0
        return {"bytes": 4 * K * N + 4 * W * N + 4 * W * (N // 32) + lists, "flops": 2 * K * N}
    if c["kind"] == "train":
        # forward: x, values, indices in, y out; backward: grad_y in, both gradients out
        return {"bytes": 4 * (2 * M * K + 2 * W * N + 2 * M * N) + index, "flops": int(3 * _flops(c))}
    return {"bytes": width * (M * K + M * N) + 4 * W * N + index, "flops": int(_flops(c))}


def tolerance(case):
    if case["kind"] == "weights":
        return "exact"                    # kept values, ranks and column lists are selected, not computed
    if case["dtype"] == "bf16":
        return {"rel": 7e-3}              # one rounding of the result to 8 bits (1.7e-3 seen), TF32 operands where asked for
    if case["path"] == "tf32":
        return {"rel": 2e-3}              # operands cut to 10 mantissa bits: 7e-4 seen against a 64-bit product
    if case["dtype"] == "f16":
        return {"rel": 1e-3}              # one rounding of the result to 11 bits (2e-4 seen)
    return {"rel": 1e-5}                  # 32-bit sums: up to 2.4e-6 seen against a 64-bit product (K = 131072)
