"""Tensor-core GEMM of the learned warm start (pot3d_tc_gemm, tcgen05 BF16).

tc_gemm(A, B) returns A @ B^T for BF16 CUDA tensors shaped [batch, M, K] and
[batch, N, K] (or without the batch axis), accumulating in FP32 on the
tensor cores.  K must be a multiple of 64 and N a multiple of 16.
"""
from __future__ import annotations

import ctypes as C

from . import _lib

_err = {}
# Kernels of the learned path launched so far (GEMMs here, the element-wise
# kernels of fno.py and warmstart.py count themselves).
LAUNCHES = [0]


def _fn():
    L = _lib.lib()
    f = L.pot3d_tc_gemm_ex
    if not getattr(f, "_typed", False):
        f.argtypes = [C.c_void_p] * 4 + [C.c_int] * 4 + [C.c_longlong, C.c_longlong] + [C.c_int] * 4 + [C.c_void_p] * 3
        f.restype = C.c_int
        f._typed = True
    return f


def _err_flag(device):
    """The error flag of a device (a torch.device or its name; without an
    index, the current one): one int32 that a timed-out wait sets."""
    import torch
    i = device.index if isinstance(device, torch.device) else torch.device(device).index
    if i is None:
        i = torch.cuda.current_device()
    flag = _err.get(i)
    if flag is None:
        flag = _err.setdefault(i, torch.zeros(1, dtype=torch.int32, device=torch.device("cuda", i)))
    return flag


def raw_stream(device_index):
    """Current stream of a device as a number: a call of the learned path is
    some fifty launches, and building torch's stream object for each made the
    host the bound of a guess (1.06 -> 0.91 ms at 255x361x721)."""
    import torch
    raw = getattr(torch._C, "_cuda_getCurrentRawStream", None)  # not a public name
    return raw(device_index) if raw else torch.cuda.current_stream(device_index).cuda_stream


def k_splits(batch, M, N, K):
    """Blocks that share the K of one output tile: a product with fewer tiles
    than half the SMs and a K of 64 or more steps, and of two or more a tile
    (the partial sums cost a pass over all tiles: 74 tiles of 64 steps 72 us
    split and 62 whole, of 256 steps 143 and 160), is split so that about two
    blocks an SM have work, each with at least 8 steps."""
    tile_n = 32 if N <= 32 else 64 if N <= 64 else 128
    tiles = batch * -(-M // 128) * -(-N // tile_n)
    steps = K // 64
    return max(1, min(steps // 8, -(-296 // tiles))) if tiles <= 74 and steps >= max(64, 2 * tiles) else 1


def tc_gemm(A, B, bias=None, out=None, out_dtype=None, ldd=None, accumulate=False, n=None, act=None):
    """out[b, m, :n] (+)= A[b] @ B[b]^T (+ bias).  `out` may be wider than N
    (row stride ldd, e.g. a zero-padded channel buffer).  act "gelu" applies
    the activation to the result."""
    import torch
    if act not in (None, "gelu"):
        raise ValueError(f"tc_gemm: unknown activation {act!r}")
    squeeze = A.dim() == 2
    assert A.dtype == torch.bfloat16 and B.dtype == torch.bfloat16 and A.is_cuda and B.is_cuda
    assert A.is_contiguous() and B.is_contiguous()
    if squeeze:
        bsz = bb = 1
        (M, K), (N, K2) = A.shape, B.shape
    else:
        (bsz, M, K), (bb, N, K2) = A.shape, B.shape
    assert bb == bsz and K2 == K
    device = A.device
    if out is None:
        out = (torch.zeros if accumulate else torch.empty)((M, N) if squeeze else (bsz, M, N),
                                                           dtype=out_dtype or torch.float32, device=device)
    lead = out.shape[:1] if squeeze else out.shape[:2]
    assert out.is_contiguous() and lead == ((M,) if squeeze else (bsz, M))
    ldd = out.shape[-1] if ldd is None else ldd
    assert ldd >= N and out.shape[-1] == ldd
    bf16 = out.dtype == torch.bfloat16
    splits = k_splits(bsz, M, N, K) if out.dtype == torch.float32 else 1
    ws = torch.empty(splits * bsz * M * N, dtype=torch.float32, device=device) if splits > 1 else None
    rc = _fn()(A.data_ptr(), B.data_ptr(), out.data_ptr(), bias.data_ptr() if bias is not None else None, bsz, M, N, K,
               ldd, M * ldd, 1 if accumulate else 0, 1 if bf16 else 0, 1 if act == "gelu" else 0, splits,
               ws.data_ptr() if ws is not None else None, _err_flag(device).data_ptr(), raw_stream(device.index))
    _lib.check(rc)
    LAUNCHES[0] += 2 if splits > 1 else 1
    return out


def check_errors(device="cuda"):
    """Raise if a tensor-core GEMM reported a timed-out wait."""
    e = _err_flag(device)
    if int(e.item()) != 0:
        raise RuntimeError("pot3d_tc_gemm: a bounded wait ran out on the device")


# Shapes of the learned operator's GEMMs at 255x361x721 (359 x 719 theta-phi
# positions) and a square reference shape.
BENCH_SHAPES = ((258121, 32, 64, "lift and pointwise layers"), (258121, 128, 64, "first projection"),
                (258121, 128, 128, "radial projection (128 channels)"), (8192, 8192, 8192, "square"))


def main(argv=None):
    """Throughput of tc_gemm (CUDA events, 3 warm-up and 20 timed launches)
    at the operator's shapes, beside torch.matmul on the same operands; with
    --one, a single 8192^3 product after warm-up (for a profiler)."""
    import argparse
    import json

    import torch
    ap = argparse.ArgumentParser()
    ap.add_argument("--one", action="store_true")
    args = ap.parse_args(argv)
    if args.one:
        A = torch.randn(8192, 8192, device="cuda").bfloat16()
        B = torch.randn(8192, 8192, device="cuda").bfloat16()
        out = torch.empty(8192, 8192, device="cuda", dtype=torch.float32)
        for _ in range(3):
            tc_gemm(A, B, out=out)
        torch.cuda.synchronize()
        check_errors()
        return 0

    def timed(fn, reps=20):
        for _ in range(3):
            fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / reps

    for M, N, K, name in BENCH_SHAPES:
        A = torch.randn(M, K, device="cuda").bfloat16()
        B = torch.randn(N, K, device="cuda").bfloat16()
        out = torch.empty(M, N, device="cuda", dtype=torch.float32)
        ms = timed(lambda: tc_gemm(A, B, out=out))
        ref = timed(lambda: torch.matmul(A, B.T))
        check_errors()
        flops, nbytes = 2.0 * M * N * K, 2.0 * (M * K + N * K) + 4.0 * M * N
        print(json.dumps(dict(shape=[M, N, K], name=name, ms=ms, tflops=flops / ms / 1e9, gbs=nbytes / ms / 1e6,
                              torch_ms=ref, torch_tflops=flops / ref / 1e9)), flush=True)
    return 0


if __name__ == "__main__":
    raise SystemExit(main())
