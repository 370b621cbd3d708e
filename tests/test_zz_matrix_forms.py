"""The forms of the FP32 matrix products (panels of 16 and of 32 rows, 64 x 64
tiles) through the library's own launch functions: sums that aren't split
(64 doesn't divide K), plain and with either operand folded, with the
butterfly about columns and about rows, float4 and single loads, one and
several steps of K, remainders of every tile.

All forms give the same bits, and each lies within the bound of any FP32 sum
of K products (Higham, Accuracy and Stability, 3.5: gamma_n |A||B| with n = K
roundings; one more for a folded operand, one for a butterfly).
"""
import ctypes

import numpy as np
import pytest
import torch

from eisenjoch_b200 import _abi

pytestmark = pytest.mark.gpu


class Op(ctypes.Structure):  # GemmOp
    _fields_ = [(n, ctypes.c_void_p) for n in ("A", "B", "C", "C2")] + \
               [(n, ctypes.c_int) for n in ("lda", "ldb", "ldc", "a_mir", "a_full", "b_mir", "b_full", "row_par",
                                            "col_split")]


class Fly(ctypes.Structure):  # FlyOp
    _fields_ = [("E", ctypes.c_void_p), ("O", ctypes.c_void_p), ("out", ctypes.c_void_p), ("sig", ctypes.c_float)]


SGEMM = "_ZN6eplace12launch_sgemmEPKNS_6GemmOpEiiiiP11CUstream_stib"
FLY = "_ZN6eplace16launch_sgemm_flyEPKNS_6GemmOpEPKNS_5FlyOpEiiiibP11CUstream_stib"
SHAPES = [(1, 1, 1), (5, 7, 9), (16, 32, 12), (17, 33, 61), (15, 36, 68), (33, 31, 130), (64, 64, 60), (67, 68, 132),
          (100, 100, 100), (131, 129, 269)]


def on_device(structs):
    raw = b"".join(bytes(s) for s in structs)
    return torch.frombuffer(bytearray(raw), dtype=torch.uint8).cuda()


def call(name, *args):
    fn = getattr(_abi.lib(), name)
    fn.restype = ctypes.c_int
    assert fn(*args) == 0
    torch.cuda.synchronize()


def gamma(n):
    u = 2.0 ** -24
    return n * u / (1 - n * u)


def product(A, B):
    a, b = A.double(), B.double()
    return a @ b, a.abs() @ b.abs()


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("fold", ["", "a", "b"])
def test_products(m, n, k, fold):
    if fold and (k % 4 or n % 4):
        pytest.skip("folded products have sides that are multiples of 4")
    g = torch.Generator().manual_seed(m * 10007 + n * 101 + k)
    A = torch.randn(2, m, 2 * k if fold == "a" else k, generator=g).cuda()
    B = torch.randn(2, 2 * k if fold == "b" else k, n, generator=g).cuda()
    want = []
    for b, sig in ((0, 1.0), (1, -1.0)):
        a64, b64 = A[b].double(), B[b].double()
        abs_a, abs_b = a64.abs(), b64.abs()
        if fold == "a":
            a64, abs_a = a64[:, :k] + sig * a64.flip(1)[:, :k], abs_a[:, :k] + abs_a.flip(1)[:, :k]
        if fold == "b":
            b64, abs_b = b64[:k] + sig * b64.flip(0)[:k], abs_b[:k] + abs_b.flip(0)[:k]
        want.append((a64 @ b64, abs_a @ abs_b))
    first = None
    for tile in (64, 32, 16, 0):
        C = torch.full((2, m, n), float("nan"), device="cuda")
        ops = on_device([Op(A[b].data_ptr(), B[b].data_ptr(), C[b].data_ptr(), None, A.shape[2], n, n,
                            sig if fold == "a" else 0, 2 * k if fold == "a" else 0,
                            sig if fold == "b" else 0, 2 * k if fold == "b" else 0, -1, 0)
                         for b, sig in ((0, 1), (1, -1))])
        call(SGEMM, ctypes.c_void_p(ops.data_ptr()), 2, m, n, k, None, tile, ctypes.c_bool(tile != 64))
        for b in range(2):
            ref, mag = want[b]
            assert bool(((C[b].double() - ref).abs() <= gamma(k + 1) * mag).all())
        first = C if first is None else first
        assert torch.equal(C.view(torch.int32), first.view(torch.int32)), tile


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("cols", [False, True])
def test_products_with_butterfly(m, n, k, cols):
    g = torch.Generator().manual_seed(m * 10007 + n * 101 + k + cols)
    A = torch.randn(4, m, k, generator=g).cuda()
    B = torch.randn(4, k, n, generator=g).cuda()
    first = None
    for tile in (64, 32, 16, 0):
        C = torch.zeros((4, m, n), device="cuda")
        out = torch.full((2, m, 2 * n) if cols else (2, 2 * m, n), float("nan"), device="cuda")
        ops = on_device([Op(A[b].data_ptr(), B[b].data_ptr(), C[b].data_ptr(), None, k, n, n, 0, 0, 0, 0, -1, 0)
                         for b in range(4)])
        fly = on_device([Fly(C[2 * b].data_ptr(), C[2 * b + 1].data_ptr(), out[b].data_ptr(), 1.0 - 2.0 * b)
                         for b in range(2)])
        call(FLY, ctypes.c_void_p(ops.data_ptr()), ctypes.c_void_p(fly.data_ptr()), 4, m, n, k, ctypes.c_bool(cols),
             None, tile, ctypes.c_bool(tile != 64))
        for b in range(2):
            e, me = product(A[2 * b], B[2 * b])
            o, mo = product(A[2 * b + 1], B[2 * b + 1])
            back = (1.0 - 2.0 * b) * (e - o)
            ref = torch.cat([e + o, back.flip(1)], 1) if cols else torch.cat([e + o, back.flip(0)], 0)
            mag = torch.cat([me + mo, (me + mo).flip(1)], 1) if cols else torch.cat([me + mo, (me + mo).flip(0)], 0)
            assert bool(((out[b].double() - ref).abs() <= gamma(k + 1) * mag).all())
        first = out if first is None else first
        assert torch.equal(out.view(torch.int32), first.view(torch.int32)), tile
