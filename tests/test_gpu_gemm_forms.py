"""Tensor-core products of all tile widths and operand orders: the TMA form (base
and rows 16-byte aligned) and the copying form against float64 and against each other,
and the layer entry points with their epilogues against product + element-wise
kernels."""
import ctypes as C

import numpy as np
import pytest
import torch

from espec_b200 import _native as N

pytestmark = pytest.mark.gpu
DEV = "cuda"


def status():
    v = C.c_int(-1)
    N.check(N.load().espec_gemm_bf16_status(C.byref(v)), "espec_gemm_bf16_status")
    return v.value


def operand(rows, cols, pad, shift, gen):
    """bf16 [rows, cols], rows cols + pad apart, first element `shift` into its buffer."""
    flat = torch.zeros(rows * (cols + pad) + shift, dtype=torch.bfloat16, device=DEV)
    x = flat[shift:].view(rows, cols + pad)[:, :cols]
    x.copy_(torch.randn((rows, cols), generator=gen, device=DEV))
    return x


def gemm(a, b, ta, tb, m, n, k):
    c = torch.full((m, n), 7.0, device=DEV)
    N.check(N.load().espec_gemm_bf16(m, n, k, 1.0, a.data_ptr(), a.stride(0), ta, b.data_ptr(),
                                     b.stride(0), tb, 0.0, c.data_ptr(), n,
                                     torch.cuda.current_stream().cuda_stream), "espec_gemm_bf16")
    return c


@pytest.mark.parametrize("m,n,k", [(1, 1, 264), (128, 32, 257), (67, 130, 320), (256, 256, 4096),
                                   (300, 33, 1000), (129, 31, 576), (32, 256, 1024), (5, 8, 1), (130, 70, 64), (1024, 1210, 100),
                                   (1100, 2400, 328), (1270, 3840, 72)])
def test_products(m, n, k):
    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    pad = -k % 8
    a, b = operand(m, k, pad, 0, gen), operand(n, k, pad, 0, gen)
    ref = a.double() @ b.double().T
    # FP32 accumulation of k products: 2^-22 sqrt(k) of the sum of magnitudes
    bound = (a.double().abs() @ b.double().abs().T) * 2.0 ** -22 * k ** 0.5 + 1e-7
    out = gemm(a, b, 0, 1, m, n, k)
    assert status() == 0 and bool(((out.double() - ref).abs() <= bound).all())
    # an operand off its alignment: the copying form; the sums and their order are the same
    a1, b1 = operand(m, k, 3, 1, gen), operand(n, k, 5, 0, gen)
    a1.copy_(a), b1.copy_(b)
    assert torch.equal(gemm(a1, b1, 0, 1, m, n, k), out)
    at, bt = operand(k, m, -m % 8, 0, gen), operand(k, n, -n % 8, 0, gen)
    at.copy_(a.T), bt.copy_(b.T)
    for got in (gemm(at, b, 1, 1, m, n, k), gemm(a, bt, 0, 0, m, n, k), gemm(at, bt, 1, 0, m, n, k)):
        assert torch.equal(got, out)
    assert status() == 0


@pytest.mark.parametrize("rows,fin,fout", [(256, 256, 4096), (33, 5, 256), (130, 264, 1000),
                                           (512, 256, 320), (100, 60, 257)])
def test_layer_epilogues(rows, fin, fout):
    lib, st = N.load(), torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device=DEV).manual_seed(rows + fin + fout)
    x, w = operand(rows, fin, 0, 0, gen), operand(fin, fout, 0, 0, gen)
    bias = torch.randn(fout, generator=gen, device=DEV)
    new = lambda r, c, t=torch.float32: torch.zeros((r, c), dtype=t, device=DEV)
    for act in (0, 1):
        z, h, h2 = new(rows, fout), new(rows, fout, torch.bfloat16), new(rows, fout, torch.bfloat16)
        N.check(lib.espec_mlp_layer(rows, fin, fout, x.data_ptr(), w.data_ptr(), bias.data_ptr(),
                                    act, z.data_ptr(), h.data_ptr(), st), "espec_mlp_layer")
        z2 = gemm(x, w, 0, 0, rows, fout, fin)
        N.check(lib.espec_mlp_bias_gelu(z2.data_ptr(), bias.data_ptr(), rows, fout, act,
                                        h2.data_ptr(), st), "espec_mlp_bias_gelu")
        assert torch.equal(z, z2) and torch.equal(h, h2)
    dz, zin = operand(rows, fout, 0, 0, gen), torch.randn((rows, fin), generator=gen, device=DEV)
    d, db = new(rows, fin), new(rows, fin, torch.bfloat16)
    N.check(lib.espec_mlp_layer_back(rows, fin, fout, dz.data_ptr(), w.data_ptr(), zin.data_ptr(),
                                     d.data_ptr(), db.data_ptr(), st), "espec_mlp_layer_back")
    d2, db2 = gemm(dz, w, 0, 1, rows, fin, fout), new(rows, fin, torch.bfloat16)
    N.check(lib.espec_mlp_gelu_back(d2.data_ptr(), zin.data_ptr(), rows * fin, db2.data_ptr(), st),
            "espec_mlp_gelu_back")
    assert torch.equal(d, d2) and torch.equal(db, db2)
    assert status() == 0
