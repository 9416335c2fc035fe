"""Symmetric int4 with bf16 activations and scales above the decode sizes: one fp16 tile per k-block, which holds every
weight exactly.  Against the oracle and against fp64, no further off than the two bf16 tiles it replaces (variant 8)."""
import numpy as np
import pytest
import torch

from oracle import check as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,g,spread", [
    (33, 1024, 512, 128, 0),      # smallest on this route
    (65, 200, 1024, 64, 0),       # ragged rows, weight tiles in tensor memory
    (200, 384, 4096, 128, 0),     # K split: planes before the activations' copy
    (257, 130, 640, 128, 0),      # CTA pairs, two accumulators
    (512, 384, 1024, 64, 12),     # scales of a row 2^12 apart, tokens 2^40 apart
    (1100, 256, 512, 256, 12),    # three token tiles
])
def test_exact_half_tiles(M, N, K, g, spread):
    import metal_native
    import mnq_workloads as workloads
    C = metal_native._C
    L = workloads.make_layer("t", M, K, N, quant_type="int4", group_size=g, act_dtype=torch.bfloat16, scale_dtype=torch.bfloat16,
                             asymmetric=False, seed=M + N + K)
    if spread:
        L.scales *= torch.logspace(-spread, 0, L.scales.shape[1], base=2.0).to(torch.bfloat16)[None, :]
        L.x *= torch.logspace(-20, 20, M, base=2.0).to(torch.bfloat16)[:, None]
    d = L.to("cuda")
    out = C.dequant_matmul(*d.args())
    out32 = C.dequant_matmul_fused(*d.args(), out_dtype=torch.float32)
    t = C.Tuning()
    t.path, t.gemv_variant = C.PATH_GEMM, 8
    two = C.dequant_matmul(*d.args(), tuning=t)
    C.synchronize()
    assert C.device_status() == 0
    W = metal_native.dequantize(d.wq, d.scales, None, g, "int4", torch.float32).double()
    ref = d.x.double() @ W.t()
    # row by row (tokens differ by many orders of magnitude): fp32 sums are good to a few 2^-24 of the terms' norm
    err32 = (out32.double() - ref).norm(dim=1) / ref.norm(dim=1)
    assert float(err32.max()) < 2e-6, float(err32.max())
    err, err2 = ((y.double() - ref).norm(dim=1) / ref.norm(dim=1) for y in (out, two))
    assert float((err - err2).max()) < 2e-5, "further off than two bf16 tiles"
    assert torch.equal(out, out32.to(torch.bfloat16))


@pytest.mark.parametrize("x_exp,s_exp", [(120, -20), (-120, 20), (-128, 100), (30, -110), (-110, 118)])
def test_the_ends_of_bf16s_range(x_exp, s_exp):
    """Activations and scales near bf16's largest and smallest values (2^-128: subnormal): the powers of two that bring them into fp16 reach."""
    import metal_native
    import mnq_workloads as workloads
    C = metal_native._C
    L = workloads.make_layer("t", 72, 512, 256, quant_type="int4", group_size=128, act_dtype=torch.bfloat16,
                             scale_dtype=torch.bfloat16, asymmetric=False, seed=9)
    L.x = (L.x.double() * 2.0 ** x_exp).to(torch.bfloat16)
    L.scales = (L.scales.double() * 2.0 ** s_exp).to(torch.bfloat16)
    d = L.to("cuda")
    out32 = C.dequant_matmul_fused(*d.args(), out_dtype=torch.float32)
    W = metal_native.dequantize(d.wq, d.scales, None, 128, "int4", torch.float32).double()
    ref = d.x.double() @ W.t()
    assert bool(torch.isfinite(out32).all())
    assert float((out32.double() - ref).norm() / ref.norm()) < 2e-6


def test_little_workspace_takes_the_two_tiles():
    """A caller that brings what mnq_workspace_bytes names gets the kernel that needs no more."""
    import metal_native
    import mnq_workloads as workloads
    C = metal_native._C
    d = workloads.make_layer("t", 128, 1024, 512, quant_type="int4", group_size=128, act_dtype=torch.bfloat16,
                             scale_dtype=torch.bfloat16, asymmetric=False, seed=1).to("cuda")
    need = C._lib.mnq_workspace_bytes(128, 512, 1024, 128, C.INT4)
    assert C._lib.mnq_workspace_bytes_for(128, 512, 1024, 128, C.INT4, 1, 1, 0) > need
    ws = torch.zeros(max(need, 1), dtype=torch.uint8, device="cuda")
    out = torch.empty((128, 512), dtype=torch.bfloat16, device="cuda")
    rc = C._lib.mnq_dequant_matmul(d.x.data_ptr(), d.wq.data_ptr(), d.scales.data_ptr(), None, out.data_ptr(), 128, 512, 1024,
                                   1024, 512, 128, C.INT4, 1, 1, ws.data_ptr() if need else None, need,
                                   torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    t = C.Tuning()
    t.path, t.gemv_variant = C.PATH_GEMM, 8
    assert torch.equal(out, C.dequant_matmul(*d.args(), tuning=t))
