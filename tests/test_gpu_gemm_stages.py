"""The tcgen05 GEMM's two rings: as many CTAs as SMs (five stages) and more
(three), K from one chunk to more than either ring holds, against FP64
products of the same BF16 operands.

Tolerance: products are exact in FP32, the K sums of them are rounded: 2e-6 of
the largest result times sqrt(K), as for the GEMM's other tests."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import _lib, engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [0, 1, 400])
@pytest.mark.parametrize("N, K", [(256, 64), (256, 72), (256, 256), (70, 333), (64, 1000)])
def test_rings_match_fp64(cuda, more, N, K):
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    cols = (N + 63) // 64
    M = 128 * (sms // cols) + more           # M + 1 rows: one more row of CTAs
    rng = np.random.default_rng(M + K)
    A = torch.tensor(rng.standard_normal((M, K)), dtype=torch.float32).bfloat16()
    W = torch.tensor(rng.standard_normal((N, K)), dtype=torch.float32).bfloat16()
    bias = torch.tensor(rng.standard_normal(N), dtype=torch.float32)
    Ad, Wd, bd = A.to(cuda), W.to(cuda), bias.to(cuda)
    C = torch.full((M, N), float("nan"), dtype=torch.float32, device=cuda)
    L = _lib.load()
    _lib.check(L.mk_gemm_tc(M, N, K, Ad.data_ptr(), K, 1, Wd.data_ptr(), 1, K, C.data_ptr(), N, bd.data_ptr(), 2,
                            None, 0, None, 0, None, None, engine._stream_handle()))
    engine.sync()
    _lib.check(L.mk_sync_status(engine._stream_handle()))
    ref = A.double() @ W.double().T + bias.double()
    assert float((C.cpu().double() - ref).abs().max()) <= 2e-6 * float(ref.abs().max()) * K ** 0.5 + 1e-6
