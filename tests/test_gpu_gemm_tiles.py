"""The tcgen05 product of quantised weights at every token-tile width: ragged rows and tokens, one superblock, odd superblock counts (the rings of a
persistent CTA go on from one unit to the next), and more units than SMs."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu
synth = cases.synth


@pytest.mark.parametrize("fmt", ["q4_k", "q6_k"])
@pytest.mark.parametrize("width", [64, 96, 128])
@pytest.mark.parametrize("m,n,k", [(65, 40, 256), (97, 129, 768), (129, 19200, 256), (200, 3000, 1792)], ids=["one-block", "odd-blocks", "many-units", "ragged"])
def test_gemm_tile_widths(ck, orc, fmt, width, m, n, k):
    import torch

    dev = torch.device("cuda", 0)
    w = synth.make_weights(fmt, n, k, seed=m + width)
    aq = cases.quantize_act(orc, "oracle_", fmt, synth.make_x(k, seed=n, rows=m), rows=m)
    bias = np.random.default_rng(k).standard_normal(n).astype(np.float32)
    want = cases.gemm_nt(orc, "oracle_", fmt, aq, w, bias, m, n, k)
    raw, taq, tb = torch.from_numpy(w).to(dev), torch.from_numpy(aq).to(dev), torch.from_numpy(bias).to(dev)
    if fmt == "q6_k":
        ck.ckb200_q6_k_planar_bytes.restype = C.c_size_t
        wdev = torch.empty(ck.ckb200_q6_k_planar_bytes(n, k), dtype=torch.uint8, device=dev)
        torch.cuda.synchronize()
        assert ck.ckb200_dev_q6_k_to_planar(C.c_void_p(wdev.data_ptr()), C.c_void_p(raw.data_ptr()), n, k, None) == 0
        fn = ck.ckb200_dev_gemm_nt_q6_k_planar_q8_k
    else:
        wdev, fn = raw, ck.ckb200_dev_gemm_nt_q4_k_q8_k
    outs = []
    try:
        ck.ckb200_tune_set(b"gemm_tc_nt", width)
        for _ in range(2):
            c = torch.full((m, n), float("nan"), device=dev)
            torch.cuda.synchronize()
            assert fn(C.c_void_p(taq.data_ptr()), C.c_void_p(wdev.data_ptr()), C.c_void_p(tb.data_ptr()), C.c_void_p(c.data_ptr()), m, n, k, None) == 0
            assert ck.ckb200_synchronize() == 0
            outs.append(c.cpu().numpy())
    finally:
        ck.ckb200_tune_set(b"gemm_tc_nt", 0)
    # the integer stage is exact on both sides; each adds K / 256 fp32 terms of three roundings, and no partial sum is larger than a few times
    # the largest result (positive and negative terms of a row cancel by less than a factor of 8 with these weights)
    bound = 2 * (k // 256 + 3) * 2.0 ** -24 * 8 * float(np.max(np.abs(want)))
    assert float(np.max(np.abs(outs[0].astype(np.float64) - want))) <= bound
    assert np.array_equal(outs[0], outs[1])
