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


def wide_scales(w, n, k, mixed, seed):
    """Q6_K scales over the whole int8 range: in every superblock, or in some superblocks of some groups of 32 rows (the rows of one warp)."""
    rng = np.random.default_rng(seed)
    w = w.reshape(n, k // 256, 210).copy()
    some = rng.integers(-128, 128, size=(n, k // 256, 16)).astype(np.int8).view(np.uint8)
    pick = np.repeat(rng.random(((n + 31) // 32, k // 256)) < 0.4, 32, axis=0)[:n] if mixed else np.ones((n, k // 256), bool)
    w[:, :, 192:208] = np.where(pick[:, :, None], some, w[:, :, 192:208])
    return w.reshape(-1)


@pytest.mark.parametrize("fmt,scales", [("q4_k", "small"), ("q6_k", "small"), ("q6_k", "whole range"), ("q6_k", "some rows")])
@pytest.mark.parametrize("width,m,n,k,slices", [(32, 17, 40, 256, 0), (32, 33, 300, 1792, 0), (32, 64, 1000, 4864, 0), (32, 64, 200, 2304, 3), (64, 65, 300, 1792, 0), (96, 97, 129, 768, 0),
                                                (128, 129, 19200, 768, 0), (128, 200, 300, 4864, 3)])
def test_gemm_tiles_are_exact_over_the_scales(ck, orc, fmt, scales, width, m, n, k, slices):
    """Products of 6-bit weights and 8-bit scales beyond 2048 do not fit an fp16 operand: they are as exact as the others.  The 32-token form is what prompts and
    batches of up to 64 tokens get where the integer-MMA kernels refuse (here they are switched off)."""
    import torch

    dev = torch.device("cuda", 0)
    w = synth.make_weights(fmt, n, k, seed=m + width)
    if scales != "small":
        w = wide_scales(w, n, k, scales == "some rows", seed=n)
    aq = cases.quantize_act(orc, "oracle_", fmt, synth.make_x(k, seed=n, rows=m), rows=m)
    want = cases.gemm_nt(orc, "oracle_", fmt, aq, w, None, m, n, k)
    raw, taq = torch.from_numpy(w).to(dev), torch.from_numpy(aq).to(dev)
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
        for key, value in ((b"gemm_tc_nt", width if width > 32 else 0), (b"gemm_tc_slices", slices), (b"gemm_q4k_mma", 0), (b"gemm_q6k_mma", 0)):
            ck.ckb200_tune_set(key, value)
        for _ in range(2):
            c = torch.full((m, n), float("nan"), device=dev)
            torch.cuda.synchronize()
            assert fn(C.c_void_p(taq.data_ptr()), C.c_void_p(wdev.data_ptr()), None, C.c_void_p(c.data_ptr()), m, n, k, None) == 0
            assert ck.ckb200_synchronize() == 0
            outs.append(c.cpu().numpy())
    finally:
        for key, value in ((b"gemm_tc_nt", 0), (b"gemm_tc_slices", 0), (b"gemm_q4k_mma", 1), (b"gemm_q6k_mma", 1)):
            ck.ckb200_tune_set(key, value)
    # as above: integer sums are the same on both sides, K / 256 fp32 terms of three roundings each; with fp16-rounded products it would be about 1e-4
    bound = 2 * (k // 256 + 3) * 2.0 ** -24 * 8 * float(np.max(np.abs(want)))
    assert float(np.max(np.abs(outs[0].astype(np.float64) - want))) <= bound
    assert np.array_equal(outs[0], outs[1])
