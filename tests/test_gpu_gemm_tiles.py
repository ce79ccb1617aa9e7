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
    """Products of 6-bit weights and 8-bit scales beyond 2048 do not fit an fp16 operand: they are as exact as the others."""
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
        for key, value in ((b"gemm_tc_nt", width if width > 32 else 0), (b"gemm_tc_small_max", 64 if width == 32 else 32), (b"gemm_tc_slices", slices), (b"gemm_q4k_mma", 0),
                           (b"gemm_q6k_mma", 0)):
            ck.ckb200_tune_set(key, value)
        for _ in range(2):
            c = torch.full((m, n), float("nan"), device=dev)
            torch.cuda.synchronize()
            assert fn(C.c_void_p(taq.data_ptr()), C.c_void_p(wdev.data_ptr()), None, C.c_void_p(c.data_ptr()), m, n, k, None) == 0
            assert ck.ckb200_synchronize() == 0
            outs.append(c.cpu().numpy())
    finally:
        for key, value in ((b"gemm_tc_nt", 0), (b"gemm_tc_small_max", 32), (b"gemm_tc_slices", 0), (b"gemm_q4k_mma", 1), (b"gemm_q6k_mma", 1)):
            ck.ckb200_tune_set(key, value)
    # as above: integer sums are the same on both sides, K / 256 fp32 terms of three roundings each; with fp16-rounded products it would be about 1e-4
    bound = 2 * (k // 256 + 3) * 2.0 ** -24 * 8 * float(np.max(np.abs(want)))
    assert float(np.max(np.abs(outs[0].astype(np.float64) - want))) <= bound
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.parametrize("fmt", ["q4_k", "q6_k"])
@pytest.mark.parametrize("m,width", [(32, 32), (64, 64), (90, 96), (128, 128)])
def test_sums_of_one_sign_beyond_the_exact_range(ck, orc, fmt, m, width):
    """Sums of a superblock whose terms have one sign, beyond the 2^24 up to which an fp32 accumulator holds every integer: up to 3.0e7 (Q4_K) and 1.3e8 (Q6_K, with operands
    that fp16 does not hold), against the same in 64 bits.  The bound: an MMA aligns its 16 products and the accumulator to the largest of them and cuts off what lies below
    its last place (Fasi, Higham, Mikaitis, Pranesh, "Numerical behavior of NVIDIA tensor cores", 2021), so 17 addends and the result lose a unit of the running sum each at
    most, and that is no larger than the last; 16 MMAs a superblock, 32 with those operands; then K / 256 terms of three fp32 roundings each.  Measured 3e-7 and 7e-7; the
    integer kernels, which round such a sum once, 2e-7."""
    import torch

    dev = torch.device("cuda", 0)
    n, nb = 200, 5
    k = 256 * nb
    rng = np.random.default_rng(m)
    w = synth.make_weights(fmt, n, k, seed=9).reshape(n, nb, -1).copy()
    if fmt == "q4_k":
        w[:, :, 2:4] = 0                                                                # no mins: nothing cancels
        w[:, :, 4:16] = 0xFF                                                            # scales of 63
        w[:, :, 16:] = 0xF0 | rng.integers(13, 16, size=w[:, :, 16:].shape, dtype=np.uint8)
        nibbles = w[:, :, 16:].reshape(n, nb, 4, 1, 32)
        weights = 63 * np.concatenate([nibbles & 15, nibbles >> 4], 3).reshape(n, nb, 256).astype(np.int64)
        d = w[:, :, 0:2].copy().view(np.float16)[..., 0].astype(np.float64)
    else:
        w[:, :, :192] = 0xFF                                                            # 63 - 32
        w[:, :, 192:208] = rng.integers(121, 128, size=(n, nb, 16), dtype=np.uint8)     # odd products beyond 2048
        weights = 31 * np.repeat(w[:, :, 192:208].astype(np.int64), 16, axis=2)
        d = w[:, :, 208:210].copy().view(np.float16)[..., 0].astype(np.float64)
    w[:, :, 1 if fmt == "q4_k" else 209] &= 0x7F                                        # d of one sign
    d = np.abs(d)
    x = rng.uniform(0.95, 1.0, size=(m, k)).astype(np.float32) * np.linspace(0.5, 2.0, m, dtype=np.float32)[:, None]
    aq = cases.quantize_act(orc, "oracle_", fmt, x, rows=m)
    rows = aq.reshape(m, nb, 292)
    q, dx = rows[:, :, 4:260].copy().view(np.int8).astype(np.int64), rows[:, :, :4].copy().view(np.float32)[..., 0].astype(np.float64)
    sums = np.einsum("mbk,nbk->mnb", q, weights)
    assert np.abs(sums).max() > (1.7e7 if fmt == "q4_k" else 1.0e8)
    want = np.einsum("mnb,nb,mb->mn", sums.astype(np.float64), d, dx)
    raw, taq = torch.from_numpy(w.reshape(-1)).to(dev), torch.from_numpy(aq).to(dev)
    if fmt == "q6_k":
        ck.ckb200_q6_k_planar_bytes.restype = C.c_size_t
        wdev = torch.empty(ck.ckb200_q6_k_planar_bytes(n, k), dtype=torch.uint8, device=dev)
        torch.cuda.synchronize()
        assert ck.ckb200_dev_q6_k_to_planar(C.c_void_p(wdev.data_ptr()), C.c_void_p(raw.data_ptr()), n, k, None) == 0
        fn = ck.ckb200_dev_gemm_nt_q6_k_planar_q8_k
    else:
        wdev, fn = raw, ck.ckb200_dev_gemm_nt_q4_k_q8_k
    c = torch.full((m, n), float("nan"), device=dev)
    try:
        for key, value in ((b"gemm_tc_nt", width if width > 32 else 0), (b"gemm_q4k_mma", 0), (b"gemm_q6k_mma", 0)):
            ck.ckb200_tune_set(key, value)
        torch.cuda.synchronize()
        assert fn(C.c_void_p(taq.data_ptr()), C.c_void_p(wdev.data_ptr()), None, C.c_void_p(c.data_ptr()), m, n, k, None) == 0
        assert ck.ckb200_synchronize() == 0
    finally:
        for key, value in ((b"gemm_tc_nt", 0), (b"gemm_q4k_mma", 1), (b"gemm_q6k_mma", 1)):
            ck.ckb200_tune_set(key, value)
    worst = float(np.max(np.abs(c.cpu().numpy().astype(np.float64) - want) / want))
    print(f"{fmt} {m}: {worst:.3g}")
    assert worst <= (16 if fmt == "q4_k" else 32) * 18 * 2.0 ** -23 + (nb + 3) * 2.0 ** -24


def tiles_from_rows(rows, nt):
    """What the operand tiles of `nt` tokens hold for Q8_K rows [tokens][superblocks][292]: halves of the quants [tile][superblock][32 chunks][token][8], the 16 sums as two more
    chunks, the scales [tile][superblock][token]; tokens past the end are left out."""
    T, nb, _ = rows.shape
    q = rows[:, :, 4:260].view(np.int8).reshape(T, nb, 32, 8)[..., [0, 2, 1, 3, 4, 6, 5, 7]].astype(np.float16)
    sums = rows[:, :, 260:292].copy().view(np.int16).reshape(T, nb, 2, 8).astype(np.float16)
    return np.concatenate([q, sums], 2), rows[:, :, :4].copy().view(np.float32)[..., 0]


def split_tiles(raw, nt, T, nb):
    blobs = raw[:((T + nt - 1) // nt) * nb * nt * 548].reshape(-1, nb, nt * 548)
    chunks = blobs[:, :, :nt * 544].copy().view(np.float16).reshape(-1, nb, 34, nt, 8)
    scales = blobs[:, :, nt * 544:].copy().view(np.float32).reshape(-1, nb, nt)
    return chunks.transpose(0, 3, 1, 2, 4).reshape(-1, nb, 34, 8)[:T], scales.transpose(0, 2, 1).reshape(-1, nb)[:T]


@pytest.mark.parametrize("nt", [64, 96, 128])
@pytest.mark.parametrize("T", [65, 96, 200])
@pytest.mark.parametrize("producer", ["norm", "swiglu", "gather"])
def test_producers_write_the_tiles_of_their_rows(ck, producer, nt, T):
    """The kernels in front of a product write its operand tiles: the same quants, sums and scales as the rows that they write elsewhere, each in its place."""
    import torch

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(T)
    p = lambda t: C.c_void_p(t.data_ptr())
    nb = 3
    rows = torch.zeros(T * nb * 292, dtype=torch.uint8, device=dev)
    tiles = torch.zeros(((T + nt - 1) // nt) * nb * nt * 548, dtype=torch.uint8, device=dev)
    if producer == "norm":
        x, delta, gamma = torch.randn(T, 768, device=dev, generator=g), torch.randn(T, 768, device=dev, generator=g), torch.rand(768, device=dev, generator=g) + 0.5
        x[:, 700:] = 0
        delta[:, 700:] = 0
        x2 = x.clone()
        torch.cuda.synchronize()
        assert ck.ckb200_dev_add_rmsnorm_q8k(p(x), p(delta), p(gamma), p(rows), None, T, 700, 768, C.c_float(1e-5), None) == 0
        assert ck.ckb_add_rmsnorm_tiles(p(x2), p(delta), p(gamma), p(tiles), nt, T, 700, 768, C.c_float(1e-5), None) == 0
    elif producer == "swiglu":
        gu = torch.randn(T, 1536, device=dev, generator=g)
        torch.cuda.synchronize()
        assert ck.ckb200_dev_swiglu_q8k(p(gu), p(rows), T, 768, None) == 0
        assert ck.ckb_swiglu_tiles(p(gu), p(tiles), nt, T, 768, None) == 0
    else:
        out = torch.randn(11, T, 64, device=dev, generator=g)          # 704 of 768 columns
        torch.cuda.synchronize()
        assert ck.ckb200_dev_prefill_gather_q8k(p(out), p(rows), T, 11, 64, 768, None) == 0
        assert ck.ckb_prefill_gather_tiles(p(out), p(tiles), nt, T, 11, 64, 768, None) == 0
    assert ck.ckb200_synchronize() == 0
    want, scales = tiles_from_rows(rows.cpu().numpy().reshape(T, nb, 292), nt)
    got, got_scales = split_tiles(tiles.cpu().numpy(), nt, T, nb)
    assert np.array_equal(got, want)
    assert np.array_equal(got_scales, scales)


@pytest.mark.parametrize("fmt", ["q4_k", "q6_k"])
@pytest.mark.parametrize("width,m,n,superblocks,launches", [
    # every remainder of the expanders' turns, of the rings and of two accumulators, in whole units and in slices of four
    (32, 20, 40, 1, 1), (32, 32, 129, 2, 1), (32, 17, 128, 3, 1), (32, 31, 200, 7, 1), (32, 32, 300, 9, 2), (64, 33, 129, 5, 1), (64, 64, 40, 10, 2), (96, 65, 130, 6, 1), (128, 97, 129, 11, 2),
    # a wave and a few tiles: the whole ones and the slices of the last rows are launches of their own, with the sum of the slices three
    (32, 19, 151 * 128, 8, 3), (64, 50, 150 * 128, 9, 3),
    # several units a CTA, the last of them of fewer superblocks
    (32, 25, 300 * 128 + 40, 2, 1), (64, 60, 299 * 128, 3, 1)])
def test_gemm_tiles_at_the_edges_of_their_deal(ck, orc, fmt, width, m, n, superblocks, launches):
    """The tcgen05 product over numbers of superblocks, tokens and row tiles at which its rings, its expander sets and its units have remainders.  Integer sums are the same on both
    sides; per superblock three fp32 roundings on either, as above."""
    import torch

    dev = torch.device("cuda", 0)
    k = 256 * superblocks
    w = synth.make_weights(fmt, n, k, seed=superblocks)
    aq = cases.quantize_act(orc, "oracle_", fmt, synth.make_x(k, seed=m, rows=m), rows=m)
    rows = np.r_[0:min(n, 256), max(n - 300, 0):n] if n > 600 else np.arange(n)          # the oracle's share of tall matrices: first and last tiles
    rows = np.unique(rows)
    want = cases.gemm_nt(orc, "oracle_", fmt, aq, np.ascontiguousarray(w.reshape(n, -1)[rows]).reshape(-1), None, m, len(rows), k)
    raw, taq = torch.from_numpy(w).to(dev), torch.from_numpy(aq).to(dev)
    if fmt == "q6_k":
        ck.ckb200_q6_k_planar_bytes.restype = C.c_size_t
        wdev = torch.empty(ck.ckb200_q6_k_planar_bytes(n, k), dtype=torch.uint8, device=dev)
        torch.cuda.synchronize()
        assert ck.ckb200_dev_q6_k_to_planar(C.c_void_p(wdev.data_ptr()), C.c_void_p(raw.data_ptr()), n, k, None) == 0
        fn = ck.ckb200_dev_gemm_nt_q6_k_planar_q8_k
    else:
        wdev, fn = raw, ck.ckb200_dev_gemm_nt_q4_k_q8_k
    ck.ckb200_launch_count.restype = C.c_longlong
    outs = []
    try:
        for key, value in ((b"gemm_tc_nt", width), (b"gemm_tc_slices", (superblocks + 3) // 4 if launches == 2 else 0), (b"gemm_q4k_mma", 0), (b"gemm_q6k_mma", 0)):
            ck.ckb200_tune_set(key, value)
        for _ in range(2):
            c = torch.full((m, n), float("nan"), device=dev)
            torch.cuda.synchronize()
            n0 = ck.ckb200_launch_count()
            assert fn(C.c_void_p(taq.data_ptr()), C.c_void_p(wdev.data_ptr()), None, C.c_void_p(c.data_ptr()), m, n, k, None) == 0
            count = ck.ckb200_launch_count() - n0
            assert ck.ckb200_synchronize() == 0
            outs.append(c.cpu().numpy())
    finally:
        for key, value in ((b"gemm_tc_nt", 0), (b"gemm_tc_slices", 0), (b"gemm_q4k_mma", 1), (b"gemm_q6k_mma", 1)):
            ck.ckb200_tune_set(key, value)
    bound = 2 * (superblocks + 3) * 2.0 ** -24 * 8 * float(np.max(np.abs(want)))
    assert float(np.max(np.abs(outs[0][:, rows].astype(np.float64) - want))) <= bound
    assert np.array_equal(outs[0], outs[1]) and np.isfinite(outs[0]).all()
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert count == 1 + launches, count          # and the launch that makes operand tiles


@pytest.mark.parametrize("m,n", [(130, 9600), (130, 9472), (129, 18944 + 40), (300, 4736)])
def test_q8_0_product_is_the_same_in_either_tile(ck, orc, m, n):
    """Wide tiles in whole rounds or a few behind them, narrow ones instead: the tile changes the deal, not a bit of the result."""
    import torch

    dev = torch.device("cuda", 0)
    k = 256
    g = torch.Generator(device=dev).manual_seed(n)
    x, w = torch.randn(m, k, device=dev, generator=g), torch.randn(n, k, device=dev, generator=g)
    p = lambda t: C.c_void_p(t.data_ptr())
    xq, wq = (torch.zeros(r * k // 32 * 34 + 64, dtype=torch.uint8, device=dev) for r in (m, n))
    torch.cuda.synchronize()
    assert ck.ckb200_dev_quantize_q8_0(p(x), p(xq), m, k, None) == 0 and ck.ckb200_dev_quantize_q8_0(p(w), p(wq), n, k, None) == 0
    outs = []
    try:
        for tile in (0, 64, 128):
            ck.ckb200_tune_set(b"gemm_q80_tile", tile)
            y = torch.full((m, n), float("nan"), device=dev)
            torch.cuda.synchronize()
            assert ck.ckb200_dev_gemm_nt_q8_0_q8_0(p(xq), p(wq), None, p(y), m, n, k, None) == 0
            assert ck.ckb200_synchronize() == 0
            outs.append(y.cpu().numpy())
    finally:
        ck.ckb200_tune_set(b"gemm_q80_tile", 0)
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
    first = min(n, 200)
    want = cases.gemm_nt(orc, "oracle_", "q8_0", xq.cpu().numpy()[:m * k // 32 * 34], np.ascontiguousarray(wq.cpu().numpy()[:first * k // 32 * 34]), None, m, first, k)
    assert np.array_equal(outs[0][:, :first], want)


@pytest.mark.parametrize("nt,m,n,n2,nb", [(32, 17, 128, 1, 1), (32, 77, 896, 128, 4), (64, 65, 256, 300, 3), (96, 96, 1280, 129, 2), (128, 129, 896, 128, 5)])
def test_two_products_over_the_same_rows_as_one_launch(ck, nt, m, n, n2, nb):
    """Rows of two matrices in one deal: the bits of the two products on their own, side by side."""
    import torch

    dev = torch.device("cuda", 0)
    k = 256 * nb
    p = lambda t: C.c_void_p(t.data_ptr())
    ws = [torch.from_numpy(synth.make_weights("q4_k", rows, k, seed=rows)).to(dev) for rows in (n, n2)]
    g = torch.Generator(device=dev).manual_seed(m)
    x, gamma = torch.randn(m, k, device=dev, generator=g), torch.ones(k, device=dev)
    tiles = torch.zeros(((m + nt - 1) // nt) * nb * nt * 548, dtype=torch.uint8, device=dev)
    both, apart = torch.full((m, n + n2), float("nan"), device=dev), [torch.full((m, rows), float("nan"), device=dev) for rows in (n, n2)]
    torch.cuda.synchronize()
    assert ck.ckb_add_rmsnorm_tiles(p(x), None, p(gamma), p(tiles), nt, m, k, k, C.c_float(1e-5), None) == 0
    if not ck.ckb_gemm_tc_pairs(nt, m, n, n2, k):
        assert ck.ckb_launch_gemm_tc_pair(p(tiles), nt, p(ws[0]), n, p(ws[1]), n2, p(both), n + n2, m, k, None) == -1
        return
    assert ck.ckb_launch_gemm_tc_pair(p(tiles), nt, p(ws[0]), n, p(ws[1]), n2, p(both), n + n2, m, k, None) == 0
    for w, out in zip(ws, apart):
        assert ck.ckb_launch_gemm_tc_tiles(0, p(tiles), nt, p(w), p(out), out.shape[1], m, out.shape[1], k, None, C.c_size_t(0), None) == 0
    assert ck.ckb200_synchronize() == 0
    assert torch.equal(both, torch.cat(apart, 1)) and torch.isfinite(both).all()


@pytest.mark.parametrize("heads,kv_heads,d,tokens", [(14, 2, 64, 77), (4, 4, 128, 17), (8, 1, 64, 129)])
def test_rotation_writes_the_pieces_that_attention_splits(ck, heads, kv_heads, d, tokens):
    """Attention over pieces from the rotation kernel gives the bits of attention that splits the cache itself; rows of q and k with gaps between them."""
    import torch

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(tokens)
    p = lambda t: C.c_void_p(t.data_ptr())
    at = lambda t, floats: C.c_void_p(t.data_ptr() + 4 * floats)
    room, wq, wk = 160, heads * d, kv_heads * d
    qk, v = torch.randn(tokens, wq + wk, device=dev, generator=g), torch.randn(tokens, wk, device=dev, generator=g)
    angle = torch.rand(room, d // 2, device=dev, generator=g) * 6
    cos, sin = angle.cos().contiguous(), angle.sin().contiguous()
    q0, k0 = qk[:, :wq].contiguous(), qk[:, wq:].contiguous()
    outs = []
    ck.ckb_attn_prefill_pieces.restype = C.c_void_p
    for own in (False, True):
        qh, kc, vc, out = torch.zeros(heads, tokens, d, device=dev), torch.zeros(kv_heads, room, d, device=dev), torch.zeros(kv_heads, room, d, device=dev), torch.zeros(heads, tokens, d, device=dev)
        torch.cuda.synchronize()
        if own:
            pieces = C.c_void_p(ck.ckb_attn_prefill_pieces(heads, kv_heads, tokens, d))
            assert pieces.value
            assert ck.ckb_prefill_rope_rows(p(qk), wq + wk, at(qk, wq), wq + wk, p(v), wk, p(qh), p(kc), p(vc), p(cos), p(sin), tokens, heads, kv_heads, d, room, 0, pieces, None) == 0
            assert ck.ckb_launch_attn_prefill_of_pieces(p(qh), pieces, p(out), heads, kv_heads, tokens, d, None) == 0
        else:
            assert ck.ckb200_dev_prefill_rope_scatter(p(q0), p(k0), p(v), p(qh), p(kc), p(vc), p(cos), p(sin), tokens, heads, kv_heads, d, room, 0, None) == 0
            assert ck.ckb200_dev_attention_prefill(p(qh), p(kc), p(vc), p(out), heads, kv_heads, tokens, d, d, room, 1, None) == 0
        assert ck.ckb200_synchronize() == 0
        outs.append((qh, kc, vc, out))
    assert all(torch.equal(a, b) for a, b in zip(*outs)) and outs[0][3].abs().sum() > 0
