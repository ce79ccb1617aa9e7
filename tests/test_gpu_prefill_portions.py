"""Batched prompt passes behind keys that are already in the cache, over 32-element formats, and at the token counts where a pass changes its kernels:
logits and every layer's new cache rows against the same tokens fed one by one through the decode step (itself checked against the CPU step)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import cases
import step_oracle as so

pytestmark = pytest.mark.gpu

QWEN = dict(embed_dim=384, num_heads=6, num_kv_heads=2, head_dim=64, intermediate_size=768, num_layers=2, vocab_size=500, max_seq_len=400, rms_eps=1e-6, rope_theta=1.0e6,
            fmt_q=0, fmt_k=0, fmt_v=1, fmt_o=0, fmt_gate_up=0, fmt_down=1, fmt_lm_head=1)
LLAMA = dict(QWEN, embed_dim=512, num_heads=8, num_kv_heads=2, head_dim=128, intermediate_size=1024, rms_eps=1e-5, rope_theta=5.0e5)
Q5_0 = dict(QWEN, fmt_q=3, fmt_k=3, fmt_v=3, fmt_o=3, fmt_gate_up=3)


def cosine(a, b):
    a, b = a.astype(np.float64).reshape(-1), b.astype(np.float64).reshape(-1)
    return float(a @ b / (np.linalg.norm(a) * np.linalg.norm(b)))


@pytest.mark.parametrize("cfg", [QWEN, LLAMA, Q5_0], ids=["qwen", "llama", "q5_0"])
@pytest.mark.parametrize("before,T", [(0, 16), (1, 17), (63, 64), (64, 65), (100, 129), (7, 300)])
def test_portion_matches_decode_steps(ck, cfg, before, T):
    so.bind_model_api(ck)
    model = so.CpuModel(cfg, seed=11)
    ids = np.random.default_rng(before + T).integers(0, cfg["vocab_size"], size=before + T).astype(np.int32)
    Hkv, S, d = cfg["num_kv_heads"], cfg["max_seq_len"], cfg["head_dim"]
    results = []
    for batched in (1, 0):
        handle = ck.ckb200_model_create(C.byref(so.make_cfg(cfg, batch=1)))
        assert handle, ck.ckb200_last_error_message()
        try:
            so.upload_whole_model(ck, handle, model, 1)
            ck.ckb200_tune_set(b"model_prefill", 0)
            if before:
                assert ck.ckb200_model_prefill(handle, cases.vptr(ids), before, None) == 0
            ck.ckb200_tune_set(b"model_prefill", batched)
            ck.ckb200_launch_count.restype = C.c_longlong
            n0 = ck.ckb200_launch_count()
            logits = np.full((1, cfg["vocab_size"]), np.nan, np.float32)
            assert ck.ckb200_model_prefill(handle, cases.vptr(ids[before:]), T, cases.vptr(logits)) == 0, ck.ckb200_last_error_message()
            if batched:
                assert ck.ckb200_launch_count() - n0 < 45 * cfg["num_layers"], "the portion ran token by token"
            assert ck.ckb200_model_get_pos(handle) == before + T
            kv = np.zeros((cfg["num_layers"], 2, Hkv, S, d), np.float32)
            assert ck.ckb200_copy_to_host(cases.vptr(kv), C.c_void_p(ck.ckb200_model_kv_device(handle, 0, 0)), kv.nbytes) == 0
            results.append((logits, kv))
        finally:
            ck.ckb200_tune_set(b"model_prefill", 1)
            ck.ckb200_model_free(handle)
    (got, kv), (want, ref) = results
    assert not kv[:, :, :, before + T:].any()
    assert np.array_equal(kv[:, :, :, :before], ref[:, :, :, :before])
    new, old = kv[:, :, :, before:before + T], ref[:, :, :, before:before + T]
    for is_v in (0, 1):                                   # layer 0 sees the same rows: fp32 summation order only
        assert float(np.max(np.abs(new[0, is_v] - old[0, is_v]))) <= 1e-4 * float(np.max(np.abs(old[0, is_v])))
    # deeper layers: the bar that the repository sets for whole steps (values that round to the other side of an 8-bit step)
    assert cosine(new, old) >= 0.9999
    assert cosine(got, want) >= 0.9999


# products on both sides of 2 M weights, with a feed-forward width that the Q6_K integer kernel refuses
WIDE = dict(LLAMA, intermediate_size=4352)


@pytest.mark.parametrize("before,T", [(0, 17), (5, 32), (0, 33), (3, 64)])
def test_portion_of_rows_and_tiles_matches_decode_steps(ck, before, T):
    """From 17 tokens large products take operand tiles, up to 32 small ones rows: both in one pass, and k and v behind q."""
    test_portion_matches_decode_steps(ck, WIDE, before, T)


@pytest.mark.parametrize("T", [17, 32, 33, 64])
def test_prompt_without_the_tcgen05_kernel(ck, T):
    """With tune gemm_tc 0 the integer kernels make all products of up to 64 tokens: how the other kernel would cut them changes no bit."""
    cfg = dict(LLAMA, embed_dim=1024, intermediate_size=2048)
    so.bind_model_api(ck)
    model = so.CpuModel(cfg, seed=3)
    ids = np.random.default_rng(T).integers(0, cfg["vocab_size"], size=T).astype(np.int32)
    outs = []
    handle = ck.ckb200_model_create(C.byref(so.make_cfg(cfg, batch=1)))
    assert handle, ck.ckb200_last_error_message()
    try:
        so.upload_whole_model(ck, handle, model, 1)
        for tc, slices in ((0, 0), (0, 2), (1, 0)):
            ck.ckb200_tune_set(b"gemm_tc", tc)
            ck.ckb200_tune_set(b"gemm_tc_slices", slices)
            assert ck.ckb200_model_reset(handle) == 0
            logits = np.full((1, cfg["vocab_size"]), np.nan, np.float32)
            assert ck.ckb200_model_prefill(handle, cases.vptr(ids), T, cases.vptr(logits)) == 0, ck.ckb200_last_error_message()
            outs.append(logits)
    finally:
        ck.ckb200_tune_set(b"gemm_tc", 1)
        ck.ckb200_tune_set(b"gemm_tc_slices", 0)
        ck.ckb200_model_free(handle)
    assert np.array_equal(outs[0], outs[1])
    assert cosine(outs[0], outs[2]) >= 0.9999


@pytest.mark.parametrize("tile", [64, 128])
@pytest.mark.parametrize("m,n,k", [(16, 40, 128), (65, 130, 384), (200, 300, 896)])
def test_q5_0_product_is_bit_identical(ck, orc, tile, m, n, k):
    """Q5_0 x Q8_0 over the planes: exact int32 block sums, fp32 in the reference's block order."""
    import torch

    dev = torch.device("cuda", 0)
    w = cases.synth.make_weights("q5_0", n, k, seed=m)
    aq = cases.quantize_act(orc, "oracle_", "q5_0", cases.synth.make_x(k, seed=n, rows=m), rows=m)
    want = cases.gemm_nt(orc, "oracle_", "q5_0", aq, w, None, m, n, k)
    raw, taq = torch.from_numpy(w).to(dev), torch.from_numpy(aq).to(dev)
    ck.ckb200_q5_0_planar_bytes.restype = ck.ckb200_q8_0_planar_bytes.restype = C.c_size_t
    wp = torch.empty(ck.ckb200_q5_0_planar_bytes(n, k) + 256, dtype=torch.uint8, device=dev)
    ap = torch.empty(ck.ckb200_q8_0_planar_bytes(m, k) + 256, dtype=torch.uint8, device=dev)
    c = torch.full((m, n + 3), float("nan"), device=dev)
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())
    assert ck.ckb200_dev_q5_0_to_planar(p(wp), p(raw), n, k, None) == 0
    assert ck.ckb200_dev_q8_0_to_planar(p(ap), p(taq), m, k, None) == 0
    try:
        ck.ckb200_tune_set(b"gemm_q80_tile", tile)
        assert ck.ckb_launch_gemm_q50_mma(p(ap), p(wp), None, p(c), n + 3, m, n, k, 0, None) == 0
    finally:
        ck.ckb200_tune_set(b"gemm_q80_tile", 0)
    assert ck.ckb200_synchronize() == 0
    got = c.cpu().numpy()
    assert np.array_equal(got[:, :n], want)
    assert np.isnan(got[:, n:]).all()


@pytest.mark.parametrize("heads,kvh,d", [(4, 1, 128), (7, 1, 64), (8, 1, 128), (3, 3, 64), (10, 2, 128)])
@pytest.mark.parametrize("before,T", [(0, 16), (1, 17), (63, 64), (64, 1), (1000, 16), (3000, 130), (129, 400)])
@pytest.mark.parametrize("spread", ["ordinary", "small values", "huge values", "large queries"])
def test_attention_behind_earlier_keys(ck, heads, kvh, d, before, T, spread):
    """Attention of a portion against softmax in 64 bits, with scores of spread 1 so that every run of keys carries weight.  In fp32 a score is two chains of 16 products
    per 32 dimensions, an output chains of 16 keys: some twenty roundings of 2^-24 at each that add like a random walk (four or five of them), the weight's own two
    and those of the sum and the division: ten roundings of the output's norm.  Sixteen-bit pieces of fp32 numbers miss that, and fp16's range: values of 0.003 as well
    as keys, values and queries beyond 65504."""
    import torch

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(before + T)
    S = before + T + 3
    q, k, v = (torch.randn(n, d, device=dev, generator=g) for n in (heads * T, kvh * S, kvh * S))
    q, k, v = q.view(heads, T, d), k.view(kvh, S, d), v.view(kvh, S, d)
    if spread == "small values":
        v *= 0.003
    elif spread == "huge values":
        v *= 1.0e6
        k *= 1.0e5
        q *= 1.0e-5
    elif spread == "large queries":
        q *= 1.0e4
        k *= 1.0e-4
    k[:, before + T:] = float("nan")                    # rows past the portion are nobody's
    v[:, before + T:] = float("nan")
    out = torch.full((heads, T, d), float("nan"), device=dev)
    ck.ckb_attn_behind_part_bytes.restype = C.c_size_t
    part = torch.empty(ck.ckb_attn_behind_part_bytes(d) // 4, device=dev)
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())
    assert ck.ckb_launch_attn_behind(p(q), p(k), p(v), p(out), heads, kvh, T, d, S, before, p(part), None) == 0, ck.ckb200_last_error_message()
    assert ck.ckb200_synchronize() == 0
    kk, vv = (t[:, :before + T].double().repeat_interleave(heads // kvh, 0) for t in (k, v))
    s = q.double() @ kk.transpose(1, 2) / d ** 0.5
    s = s.masked_fill(torch.arange(before + T, device=dev)[None, :] > torch.arange(before, before + T, device=dev)[:, None], -float("inf"))
    want = torch.softmax(s, -1) @ vv
    assert float((out.double() - want).norm() / want.norm()) <= 10 * 2.0 ** -24
    # a value that a query may not see does not reach it, whatever it is
    if T > 1:
        v[:, before + T - 1] = float("inf")
        torch.cuda.synchronize()
        assert ck.ckb_launch_attn_behind(p(q), p(k), p(v), p(out), heads, kvh, T, d, S, before, p(part), None) == 0
        assert ck.ckb200_synchronize() == 0
        assert torch.isfinite(out[:, :T - 1]).all()


@pytest.mark.parametrize("before", [0, 40])
def test_prompt_without_room_for_its_buffers_runs_as_steps(ck, before):
    """A batched pass takes device memory that decode steps do without: where there is none, the prompt goes through as steps, with their results."""
    so.bind_model_api(ck)
    ids = np.random.default_rng(5).integers(0, QWEN["vocab_size"], size=before + 100).astype(np.int32)
    ck.ckb200_launch_count.restype = C.c_longlong
    results, launches = [], []
    for max_mb, batched in ((1, 1), (0, 0), (64, 1)):
        handle = ck.ckb200_model_create(C.byref(so.make_cfg(QWEN, batch=1)))
        assert handle, ck.ckb200_last_error_message()
        try:
            assert ck.ckb200_model_fill_synthetic(handle, 9) == 0
            ck.ckb200_tune_set(b"model_prefill", 0)
            if before:
                assert ck.ckb200_model_prefill(handle, cases.vptr(ids), before, None) == 0
            ck.ckb200_tune_set(b"model_prefill", batched)
            ck.ckb200_tune_set(b"model_prefill_max_mb", max_mb)
            ck.ckb200_tune_set(b"model_graph", 0)                  # replays of a graph are not counted
            n0 = ck.ckb200_launch_count()
            logits = np.full((1, QWEN["vocab_size"]), np.nan, np.float32)
            assert ck.ckb200_model_prefill(handle, cases.vptr(ids[before:]), 100, cases.vptr(logits)) == 0, ck.ckb200_last_error_message()
            launches.append(ck.ckb200_launch_count() - n0)
            assert ck.ckb200_model_get_pos(handle) == before + 100
            results.append(logits)
        finally:
            ck.ckb200_tune_set(b"model_prefill", 1)
            ck.ckb200_tune_set(b"model_prefill_max_mb", 0)
            ck.ckb200_tune_set(b"model_graph", 1)
            ck.ckb200_model_free(handle)
    assert launches[0] == launches[1] >= 100 > launches[2], launches
    assert np.array_equal(results[0], results[1])
