"""The decode step as one launch against the same step as a launch per operation, at the places where its deal can go wrong: rows that are no
multiple of an item, rows of one and of several passes, every number of heads to a kv head, one run of keys, several, and more than are merged at a time."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import cases
import step_oracle as so

pytestmark = pytest.mark.gpu

KQ = dict(fmt_q=0, fmt_k=0, fmt_v=1, fmt_o=0, fmt_gate_up=0, fmt_down=1, fmt_lm_head=1)
BASE = dict(rms_eps=1e-5, rope_theta=5.0e5, num_layers=2, max_seq_len=256)
CONFIGS = {
    # Q4_K rows of 17 superblocks (two passes, the second of one), an odd number of logits, one head per kv head
    "two passes, odd vocabulary": (dict(BASE, embed_dim=4352, num_heads=4, num_kv_heads=4, head_dim=128, intermediate_size=512, vocab_size=777, **KQ), 0, 100),
    # Q6_K everywhere, rows long enough that passes go to different warps; eight heads per kv head
    "q6_k": (dict(BASE, embed_dim=2304, num_heads=8, num_kv_heads=1, head_dim=64, intermediate_size=4864, vocab_size=515, **dict.fromkeys(KQ, 1)), 0, 31),
    # Q4_K down projection of few rows over many superblocks, and as LM head; nothing in the cache
    "q4_k, first token": (dict(BASE, embed_dim=512, num_heads=6, num_kv_heads=2, head_dim=64, intermediate_size=8192, vocab_size=1001, **dict(KQ, fmt_v=0, fmt_down=0, fmt_lm_head=0)), 0, 0),
    "q5_0": (dict(BASE, embed_dim=896, num_heads=14, num_kv_heads=2, head_dim=64, intermediate_size=1280, vocab_size=300,
                  **dict(dict.fromkeys(KQ, 3), fmt_down=1, fmt_lm_head=1)), 0, 64),
    # 36 runs of keys: two batches of the merge
    "long context": (dict(BASE, embed_dim=512, num_heads=4, num_kv_heads=1, head_dim=128, intermediate_size=512, vocab_size=300, **dict(KQ, max_seq_len=9216)), 0, 9001),
    "half cache": (dict(BASE, embed_dim=512, num_heads=4, num_kv_heads=2, head_dim=128, intermediate_size=512, vocab_size=300, **KQ), 1, 200),
    "half cache, 64": (dict(BASE, embed_dim=512, num_heads=8, num_kv_heads=2, head_dim=64, intermediate_size=512, vocab_size=300, **dict(KQ, max_seq_len=2048)), 1, 1500),
}


@pytest.mark.parametrize("name", CONFIGS)
def test_one_launch_step_matches_the_launch_per_op_step(ck, name):
    """The pieces round alike; sums over warps and over runs of keys are taken in another order (1e-6), which now and then turns an 8-bit activation to its
    neighbour: 1/127 of its block's largest, one in a hundred thousand of them or so.  A flip in one of 512 elements moves a row of products by 1/127/sqrt(512) of
    its norm = 3.5e-4; the bound allows a dozen at once."""
    cfg, f16, ctx = CONFIGS[name]
    so.bind_model_api(ck)
    ck.ckb200_launch_count.restype = C.c_longlong
    V, got, launches = cfg["vocab_size"], {}, {}
    try:
        for one in (1, 0):
            ck.ckb200_tune_set(b"model_fused_step", one)
            ck.ckb200_tune_set(b"model_kv_f16", f16)
            handle = ck.ckb200_model_create(C.byref(so.make_cfg(cfg, batch=1)))
            ck.ckb200_tune_set(b"model_kv_f16", 0)
            assert handle, ck.ckb200_last_error_message()
            try:
                assert ck.ckb200_model_fill_synthetic(handle, 5) == 0
                assert ck.ckb200_model_fill_kv_synthetic(handle, ctx, 6) == 0
                assert ck.ckb200_model_set_pos(handle, ctx) == 0
                outs = []
                for i, tok in enumerate((3, 250, 77, 8)):
                    logits = np.full((1, V), np.nan, np.float32)
                    n0 = ck.ckb200_launch_count()
                    assert ck.ckb200_model_decode(handle, cases.vptr(np.array([tok], np.int32)), cases.vptr(logits)) == 0, ck.ckb200_last_error_message()
                    if i == 0:
                        launches[one] = ck.ckb200_launch_count() - n0
                    outs.append(logits[0].astype(np.float64))
                    assert ck.ckb200_model_get_pos(handle) == ctx + i + 1
                got[one] = outs
            finally:
                ck.ckb200_model_free(handle)
    finally:
        ck.ckb200_tune_set(b"model_fused_step", 1)
    assert 2 * launches[1] < launches[0], launches           # it is the other step
    for a, b in zip(got[1], got[0]):
        assert np.isfinite(b).all()
        assert np.linalg.norm(a - b) <= 5e-3 * np.linalg.norm(b), np.linalg.norm(a - b) / np.linalg.norm(b)


def steps_of(ck, name, tokens, tunes=()):
    """logits and positions of a few decode steps of a configuration, with tune keys set while they run"""
    cfg, f16, ctx = CONFIGS[name]
    so.bind_model_api(ck)
    outs, pos = [], []
    try:
        ck.ckb200_tune_set(b"model_kv_f16", f16)
        handle = ck.ckb200_model_create(C.byref(so.make_cfg(cfg, batch=1)))
        assert handle, ck.ckb200_last_error_message()
        ck.ckb200_tune_set(b"model_kv_f16", 0)
        assert ck.ckb200_model_fill_synthetic(handle, 5) == 0
        assert ck.ckb200_model_fill_kv_synthetic(handle, ctx, 6) == 0
        for key, value, _ in tunes:
            ck.ckb200_tune_set(key, value)
        for tok in tokens:
            logits = np.full((1, cfg["vocab_size"]), np.nan, np.float32)
            assert ck.ckb200_model_decode(handle, cases.vptr(np.array([tok], np.int32)), cases.vptr(logits)) == 0, ck.ckb200_last_error_message()
            outs.append(logits)
            pos.append(ck.ckb200_model_get_pos(handle) - ctx)
        ck.ckb200_model_free(handle)
    finally:
        ck.ckb200_tune_set(b"model_kv_f16", 0)
        for key, _, back in tunes:
            ck.ckb200_tune_set(key, back)
    return np.concatenate(outs), pos


@pytest.mark.parametrize("name", ["two passes, odd vocabulary", "q6_k", "q5_0", "half cache, 64"])
@pytest.mark.parametrize("missing", [1, 80, "all but one"])
def test_step_with_fewer_ctas_than_shares(ck, name, missing):
    """CTAs that find no SM while the others start: those that are there do all the work, with the same bits."""
    import torch

    if missing == "all but one":
        missing = torch.cuda.get_device_properties(0).multi_processor_count - 1
    whole = steps_of(ck, name, (3, 250, 77))
    assert whole[1] == [1, 2, 3]
    few = steps_of(ck, name, (3, 250, 77), [(b"step_missing_ctas", missing, 0)])
    assert few[1] == [1, 2, 3]
    assert np.array_equal(whole[0], few[0])


def test_barrier_that_runs_out_is_reported_and_leaves_the_positions_agreed(ck):
    """Barriers that wait for arrivals that nobody makes: every CTA gives up after the shortened limit and leaves, the call reports it, device and host agree where
    the sequence stands, and the steps behind it are those of a model that never failed."""
    import time

    name = "q6_k"
    cfg, _, ctx = CONFIGS[name]
    want, _ = steps_of(ck, name, (3, 250))
    so.bind_model_api(ck)
    handle = ck.ckb200_model_create(C.byref(so.make_cfg(cfg, batch=1)))
    assert handle, ck.ckb200_last_error_message()
    tok = lambda t: cases.vptr(np.array([t], np.int32))
    try:
        assert ck.ckb200_model_fill_synthetic(handle, 5) == 0
        assert ck.ckb200_model_fill_kv_synthetic(handle, ctx, 6) == 0
        logits = np.full((1, cfg["vocab_size"]), np.nan, np.float32)
        for key, value in ((b"model_graph", 0), (b"wait_limit_ms", 1), (b"step_extra_arrivals", 1)):
            ck.ckb200_tune_set(key, value)
        t0 = time.perf_counter()
        assert ck.ckb200_model_decode(handle, tok(3), cases.vptr(logits)) == 5         # CKB_ERR_DEVICE_WAIT
        assert time.perf_counter() - t0 < 1.0
        for key, value in ((b"model_graph", 1), (b"wait_limit_ms", 10000), (b"step_extra_arrivals", 0)):
            ck.ckb200_tune_set(key, value)
        ck.ckb200_clear_error()
        assert ck.ckb200_model_get_pos(handle) == ctx + 1
        # a batched pass goes by the host's position and leaves the device's behind its own tokens
        ids = np.arange(16, dtype=np.int32)
        assert ck.ckb200_model_prefill(handle, cases.vptr(ids), 16, None) == 0, ck.ckb200_last_error_message()
        assert ck.ckb200_model_get_pos(handle) == ctx + 17
        assert ck.ckb200_model_set_pos(handle, ctx) == 0
        for i, t in enumerate((3, 250)):
            assert ck.ckb200_model_decode(handle, tok(t), cases.vptr(logits)) == 0, ck.ckb200_last_error_message()
            assert ck.ckb200_model_get_pos(handle) == ctx + i + 1
            assert np.array_equal(logits[0], want[i])
    finally:
        for key, value in ((b"model_graph", 1), (b"wait_limit_ms", 10000), (b"step_extra_arrivals", 0)):
            ck.ckb200_tune_set(key, value)
        ck.ckb200_clear_error()
        ck.ckb200_model_free(handle)


# ---------------------------------------------------------------- the step against the CPU's, with weights and caches that let every run of keys count

def conditioned(fmt, rows, cols, seed, scale):
    """Blocks with values of mean 0 and variance scale^2 / cols, as trained weights have, so that scores stay of spread 1 and the softmax spreads over the keys."""
    name, size, unit, at, spread = {0: ("q4_k", 144, 256, 0, 258.0), 1: ("q6_k", 210, 256, 208, 342.0), 3: ("q5_0", 22, 32, 0, 9.2)}[fmt]
    w = cases.synth.make_weights(name, rows, cols, seed=seed).reshape(-1, size).copy()
    d = np.random.default_rng(seed).uniform(0.5, 1.5, len(w)) * scale / (spread * np.sqrt(cols))
    w[:, at:at + 2] = d.astype(np.float16).view(np.uint8).reshape(-1, 2)
    if fmt == 0:
        w[:, 2:4] = (7.5 * d).astype(np.float16).view(np.uint8).reshape(-1, 2)
    return w.reshape(-1)


def conditioned_model(cfg, ctx, attention):
    """A CpuModel of such weights, its cache filled.  Values change from 64 keys to the next 64 only, so that a row of attention is a mean of many such stretches, each with
    its share; `attention` scales the o projection so that the row is as large as the residual."""
    model = so.CpuModel(cfg, seed=3)
    scales = dict(WO=attention, W2=0.1)
    for i, lay in enumerate(model.layers):
        for j, (name, entry) in enumerate([(n, e) for n, e in lay.items() if isinstance(e, tuple)]):
            fmt, rows, cols, _ = entry
            lay[name] = (fmt, rows, cols, conditioned(fmt, rows, cols, 10 * i + j, scales.get(name, 1.0)))
    fmt, rows, cols, _ = model.lm_head
    model.lm_head = (fmt, rows, cols, conditioned(fmt, rows, cols, 99, np.sqrt(cols)))
    rng = np.random.default_rng(8)
    L, H, S, d = model.kc.shape
    model.kc[:, :, :ctx] = rng.standard_normal((L, H, ctx, d))
    model.vc[:, :, :ctx] = np.repeat(rng.standard_normal((L, H, (ctx + 63) // 64, d)), 64, axis=2)[:, :, :ctx]
    return model


def second_layer_rows(model, orc, token, pos, left_out=slice(0, 0)):
    """k and v of the new token in layer 1 by the CPU's kernels: what layer 0 made of its attention.  left_out: keys of layer 0 that attention forgets."""
    c = model.cfg
    D, H, G, d = c["embed_dim"], c["num_heads"], c["num_kv_heads"], c["head_dim"]
    cos, sin = cases.rope_cache(orc, "oracle_", c["max_seq_len"], d, c["rope_theta"])
    fmt, _, cols, table = model.lm_head
    x = so.embed_row(orc, fmt, table, token, c["vocab_size"], D, cols, model.Da)

    def qkv(lay, x):
        h = cases.rmsnorm(orc, "oracle_", x.reshape(1, -1), lay["LN1"], D, c["rms_eps"])[0]
        q, k = model._matvec(orc, lay["WQ"], h).reshape(H, 1, d).copy(), model._matvec(orc, lay["WK"], h).reshape(G, 1, d).copy()
        cases.rope_qk(orc, "oracle_", q, k, cos, sin, pos)
        return q.reshape(H, d), k.reshape(G, d), model._matvec(orc, lay["WV"], h).reshape(G, d).copy()

    lay = model.layers[0]
    q, k, v = qkv(lay, x)
    keep = np.ones(pos + 1, bool)
    keep[left_out] = False
    kc, vc = (np.ascontiguousarray(np.concatenate([cache[0][:, :pos], new[:, None]], 1)[:, keep]) for cache, new in ((model.kc, k), (model.vc, v)))
    x[:D] += model._matvec(orc, lay["WO"], cases.attention_decode(orc, "oracle_", np.ascontiguousarray(q), kc, vc, int(keep.sum())).reshape(-1))
    h = cases.rmsnorm(orc, "oracle_", x.reshape(1, -1), lay["LN2"], D, c["rms_eps"])[0]
    x[:D] += model._matvec(orc, lay["W2"], cases.swiglu(orc, "oracle_", model._matvec(orc, lay["W1"], h).reshape(1, -1), c["intermediate_size"])[0])
    _, k, v = qkv(model.layers[1], x)
    return np.stack([k, v])


@pytest.mark.parametrize("cfg,ctx,left_out", [
    # 36 runs of 256 keys: the second batch of the merge, one run in the first batch
    (dict(BASE, embed_dim=512, num_heads=4, num_kv_heads=1, head_dim=128, intermediate_size=512, vocab_size=300, **dict(KQ, max_seq_len=9216)), 9001, (slice(32 * 256, 9001), slice(1024, 1280))),
    # a few runs: the last, the first keys of a warp
    (dict(BASE, embed_dim=512, num_heads=8, num_kv_heads=2, head_dim=64, intermediate_size=512, vocab_size=300, **dict(dict.fromkeys(KQ, 1), max_seq_len=1024)), 700, (slice(640, 700), slice(0, 32))),
    (dict(BASE, embed_dim=896, num_heads=14, num_kv_heads=2, head_dim=64, intermediate_size=1280, vocab_size=300, **dict(dict.fromkeys(KQ, 3), fmt_down=1, fmt_lm_head=1)), 130, (slice(64, 96),)),
], ids=["two batches of runs", "runs", "q5_0"])
def test_one_launch_step_matches_the_cpu_where_every_run_of_keys_counts(ck, orc, cfg, ctx, left_out):
    """The new k and v of layer 1 show layer 0's attention directly.  Both sides round activations to 8 bits between products; a value of 1 / 127 of its block's largest to
    the other side of a step is the most that their orders of summation can do, 2e-3 of a row or less.  Forgetting a run of keys, or a batch of them in the merge, is
    several times the bound: checked with the oracle."""
    so.bind_model_api(ck)
    # the mean of n stretches of 64 equal values has 1 / sqrt(n) of their size
    model = conditioned_model(cfg, ctx, attention=np.sqrt((ctx + 63) // 64))
    want = second_layer_rows(model, orc, 7, ctx)
    for keys in left_out:
        assert np.linalg.norm(second_layer_rows(model, orc, 7, ctx, keys) - want) > 5 * 5e-3 * np.linalg.norm(want), keys
    G, S, d = cfg["num_kv_heads"], cfg["max_seq_len"], cfg["head_dim"]
    handle = ck.ckb200_model_create(C.byref(so.make_cfg(cfg, batch=1)))
    assert handle, ck.ckb200_last_error_message()
    try:
        so.upload_whole_model(ck, handle, model, 1)
        assert ck.ckb200_model_set_pos(handle, ctx) == 0
        assert ck.ckb200_model_decode(handle, cases.vptr(np.array([7], np.int32)), None) == 0
        kv = np.zeros((2, 2, G, S, d), np.float32)
        assert ck.ckb200_copy_to_host(cases.vptr(kv), C.c_void_p(ck.ckb200_model_kv_device(handle, 0, 0)), kv.nbytes) == 0
    finally:
        ck.ckb200_model_free(handle)
    got = kv[1, :, :, ctx]
    assert np.linalg.norm(got - want) <= 5e-3 * np.linalg.norm(want), np.linalg.norm(got - want) / np.linalg.norm(want)
