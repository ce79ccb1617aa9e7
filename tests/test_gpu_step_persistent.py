"""The decode step as one cooperative launch against the same step as a launch per operation, at the places where its deal can go wrong: rows that are no
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
