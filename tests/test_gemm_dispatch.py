"""Which kernel takes a product of 17 to 64 tokens, and what its callers may rely on: the integer-MMA kernels need no workspace, so such a product is right on any
stream, from any thread and in a graph; the tcgen05 kernel, which is faster from some size on, makes it where that stays so."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

import cases

synth = cases.synth

N, K = 18944, 4096                       # one round of 128-row tiles on 148 SMs: the tcgen05 kernel is the faster one from 17 tokens up, for either format
ALIGNED = C.c_void_p(1 << 20)            # never read


@pytest.mark.parametrize("fmt", ["q4k", "q6k"])
@pytest.mark.parametrize("m", [17, 32, 33, 64])
def test_integer_kernels_take_products_that_are_faster_elsewhere(pkg, fmt, m):
    lib = pkg.load_lib()
    takes, best = getattr(lib, f"ckb_gemm_{fmt}_mma_takes"), getattr(lib, f"ckb_gemm_{fmt}_mma_best")
    assert takes(ALIGNED, ALIGNED, m, N, K) == 1 and best(ALIGNED, ALIGNED, m, N, K) == 0
    assert takes(ALIGNED, ALIGNED, m, 512, 1024) == 1 and best(ALIGNED, ALIGNED, m, 512, 1024) == 1


@pytest.mark.parametrize("fmt", ["q4k", "q6k"])
def test_fewest_tokens_of_the_tcgen05_kernel(pkg, fmt):
    """A product that tune gemm_tc_min_tokens keeps from the tcgen05 kernel stays with the integer kernel."""
    lib = pkg.load_lib()
    best = getattr(lib, f"ckb_gemm_{fmt}_mma_best")
    try:
        lib.ckb200_tune_set(b"gemm_tc_min_tokens", 33)
        assert [best(ALIGNED, ALIGNED, m, N, K) for m in (17, 32, 33, 64)] == [1, 1, 0, 0]
    finally:
        lib.ckb200_tune_set(b"gemm_tc_min_tokens", 16)
    assert best(ALIGNED, ALIGNED, 32, N, K) == 0


@pytest.mark.parametrize("wf,m,n,k,width", [
    # one wave of 128-token tiles and a few behind it: no tokens computed for nothing where a narrower tile holds them all
    (0, 40, 19072, 2048, 64), (0, 64, 22016, 4096, 64), (0, 77, 22016, 4096, 96), (0, 96, 23552, 2048, 96), (1, 64, 22016, 2048, 64), (1, 96, 22016, 4096, 96),
    (0, 112, 22016, 2048, 128), (0, 128, 23552, 2048, 128), (1, 128, 23552, 8192, 128),
    (0, 130, 9600, 2048, 128)])
def test_width_of_token_tiles(pkg, wf, m, n, k, width):
    assert pkg.load_lib().ckb_gemm_tc_width(wf, m, n, k) == width


@pytest.mark.parametrize("name", ["ckb200_dev_gemm_nt_q4_k_q8_k", "ckb200_dev_gemm_nt_q6_k_planar_q8_k"])
@pytest.mark.parametrize("m", [16, 32, 64, 65, 200])
def test_first_call_initialises(pkg, name, m):
    """Whichever kernel takes it, a product comes behind the library's initialisation (its stream, the error word of the waits): without a device it ends there."""
    import torch

    if torch.cuda.is_available():
        pytest.skip("needs a machine without a GPU")
    lib = pkg.load_lib()
    try:
        assert getattr(lib, name)(ALIGNED, ALIGNED, None, ALIGNED, m, N, K, None) == 4          # CKB_ERR_NO_DEVICE
    finally:
        lib.ckb200_clear_error()


class Product:
    """Resident weights, rows of activations, and the device entry over them."""

    def __init__(self, ck, orc, fmt, m, n=N, k=K, seed=0):
        import torch

        self.ck, self.shape = ck, (m, n, k)
        dev = torch.device("cuda", 0)
        unit = synth.make_weights(fmt, 128, k, seed=seed)                        # repeated: what is compared are runs of one product
        raw = torch.from_numpy(np.tile(unit.reshape(128, -1), (n // 128, 1)).reshape(-1)).to(dev)
        self.a = torch.from_numpy(cases.quantize_act(orc, "oracle_", fmt, synth.make_x(k, seed=seed + m, rows=m), rows=m)).to(dev)
        if fmt == "q6_k":
            ck.ckb200_q6_k_planar_bytes.restype = C.c_size_t
            self.w = torch.empty(ck.ckb200_q6_k_planar_bytes(n, k), dtype=torch.uint8, device=dev)
            torch.cuda.synchronize()
            assert ck.ckb200_dev_q6_k_to_planar(C.c_void_p(self.w.data_ptr()), C.c_void_p(raw.data_ptr()), n, k, None) == 0
            self.fn = ck.ckb200_dev_gemm_nt_q6_k_planar_q8_k
        else:
            self.w, self.fn = raw, ck.ckb200_dev_gemm_nt_q4_k_q8_k
        self.c = torch.empty(m, n, device=dev)
        assert ck.ckb200_synchronize() == 0
        torch.cuda.synchronize()

    def run(self, stream=None):
        p = lambda t: C.c_void_p(t.data_ptr())
        return self.fn(p(self.a), p(self.w), None, p(self.c), *self.shape, C.c_void_p(stream.cuda_stream) if stream else None)

    def alone(self, stream=None):
        import torch

        self.c.fill_(float("nan"))
        torch.cuda.synchronize()
        assert self.run(stream) == 0
        torch.cuda.synchronize()
        assert self.ck.ckb200_synchronize() == 0
        return self.c.clone()


def launches(ck, call):
    ck.ckb200_launch_count.restype = C.c_longlong
    n0 = ck.ckb200_launch_count()
    out = call()
    return ck.ckb200_launch_count() - n0, out


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["q4_k", "q6_k"])
@pytest.mark.parametrize("m", [32, 64])
def test_products_on_several_streams_at_once(ck, orc, fmt, m):
    """Two streams of a caller and the library's own, different activations: every result has the bits of the call on its own, and a caller's stream those of the
    integer kernel."""
    import torch

    streams = [torch.cuda.Stream(), torch.cuda.Stream(), None]
    products = [Product(ck, orc, fmt, m, seed=s) for s in range(3)]
    want = [p.alone(s) for p, s in zip(products, streams)]
    try:
        ck.ckb200_tune_set(b"gemm_tc", 0)
        assert torch.equal(products[0].alone(), want[0])
    finally:
        ck.ckb200_tune_set(b"gemm_tc", 1)
    for _ in range(20):
        for p in products:
            p.c.fill_(float("nan"))
        torch.cuda.synchronize()
        for _ in range(4):
            for p, s in zip(products, streams):
                assert p.run(s) == 0
        torch.cuda.synchronize()
        assert ck.ckb200_synchronize() == 0
        for p, w in zip(products, want):
            assert torch.equal(p.c, w)


@pytest.mark.gpu
def test_products_of_several_threads(ck, orc):
    """Threads that share the library's stream: operand tiles of one call are read before those of the next are written, at sizes for which the workspace grows."""
    import torch

    products = [Product(ck, orc, "q4_k", m, n, k, seed=m) for m, n, k in ((32, N, K), (64, N, K), (64, 4992, 14336), (48, 2 * N, 8192))]
    gate, rcs = threading.Barrier(len(products)), []

    def work(p):
        gate.wait()
        rcs.extend(p.run() for _ in range(30))

    threads = [threading.Thread(target=work, args=(p,)) for p in products]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert ck.ckb200_synchronize() == 0 and not any(rcs)
    got = [p.c.clone() for p in products]
    for p, g in zip(products, got):
        assert torch.equal(p.alone(), g)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["q4_k", "q6_k"])
@pytest.mark.parametrize("own", [False, True], ids=["stream of the caller", "stream of the library"])
def test_product_in_a_graph(ck, orc, fmt, own):
    """Recorded on either kind of stream, and replayed after calls that need more workspace: the bits of the integer kernel.  A call on the library's stream beside a
    capture does what it does without one, its workspace growing."""
    import torch

    ck.ckb200_stream.restype = C.c_void_p
    stream = torch.cuda.ExternalStream(ck.ckb200_stream()) if own else torch.cuda.Stream()
    p, beside = Product(ck, orc, fmt, 32), Product(ck, orc, "q4_k", 64, N, 28672 if fmt == "q4_k" else 36864)          # more workspace than any test before
    try:
        ck.ckb200_tune_set(b"gemm_tc", 0)
        want = p.alone()
    finally:
        ck.ckb200_tune_set(b"gemm_tc", 1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        assert p.run(None if own else stream) == 0
        if not own:
            assert beside.run() == 0
    assert ck.ckb200_synchronize() == 0
    other = beside.c.clone()
    if not own:
        assert torch.equal(beside.alone(), other)
    beside.alone()
    Product(ck, orc, fmt, 200).alone()
    for _ in range(3):
        p.c.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(p.c, want)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["q4_k", "q6_k"])
def test_fewest_tokens_of_the_entry_points(ck, orc, fmt):
    """With gemm_tc_min_tokens above the call's tokens: the integer kernel in one launch or two, not a GEMV per token."""
    import torch

    p = Product(ck, orc, fmt, 32)
    try:
        ck.ckb200_tune_set(b"gemm_tc", 0)
        want = p.alone()
        ck.ckb200_tune_set(b"gemm_tc", 1)
        ck.ckb200_tune_set(b"gemm_tc_min_tokens", 65)
        count, got = launches(ck, p.alone)
    finally:
        ck.ckb200_tune_set(b"gemm_tc", 1)
        ck.ckb200_tune_set(b"gemm_tc_min_tokens", 16)
    assert count <= 2 and torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["q4_k", "q6_k"])
def test_own_stream_takes_the_faster_kernel(ck, orc, fmt):
    """On the library's stream the tcgen05 kernel and the launch that makes its operand tiles; the same values within fp32 rounding as the integer kernel."""
    import torch

    p, stream = Product(ck, orc, fmt, 32), torch.cuda.Stream()
    fast = p.alone()
    count, _ = launches(ck, p.alone)
    integer = p.alone(stream)
    assert float((fast - integer).abs().max()) <= 2 * (K // 256 + 3) * 2.0 ** -24 * 8 * float(integer.abs().max())
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert count == 2, count
