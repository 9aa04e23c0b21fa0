"""The bf16 tcgen05 form of the W4A8 product (17 to 64 sequences) against the double-precision oracle and, where all sums are
exact integers, bit for bit against the dp4a kernel."""
import numpy as np
import pytest

import oracle
from blackwell_b200 import synth
from tests.util import max_abs_rel, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def k(cuda):
    """The kernels with every call of more than 16 sequences on this form."""
    from blackwell_b200 import kernels

    kernels.set_tuning(24, 1)
    yield kernels
    kernels.set_tuning(24, 0)


# rows around a tile of 256 and its halves; K of one, a part of one and many chunks of 256, scale rows of 4-, 8- and 16-byte
# pitch; every number of columns; shares that begin and end inside a tile, clusters (split 2..8), whole tiles (split 1)
@pytest.mark.parametrize("M,K,N,split", [
    (17, 32, 1, 0), (32, 256, 128, 0), (33, 288, 255, 0), (48, 544, 257, 9), (49, 4096, 129, 0), (64, 4096, 4096, 0),
    (40, 10944, 512, 9), (64, 10944, 300, 9), (24, 2080, 40000, 9), (64, 1024, 40000, 1), (32, 4096, 700, 2), (48, 4096, 511, 5),
    (64, 2048, 256, 8), (65, 1024, 256, 0), (100, 256, 130, 0)])
def test_matches_the_oracle(k, M, K, N, split):
    import torch

    W, sc16, _ = synth.int4_weights(N, K, seed=M + K + N, full_range=True)
    x32 = synth.activations_f16(M, K, 901).astype(np.float32) * 2.0
    xq, xs = oracle.quantize_int8(x32)
    args = [to_dev(xq), to_dev(xs), to_dev(W), to_dev(sc16.view(np.uint16)), K, N, M]
    y = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    y2 = torch.full_like(y, float("nan"))
    k.set_tuning(6, split)
    try:
        k.gemv_w4a8(y, *args)
        k.gemv_w4a8(y2, *args)
    finally:
        k.set_tuning(6, 0)
    torch.cuda.synchronize()
    assert k.device_status() == 0
    assert torch.equal(y, y2)
    # fp32 sums of K / 16 block terms in K order: K / 16 roundings of 2^-24 at most, far less than the bar
    assert max_abs_rel(y.cpu().numpy(), oracle.gemv_w4a8_f64(xq, xs, W, sc16)) < 2e-5


@pytest.mark.parametrize("M", [32, 48, 64])
def test_scales_of_every_kind_are_split_without_rounding(k, M):
    """Subnormal, negative, largest and full-mantissa binary16 scales: one k-block per output and an activation scale of 1, so
    that the output is w_sc * dot, at most 25 bits, to one rounding."""
    import torch

    K, N = 32, 4096
    r = synth.rng(77)
    bits = r.integers(0, 1 << 16, size=(N, 2), dtype=np.uint16)
    bits[(bits & 0x7C00) == 0x7C00] ^= 0x4000            # no infinities or NaN
    bits[:64, 0] = np.arange(64)                          # subnormals
    bits[64:68, 0] = [0x7BFF, 0xFBFF, 0x0400, 0x8001]
    bits[:, 1] = 0
    W, _, _ = synth.int4_weights(N, K, seed=5, full_range=True)
    xq = r.integers(-127, 128, size=(M, K), dtype=np.int8)
    xs = np.ones((M, 2), np.float32)
    y = torch.empty((M, N), dtype=torch.float32, device="cuda")
    k.gemv_w4a8(y, to_dev(xq), to_dev(xs), to_dev(W), to_dev(bits), K, N, M)
    ref = oracle.gemv_w4a8_f64(xq, xs, W, bits.view(np.float16))
    assert (np.abs(y.cpu().numpy() - ref) <= 2.0 ** -23 * np.abs(ref)).all()


def test_integers_match_the_small_batch_kernel(k):
    import torch

    K, N = 1024, 300
    W, _, _ = synth.int4_weights(N, K, seed=79, full_range=True)
    ones16 = np.ones((N, K // 16), np.float16)
    xq = synth.rng(907).integers(-127, 128, size=(64, K), dtype=np.int8)
    xs = np.ones((64, K // 16), np.float32)
    Wd, sd = to_dev(W), to_dev(ones16.view(np.uint16))
    y4 = torch.empty((4, N), dtype=torch.float32, device="cuda")
    k.gemv_w4a8(y4, to_dev(xq[:4]), to_dev(xs[:4]), Wd, sd, K, N, 4)
    for M in (17, 48, 64):
        y = torch.empty((M, N), dtype=torch.float32, device="cuda")
        k.gemv_w4a8(y, to_dev(xq[:M]), to_dev(xs[:M]), Wd, sd, K, N, M)
        assert torch.equal(y[:4], y4), M


def test_prologues_strides_and_residual(k):
    import torch

    M, K, N = 40, 4096, 300
    W, sc16, _ = synth.int4_weights(N, K, seed=78)
    x32 = synth.activations_f16(M, K, 903).astype(np.float32)
    nw = synth.norm_weight(K, 904)
    res = synth.activations_f16(M, N + 4, 905).astype(np.float32)
    Wd, sd = to_dev(W), to_dev(sc16.view(np.uint16))
    y = to_dev(res.copy())
    k.gemv_w4a8_decode(y, N + 4, y, to_dev(x32), None, 0, to_dev(nw), 1e-6, Wd, sd, K, N, M)
    xq, xs = oracle.quantize_int8(oracle.rmsnorm(x32, nw))
    ref = res.copy()
    ref[:, :N] += oracle.gemv_w4a8_f64(xq, xs, W, sc16)
    assert max_abs_rel(y.cpu().numpy(), ref) < 1e-3
    assert np.array_equal(y.cpu().numpy()[:, N:], res[:, N:])
    gud = to_dev(synth.activations_f16(M, 2 * K, 906).astype(np.float32))
    y2 = torch.empty((M, N), dtype=torch.float32, device="cuda")
    k.gemv_w4a8_decode(y2, 0, None, gud, gud[:, K:], 2 * K, None, 0.0, Wd, sd, K, N, M)
    gu = gud.cpu().numpy()
    xq, xs = oracle.quantize_int8(oracle.swiglu(np.ascontiguousarray(gu[:, :K]), np.ascontiguousarray(gu[:, K:])))
    assert max_abs_rel(y2.cpu().numpy(), oracle.gemv_w4a8_f64(xq, xs, W, sc16)) < 1e-3
    # binary16 input: the integers of the unfused quantizer
    x16 = synth.activations_f16(M, K, 907)
    k.gemv_w4a8_f16in(y2, to_dev(x16.view(np.uint16)), Wd, sd, K, N, M)
    xq, xs = oracle.quantize_int8(x16.astype(np.float32))
    assert max_abs_rel(y2.cpu().numpy(), oracle.gemv_w4a8_f64(xq, xs, W, sc16)) < 2e-5
    assert k.device_status() == 0


def test_both_forms_in_turn_on_the_block_they_share(k):
    """K split of the int8 form (-1) and equal shares of the bf16 form (1), with few tiles and with many."""
    import torch

    K = 2048
    try:
        for form, M, N in [(-1, 32, 256), (1, 48, 9000), (-1, 64, 384), (1, 17, 12800), (-1, 64, 1100), (1, 64, 700), (-1, 20, 130)]:
            W, sc16, _ = synth.int4_weights(N, K, seed=N)
            xq, xs = oracle.quantize_int8(synth.activations_f16(M, K, N + 1).astype(np.float32))
            y = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
            k.set_tuning(24, form)
            k.set_tuning(6, 9 if form > 0 else 0)
            k.gemv_w4a8(y, to_dev(xq), to_dev(xs), to_dev(W), to_dev(sc16.view(np.uint16)), K, N, M)
            torch.cuda.synchronize()
            assert k.device_status() == 0
            assert max_abs_rel(y.cpu().numpy(), oracle.gemv_w4a8_f64(xq, xs, W, sc16)) < 2e-5, (form, M, N)
    finally:
        k.set_tuning(6, 0)
        k.set_tuning(24, 1)


def test_a_form_with_longer_chains_of_sums_is_not_chosen(k):
    """A narrow matrix of long rows, which the int8 form splits finer."""
    import torch

    M, K, N = 32, 32768, 300
    W, sc16, _ = synth.int4_weights(N, K, seed=93)
    xq, xs = oracle.quantize_int8(synth.activations_f16(M, K, 94).astype(np.float32))
    args = [to_dev(xq), to_dev(xs), to_dev(W), to_dev(sc16.view(np.uint16)), K, N, M]
    out = []
    try:
        for form in (-1, 0):
            k.set_tuning(24, form)
            out.append(torch.empty((M, N), dtype=torch.float32, device="cuda"))
            k.gemv_w4a8(out[-1], *args)
    finally:
        k.set_tuning(24, 1)
    assert torch.equal(*out)


# (form, key 6): equal shares of the bf16 form, K split of the int8 form
@pytest.mark.parametrize("form,split", [(1, 9), (-1, 5)])
def test_counters_of_a_call_that_gave_up_do_not_reach_the_next(k, form, split):
    """A product that gives up in a wait leaves tiles half counted in the block that both forms share."""
    import ctypes as C

    import torch

    from blackwell_b200 import _lib

    M, K, N = 40, 4096, 700
    W, sc16, _ = synth.int4_weights(N, K, seed=91)
    xq, xs = oracle.quantize_int8(synth.activations_f16(M, K, 92).astype(np.float32))
    args = [to_dev(xq), to_dev(xs), to_dev(W), to_dev(sc16.view(np.uint16)), K, N, M]
    y = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    block = C.c_void_p()
    L = _lib.load()
    assert L["_ZN2bw2tc7scratchEmP11CUstream_stPPh"](C.c_size_t(1), None, C.byref(block)) == 0
    k.set_tuning(24, form)
    k.set_tuning(6, split)
    try:
        k.gemv_w4a8(y, *args)
        torch.cuda.synchronize()
        half = type("_View", (), {"__cuda_array_interface__": {"shape": (16384,), "typestr": "<i4", "data": (block.value, False), "version": 2}})()
        torch.as_tensor(half, device="cuda").fill_(1)
        want = y.clone()
        y.fill_(float("nan"))
        k.gemv_w4a8(y, *args)
        torch.cuda.synchronize()
    finally:
        k.set_tuning(6, 0)
        k.set_tuning(24, 1)
    assert k.device_status() == 0
    assert torch.equal(y, want)
    assert max_abs_rel(y.cpu().numpy(), oracle.gemv_w4a8_f64(xq, xs, W, sc16)) < 2e-5


# Halves of a chunk that K ends in, six products (K up to 3,072) and five, one and many chunks, whole tiles and shares.
@pytest.mark.parametrize("M,K,N,split", [(17, 96, 40, 0), (48, 128, 513, 0), (64, 160, 256, 0), (33, 3072, 300, 0), (32, 3104, 300, 0),
                                         (64, 4096, 2000, 0), (20, 4128, 2000, 9), (48, 2080, 700, 1)])
def test_error_against_64_bits(k, M, K, N, split):
    """Neighbouring blocks and weights of very different size.  What is lost beside the fp32 sums: sl x3, 8e-8 (2-norm) where it is
    left out, and the fp32 additions, at most K / 256 + 2 roundings of 2^-24.  Without any other of the products: 6e-6 or more."""
    import torch

    r = synth.rng(K + N)
    W, sc16, _ = synth.int4_weights(N, K, seed=K, full_range=True)
    sc16 = (sc16.astype(np.float32) * 2.0 ** r.integers(-6, 7, size=sc16.shape)).astype(np.float16)
    x = synth.activations_f16(M, K, 95).astype(np.float32) * np.repeat(2.0 ** r.integers(-6, 7, size=(M, K // 16)), 16, 1).astype(np.float32)
    xq, xs = oracle.quantize_int8(x)
    y = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    k.set_tuning(6, split)
    try:
        k.gemv_w4a8(y, to_dev(xq), to_dev(xs), to_dev(W), to_dev(sc16.view(np.uint16)), K, N, M)
    finally:
        k.set_tuning(6, 0)
    ref = oracle.gemv_w4a8_f64(xq, xs, W, sc16)
    err = np.linalg.norm(y.cpu().numpy() - ref) / np.linalg.norm(ref)
    assert err < (1e-7 if K <= 3072 else 2e-7) + (K // 256 + 2) ** 0.5 * 2.0 ** -25


# whole tiles, clusters and shares; rows that end in either half of a chunk; scale rows of every pitch
@pytest.mark.parametrize("M,K,N,split", [(9, 2048, 300, 0), (16, 4096, 257, 0), (12, 10944, 512, 9), (10, 5632, 2000, 2), (13, 2080, 40000, 1),
                                         (16, 2208, 700, 9), (11, 704, 12000, 0), (75, 2048, 256, 0)])
def test_nine_to_sixteen_sequences(k, M, K, N, split):
    import torch

    W, sc16, _ = synth.int4_weights(N, K, seed=K, full_range=True)
    x16 = synth.activations_f16(M, K, 96)
    xq, xs = oracle.quantize_int8(x16.astype(np.float32))
    y = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    k.set_tuning(6, split)
    try:
        k.gemv_w4a8_f16in(y, to_dev(x16.view(np.uint16)), to_dev(W), to_dev(sc16.view(np.uint16)), K, N, M)
    finally:
        k.set_tuning(6, 0)
    torch.cuda.synchronize()
    assert k.device_status() == 0
    ref = oracle.gemv_w4a8_f64(xq, xs, W, sc16)
    # six products: the fp32 additions are all that is lost (see above)
    assert np.linalg.norm(y.cpu().numpy() - ref) / np.linalg.norm(ref) < (K // 256 + 2) ** 0.5 * 2.0 ** -24


@pytest.mark.parametrize("M,K", [(16, 499968), (40, 119968)])
def test_a_call_that_may_not_grow_the_scratch_is_still_taken(k, M, K):
    """Under capture, 48 / 34 MB of prepared activations against 10 MB of quantized ones."""
    import torch

    N = 32
    W, sc16, _ = synth.int4_weights(N, K, seed=97)
    x16 = synth.activations_f16(M, K, 98)
    args = [to_dev(x16.view(np.uint16)), to_dev(W), to_dev(sc16.view(np.uint16)), K, N, M]
    y = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    k.gemv_w4a8_f16in(torch.empty((2, N), dtype=torch.float32, device="cuda"), *args[:5], 2)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        k.gemv_w4a8_f16in(y, *args)
    g.replay()
    torch.cuda.synchronize()
    xq, xs = oracle.quantize_int8(x16.astype(np.float32))
    assert max_abs_rel(y.cpu().numpy(), oracle.gemv_w4a8_f64(xq, xs, W, sc16)) < 2e-5


@pytest.mark.parametrize("M,K,N,factor", [(17, 1024, 300, 64), (12, 2048, 300, 1024), (20, 3104, 300, 4), (32, 4096, 300, 64), (64, 4096, 300, 1024)])
def test_blocks_far_below_the_largest_of_their_chunk(k, M, K, N, factor):
    """One block in 16 carries larger activations on weights that are zero.  Of an element min(2^-19 u, 2^-18 |x|) is lost, u = 2^-7 of
    the power of two below the chunk's largest |x|; with five products min(2^-15 p, 2^-14 |x|) + 2^-23 |x| more, p the lesser of u and 2^-5 of
    the power of two below the block's mean |x|.  These roundings are independent and of both signs: their 2-norm bounds that of the error,
    beside the fp32 sums.  Without x3 at all 2^-9 |x| would be lost."""
    import torch

    W, sc16, _ = synth.int4_weights(N, K, seed=K, full_range=True)
    large = np.arange(K // 16) % 16 == 5
    W.reshape(N, K // 16, 8)[:, large] = 0x88
    x16 = synth.activations_f16(M, K, 99).astype(np.float32)
    x16.reshape(M, K // 16, 16)[:, large] *= factor
    x16 = x16.astype(np.float16)
    y = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
    k.gemv_w4a8_f16in(y, to_dev(x16.view(np.uint16)), to_dev(W), to_dev(sc16.view(np.uint16)), K, N, M)
    xq, xs = oracle.quantize_int8(x16.astype(np.float32))
    ref = oracle.gemv_w4a8_f64(xq, xs, W, sc16)
    x = np.abs(xq.astype(np.float64) * np.repeat(xs, 16, 1))
    q = np.stack([W & 15, W >> 4], 2).reshape(N, K).astype(np.float64) - 8
    w = q * np.repeat(sc16.astype(np.float64), 16, 1)
    top = np.maximum.reduceat(x, np.arange(0, K, 256), axis=1)
    u = np.repeat(2.0 ** (np.floor(np.log2(top)) - 7), 256, 1)[:, :K]
    lost = np.minimum(2.0 ** -19 * u, 2.0 ** -18 * x)
    if M > 16 and K > 3072:
        mean = np.repeat(x.reshape(M, -1, 16).mean(2), 16, 1)
        p = np.minimum(u, 2.0 ** (np.floor(np.log2(mean)) - 5))
        lost += np.minimum(2.0 ** -15 * p, 2.0 ** -14 * x) + 2.0 ** -23 * x
    bound = np.sqrt((lost ** 2 @ (w ** 2).T).sum()) + (K // 256 + 2) ** 0.5 * 2.0 ** -24 * np.linalg.norm(ref)
    assert np.linalg.norm(y.cpu().numpy() - ref) < bound
    assert bound < 2.0 ** -12 * np.linalg.norm(ref)


@pytest.mark.parametrize("kind", ["normal", "silu", "channels", "tails", "lognormal"])
@pytest.mark.parametrize("M,K,N", [(48, 2048, 3072), (64, 5632, 2048), (20, 12288, 1000)])
def test_no_further_from_64_bits_than_the_form_that_scales_every_block(k, M, K, N, kind):
    """Activations as the products meet them: after a norm, silu(g) u, a few large channels, long tails, channels of many sizes."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(K + M)
    n = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    x = n(M, K)
    if kind == "silu":
        x = torch.nn.functional.silu(x) * n(M, K)
    elif kind == "channels":
        x[:, ::200] *= 30
    elif kind == "tails":
        x = x / ((n(M, K) ** 2 + n(M, K) ** 2 + n(M, K) ** 2) / 3).sqrt()
    elif kind == "lognormal":
        x = x * n(1, K).exp()
    W, sc = synth.int4_weights_device(N, K, 41)
    xq, xs = torch.empty((M, K), dtype=torch.int8, device="cuda"), torch.empty((M, K // 16), device="cuda")
    k.quantize_int8(xq, xs, x.contiguous(), M * K)
    q = torch.stack([W & 15, W >> 4], 2).view(N, K).double() - 8
    each = lambda v, s: (v.double().view(len(v), -1, 16) * s.double()[..., None]).view(len(v), K)
    want, err = each(xq, xs) @ each(q, sc).T, []
    for form in (1, -1):
        y = torch.empty((M, N), device="cuda")
        k.set_tuning(24, form)
        try:
            k.gemv_w4a8(y, xq, xs, W, sc, K, N, M)
        finally:
            k.set_tuning(24, 1)
        err.append(float((y.double() - want).norm() / want.norm()))
    assert err[0] < err[1] < 4e-7, err
