"""Sizes at which the kernels chosen by row count, alignment and type can go wrong: tile and stage remainders, the
smallest and the largest of a range, cut work items, row pitches that no 16-byte copy can start at."""
import numpy as np
import pytest
import torch

from oracle import qx_oracle as O
from tests._util import FMTS, assert_close_dtype, check_ids, dev, host, rounded

pytestmark = pytest.mark.gpu

tk = pytest.importorskip("quixicore_metal_b200.tk")
tk_torch = pytest.importorskip("quixicore_metal_b200.tk_torch")


def _linear(fmt, M, K, N, dtype, seed, pack="synth"):
    rng = np.random.default_rng(seed)
    x = rounded(rng.standard_normal((M, K)), dtype)
    W = O.synth_pack(fmt, (0.02 * rng.standard_normal((N, K))).astype(np.float32)) if pack == "synth" else O.random_packed(fmt, N, K, seed)
    return x, W, rounded(0.01 * rng.standard_normal(N), dtype), rounded(rng.standard_normal((M, N)), dtype)


# rows around the chunks of 16 / 32 / 64 / 128 activation rows; 1031 = 8 * 128 + 7 weight rows; K = 1056 and 4640: row
# pitches that are no multiple of 16 bytes and a last stage that is not full; 8192: items cut between CTAs
@pytest.mark.parametrize("M,K,N", [(17, 256, 8), (32, 1056, 129), (33, 8192, 1031), (64, 4640, 35), (65, 512, 257), (128, 2048, 128),
                                   (129, 1056, 1), (256, 768, 300)])
@pytest.mark.parametrize("fmt", FMTS)
def test_linear_above_16_rows(fmt, M, K, N):
    K = K - K % O.FORMATS[fmt][0] if K % O.FORMATS[fmt][0] else K
    dtype = "f16" if M == 65 else "bf16"
    x, W, bias, res = _linear(fmt, M, K, N, dtype, M + K)
    got = tk.decode_linear_epilogue(dev(x, dtype), dev(W), dev(bias, dtype), dev(res, dtype), activation="silu", format=fmt)
    assert_close_dtype(host(got), O.decode_linear_epilogue(x, W, fmt, bias, res, 2, dtype), dtype)


# random bytes: every code; e8m0 scales far from that of the row's first block, whose blocks are added apart
@pytest.mark.parametrize("fmt,K", [("q4_0", 1024), ("q8_0", 1056), ("q6_K", 512), ("mxfp8", 4096), ("mxfp4", 1056)])
def test_rows_with_extreme_scales(fmt, K):
    x, W, _, _ = _linear(fmt, 40, K, 136, "bf16", 5, pack="random")
    ref = O.decode_linear_epilogue(x, W, fmt, None, None, 0, "bf16")
    got = host(tk.decode_linear_epilogue(dev(x, "bf16"), dev(W), None, None, format=fmt))
    ok = np.isfinite(ref).all(0)
    assert ok.any()
    for n in np.nonzero(ok)[0]:                              # every row of weights at its own scale
        assert_close_dtype(got[:, n], ref[:, n], "bf16", scale=float(np.abs(O.dequantize(fmt, W[n:n + 1])).max()) * 30)


@pytest.mark.parametrize("M,K,N", [(17, 1056, 96), (64, 2048, 1056), (130, 768, 160)])
@pytest.mark.parametrize("fmt", ["q4_0", "nvfp4", "mxfp8"])
def test_swiglu_and_mxfp8_rows_above_16(fmt, M, K, N):
    x, g, gb, _ = _linear(fmt, M, K, N, "bf16", M)
    _, u, ub, _ = _linear(fmt, M, K, N, "bf16", M + 1)
    y, blocks = tk_torch.decode_swiglu(dev(x, "bf16"), dev(g), dev(u), dev(gb, "bf16"), dev(ub, "bf16"), fmt, True,
                                       output_quant="mxfp8", with_output=True)
    assert_close_dtype(host(y), O.decode_swiglu(x, g, u, fmt, gb, ub, "bf16"), "bf16")
    np.testing.assert_array_equal(host(blocks), O.quantize_mxfp8_rows(host(y)))


# the fixed summation order of the decoder stack: one row, passes of 16 and 32 rows, the uncut form above
@pytest.mark.parametrize("M,K,N", [(1, 1024, 48), (5, 512, 257), (17, 2048, 129), (32, 1024, 256), (33, 512, 40)])
@pytest.mark.parametrize("fmt", ["nvfp4", "q4_0", "q6_K"])
def test_ordered_entries(fmt, M, K, N):
    x, W, bias, res = _linear(fmt, M, K, N, "bf16", M)
    _, u, _, _ = _linear(fmt, M, K, N, "bf16", M + 1)
    lin = lambda: tk_torch.decode_linear_epilogue(dev(x, "bf16"), dev(W), dev(bias, "bf16"), dev(res, "bf16"), fmt, 0, True, True, ordered=True)
    got = lin()
    assert_close_dtype(host(got), O.decode_linear_epilogue(x, W, fmt, bias, res, 0, "bf16"), "bf16")
    assert torch.equal(got, lin())
    got = tk_torch.decode_swiglu(dev(x, "bf16"), dev(W), dev(u), dev(x, "bf16"), dev(x, "bf16"), fmt, False, ordered=True)
    assert_close_dtype(host(got), O.decode_swiglu(x, W, u, fmt, None, None, "bf16"), "bf16")


# fp32 (and 16-bit activations that start between 16-byte boundaries): K shorter than a warp's step and with a
# remainder, row groups of every size, K slices
@pytest.mark.parametrize("M,K,N", [(1, 256, 1), (2, 512, 35), (3, 1280, 129), (4, 8192, 64), (8, 4352, 33), (9, 768, 17)])
@pytest.mark.parametrize("fmt", FMTS)
def test_fp32_and_unaligned_activations(fmt, M, K, N):
    x, W, bias, res = _linear(fmt, M, K, N, "f32", M + K)
    _, u, _, _ = _linear(fmt, M, K, N, "f32", M + 1)
    got = tk.decode_linear_epilogue(dev(x), dev(W), dev(bias), dev(res), activation="gelu", format=fmt)
    assert_close_dtype(host(got), O.decode_linear_epilogue(x, W, fmt, bias, res, 1, "f32"), "f32")
    got = tk.decode_swiglu(dev(x), dev(W), dev(u), format=fmt)
    assert_close_dtype(host(got), O.decode_swiglu(x, W, u, fmt, None, None, "f32"), "f32")
    xb = rounded(x, "bf16")
    shifted = torch.zeros(M * K + 1, dtype=torch.bfloat16, device="cuda")[1:].view(M, K).copy_(dev(xb, "bf16"))
    assert shifted.data_ptr() % 16 == 2
    got = tk.decode_linear_epilogue(shifted, dev(W), None, None, format=fmt)
    assert_close_dtype(host(got), O.decode_linear_epilogue(xb, W, fmt, None, None, 0, "bf16"), "bf16")


# q6_K gate and up rows in paired warps: fewer tiles than pairs, a tile remainder, ranges that end inside a tile
@pytest.mark.parametrize("M,K,N", [(1, 256, 16), (4, 2048, 33), (8, 512, 4099), (16, 4096, 200)])
def test_q6k_swiglu_pairs(M, K, N):
    x, g, gb, _ = _linear("q6_K", M, K, N, "bf16", N)
    _, u, ub, _ = _linear("q6_K", M, K, N, "bf16", N + 1)
    got = tk.decode_swiglu(dev(x, "bf16"), dev(g), dev(u), dev(gb, "bf16"), dev(ub, "bf16"), format="q6_K")
    assert_close_dtype(host(got), O.decode_swiglu(x, g, u, "q6_K", gb, ub, "bf16"), "bf16")


@pytest.mark.parametrize("T", [17, 64])
@pytest.mark.parametrize("fmt,K", [("q6_K", 512), ("q4_0", 1056), ("mxfp8", 1056)])
def test_lm_head_above_16_rows(fmt, K, T):
    rng = np.random.default_rng(T)
    W = O.synth_pack(fmt, (0.3 * rng.standard_normal((4003, K))).astype(np.float32))
    h = rounded(0.5 * rng.standard_normal((T, K)), "bf16")
    for mode, code, kw in (("argmax", 0, {}), ("topk", 2, dict(k=64)), ("topp", 3, dict(k=32, top_p=0.9))):
        tok = host(tk.lm_head_sample(dev(h, "bf16"), dev(W), mode=mode, format=fmt, temperature=0.8, seed=3, **kw))
        want, margin = O.lm_head_sample(h, W, fmt, code, temperature=0.8, seed=3, return_detail=True, **kw)
        check_ids(tok, want, margin, 1e-4, f"{fmt}/{mode}")


# rows in registers: one vector, a partial last warp, two and four vectors per thread, one row past what is resident
# (the ring), a row too long for registers
@pytest.mark.parametrize("rows,D", [(1, 8), (4800, 264), (299, 8192), (600, 4088), (3, 8200), (151, 16384), (2, 16392)])
def test_seam_rows(rows, D):
    rng = np.random.default_rng(D)
    x, r = (rounded(rng.standard_normal((rows, D)), "bf16") for _ in range(2))
    x[0, :] = -0.0
    x[-1, : D // 2] *= 100.0                                  # exponents beyond the paired form's range
    x = rounded(x, "bf16")
    w = rounded(1 + 0.1 * rng.standard_normal(D), "bf16")
    n, added_ref = O.rms_norm_add(x, r, w, 1e-5, "bf16")
    act = O.gated_act("swiglu", x, r)
    pick = np.unique(np.r_[0, rows // 2, rows - 1])
    for kind in ("fp8", "int8"):
        norm = tk.rms_norm_add_fp8 if kind == "fp8" else tk_torch.rms_norm_add_int8_dyn
        silu = tk.silu_mul_quant_fp8 if kind == "fp8" else tk.silu_mul_quant_int8
        codes, added, scale = norm(dev(x, "bf16"), dev(r, "bf16"), dev(w, "bf16"))
        np.testing.assert_array_equal(host(added), added_ref)
        for ref, (c, s) in ((n, (codes, scale)), (act, silu(dev(x, "bf16"), dev(r, "bf16")))):
            rc, rs = O.quantize_groups(ref[pick], D, kind)
            np.testing.assert_allclose(host(s).reshape(-1)[pick], rs.reshape(-1), rtol=1e-5)
            same = (host(c)[pick].astype(np.int32) & 0xFF) == (rc.astype(np.int32) & 0xFF)
            assert same.mean() >= 0.99, (kind, float(same.mean()))


# ---- block scales at the ends of their range ------------------------------------------------------------------
# e8m0 scales of 2^120 and more against small codes and codes of zero, on the generic kernel (fp32 activations, and
# 16-bit ones that start between 16-byte boundaries): products that fp32 holds stay finite
@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4"])
@pytest.mark.parametrize("e", [0, 1, 246, 247, 254])
def test_generic_kernel_block_scales(fmt, e):
    K, N = 96, 35
    x, W, _, _ = _linear(fmt, 3, K, N, "bf16", e, pack="random")
    x = x * np.float32(2.0 ** -8)                        # 32 products of up to 2^126 stay below 2^128
    W[:, 1, 0] = e
    W[:, 1, 1:] &= 0x88 if fmt == "mxfp8" else 0x11      # 0, 2^-6 and their negatives; 0 and 0.5
    W[0, 1, 1:] = 0                                      # a block of zeros
    shifted = torch.zeros(3 * K + 1, dtype=torch.bfloat16, device="cuda")[1:].view(3, K).copy_(dev(x, "bf16"))
    ref = x.astype(np.float64) @ O.dequantize(fmt, W).astype(np.float64).T
    size = np.abs(x).astype(np.float64) @ np.abs(O.dequantize(fmt, W)).astype(np.float64).T
    for xs, ulp in ((dev(x), 2.0 ** -22), (shifted, 2.0 ** -8)):
        got = host(tk.decode_linear_epilogue(xs, dev(W), None, None, format=fmt)).astype(np.float64)
        assert np.isfinite(got).all()
        # one rounding of the output and, below, at most K + 8 of the sum's (2^-24 of the terms each)
        assert (np.abs(got - ref) <= ulp * np.abs(ref) + (K + 8) * 2.0 ** -24 * size).all()


# activations near the end of fp32: a weight times an activation is in range, its code times the activation is not
@pytest.mark.parametrize("fmt", FMTS)
def test_generic_kernel_large_activations(fmt):
    x, W, _, _ = _linear(fmt, 2, 512, 19, "f32", 1)
    x = (x * 2.0 ** 125).astype(np.float32)              # |x| up to 2^127; sums below 2^127 * 0.02 * 2 * 23
    w = O.dequantize(fmt, W).astype(np.float64)
    ref, size = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    got = host(tk.decode_linear_epilogue(dev(x), dev(W), None, None, format=fmt)).astype(np.float64)
    assert (np.abs(got - ref) <= 520 * 2.0 ** -24 * size).all()


def test_mxfp8_rows_of_infinities():
    x = rounded(np.random.default_rng(2).standard_normal((4, 96)), "bf16")
    x[0, 5], x[1, 40], x[2, :32], x[3, 64:] = np.inf, -np.inf, np.inf, 3.3e38
    x = rounded(x, "bf16")
    for dtype in ("bf16", "f32"):
        np.testing.assert_array_equal(host(tk_torch.quantize_mxfp8_rows(dev(x, dtype))), O.quantize_mxfp8_rows(x))


# ---- host side -------------------------------------------------------------------------------------------------
def test_other_threads_run_while_a_launch_blocks():
    """The launch queue behind a long kernel fills up; the thread that blocks on it must not hold the interpreter."""
    import threading
    import time
    x, W, _, _ = _linear("q4_0", 1, 512, 64, "bf16", 1)
    x, W = dev(x, "bf16"), dev(W)
    run = lambda: tk.decode_linear_epilogue(x, W, None, None, format="q4_0")
    run(); torch.cuda.synchronize()
    done = threading.Event()

    def work():
        torch.cuda._sleep(int(1.5e9))                    # below a second
        for _ in range(3000):
            run()
        done.set()
    t = threading.Thread(target=work)
    gap, last = 0.0, time.perf_counter()
    t.start()
    while not done.is_set():
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
        time.sleep(0)
    t.join(); torch.cuda.synchronize()
    assert gap < 0.25, gap


def test_workspace_of_a_captured_graph_survives_larger_calls():
    """A graph keeps the addresses of the workspace that its calls used; later calls may not give that memory away."""
    rng = np.random.default_rng(2)
    V, K = 6000, 512
    W = dev(O.synth_pack("q4_0", (0.3 * rng.standard_normal((V, K))).astype(np.float32)))
    h = dev(rounded(rng.standard_normal((64, K)), "bf16"), "bf16")
    call = lambda T: tk.lm_head_sample(h[:T], W, mode="topk", k=8, temperature=0.8, seed=3, format="q4_0")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        want = call(2)
        g = torch.cuda.CUDAGraph()
        s.synchronize()
        with torch.cuda.graph(g, stream=s):
            got = call(2)
        call(64)                                         # a larger workspace on the same stream
        keep = [torch.full((4 << 20,), 90, dtype=torch.uint8, device="cuda") for _ in range(32)]
        g.replay()
        s.synchronize()
        assert torch.equal(got, want)
        assert all(bool((t == 90).all()) for t in keep)


# MXFP8 rows of one projection as the packed weight of the next, nothing in between: the second kernel may start before
# the first has finished, its weight loads may not
def _rows_as_weight(producer_rows, consumer_rows, K=2048, N=4096, reps=12):
    gen = torch.Generator("cuda").manual_seed(producer_rows)
    W = dev(O.synth_pack("q8_0", (0.02 * np.random.default_rng(1).standard_normal((N, K))).astype(np.float32)))
    x = torch.randn(reps, producer_rows, K, generator=gen, device="cuda").bfloat16()
    z = torch.randn(consumer_rows, N, generator=gen, device="cuda").bfloat16()
    tk.decode_linear_epilogue(z, tk.decode_linear_epilogue(x[0], W, output_quant="mxfp8", format="q8_0"), format="mxfp8")
    torch.cuda.synchronize()
    rows, got = [], []
    for r in range(reps):
        rows.append(tk.decode_linear_epilogue(x[r], W, output_quant="mxfp8", format="q8_0"))
        got.append(tk.decode_linear_epilogue(z, rows[-1], format="mxfp8"))
    torch.cuda.synchronize()
    for w, y in zip(rows, got):
        assert torch.equal(y, tk.decode_linear_epilogue(z, w, format="mxfp8"))
        torch.cuda.synchronize()


@pytest.mark.parametrize("producer_rows", [16, 64, 256])
def test_fresh_rows_as_weight_above_16_rows(producer_rows):
    _rows_as_weight(producer_rows, 40)


# one row: its kernel follows the producer directly; the producers are the streaming kernel and its passes, the
# tensor-memory form and (few bytes, many weight rows) the in-place pipeline
@pytest.mark.parametrize("producer_rows,K,N", [(1, 2048, 4096), (16, 2048, 4096), (32, 2048, 4096), (64, 2048, 4096), (32, 512, 28672)])
def test_fresh_rows_as_weight_of_one_row(producer_rows, K, N):
    _rows_as_weight(producer_rows, 1, K, N)


# Blocks whose scale leaves the range in which the decoded f16 operand is exact are added apart in fp32, rows that lie
# outside it as a whole are shifted.  Such blocks in the first and the last stage, in neighbouring rows and in a
# whole group of 32, above and below the range; K = 256 leaves items whole, the others are cut between CTAs; K = 256
# and 768 of the mx formats have pitches that are no multiple of 16 bytes (rows interleaved in 2, 4 or 8 boxes).
def _wild(fmt, W, n, big):
    last = W.shape[1] - 1
    rows = [r for r in (0, 1, 33, *range(64, 96), 127, 130, n - 1) if r < n]
    for i, r in enumerate(rows):
        for b in ((0,), (last,), (0, last))[i % 3]:
            if fmt in ("q4_0", "q8_0"):
                W[r, b, :2] = np.array([600.0 + i if big else 65504.0], np.float16).view(np.uint8)
            elif fmt == "q6_K":
                W[r, b, 208:210] = np.array([16.0 + i if big else 3000.0], np.float16).view(np.uint8)
            else:
                W[r, b, 0] = 127 + i % 12 if big else 60 + i % 40
    return rows


@pytest.mark.parametrize("big", [False, True])
@pytest.mark.parametrize("M,K,N", [(17, 256, 131), (40, 768, 300), (64, 4096, 136), (129, 2048, 40)])
@pytest.mark.parametrize("fmt", ["q4_0", "q8_0", "q6_K", "mxfp8", "mxfp4"])
def test_rows_with_scales_outside_the_exact_range(fmt, M, K, N, big):
    from quixicore_metal_b200 import _lib
    x, W, _, _ = _linear(fmt, M, K, N, "bf16", 5, pack="random")
    rows = _wild(fmt, W, N, big)
    for r in rows[3:8]:                                  # whole rows out of range, nothing larger beside it
        W[r, :, :] = W[r, :1, :]
        if fmt in ("mxfp8", "mxfp4"):
            W[r, :, 0] = 40 + r % 50
    if fmt in ("mxfp8", "mxfp4"):
        W[rows[-1], 0, 1:] = 0                           # a first block that holds nothing
    w = O.dequantize(fmt, W).astype(np.float64)
    ref = x.astype(np.float64) @ w.T
    size = np.abs(x).astype(np.float64) @ np.abs(w).T
    _, U, _, _ = _linear(fmt, M, K, N, "bf16", 6)
    _lib.set_option("ts_min_rows", 1)                    # the kernel with that operand at every row count
    try:
        got = host(tk.decode_linear_epilogue(dev(x, "bf16"), dev(W), None, None, format=fmt)).astype(np.float64)
        # half an ulp of bf16 and the noise of the sums: at most 2^-24 of the terms for each of the K / 16 x 3
        # products of a chunk and the K / 256 sums over chunks
        assert (np.abs(got - ref) <= 2.0 ** -8 * np.abs(ref) + 2e-5 * size).all()
        part = host(tk_torch.decode_linear_partial(dev(x, "bf16"), dev(W), fmt)).astype(np.float64)
        assert (np.abs(part - ref) <= 2e-5 * size).all()
        for gate, up in ((W, U), (U, W)):                # marked rows in either matrix of a pair
            want = O.decode_swiglu(x, gate, up, fmt, None, None, "f32")
            y = host(tk.decode_swiglu(dev(x, "bf16"), dev(gate), dev(up), format=fmt))
            dots = [x.astype(np.float64) @ O.dequantize(fmt, v).astype(np.float64).T for v in (gate, up)]
            sums = [np.abs(x).astype(np.float64) @ np.abs(O.dequantize(fmt, v)).astype(np.float64).T for v in (gate, up)]
            tol = 2.0 ** -8 * np.abs(want) + 2e-5 * 1.1 * (sums[0] * np.abs(dots[1]) + sums[1] * np.abs(dots[0]))  # |silu'| < 1.1, |silu(g)| <= |g|
            ok = np.isfinite(want) & (np.abs(want) < 1e38)
            assert (np.abs(y - want)[ok] <= tol[ok] + 1e-30).all()
    finally:
        _lib.set_option("ts_min_rows", 0)


# A cut item's part is handed over only when the shares of all its marked rows are in: blocks left out only in the rows that
# output warps 1 - 3 add (32 - 127 of every 128) and only in the last stages of K, which are the part of a CTA that starts
# inside an item and goes on with the next one.
def _marked_parts(fmt, K, seed):
    x, W, _, _ = _linear(fmt, 64, K, 256, "bf16", seed)
    nb = W.shape[1]
    for r in (r for r in range(256) if r % 128 >= 32):
        for j in range(6):
            b = nb // 2 + (7 * r + 11 * j) % (nb // 2)
            if fmt in ("q4_0", "q8_0"):
                W[r, b, :2] = np.array([600.0 + r], np.float16).view(np.uint8)
            elif fmt == "q6_K":
                W[r, b, 208:210] = np.array([16.0 + r], np.float16).view(np.uint8)
            else:
                W[r, b, 0] = 130 + r % 8
    return x, W, O.dequantize(fmt, W).astype(np.float64)


def _assert_parts_handed_over(tiles, stages, groups):
    """Some CTAs hold the end of an item and then the start of another."""
    ctas = torch.cuda.get_device_properties(0).multi_processor_count // groups
    first = [tiles * stages * c // ctas for c in range(ctas + 1)]
    assert sum(a % stages != 0 and b > -(-a // stages) * stages for a, b in zip(first, first[1:])) > 30


@pytest.mark.parametrize("fmt", ["q4_0", "q8_0", "q6_K", "mxfp8", "mxfp4"])
def test_marked_rows_of_parts_handed_over(fmt):
    M, K, N, reps = 64, 4096, 14336, 8
    _assert_parts_handed_over(N // 128, K // 256, 1)
    _assert_parts_handed_over(N // 128, K // 256, 2 if fmt == "q6_K" else 1)     # gate / up pairs
    x, W, w = _marked_parts(fmt, K, 7)
    _, U, _, _ = _linear(fmt, M, K, 256, "bf16", 8)
    wide = lambda a: dev(a).repeat(N // 256, 1, 1)
    X, Wd, Ud = dev(x, "bf16"), wide(W), wide(U)
    x = x.astype(np.float64)
    dots = [x @ w.T, x @ O.dequantize(fmt, U).astype(np.float64).T]
    sums = [np.abs(x) @ np.abs(w).T, np.abs(x) @ np.abs(O.dequantize(fmt, U)).astype(np.float64).T]
    # half an ulp of bf16 and the noise of the sums, as in the test above
    got = [tk.decode_linear_epilogue(X, Wd, None, None, format=fmt) for _ in range(reps)]
    err = np.abs(host(got[0]).reshape(M, -1, 256) - dots[0][:, None])
    assert (err <= (2.0 ** -8 * np.abs(dots[0]) + 2e-5 * sums[0])[:, None]).all()
    assert all(torch.equal(g, got[0]) for g in got)
    for gate, up, (a, b) in ((Wd, Ud, (0, 1)), (Ud, Wd, (1, 0))):
        want = dots[a] / (1 + np.exp(-np.clip(dots[a], -700, 700))) * dots[b]
        tol = 2.0 ** -8 * np.abs(want) + 2e-5 * 1.1 * (sums[a] * np.abs(dots[b]) + sums[b] * np.abs(dots[a]))
        got = [tk.decode_swiglu(X, gate, up, format=fmt) for _ in range(reps)]
        assert (np.abs(host(got[0]).reshape(M, -1, 256) - want[:, None]) <= tol[:, None] + 1e-30).all()
        assert all(torch.equal(g, got[0]) for g in got)


@pytest.mark.parametrize("fmt", ["q4_0", "q8_0", "q6_K", "mxfp8", "mxfp4"])
def test_marked_rows_of_head_parts_handed_over(fmt):
    T, K, V, reps = 64, 4096, 64 * 256, 8
    _assert_parts_handed_over(V // 256, K // 256, 2 if fmt == "q6_K" else 1)
    h, W, w = _marked_parts(fmt, K, 9)
    h = (h * 2.0 ** -16).astype(np.float32)                  # logits of up to about 100
    pick = [32, 63, 64, 127, 160, 197, 233, 255]
    allowed = [[256 * t + r for r in pick] for t in range(T)]                    # hidden row t looks at tile t
    mask = dev(O.packed_allow_mask(allowed, V).view(np.int32))
    H, Wd = dev(h, "bf16"), dev(W).repeat(V // 256, 1, 1)
    got = [tk.lm_head_masked(H, Wd, mask, format=fmt, topk=len(pick)) for _ in range(reps)]
    logits = h.astype(np.float64) @ w[pick].T
    noise = 2e-5 * (np.abs(h).astype(np.float64) @ np.abs(w[pick]).T).max(1, keepdims=True)
    top = np.sort(logits, 1)[:, ::-1]
    want = top - top[:, :1] - np.log(np.exp(top - top[:, :1]).sum(1, keepdims=True))
    assert (np.abs(host(got[0][1]) - want) <= 2 * noise + 1e-5 * np.abs(want) + 1e-6).all()
    assert all(torch.equal(a, b) for g in got for a, b in zip(g, got[0]))


# results that fp32 does not hold in units of the scaled activations and weights (2^26 and 2^23 of them, unit
# activations) from blocks with large e8m0 scales: whole items and cut ones
@pytest.mark.parametrize("K", [256, 4096])
@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4"])
def test_large_results_of_shifted_rows(fmt, K):
    x, W, _, _ = _linear(fmt, 40, K, 136, "bf16", 8, pack="random")
    W[:100, :, 0] = 127 + (100 if fmt == "mxfp8" else 108)
    w = O.dequantize(fmt, W).astype(np.float64)
    ref, size = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    assert np.abs(ref).max() > 2.0 ** 110 and size.max() < 2.0 ** 127
    got = host(tk.decode_linear_epilogue(dev(x, "bf16"), dev(W), None, None, format=fmt)).astype(np.float64)
    assert (np.abs(got - ref) <= 2.0 ** -8 * np.abs(ref) + 2e-5 * size).all()


# an LM head with rows far below the others (tokens that no training step has touched) and a few far above
@pytest.mark.parametrize("fmt", ["mxfp8", "mxfp4", "q8_0"])
@pytest.mark.parametrize("T,V,K", [(17, 4003, 512), (64, 700, 4096)])
def test_lm_head_rows_outside_the_exact_range(fmt, T, V, K):
    rng = np.random.default_rng(T)
    W = O.synth_pack(fmt, (0.3 * rng.standard_normal((V, K))).astype(np.float32))
    h = rounded(0.5 * rng.standard_normal((T, K)), "bf16")
    if fmt == "q8_0":
        W[300:310, 1, :2] = np.array([600.0], np.float16).view(np.uint8)
    else:
        W[256:512, :, 0] = 60
        W[600, 1, 0] = 140
    for mode, code, kw in (("argmax", 0, {}), ("topk", 2, dict(k=64)), ("topp", 3, dict(k=32, top_p=0.9))):
        tok = host(tk.lm_head_sample(dev(h, "bf16"), dev(W), mode=mode, format=fmt, temperature=0.8, seed=3, **kw))
        want, margin = O.lm_head_sample(h, W, fmt, code, temperature=0.8, seed=3, return_detail=True, **kw)
        check_ids(tok, want, margin, 1e-4 if fmt != "q8_0" else 0.5, f"{fmt}/{mode}")


def _elapsed(fn, n=3):
    fn(); fn()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    for _ in range(n):
        fn()
    b.record(); b.synchronize()
    return a.elapsed_time(b) / n


# 148 groups of 64 rows fill one launch of the LM head's tensor-memory form; one row more is a second launch (the
# scalar kernel took 40 times as long)
def test_lm_head_rows_past_one_launch():
    rng = np.random.default_rng(1)
    V, K = 3000, 1024
    W = dev(O.synth_pack("q8_0", (0.3 * rng.standard_normal((V, K))).astype(np.float32)))
    h = torch.randn(148 * 64 + 1, K, generator=torch.Generator("cuda").manual_seed(1), device="cuda").bfloat16()
    call = lambda rows, mode="categorical": tk.lm_head_sample(h[rows], W, mode=mode, k=0, temperature=0.8, seed=3, format="q8_0")
    got, first = call(slice(None)), call(slice(0, 9472))
    assert (got[:9472] != first).float().mean() < 1e-3            # the noise of a row goes by its index in the call; near-ties
    want, margin = O.lm_head_sample(host(h[-8:]), host(W), "q8_0", 0, temperature=0.8, seed=3, return_detail=True)
    check_ids(host(call(slice(None), "argmax"))[-8:], want, margin, 1e-4, "last rows")
    assert _elapsed(lambda: call(slice(None))) < 5 * _elapsed(lambda: call(slice(0, 9472)))


# The one-accumulator form of the ordered entries is for nvfp4; other formats keep rounded chunk sums.  Mean signed error
# of 32 x 136 f16 outputs in units of the output: rounding to f16 averages to below 1e-5 (2^-11 / sqrt(12 * 4352)), a
# truncating accumulator over the 5184 steps of this K leaves 1e-4 towards zero.
def test_ordered_sums_are_not_biased():
    x, W, _, _ = _linear("q6_K", 32, 27648, 136, "f16", 3)
    ref = x.astype(np.float64) @ O.dequantize("q6_K", W).astype(np.float64).T
    got = host(tk_torch.decode_linear_epilogue(dev(x, "f16"), dev(W), None, None, "q6_K", ordered=True)).astype(np.float64)
    big = np.abs(ref) > 0.5
    assert abs(np.mean(((got - ref) / ref)[big])) < 3e-5


# nvfp4 above the passes: the uncut form against the in-place pipeline whose sums it continues, bit for bit
@pytest.mark.parametrize("M,K,N", [(70, 2048, 300), (128, 4096, 257), (32, 512, 24640)])
def test_ordered_nvfp4_equals_the_pipeline(M, K, N):
    from quixicore_metal_b200 import _lib
    x, W, _, _ = _linear("nvfp4", M, K, N, "bf16", M)
    _, U, _, _ = _linear("nvfp4", M, K, N, "bf16", M + 1)
    x, W, U = dev(x, "bf16"), dev(W), dev(U)
    run = lambda: (tk_torch.decode_linear_epilogue(x, W, None, None, "nvfp4", ordered=True),
                   tk_torch.decode_swiglu(x, W, U, None, None, "nvfp4", ordered=True))
    got = run()
    _lib.set_option("ts_min_rows", 1 << 20)
    try:
        want = run()
    finally:
        _lib.set_option("ts_min_rows", 0)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


# Activation preparation: an infinity, a NaN or a bf16 value past 3e38 in one row chooses no scale and reaches no other
# row; a row of zeros; orders of magnitude between rows; rows of one and of several passes over K.
@pytest.mark.parametrize("M,K", [(5, 512), (5, 12288), (20, 768), (20, 4352)])
@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("fmt", FMTS)
def test_prepared_rows_with_special_values(fmt, dtype, M, K):
    x, W, _, _ = _linear(fmt, M, K, 80, dtype, M + K)
    x[0, K - 1], x[1, 3], x[2, 7] = np.inf, np.nan, 3.3e38 if dtype == "bf16" else -np.inf
    x[3] = 0.0
    x[4] = rounded(x[4] * 2.0 ** (-60 if dtype == "bf16" else -9), dtype)
    got = host(tk.decode_linear_epilogue(dev(x, dtype), dev(W), None, None, format=fmt))
    ref = O.decode_linear_epilogue(x[3:], W, fmt, None, None, 0, dtype)
    # one ulp, fp32 noise of the row's largest output, one step of f16 subnormals
    ulp, step = (2.0 ** -7, 0.0) if dtype == "bf16" else (2.0 ** -10, 2.0 ** -24)
    assert np.all(np.abs(got[3:] - ref) <= np.abs(ref) * ulp * 1.01 + 2e-5 * np.abs(ref).max(1, keepdims=True) + step)
    assert not np.isfinite(got[:2]).any() and np.all(got[3] == 0)


# Items of one stage each, several per CTA, with marked rows in all of them: the marks travel from the workers to the output
# warps, up to eight items behind, and the last item is shared by more warps.
@pytest.mark.parametrize("M,N", [(40, 148 * 128 * 9 + 5), (64, 4000)])
@pytest.mark.parametrize("fmt", ["q4_0", "q8_0", "q6_K", "mxfp8", "mxfp4"])
def test_marked_rows_of_short_items(fmt, M, N):
    K = 256
    x, W, _, _ = _linear(fmt, M, K, 64, "bf16", M, pack="random")
    _wild(fmt, W, 64, True)
    W = np.tile(W, (-(-N // 64), 1, 1))[:N]                  # 64 rows over and over: the same outputs wherever a row lies
    got = host(tk.decode_linear_epilogue(dev(x, "bf16"), dev(W), None, None, format=fmt)).astype(np.float64)
    w, x = O.dequantize(fmt, W[:64]).astype(np.float64), x.astype(np.float64)
    ref, size = x @ w.T, np.abs(x) @ np.abs(w).T
    assert (np.abs(got[:, :64] - ref) <= 2.0 ** -8 * np.abs(ref) + 2e-5 * size).all()
    for n in range(64):
        assert np.all(got[:, n::64] == got[:, n:n + 1])


# Selection above 16 hidden rows: whole logits with many equals at every threshold (lowest ids win), fewer rows than output
# warps, one more than a pair per warp, a ragged last tile, candidates of -inf.
@pytest.mark.parametrize("T", [17, 25, 64])
@pytest.mark.parametrize("mode,k", [("argmax", 0), ("categorical", 0), ("topk", 1), ("topk", 33), ("topp", 5), ("topp", 64)])
def test_lm_head_ties_above_16_rows(T, mode, k):
    rng = np.random.default_rng(T + k)
    V, K = 5 * 256 + 100, 256
    W = np.zeros((V, K // 32, 34), np.uint8)
    W[..., 1] = 0x3C                                                          # scale 1.0
    W[..., 2:] = rng.integers(-2, 3, (V, K // 32, 32)).astype(np.int8).view(np.uint8)
    h = np.zeros((T, K), np.float32)
    h[:, ::32] = rng.integers(-1, 2, (T, 8))                                  # logits are whole numbers, about -10 .. 10
    bias = np.zeros(V, np.float32)
    bias[rng.integers(0, V, 300)] = -np.inf
    m = ("argmax", "categorical", "topk", "topp").index(mode)
    kw = dict(temperature=1.0, seed=11, top_p=0.9)
    got = host(tk.lm_head_sample(dev(h, "bf16"), dev(W), mode=mode, k=k, bias=dev(bias), format="q8_0", **kw))
    L = O.lm_head_logits(h, W, "q8_0")
    want, margin = O.lm_head_sample_from_logits(L, m, k=k if m >= 2 else 0, bias=bias, return_detail=True, **kw)
    if mode == "argmax":
        np.testing.assert_array_equal(got, want)
    check_ids(got, want, margin, 1e-4, mode)


# The merge of top-k candidates: one warp's search up to 512 tiles and 512 candidates, the block's above, ties at the threshold
# (whole logits) that send it to the exact search by id.
@pytest.mark.parametrize("V", [2 * 256 + 1, 9 * 256, 512 * 256, 513 * 256 - 5])
@pytest.mark.parametrize("k,ties", [(1, False), (9, False), (9, True), (64, True), (64, False)])
def test_top_k_merge(V, k, ties):
    rng = np.random.default_rng(V + k)
    T, K = 3, 256
    W = np.zeros((V, K // 32, 34), np.uint8)
    W[..., 1] = 0x3C if ties else 0x24                                        # scale 1, 2^-6
    W[..., 2:] = rng.integers(-3, 4, (V, K // 32, 32)).astype(np.int8).view(np.uint8)
    h = np.zeros((T, K), np.float32)
    if ties: h[:, ::32] = rng.integers(-1, 2, (T, 8))
    else: h = rounded(rng.standard_normal((T, K)), "bf16")
    got = host(tk.lm_head_sample(dev(h, "bf16"), dev(W), mode="topk", k=k, format="q8_0", temperature=1.0, seed=5))
    want, margin = O.lm_head_sample_from_logits(O.lm_head_logits(h, W, "q8_0"), 2, k=k, temperature=1.0, seed=5, return_detail=True)
    check_ids(got, want, margin, 1e-4, "top-k")


# The same results on both sides of a line between the streaming kernel and the tensor-memory one
@pytest.mark.parametrize("fmt,M,K,N", [("mxfp4", 11, 8192, 6784), ("mxfp4", 12, 8192, 6784), ("q6_K", 20, 8192, 4608), ("q6_K", 21, 8192, 4608)])
def test_lines_between_the_kernels(fmt, M, K, N):
    x, W, _, _ = _linear(fmt, M, K, 64, "bf16", M)
    W = np.tile(W, (N // 64, 1, 1))
    got = host(tk.decode_linear_epilogue(dev(x, "bf16"), dev(W), None, None, format=fmt))
    ref = O.decode_linear_epilogue(x, W[:64], fmt, None, None, 0, "bf16")
    for n in range(0, N, 64):
        assert_close_dtype(got[:, n:n + 64], ref, "bf16")


# Which kernel serves a call, on both sides of the lines in bytes and rows: its sums are those of the streaming kernel (and its
# passes) or those of the tensor-memory one, which differ in their order.
def _line(fmt, pair, M, mib, above):
    from quixicore_metal_b200 import _lib
    K = 8192
    bk, bb = O.FORMATS[fmt]
    N = -(-(mib << 20) // (K // bk * bb * (1 + pair))) - (not above)      # the first number of rows with that many bytes, the last below
    x, W, _, _ = _linear(fmt, M, K, 64, "f16", M)
    _, U, _, _ = _linear(fmt, M, K, 64, "f16", M + 1)
    wide = lambda a, *one: dev(a).repeat(-(-N // 64), *one)[:N]
    X, Wd, Ud = dev(x, "f16"), wide(W, 1, 1), wide(U, 1, 1) if pair else None
    # up biases that leave the low bits of the first row's dot products: elsewhere rounding hides the order of the sums
    gb, ub = np.zeros(64, np.float32), rounded(-(x[0].astype(np.float64) @ O.dequantize(fmt, U).astype(np.float64).T), "f16")
    run = lambda: (tk.decode_swiglu(X, Wd, Ud, wide(gb).half(), wide(ub).half(), format=fmt) if pair
                   else tk_torch.decode_linear_partial(X, Wd, fmt))
    got, kinds = run(), {}
    try:
        for kind, rows in (("streaming", 1 << 20), ("tensor memory", 1)):
            _lib.set_option("ts_min_rows", rows)
            kinds[kind] = run()
    finally:
        _lib.set_option("ts_min_rows", 0)
    of, x = np.arange(N) % 64, x.astype(np.float64)
    dots = [x @ O.dequantize(fmt, w).astype(np.float64).T for w in (W, U)]
    noise = [2e-5 * (np.abs(x) @ np.abs(O.dequantize(fmt, w)).astype(np.float64).T) for w in (W, U)]
    want, tol = dots[0], noise[0]
    if pair:                                                 # half an ulp of f16, half a step of its subnormals; |silu'| < 1.1, |silu(g)| <= |g|
        up = dots[1] + ub
        want = dots[0] / (1 + np.exp(-dots[0])) * up
        tol = 2.0 ** -11 * np.abs(want) + 2.0 ** -25 + 1.1 * (noise[0] * np.abs(up) + noise[1] * np.abs(dots[0]))
    assert (np.abs(host(got) - want[:, of]) <= tol[:, of]).all()
    assert not torch.equal(kinds["streaming"], kinds["tensor memory"])
    return [k for k, y in kinds.items() if torch.equal(y, got)]


# (format, gate / up pair, rows, MiB of weights)
@pytest.mark.parametrize("fmt,pair,M,mib", [("mxfp4", 0, 12, 28), ("mxfp4", 0, 9, 56), ("mxfp8", 0, 9, 56), ("nvfp4", 0, 12, 64),
                                            ("nvfp4", 0, 9, 100), ("q8_0", 0, 12, 200), ("q6_K", 0, 21, 28), ("nvfp4", 1, 9, 100),
                                            ("mxfp4", 1, 16, 100), ("mxfp8", 1, 9, 100)]
                         + [(f, 0, 17, 28) for f in FMTS if f != "q6_K"] + [(f, 1, 17, 16) for f in FMTS])
def test_kernel_at_the_lines(fmt, pair, M, mib):
    assert _line(fmt, pair, M, mib, True) == ["tensor memory"]
    assert _line(fmt, pair, M, mib, False) == ["streaming"]


# one row fewer, or a format whose streaming kernel is the faster one up to 16 rows
@pytest.mark.parametrize("fmt,pair,M,mib", [("mxfp4", 0, 11, 28), ("mxfp4", 0, 8, 56), ("mxfp8", 0, 8, 56), ("nvfp4", 0, 11, 64),
                                            ("nvfp4", 1, 8, 100), ("q8_0", 0, 11, 200), ("q8_0", 1, 16, 200), ("q6_K", 0, 20, 28),
                                            ("q4_0", 0, 16, 112), ("q4_0", 1, 16, 200), ("q6_K", 1, 16, 100)])
def test_kernel_one_row_below_the_lines(fmt, pair, M, mib):
    assert _line(fmt, pair, M, mib, True) == ["streaming"]
