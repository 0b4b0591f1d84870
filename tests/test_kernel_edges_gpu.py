"""GPU tests of the edges of the kernels' tiles, splits and copies: where a store is clipped, a tile is cut between CTAs, a row does
not start on a whole word.  Integer-valued operands make the products exact in f32 (every partial sum is an integer below 2^24), so
those comparisons are bit for bit; the others state their bound.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 512


def ints(rng, *shape, lim=4):
    return rng.integers(-lim, lim + 1, shape).astype(np.float32)


def bf16_bits(v):
    u = np.ascontiguousarray(v, np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)


def from_bf16(u):
    return (u.astype(np.uint32) << 16).view(np.float32)


def run_gemm(t0, rt, x, b, m, n, k, out_bf16=False, bias=None, x_skip=0, b_skip=0, **kw):
    """x [m,k] and b as given (f32 values that bf16 holds exactly), *_skip elements into their buffers; the output and its guard."""
    xd = rt.upload(np.concatenate([np.zeros(x_skip, np.uint16), bf16_bits(x).ravel()]))
    bd = rt.upload(np.concatenate([np.zeros(b_skip, np.uint16), bf16_bits(b).ravel()]))
    size = 2 if out_bf16 else 4
    y = rt.alloc(m * n * size + GUARD)
    y.write(np.full(m * n * size + GUARD, 0xA5, np.uint8))
    bb = rt.upload(bias) if bias is not None else None
    rt.gemm(xd.gpu_addr() + 2 * x_skip, bd.gpu_addr() + 2 * b_skip, y.gpu_addr(), m, n, k, out_bf16=out_bf16, bias=bb.gpu_addr() if bb else 0, **kw)
    rt.synchronize()
    raw = y.read(m * n * size + GUARD, np.uint8)
    for buf in [xd, bd, y] + ([bb] if bb else []):
        buf.free()
    assert np.all(raw[m * n * size:] == 0xA5), "wrote past the output"
    body = raw[:m * n * size]
    return from_bf16(body.view(np.uint16)).reshape(m, n) if out_bf16 else body.view(np.float32).reshape(m, n)


@pytest.mark.parametrize("out_bf16", [False, True])
@pytest.mark.parametrize("n", [8, 33, 36, 72, 130, 264, 520])
@pytest.mark.parametrize("pair,tile_n", [(2, 32), (2, 64), (2, 128), (2, 256), (1, 128), (1, 256)])
def test_output_edges_of_every_tile(t0, rt, pair, tile_n, n, out_bf16):
    # widths that end inside a 32-column chunk, after an even chunk of a bf16 block, and that no 16-byte rule fits
    m, k = 150, 96
    rng = np.random.default_rng(n)
    x, b, bias = ints(rng, m, k), ints(rng, n, k), ints(rng, n, lim=100)
    got = run_gemm(t0, rt, x, b, m, n, k, out_bf16, bias, tile_n=tile_n, pair_cta=pair, epilogue=t0.EPI_BIAS_ADD_RELU_STORE_F32)
    want = np.maximum(x @ b.T + bias, 0)
    assert np.array_equal(got, from_bf16(bf16_bits(want)) if out_bf16 else want)


@pytest.mark.parametrize("pair,tile_n,split_k", [(2, 64, 1), (2, 256, 1), (1, 256, 1), (2, 128, 4)])
@pytest.mark.parametrize("out_bf16", [False, True])
def test_epilogue_chain_on_every_kernel(t0, rt, pair, tile_n, split_k, out_bf16):
    m, n, k = 150, 328, 512
    rng = np.random.default_rng(5)
    x, b = ints(rng, m, k, lim=1), ints(rng, n, k, lim=1)
    bias = rng.uniform(-2, 2, n).astype(np.float32)
    got = run_gemm(t0, rt, x, b, m, n, k, out_bf16, bias, tile_n=tile_n, pair_cta=pair, split_k=split_k, scale=0.125,
                   tile_epilogue=["scale", "bias", "silu", "neg", "gelu"])
    v = (x @ b.T).astype(np.float64) * 0.125 + bias
    v = -(v / (1 + np.exp(-v)))
    v = v / (1 + np.exp(-1.702 * v))
    # f32 elementwise: a few roundings of 2^-24 each, exp2 of an argument of up to ~40 adds |argument| * 2^-24 to the relative error
    tol = 1e-5 * np.abs(v) + 1e-6
    assert np.all(np.abs(got - v) <= tol + (2.0 ** -8 * np.abs(v) if out_bf16 else 0))


@pytest.mark.parametrize("m,k,n", [(3, 5, 7), (64, 64, 64), (100, 72, 200), (513, 264, 1000), (2048, 384, 640), (1024, 1024, 2056), (65, 1001, 30)])
def test_f32_products_are_exact_on_integers(t0, rt, m, k, n):
    # forward and both gradients; X^T is read as it lies (the tensor cores take it M-major), widths off the 16-byte rule are padded
    rng = np.random.default_rng(m)
    x, w, dy = ints(rng, m, k), ints(rng, k, n), ints(rng, m, n)
    xd, wd, dyd = rt.upload(x), rt.upload(w), rt.upload(dy)
    for call, rows, cols, want in ((lambda y: rt.matmul_f32(xd.gpu_addr(), wd.gpu_addr(), y, m, k, n), m, n, x @ w),
                                   (lambda y: rt.matmul_f32_backward_data(dyd.gpu_addr(), wd.gpu_addr(), y, m, k, n), m, k, dy @ w.T),
                                   (lambda y: rt.matmul_f32_backward_weight(xd.gpu_addr(), dyd.gpu_addr(), y, m, k, n), k, n, x.T @ dy)):
        y = rt.alloc(rows * cols * 4 + GUARD)
        y.write(np.full(rows * cols * 4 + GUARD, 0xA5, np.uint8))
        call(y.gpu_addr())
        rt.synchronize()
        raw = y.read(rows * cols * 4 + GUARD, np.uint8)
        assert np.array_equal(raw[:rows * cols * 4].view(np.float32).reshape(rows, cols), want)
        assert np.all(raw[rows * cols * 4:] == 0xA5), "wrote past the output"
        y.free()
    for b in (xd, wd, dyd):
        b.free()


@pytest.mark.parametrize("layout", ["nt", "nn"])
@pytest.mark.parametrize("m,n,k", [(5, 9, 3), (64, 65, 77), (130, 111, 250), (257, 1030, 129)])
@pytest.mark.parametrize("x_skip,b_skip", [(0, 0), (1, 0), (0, 3), (1, 1), (2, 4)])
def test_operands_at_any_element_address(t0, rt, layout, m, n, k, x_skip, b_skip):
    # rows that start at odd elements, bases inside a word: the staging copy reads whole words and shifts
    rng = np.random.default_rng(m + k)
    x, b = ints(rng, m, k), ints(rng, n, k)
    nn = layout == "nn"
    got = run_gemm(t0, rt, x, b.T if nn else b, m, n, k, x_skip=x_skip, b_skip=b_skip, transpose=t0.NN if nn else t0.NT)
    assert np.array_equal(got, x @ b.T)


@pytest.mark.parametrize("entry", ["tiled", "row"])
@pytest.mark.parametrize("M,K,N,count", [(17, 8192, 512, 2), (33, 4096, 768, 1), (128, 4096, 2560, 2), (107, 4352, 7936, 2), (40, 4096, 11008, 2), (1, 4096, 2592, 3)])
def test_w4a16_tiles_cut_between_ctas(t0, oracle, rt, entry, M, K, N, count):
    # tiles that do not fill the GPU evenly: they are cut into the ranges of two or more CTAs, whose parts are added in k order whoever finishes: repeated
    # calls agree bit for bit.  Bound: f32 sums of K exact products in another order, K * 2^-24 of the sum of their magnitudes at most
    if entry == "row" and M <= 16:
        pytest.skip("the row layout runs another kernel for M <= 16")
    G = 128
    calls, bufs, ys, refs = [], [], [], []
    for i in range(count):
        packed, scales, zeros = oracle.fill_u32((K // 8) * N, 10 + i), oracle.fill_range_bf16((K // G) * N, 20 + i, 0.001, 0.02), oracle.fill_u32((K // G) * (N // 8), 30 + i)
        a = oracle.fill_normal_bf16(M * K, 40 + i)
        ref = oracle.w4a16_gemm(a, packed, scales, zeros, M, N, K, G).astype(np.float64)
        w = np.abs(oracle.bf16_to_f32(oracle.dequant_w4_b200(packed, scales, zeros, K, N, G)).reshape(K, N))
        refs.append((ref, np.abs(oracle.bf16_to_f32(a).reshape(M, K)).astype(np.float64) @ w * (K * 2.0 ** -24)))
        xp, xs, xz, xa, y = rt.upload(packed), rt.upload(scales), rt.upload(zeros), rt.upload(a), rt.alloc(M * N * 4)
        bufs += [xp, xs, xz, xa, y]
        ys.append(y)
        if entry == "tiled":
            t = rt.w4_to_tiled(xp.gpu_addr(), xs.gpu_addr(), xz.gpu_addr(), K, N, G)
            bufs.append(t)
            calls.append(t0.W4A16Args(xa.gpu_addr(), t.gpu_addr(), 0, 0, y.gpu_addr(), M, N, K, G))
        else:
            calls.append(t0.W4A16Args(xa.gpu_addr(), xp.gpu_addr(), xs.gpu_addr(), xz.gpu_addr(), y.gpu_addr(), M, N, K, G))
    run = rt.w4a16_gemm_tiled_grouped if entry == "tiled" else rt.w4a16_gemm_grouped
    first = None
    for _ in range(4):
        for y in ys:
            y.write(np.full(M * N, np.nan, np.float32))
        run(calls)
        rt.synchronize()
        got = [y.read(M * N * 4, np.float32).reshape(M, N) for y in ys]
        if first is None:
            first = got
            for g, (ref, tol) in zip(got, refs):
                assert np.all(np.abs(g - ref) <= tol)
        for g, f in zip(got, first):
            assert np.array_equal(g.view(np.uint32), f.view(np.uint32))
    for b in bufs:
        b.free()


@pytest.mark.parametrize("layout", ["nt", "nn"])
@pytest.mark.parametrize("tile_n,split_k", [(64, 2), (64, 8), (128, 2), (128, 4)])
@pytest.mark.parametrize("m,n,k", [(40, 72, 512), (129, 200, 1024), (300, 640, 4096)])
@pytest.mark.parametrize("out_bf16", [False, True])
def test_cluster_split_k_in_both_layouts(t0, rt, layout, tile_n, split_k, m, n, k, out_bf16):
    rng = np.random.default_rng(n)
    x, b, bias = ints(rng, m, k), ints(rng, n, k), ints(rng, n, lim=100)
    nn = layout == "nn"
    before = rt.launch_count()
    got = run_gemm(t0, rt, x, b.T if nn else b, m, n, k, out_bf16, bias, tile_n=tile_n, split_k=split_k, pair_cta=2,
                   transpose=t0.NN if nn else t0.NT, epilogue=t0.EPI_BIAS_ADD_STORE_F32)
    assert rt.launch_count() - before == 1
    want = x @ b.T + bias
    assert np.array_equal(got, from_bf16(bf16_bits(want)) if out_bf16 else want)


@pytest.mark.parametrize("layout", ["nt", "nn"])
@pytest.mark.parametrize("m,n,k", [(32, 752, 3984), (16, 2048, 2048), (100, 296, 8192), (512, 512, 2048), (1024, 512, 4096), (2048, 1024, 4096), (128, 4096, 1024),
                                   (1, 8, 64), (64, 1024, 200), (130, 136, 72), (64, 5056, 6656), (16, 8, 10240)])
def test_library_chosen_kernel(t0, rt, layout, m, n, k):
    # nothing fixed by the caller: parts of K that are not of one length, sums in two accumulators, pairs, and tiny products
    rng = np.random.default_rng(k)
    x, b, bias = ints(rng, m, k), ints(rng, n, k), ints(rng, n, lim=100)
    nn = layout == "nn"
    for out_bf16 in (False, True):
        got = run_gemm(t0, rt, x, b.T if nn else b, m, n, k, out_bf16, bias, transpose=t0.NN if nn else t0.NT, epilogue=t0.EPI_BIAS_ADD_STORE_F32)
        want = x @ b.T + bias
        assert np.array_equal(got, from_bf16(bf16_bits(want)) if out_bf16 else want)


def test_parts_added_in_order_whoever_is_last(t0, rt):
    # real-valued operands: the parts of a tile are added in split order, so repeated launches agree bit for bit
    rng = np.random.default_rng(3)
    m, n, k = 48, 512, 6144
    x, b = from_bf16(bf16_bits(rng.uniform(-1, 1, (m, k)))), from_bf16(bf16_bits(rng.uniform(-1, 1, (n, k))))
    first = run_gemm(t0, rt, x, b, m, n, k)
    for _ in range(5):
        assert np.array_equal(run_gemm(t0, rt, x, b, m, n, k), first)


@pytest.mark.parametrize("op,factor", [("silu", 1.0), ("gelu", 1.702)])
def test_sigmoid_over_its_whole_range(t0, rt, op, factor):
    # v arrives exactly, as the bias of a product of zeros: small and large arguments, beyond the exponential's range on both sides (from v = -88.7 on
    # 1 + e overflows), infinities, NaN
    import torch
    rng = np.random.default_rng(8)
    edges = np.array([0.0, -0.0, 87.2, 87.4, 88.0, 88.72, 88.73, 89.0, 103.0, 104.0, 1e4, 3e38, np.inf, 1e-30, 1e-40], np.float32) / np.float32(factor)
    v = np.concatenate([edges, -edges, [np.nan], rng.uniform(-110, 110, 6000), rng.uniform(-90, -86, 1000) / factor,
                        np.exp(rng.uniform(-80, 6, 1000)) * rng.choice([-1, 1], 1000)]).astype(np.float32)
    n = v.size + -v.size % 8
    v = np.pad(v, (0, n - v.size))
    got = run_gemm(t0, rt, np.zeros((1, 64), np.float32), np.zeros((n, 64), np.float32), 1, n, 64, bias=v, tile_epilogue=["bias", op])[0]
    # CUDA's exp2 and its correctly rounded quotient: the reciprocal is one unit off at most, the product rounds once more
    x = torch.from_numpy(v).cuda()
    z = x * factor if factor != 1.0 else x
    s = 1.0 / (torch.exp2(-z * 1.4426950408889634) + 1.0)
    want, s = (x * s).cpu().numpy(), s.cpu().numpy()
    with np.errstate(invalid="ignore", over="ignore", under="ignore"):
        assert np.array_equal(np.isnan(got), np.isnan(want))
        fin = np.isfinite(want)
        assert np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)])
        gap = np.abs(v[fin]).astype(np.float64) * np.spacing(s[fin]) + np.spacing(np.abs(want[fin]))
        assert np.all(np.abs(got[fin].astype(np.float64) - want[fin]) <= gap)
        # and 64 bits: the exponential's argument carries |z| roundings of 2^-24 (its factor another quarter, GELU's product another whole one), its value
        # 2 units, the sum, the reciprocal and the product one each; where 1 + e overflows (z < -88.7) a sigmoid below 2^-127.9 becomes zero
        x64, z64 = v[fin].astype(np.float64), v[fin].astype(np.float64) * factor
        exact = x64 / (1.0 + np.exp(-np.clip(z64, -700, 700)))
        assert np.all(np.abs(got[fin] - exact) <= np.abs(exact) * (1.25 * np.abs(z64) + 4) * 2.0 ** -23
                      + np.where(z64 < -88.7, np.abs(x64) * 2.0 ** -127.9, (np.abs(x64) + 1) * 2.0 ** -149))


@pytest.mark.parametrize("tile_n,split_k", [(64, 2), (64, 4), (64, 8), (128, 2), (128, 8)])
@pytest.mark.parametrize("m,n,k", [(40, 72, 1088), (150, 330, 1088), (1500, 1300, 512)])
@pytest.mark.parametrize("out_bf16", [False, True])
def test_split_k_with_several_tiles_per_cluster(t0, rt, tile_n, split_k, m, n, k, out_bf16):
    # the form in which a cluster walks a list of tiles: parts that are not whole 64-deep blocks of K (1088 / split), and more clusters than run at
    # once (64- and 128-wide tiles of 1500 x 1300)
    rng = np.random.default_rng(n)
    x, b, bias = ints(rng, m, k), ints(rng, n, k), ints(rng, n, lim=100)
    before = rt.launch_count()
    got = run_gemm(t0, rt, x, b, m, n, k, out_bf16, bias, tile_n=tile_n, split_k=split_k, pair_cta=2, epilogue=t0.EPI_BIAS_ADD_STORE_F32)
    assert rt.launch_count() - before == 1
    want = x @ b.T + bias
    assert np.array_equal(got, from_bf16(bf16_bits(want)) if out_bf16 else want)


# Pair tiles of 128 columns: as asked for (B[N,K]; over B[K,N] single CTAs run in their place), and as the library's own choice in either layout, which sums K
# in two accumulators (odd numbers of k blocks, one ragged; more tiles than pairs, the last wave cut).  Integer operands: exact whatever the order.
@pytest.mark.parametrize("layout", ["nt", "nn"])
@pytest.mark.parametrize("m,n,k,fixed", [(300, 264, 64, True), (257, 1000, 200, True), (1500, 2056, 136, True), (2048, 1024, 4096, False), (1664, 1056, 3248, False)])
def test_pair_tiles_128_wide(t0, rt, layout, m, n, k, fixed):
    rng = np.random.default_rng(n)
    x, b = ints(rng, m, k), ints(rng, *((k, n) if layout == "nn" else (n, k)))
    kw = {"tile_n": 128, "pair_cta": 1} if fixed else {}
    got = run_gemm(t0, rt, x, b, m, n, k, transpose=t0.NN if layout == "nn" else t0.NT, **kw)
    assert np.array_equal(got, x @ (b if layout == "nn" else b.T))


# The library's own choice of those tiles with two accumulators (test_kernel_choice.py asserts it for these shapes): a bias and ReLU on the sum of both, bf16
# results, odd N, a ragged last k block; more tiles than pairs, the tiles of the last wave cut in two.
@pytest.mark.parametrize("layout,m,n,k,out_bf16", [("nt", 280, 3339, 2036, True), ("nn", 280, 3339, 2040, True), ("nt", 263, 3318, 2218, True), ("nn", 263, 3320, 2218, False),
                                                   ("nn", 768, 2048, 4096, True), ("nt", 645, 7493, 4864, False)])
def test_pair_tiles_128_wide_with_two_accumulators(t0, rt, layout, m, n, k, out_bf16):
    rng = np.random.default_rng(m + n)
    x, b, bias = ints(rng, m, k), ints(rng, *((k, n) if layout == "nn" else (n, k))), ints(rng, n, lim=100)
    got = run_gemm(t0, rt, x, b, m, n, k, out_bf16, bias, transpose=t0.NN if layout == "nn" else t0.NT, epilogue=t0.EPI_BIAS_ADD_RELU_STORE_F32)
    want = np.maximum(x @ (b if layout == "nn" else b.T) + bias, 0)
    assert np.array_equal(got, from_bf16(bf16_bits(want)) if out_bf16 else want)


# The same tiles over a first operand that is read transposed: dW = X^T dY, [k, n] summed over m.
@pytest.mark.parametrize("m,k,n", [(4096, 2048, 1024), (2218, 263, 3320)])
def test_transposed_operand_on_pair_tiles_128_wide(t0, rt, m, k, n):
    rng = np.random.default_rng(m)
    x, dy = ints(rng, m, k), ints(rng, m, n)
    xd, yd, dw = rt.upload(x), rt.upload(dy), rt.alloc(k * n * 4)
    rt.matmul_f32_backward_weight(xd.gpu_addr(), yd.gpu_addr(), dw.gpu_addr(), m, k, n)
    assert np.array_equal(rt.read_f32(dw, k * n).reshape(k, n), x.T @ dy)
    for buf in (xd, yd, dw):
        buf.free()
