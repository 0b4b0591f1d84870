"""GPU tests of launches recorded into a CUDA graph (stream capture of the runtime's stream) and replayed: later calls of the runtime may
run larger products first, the replay may run on another stream beside the runtime's own, and nothing may be allocated while recording.
"""
import contextlib
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Driver:
    """The few driver calls a program needs to record a stream and replay the graph (the library has no entry for it)."""

    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        ctx = C.c_void_p()
        self.call("cuDevicePrimaryCtxRetain", C.byref(ctx), 0)
        self.call("cuCtxSetCurrent", ctx)

    def call(self, name, *args):
        rc = getattr(self.cu, name)(*args)
        assert rc == 0, f"{name} returned {rc}"

    @contextlib.contextmanager
    def record(self, rt):
        """Records what the block launches on the runtime's stream; the yielded list then holds the executable graph."""
        out, graph, stream = [], C.c_void_p(), C.c_void_p(rt.stream())
        self.call("cuStreamBeginCapture_v2", stream, 0)                      # 0 = global mode: an allocation would be refused
        try:
            yield out
        finally:
            rc = self.cu.cuStreamEndCapture(stream, C.byref(graph))
        assert rc == 0, f"the capture was invalidated ({rc})"
        ex = C.c_void_p()
        self.call("cuGraphInstantiateWithFlags", C.byref(ex), graph, C.c_ulonglong(0))
        self.call("cuGraphDestroy", graph)
        out.append(ex)

    def replay(self, ex, stream):
        self.call("cuGraphLaunch", ex, C.c_void_p(stream))

    def stream(self):
        s = C.c_void_p()
        self.call("cuStreamCreate", C.byref(s), 1)                           # 1 = does not synchronise with the default stream
        return s.value

    def sync(self, stream):
        self.call("cuStreamSynchronize", C.c_void_p(stream))

    def drop(self, ex=None, stream=None):
        if ex is not None:
            self.call("cuGraphExecDestroy", ex)
        if stream is not None:
            self.call("cuStreamDestroy_v2", C.c_void_p(stream))


@pytest.fixture()
def driver(rt):
    return Driver()


@pytest.fixture()
def fresh(t0):
    """A runtime of its own: no buffer has grown yet."""
    r = t0.GpuRuntime(0)
    yield r
    r.close()


def bf16_bits(v):
    u = np.ascontiguousarray(v, np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)


class Product:
    """One bf16 product on the runtime: real-valued operands, so that another order of the sums would show in the bits."""

    def __init__(self, t0, rt, m, n, k, seed, layout="nt", out_bf16=False, **kw):
        rng = np.random.default_rng(seed)
        self.rt, self.dims, self.words = rt, (m, n, k), m * n // (2 if out_bf16 else 1)
        self.kw = dict(kw, out_bf16=out_bf16, transpose=t0.NN if layout == "nn" else t0.NT)
        self.x, self.b = (rt.upload(bf16_bits(rng.uniform(-1, 1, c))) for c in (m * k, n * k))
        self.ys = []

    def out(self):
        self.ys.append(self.rt.alloc(self.words * 4))
        self.ys[-1].write(np.full(self.words, 0xFFFFFFFF, np.uint32))
        return self.ys[-1]

    def launch(self, y):
        self.rt.gemm(self.x.gpu_addr(), self.b.gpu_addr(), y.gpu_addr(), *self.dims, **self.kw)

    def eager(self):
        y = self.out()
        self.launch(y)
        self.rt.synchronize()
        return self.bits(y)

    def bits(self, y):
        return y.read(self.words * 4, np.uint32)

    def free(self):
        for buf in [self.x, self.b] + self.ys:
            buf.free()


# products whose K the library cuts: two to eight parts, tiles of 32, 64 and 128 columns, an odd number of k blocks, a ragged last chunk
CUT = [(16, 2048, 2048), (64, 4096, 4096), (32, 752, 3984), (128, 4096, 2048), (128, 4096, 4096), (512, 512, 2048), (100, 296, 8192), (64, 512, 8192), (16, 40, 10240)]


@pytest.mark.parametrize("layout", ["nt", "nn"])
@pytest.mark.parametrize("out_bf16", [False, True])
def test_recorded_products_equal_eager_ones(t0, fresh, driver, layout, out_bf16):
    # recorded on a fresh runtime (nothing reserved, nothing run), then larger products on the runtime, then the replay
    cases = [Product(t0, fresh, m, n, k, seed=m + n, layout=layout, out_bf16=out_bf16) for m, n, k in CUT]
    ys = [p.out() for p in cases]
    with driver.record(fresh) as graphs:
        for p, y in zip(cases, ys):
            p.launch(y)
    larger = [Product(t0, fresh, m, n, k, seed=1, layout=layout) for m, n, k in [(128, 4736, 8192), (256, 2048, 8192), (2048, 2048, 4096)]]
    for p in larger:
        p.eager()
    want = [p.eager() for p in cases]
    for _ in range(3):
        for y, p in zip(ys, cases):
            y.write(np.full(p.words, 0xFFFFFFFF, np.uint32))
        driver.replay(graphs[0], fresh.stream())
        fresh.synchronize()
        for p, y, w in zip(cases, ys, want):
            assert np.array_equal(p.bits(y), w), p.dims
    driver.drop(graphs[0])
    for p in cases + larger:
        p.free()


@pytest.mark.parametrize("layout,kw", [("nt", dict(tile_n=32, split_k=4)), ("nt", dict(tile_n=64, split_k=2)), ("nt", dict(tile_n=64, split_k=8)), ("nt", dict(tile_n=128, split_k=8)),
                                       ("nt", dict(tile_n=256, split_k=4)), ("nn", dict(tile_n=64, split_k=4)), ("nn", dict(tile_n=128, split_k=2)),
                                       ("nn", dict(tile_n=256, split_k=2)), ("nt", dict(tile_n=128, split_k=4))])
@pytest.mark.parametrize("m,n,k", [(40, 328, 2048), (200, 520, 1024)])
def test_recorded_splits_of_the_caller(t0, fresh, driver, layout, kw, m, n, k):
    p = Product(t0, fresh, m, n, k, seed=3, layout=layout, pair_cta=2, **kw)
    y = p.out()
    with driver.record(fresh) as graphs:
        p.launch(y)
    want = p.eager()
    driver.replay(graphs[0], fresh.stream())
    fresh.synchronize()
    assert np.array_equal(p.bits(y), want)
    driver.drop(graphs[0])
    p.free()


@pytest.mark.parametrize("kw", [dict(tile_n=64, split_k=2), dict(tile_n=128, split_k=4), dict(tile_n=128, split_k=8)])
def test_recorded_splits_of_narrow_pairs_over_kn(t0, fresh, driver, kw):
    # pair tiles of 128 columns or less asked for over B[K,N], K cut: one launch that needs no buffer, so it is recorded on a runtime that has none
    p = Product(t0, fresh, 300, 520, 1024, seed=13, layout="nn", pair_cta=1, **kw)
    y = p.out()
    before = fresh.launch_count()
    with driver.record(fresh) as graphs:
        p.launch(y)
    assert fresh.launch_count() - before == 1
    want = p.eager()
    driver.replay(graphs[0], fresh.stream())
    fresh.synchronize()
    assert np.array_equal(p.bits(y), want)
    driver.drop(graphs[0])
    p.free()


@pytest.mark.parametrize("layout", ["nt", "nn"])
def test_replays_beside_the_runtime_s_own_stream(t0, fresh, driver, layout):
    # two graphs of the same product on two streams, and the product itself on the runtime's stream, all under way together
    m, n, k = 16, 1024, 4096
    p = Product(t0, fresh, m, n, k, seed=9, layout=layout)
    want = p.eager()
    streams, execs, outs = [driver.stream() for _ in range(2)], [], []
    for _ in range(2):
        ys = [p.out() for _ in range(20)]
        with driver.record(fresh) as graphs:
            for y in ys:
                p.launch(y)
        execs.append(graphs[0])
        outs.append(ys)
    own = [p.out() for _ in range(20)]
    for _ in range(5):
        for ex, s in zip(execs, streams):
            driver.replay(ex, s)
        for y in own:
            p.launch(y)
    for s in streams:
        driver.sync(s)
    fresh.synchronize()
    for y in outs[0] + outs[1] + own:
        assert np.array_equal(p.bits(y), want)
    for ex, s in zip(execs, streams):
        driver.drop(ex, s)
    p.free()


def test_recorded_training_step(t0, fresh, driver):
    # dW reads X as [K, M]; the eager step before the recording makes the conversion buffers
    m, k, n = 2048, 128, 256
    rng = np.random.default_rng(2)
    x, w, dy = (fresh.upload(rng.uniform(-1, 1, s).astype(np.float32)) for s in ((m, k), (k, n), (m, n)))
    sizes = (m * n, m * k, k * n)
    eager, replayed = ([fresh.alloc(4 * c) for c in sizes] for _ in range(2))

    def step(ys):
        fresh.matmul_f32(x.gpu_addr(), w.gpu_addr(), ys[0].gpu_addr(), m, k, n)
        fresh.matmul_f32_backward_data(dy.gpu_addr(), w.gpu_addr(), ys[1].gpu_addr(), m, k, n)
        fresh.matmul_f32_backward_weight(x.gpu_addr(), dy.gpu_addr(), ys[2].gpu_addr(), m, k, n)

    step(eager)
    with driver.record(fresh) as graphs:
        step(replayed)
    driver.replay(graphs[0], fresh.stream())
    fresh.synchronize()
    for a, b, c in zip(eager, replayed, sizes):
        assert np.array_equal(a.read(4 * c, np.uint32), b.read(4 * c, np.uint32))
    driver.drop(graphs[0])
    for buf in [x, w, dy] + eager + replayed:
        buf.free()


def test_recorded_part_that_never_arrives_ends_with_an_error(t0, fresh, driver):
    # the first operand load of one part is left out: its cluster gives up after the wait limit, in every CTA, and the error is reported
    p = Product(t0, fresh, 16, 2048, 2048, seed=4)
    y = p.out()
    fresh.set_wait_limit_ns(20_000_000)
    fresh.selftest_drop_one_load()
    with driver.record(fresh) as graphs:
        p.launch(y)
    driver.replay(graphs[0], fresh.stream())
    with pytest.raises(t0.T0Error):
        fresh.synchronize()
    assert fresh.is_poisoned()
    driver.drop(graphs[0])
    p.free()


def test_recording_without_room_is_refused_and_goes_on(t0, fresh, driver):
    # a split into planes (no one-launch form: pair tiles) and a product with a padded operand need buffers: refused while recording, the capture
    # and the runtime stay usable; reserved, they are recorded and replay like the eager calls
    planes = Product(t0, fresh, 300, 512, 1024, seed=5, pair_cta=1, tile_n=256, split_k=2)
    padded = Product(t0, fresh, 40, 72, 1001, seed=6)
    plain = Product(t0, fresh, 64, 64, 512, seed=7)
    outs = [p.out() for p in (planes, padded, plain)]
    with driver.record(fresh) as graphs:
        for p, y in ((planes, outs[0]), (padded, outs[1])):
            with pytest.raises(t0.T0Error) as e:
                p.launch(y)
            assert e.value.code == 6
        plain.launch(outs[2])
    driver.replay(graphs[0], fresh.stream())
    fresh.synchronize()
    assert np.array_equal(plain.bits(outs[2]), plain.eager())
    driver.drop(graphs[0])
    fresh.reserve_scratch("splitk_planes", 300 * 512 * 2 * 4)
    fresh.reserve_scratch("operand_a", 40 * 1008 * 2)
    fresh.reserve_scratch("operand_b", 72 * 1008 * 2)
    with driver.record(fresh) as graphs:
        planes.launch(outs[0])
        padded.launch(outs[1])
    want = planes.eager(), padded.eager()
    driver.replay(graphs[0], fresh.stream())
    fresh.synchronize()
    assert np.array_equal(planes.bits(outs[0]), want[0]) and np.array_equal(padded.bits(outs[1]), want[1])
    driver.drop(graphs[0])
    for p in (planes, padded, plain):
        p.free()


class Group:
    """W4A16 problems of one shape whose column tiles are cut between CTAs in an eager call; `bound` = f32 sums in any order."""

    def __init__(self, t0, oracle, rt, M, K, N, count, G=128):
        self.rt, self.M, self.N, self.K, self.bufs, self.args, self.refs = rt, M, N, K, [], [], []
        for i in range(count):
            packed, scales, zeros = oracle.fill_u32((K // 8) * N, 10 + i), oracle.fill_range_bf16((K // G) * N, 20 + i, 0.001, 0.02), oracle.fill_u32((K // G) * (N // 8), 30 + i)
            a = oracle.fill_normal_bf16(M * K, 40 + i)
            w = np.abs(oracle.bf16_to_f32(oracle.dequant_w4_b200(packed, scales, zeros, K, N, G)).reshape(K, N))
            bound = np.abs(oracle.bf16_to_f32(a).reshape(M, K)).astype(np.float64) @ w * (K * 2.0 ** -24)
            self.refs.append((oracle.w4a16_gemm(a, packed, scales, zeros, M, N, K, G).astype(np.float64), bound))
            p, s, z, x = rt.upload(packed), rt.upload(scales), rt.upload(zeros), rt.upload(a)
            t = rt.w4_to_tiled(p.gpu_addr(), s.gpu_addr(), z.gpu_addr(), K, N, G)
            self.bufs += [p, s, z, x, t]
            self.rows = p, s, z, x
            self.args.append(lambda y, x=x, t=t: t0.W4A16Args(x.gpu_addr(), t.gpu_addr(), 0, 0, y.gpu_addr(), M, N, K, G))

    def outs(self):
        ys = [self.rt.alloc(self.M * self.N * 4) for _ in self.args]
        for y in ys:
            y.write(np.full(self.M * self.N, np.nan, np.float32))
        self.bufs += ys
        return ys

    def launch(self, ys):
        self.rt.w4a16_gemm_tiled_grouped([a(y) for a, y in zip(self.args, ys)])

    def launch_row_layout(self, y):
        p, s, z, x = self.rows
        self.rt.w4a16_gemm(x.gpu_addr(), p.gpu_addr(), s.gpu_addr(), z.gpu_addr(), y.gpu_addr(), self.M, self.N, self.K, 128)

    def check(self, ys):
        for y, (ref, bound) in zip(ys, self.refs):
            assert np.all(np.abs(y.read(self.M * self.N * 4, np.float32).reshape(self.M, self.N) - ref) <= bound)

    def free(self):
        for b in self.bufs:
            b.free()


def test_recorded_w4a16_group_beside_eager_ones(t0, oracle, fresh, driver):
    # recorded before the runtime has cut a tile, and again after: the replays run on another stream beside eager calls
    g = Group(t0, oracle, fresh, 40, 4096, 2560, 2)
    stream, execs, outs = driver.stream(), [], []
    for _ in range(2):
        ys = g.outs()
        with driver.record(fresh) as graphs:
            for _ in range(5):
                g.launch(ys)
        execs.append(graphs[0])
        outs.append(ys)
        outs.append(g.outs())
        g.launch(outs[-1])                                                    # eager
    for _ in range(10):
        for ex in execs:
            driver.replay(ex, stream)
        g.launch(outs[-1])
    driver.sync(stream)
    fresh.synchronize()
    for ys in outs:
        g.check(ys)
    driver.drop(execs[0])
    driver.drop(execs[1], stream)
    g.free()


@pytest.mark.parametrize("row_layout", [False, True])
def test_recorded_single_w4a16_problem_beside_eager_ones(t0, oracle, fresh, driver, row_layout):
    # one problem that an eager call cuts between CTAs: recorded it runs as clusters, without the buffer, so its replays may run beside eager calls
    g = Group(t0, oracle, fresh, 20, 2048, 2560, 1)
    launch = (lambda ys: g.launch_row_layout(ys[0])) if row_layout else g.launch
    stream, recorded, eager = driver.stream(), g.outs(), g.outs()
    with driver.record(fresh) as graphs:
        for _ in range(5):
            launch(recorded)
    for _ in range(10):
        driver.replay(graphs[0], stream)
        for _ in range(5):
            launch(eager)
    driver.sync(stream)
    fresh.synchronize()
    g.check(recorded), g.check(eager)
    driver.drop(graphs[0], stream)
    g.free()


def test_reserved_w4a16_calls_allocate_nothing(t0, oracle, rt, driver):
    # what t0_rt_w4_fused_scratch_bytes names covers every fused call of a runtime; a smaller reservation the calls with M <= 16
    def free_bytes():
        rt.synchronize()
        f, t = C.c_size_t(), C.c_size_t()
        driver.call("cuMemGetInfo_v2", C.byref(f), C.byref(t))
        return f.value

    one, many = Group(t0, oracle, rt, 4, 4096, 2560, 1), Group(t0, oracle, rt, 128, 4096, 2560, 2)
    ys = [g.outs() for g in (one, many)]
    one.launch_row_layout(ys[0][0]), many.launch(ys[1])                       # (the kernels are loaded)
    rt.synchronize()
    r = t0.GpuRuntime(0)
    whole, before = r.w4_fused_scratch_bytes(), free_bytes()
    r.reserve_scratch("w4_fused", 0)
    small = before - free_bytes()
    assert small < whole // 4                                                 # (the room for cut tiles was made with the runtime)
    one.rt = many.rt = r
    at = free_bytes()
    one.launch_row_layout(ys[0][0])
    r.synchronize()
    assert free_bytes() == at
    r.reserve_scratch("w4_fused", whole)
    at = free_bytes()
    assert before - at <= whole + (8 << 20)                                   # (buffers are whole megabytes)
    one.launch_row_layout(ys[0][0]), many.launch(ys[1])
    r.synchronize()
    assert free_bytes() == at
    one.check(ys[0]), many.check(ys[1])
    r.close()
    one.rt = many.rt = rt
    one.free(), many.free()


@pytest.mark.parametrize("M,K,N", [(20, 2048, 2560), (128, 4096, 11008)])
def test_single_w4a16_calls_allocate_nothing(t0, oracle, rt, driver, M, K, N):
    # one problem of 16 < M <= 128, cut between CTAs or as clusters: the first call of a new runtime takes no memory, and further calls give the same bits
    def free_bytes():
        rt.synchronize()
        f, t = C.c_size_t(), C.c_size_t()
        driver.call("cuMemGetInfo_v2", C.byref(f), C.byref(t))
        return f.value

    g = Group(t0, oracle, rt, M, K, N, 1)
    ys = [g.outs() for _ in range(4)]
    g.launch(ys[0]), g.launch_row_layout(ys[0][0])                            # (the kernels are loaded)
    r = t0.GpuRuntime(0)
    g.rt = r
    at = free_bytes()
    for y in ys[:2]:
        g.launch(y)
    for y in ys[2:]:
        g.launch_row_layout(y[0])
    r.synchronize()
    assert free_bytes() == at
    for y in ys:
        g.check(y)
        assert np.array_equal(y[0].read(M * N * 4, np.uint32), ys[0][0].read(M * N * 4, np.uint32))
    r.close()
    g.rt = rt
    g.free()
