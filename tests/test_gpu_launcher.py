"""Repeated operator calls with packed weights run through the launcher (unit_b200/csrc/host_ext.cpp): a call
of a geometry it has seen must read the buffers it is given, and calls it does not know must be checked as before."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def U():
    import unit_b200
    return unit_b200


def gen(seed):
    return torch.Generator(device='cuda').manual_seed(seed)


def u8(shape, g):
    return torch.randint(0, 256, shape, dtype=torch.uint8, device='cuda', generator=g)


# operands described by a tensor map (re-addressed on each call), below its size limit (gathered), folded through
# scratch, and the operators with float outputs
CONV = [dict(x=(1, 4, 56, 56, 16), w=(4, 4, 3, 3, 4, 16, 4), stride=1, padding=1),
        dict(x=(2, 4, 9, 9, 16), w=(4, 4, 3, 3, 4, 16, 4), stride=2, padding=(1, 1)),
        dict(x=(3, 1, 64, 64, 4), w=(4, 1, 7, 7, 1, 16, 4), stride=2, padding=3)]


@pytest.mark.parametrize('case', CONV)
@pytest.mark.parametrize('form', ['raw', 'requant', 'residual'])
def test_conv2d_calls_read_their_own_buffers(U, case, form):
    g = gen(5)
    w = torch.randint(-128, 128, case['w'], dtype=torch.int8, device='cuda', generator=g)
    kw = dict(stride=case['stride'], padding=case['padding'])
    pw = U.pack_conv_weights_int8(w, **kw)
    for i in range(4):
        x = u8(case['x'], g)
        opt = dict(kw)
        if form != 'raw':
            opt.update(bias=torch.randint(-2 ** 12, 2 ** 12, (64,), dtype=torch.int32, device='cuda', generator=g),
                       out_dtype='uint8', requant_shift=9)
        if form == 'residual':
            acc = U.conv2d_NCHWc_int8(x, pw, **kw)
            opt['residual'] = u8(tuple(acc.shape), g)
        got = U.conv2d_NCHWc_int8(x, pw, **opt)
        want = U.conv2d_NCHWc_int8_plan(x, pw, **opt).run()     # planned anew for these buffers
        named = torch.empty_like(got)
        assert U.conv2d_NCHWc_int8(x, pw, out=named, **opt) is named
        assert U.conv2d_NCHWc_int8(x, pw, out=named, **opt) is named
        assert torch.equal(got, want) and torch.equal(named, want)
        assert got.data_ptr() != x.data_ptr()
    with torch.cuda.stream(torch.cuda.Stream()) as _:           # another stream waits for the weights first
        torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
        for _ in range(2):
            assert torch.equal(U.conv2d_NCHWc_int8(x, pw, **opt), want)
    with pytest.raises(ValueError):
        U.conv2d_NCHWc_int8(x[..., :4].contiguous() if x.shape[-1] == 16 else x.repeat(1, 1, 1, 1, 4), pw, **kw)
    U.device_status()


@pytest.mark.parametrize('m', [1, 70, 300])
def test_products_and_fp16_convolutions_read_their_own_buffers(U, m):
    g = gen(6)
    wq = torch.randint(-128, 128, (4, 256, 16, 4), dtype=torch.int8, device='cuda', generator=g)
    pd = U.pack_dense_weights_int8(wq)
    dense = wq.permute(0, 2, 1, 3).reshape(64, 1024)
    bf = torch.randn((512, 64), device='cuda', generator=g).half()
    pg = U.pack_gemm_weights_f16(bf)
    wf = torch.randn((2, 2, 3, 3, 16, 16), device='cuda', generator=g).half()
    pf = U.pack_conv_weights_f16(wf)
    wc = wf.permute(0, 5, 1, 4, 2, 3).reshape(32, 32, 3, 3).double()
    for i in range(3):
        a = u8((m, 1024), g)
        assert np.array_equal(U.dense_dotprod(a, pd).cpu().numpy(), (a.cpu().to(torch.int64) @ dense.cpu().to(torch.int64).T).numpy())
        ah = torch.randn((m, 512), device='cuda', generator=g).half()
        # 512 products of fp16 values are exact in fp32; their fp32 sum is off by at most 512 * 2^-24 of the absolute sum
        bound = 512 * 2.0 ** -24 * (ah.double().abs() @ bf.double().abs()) + 1e-30
        assert bool(((U.gemm_f16f32(ah, pg).double() - ah.double() @ bf.double()).abs() <= bound).all())
        x = torch.randn((m % 7 + 1, 2, 12, 12, 16), device='cuda', generator=g).half()
        xc = x.permute(0, 1, 4, 2, 3).reshape(x.shape[0], 32, 12, 12).double()
        got = U.conv2d_NCHW16c_OHWI16o(x, pf, 1, 1, padding=1).permute(0, 1, 4, 2, 3).reshape(x.shape[0], 32, 12, 12).double()
        want = torch.nn.functional.conv2d(xc, wc, padding=1)
        bound = 288 * 2.0 ** -24 * torch.nn.functional.conv2d(xc.abs(), wc.abs(), padding=1) + 1e-30
        assert bool(((got - want).abs() <= bound).all())
    U.device_status()


class Calls:
    """Counts the calls that take the operator's own checks instead of a kept plan."""

    def __init__(self, monkeypatch):
        from unit_b200 import ops
        self.n = 0
        prepare = ops._conv_int8_prepare

        def counted(*a):
            self.n += 1
            return prepare(*a)
        monkeypatch.setattr(ops, '_conv_int8_prepare', counted)


def conv_case(U, case, g):
    w = torch.randint(-128, 128, case['w'], dtype=torch.int8, device='cuda', generator=g)
    kw = dict(stride=case['stride'], padding=case['padding'])
    return U.pack_conv_weights_int8(w, **kw), kw


@pytest.mark.parametrize('case', CONV)
def test_any_number_of_named_outputs_and_inputs(U, case, monkeypatch):
    g = gen(7)
    pw, kw = conv_case(U, case, g)
    xs = [u8(case['x'], g) for _ in range(3)]
    want = [U.conv2d_NCHWc_int8_plan(x, pw, **kw).run() for x in xs]
    ring = [torch.empty_like(want[0]) for _ in range(40)]
    calls = Calls(monkeypatch)
    for _ in range(2):
        for i, out in enumerate(ring):
            out.zero_()
            assert U.conv2d_NCHWc_int8(xs[i % 3], pw, out=out, **kw) is out
        for i, out in enumerate(ring):
            assert torch.equal(out, want[i % 3])
    assert calls.n == 1
    U.device_status()


@pytest.mark.parametrize('case', CONV)
@pytest.mark.parametrize('named', [False, True])
def test_streams_that_take_turns(U, case, named, monkeypatch):
    """One plan serves every stream; the folded stem's scratch is each stream's own."""
    g = gen(8)
    pw, kw = conv_case(U, case, g)
    x = [u8(case['x'], g) for _ in range(2)]
    want = [U.conv2d_NCHWc_int8_plan(t, pw, **kw).run() for t in x]
    out = [torch.empty_like(t) for t in want]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    calls = Calls(monkeypatch)
    for _ in range(6):
        for s in (0, 1):
            with torch.cuda.stream(streams[s]):
                got = U.conv2d_NCHWc_int8(x[s], pw, out=out[s] if named else None, **kw)
                assert torch.equal(got, want[s])
    assert calls.n == 2     # each stream's first call (it waits for the weights and gets its scratch)
    U.device_status()


def test_an_allocation_that_fails_is_torch_s_out_of_memory_error(U):
    """On repeated calls as on the first, so that a caller can free memory and try again."""
    g = gen(9)
    pw, kw = conv_case(U, dict(w=(4, 4, 3, 3, 4, 16, 4), stride=1, padding=1), g)
    x = u8((64, 4, 56, 56, 16), g)
    nchw = u8((64, 64, 56, 56), g)
    runs = [lambda: U.conv2d_NCHWc_int8(x, pw, **kw), lambda: U.pack_data_nchwc(nchw), lambda: U.unpack_data_nchwc(x)]
    want = [f().cpu() for f in runs]
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + 2 ** 20) / total)
    try:
        for f in runs:
            with pytest.raises(torch.OutOfMemoryError):
                f()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for f, t in zip(runs, want):
        assert torch.equal(f().cpu(), t)
    U.device_status()


def test_only_calls_with_packed_weights_pay_for_a_launcher(U):
    """Packing makes none, nor does a call that packs raw weights itself (its next call cannot use it)."""
    from unit_b200 import ops
    g = gen(10)
    w8 = torch.randint(-128, 128, (4, 4, 3, 3, 4, 16, 4), dtype=torch.int8, device='cuda', generator=g)
    wd = torch.randint(-128, 128, (4, 256, 16, 4), dtype=torch.int8, device='cuda', generator=g)
    wf = torch.randn((2, 2, 3, 3, 16, 16), device='cuda', generator=g).half()
    bg = torch.randn((512, 64), device='cuda', generator=g).half()
    x8, xd = u8((2, 4, 20, 20, 16), g), u8((70, 1024), g)
    xf, xg = torch.randn((2, 2, 12, 12, 16), device='cuda', generator=g).half(), torch.randn((70, 512), device='cuda', generator=g).half()
    for pack, w, call in ((lambda w: U.pack_conv_weights_int8(w, 1, 1), w8, lambda w: U.conv2d_NCHWc_int8(x8, w, padding=1)),
                          (U.pack_dense_weights_int8, wd, lambda w: U.dense_dotprod(xd, w)),
                          (U.pack_conv_weights_f16, wf, lambda w: U.conv2d_NCHW16c_OHWI16o(xf, w, 1, 1, padding=1)),
                          (U.pack_gemm_weights_f16, bg, lambda w: U.gemm_f16f32(xg, w))):
        raw = [call(w) for _ in range(2)]
        pw = pack(w)                                  # (the tensor's packed copy is cached: the one these calls used)
        assert pw._launcher is None
        n = ops.launch_count()
        packed = [call(pw) for _ in range(3)]
        assert ops.launch_count() == n + 3 and pw._launcher is not None
        for t in raw + packed:
            assert torch.equal(t, raw[0])
    U.device_status()


@pytest.mark.parametrize('case', CONV)
def test_the_first_call_of_a_thread_runs_the_kept_plan(U, case, monkeypatch):
    """A thread that has not used CUDA yet has no current context, which re-addressing a tensor map needs."""
    import threading
    g = gen(15)
    pw, kw = conv_case(U, case, g)
    xs = [u8(case['x'], g) for _ in range(4)]
    want = [U.conv2d_NCHWc_int8_plan(x, pw, **kw).run() for x in xs]
    U.conv2d_NCHWc_int8(xs[0], pw, **kw)
    torch.cuda.synchronize()
    calls, got = Calls(monkeypatch), {}
    for i, x in enumerate(xs):
        t = threading.Thread(target=lambda: got.update({i: U.conv2d_NCHWc_int8(x, pw, **kw)}))
        t.start()
        t.join()
        assert torch.equal(got[i], want[i])
    assert calls.n == 0
    U.device_status()


def test_a_stream_that_syncs_while_the_launcher_is_made(U, monkeypatch):
    """Two threads make their first calls with the same weights at once: the launcher knows both streams."""
    import threading
    g = gen(16)
    pw, kw = conv_case(U, CONV[0], g)
    x = u8(CONV[0]['x'], g)
    want = U.conv2d_NCHWc_int8_plan(x, pw, **kw).run()
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    calls = Calls(monkeypatch)

    def on_other():
        with torch.cuda.stream(other):
            assert torch.equal(U.conv2d_NCHWc_int8(x, pw, **kw), want)

    class Streams(set):
        thread = None

        def __iter__(self):     # (the launcher is being told the streams: the other thread's first call comes now)
            known = list(set.__iter__(self))
            if Streams.thread is None:
                Streams.thread = threading.Thread(target=on_other)
                Streams.thread.start()
                Streams.thread.join(0.5)
            return iter(known)

    pw._synced = Streams(pw._synced)
    U.conv2d_NCHWc_int8(x, pw, **kw)
    Streams.thread.join()
    n = calls.n
    for _ in range(3):
        on_other()
    assert n == 2 and calls.n == n
    U.device_status()


@pytest.mark.parametrize('case', CONV)
def test_threads_share_packed_weights(U, case, monkeypatch):
    """Each on its own stream with its own buffers, from the first call on; afterwards all of them run kept plans."""
    import threading
    g = gen(11)
    xs = [u8(case['x'], g) for _ in range(4)]
    calls = Calls(monkeypatch)
    for round_ in range(4):
        pw, kw = conv_case(U, case, g)
        want = [U.conv2d_NCHWc_int8_plan(x, pw, **kw).run() for x in xs]
        torch.cuda.synchronize()
        barrier, errors, streams = threading.Barrier(4), [], [torch.cuda.Stream() for _ in range(4)]

        def work(i, reps):
            try:
                with torch.cuda.stream(streams[i]):
                    barrier.wait()
                    for _ in range(reps):
                        assert torch.equal(U.conv2d_NCHWc_int8(xs[i], pw, **kw), want[i])
            except Exception as e:   # noqa: BLE001  (a thread's failure is the test's)
                errors.append(e)

        for reps in (3, 20):
            n = calls.n
            threads = [threading.Thread(target=work, args=(i, reps)) for i in range(4)]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
            assert not errors, errors
        assert calls.n == n     # the second time no call needed the checks
    U.device_status()


def test_calls_of_a_known_geometry_are_captured(U):
    g = gen(12)
    for case in CONV:
        pw, kw = conv_case(U, case, g)
        x = u8(case['x'], g)
        out = torch.empty_like(U.conv2d_NCHWc_int8(x, pw, **kw))
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            U.conv2d_NCHWc_int8(x, pw, **kw)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            inner = U.conv2d_NCHWc_int8(x, pw, **kw)
            U.conv2d_NCHWc_int8(x, pw, out=out, **kw)
        for _ in range(2):
            x.copy_(u8(case['x'], g))
            graph.replay()
            want = U.conv2d_NCHWc_int8_plan(x, pw, **kw).run()
            assert torch.equal(inner, want) and torch.equal(out, want)
    U.device_status()


def test_more_geometries_than_are_kept(U, monkeypatch):
    g = gen(13)
    pw, _ = conv_case(U, dict(w=(4, 4, 3, 3, 4, 16, 4), stride=1, padding=1), g)
    calls = Calls(monkeypatch)
    for n_seen, h in enumerate(list(range(5, 75)) + [5, 74]):
        x = u8((1, 4, h, 7, 16), g)
        for _ in range(2):
            assert torch.equal(U.conv2d_NCHWc_int8(x, pw, padding=1), U.conv2d_NCHWc_int8_plan(x, pw, padding=1).run())
    # per geometry one call with the checks (the other prepared launch is the reference); the oldest one was evicted
    assert calls.n == 72 * 2 + 71
    U.device_status()


def test_a_new_tile_table_plans_anew(U, monkeypatch):
    from unit_b200 import tile_table
    g = gen(14)
    pw, kw = conv_case(U, dict(w=(4, 4, 3, 3, 4, 16, 4), stride=1, padding=1), g)
    x = u8((2, 4, 28, 28, 16), g)
    want = U.conv2d_NCHWc_int8(x, pw, **kw)
    calls = Calls(monkeypatch)
    try:
        tile_table.set_table([dict(c_in=64, c_out=64, kh=3, kw=3, stride_h=1, stride_w=1, n=2, h=28, w=28, mt=1, ksplit=1)])
        for _ in range(2):
            assert torch.equal(U.conv2d_NCHWc_int8(x, pw, **kw), want)
        assert calls.n == 1
    finally:
        tile_table.load_default_table()
    assert torch.equal(U.conv2d_NCHWc_int8(x, pw, **kw), want) and calls.n == 2
    U.device_status()
