"""How the contraction kernel's work is cut, at the sizes where a cut can go wrong: reductions that end inside a
pipeline stage, row blocks and column blocks that are partly empty, the smallest and largest grids of a form."""
import numpy as np
import pytest
import torch

from oracle import np_oracle as no

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def U():
    import unit_b200
    return unit_b200


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def launched(run):
    """The result of run() and the names of the kernel variants it launched."""
    from unit_b200 import _lib
    L = _lib.lib()
    count = lambda: {i: L.unit_variant_launches(i) for i in range(L.unit_variant_count())}  # noqa: E731
    before = count()
    out = run()
    torch.cuda.synchronize()
    return out, [L.unit_variant_name(i).decode() for i, v in count().items() if v != before[i]]


def dense_case(U, m, n, k, seed=0):
    rng = np.random.default_rng(m + n + k + seed)
    a = rng.integers(0, 256, (m, k), dtype=np.uint8)
    b = rng.integers(-128, 128, (n, k), dtype=np.int8)
    got, names = launched(lambda: U.dense_dotprod(dev(a), dev(no.pack_dense_weights(b, 16))))
    U.device_status()
    # (float64 holds these integer sums exactly: |sum| <= 255 * 128 * k < 2^53)
    want = (dev(a).double() @ dev(b).double().t()).to(torch.int32)
    assert torch.equal(got, want)
    return names


def gemm_case(U, m, n, k):
    g = torch.Generator(device='cuda').manual_seed(m + n + k)
    a = torch.randn(m, k, device='cuda', generator=g).half()
    b = (torch.randn(k, n, device='cuda', generator=g) * 0.05).half()
    got, names = launched(lambda: U.gemm_f16f32(a, b))
    U.device_status()
    # fp32 sums of k exact products: |error| <= k 2^-24 sum |a b| in any order
    bound = k * 2.0 ** -24 * (a.double().abs() @ b.double().abs())
    assert bool(((got.double() - a.double() @ b.double()).abs() <= bound + 1e-30).all())
    return names


# reductions of whole 128-byte stages, one K step more, one column less, shorter than a stage
@pytest.mark.parametrize('m', [150, 2050])
@pytest.mark.parametrize('n,k', [(272, 1024), (272, 1040), (48, 1008), (2064, 1104), (16, 112), (528, 144)])
def test_dense_reductions_that_end_inside_a_stage(U, m, n, k):
    dense_case(U, m, n, k)


@pytest.mark.parametrize('m', [150, 2050])
@pytest.mark.parametrize('n,k', [(272, 1024), (272, 1032), (48, 1016), (2064, 520), (16, 56), (528, 72), (528, 456)])
def test_gemm_reductions_that_end_inside_a_stage(U, m, n, k):
    gemm_case(U, m, n, k)


# Reductions below one 128-byte stage arrive as 16-byte columns, two per K step.  With an odd number of columns the
# last step's second one exists in no matrix: it must read as zero whatever an earlier kernel left in shared memory
# (here: bytes that are NaN in fp16).  One and two sub-tiles per tile, a ragged last row block; even counts beside odd.
@pytest.mark.parametrize('m,n,k', [(8200, 64, 8), (40007, 64, 8), (2800, 272, 24), (40007, 32, 24), (1700, 48, 40), (20011, 128, 40),
                                   (8200, 64, 16), (2050, 528, 32), (1501, 64, 48)])
def test_gemm_column_copies_after_another_kernel(U, m, n, k):
    from unit_b200 import _lib
    # (the packed form shows which one runs: a 128-byte stage holds 8 columns of 16 bytes)
    assert m * k * 2 >= 131072 and _lib.lib().unit_packed_weights_bytes_gemm_f16(n, k) < n * 128
    a = torch.full((3000, 4096), 0x7c, dtype=torch.uint8, device='cuda')
    wq = U.pack_dense_weights_int8(torch.ones((16, 1024, 16, 4), dtype=torch.int8, device='cuda'))
    for _ in range(3):
        U.dense_dotprod(a, wq)
        gemm_case(U, m, n, k)


# the same form on bytes: every reduction below 128 bytes with a matrix of 128 KB and more
@pytest.mark.parametrize('m,n,k', [(8200, 64, 16), (40007, 64, 16), (4100, 272, 32), (2800, 48, 48), (40007, 128, 64), (1700, 528, 80),
                                   (1400, 16, 96), (1200, 64, 112)])
def test_dense_column_copies(U, m, n, k):
    from unit_b200 import _lib
    columns = (k // 16 + 1) & ~1
    per_row = _lib.lib().unit_packed_weights_bytes_dense_i8(n, k) // 16
    assert m * k >= 131072 and (per_row < n * 8 if k < 112 else per_row % (n * columns) == 0)   # (112: a stage of 8 columns)
    names = dense_case(U, m, n, k)
    assert all('A_DENSE_TMA' in v for v in names), names


# rows further apart than they are long, reductions that end inside a 128-byte stage and inside a K step
@pytest.mark.parametrize('m,n,k,gap', [(700, 272, 1040, 48), (2050, 64, 208, 16), (300, 528, 1104, 1024), (9000, 48, 80, 32)])
def test_dense_rows_with_a_gap(U, m, n, k, gap):
    import ctypes
    from unit_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(m + k)
    a = rng.integers(0, 256, (m, k + gap), dtype=np.uint8)     # (what lies in the gap must not enter the sums)
    b = rng.integers(-128, 128, (n, k), dtype=np.int8)
    ad, pw = dev(a), U.pack_dense_weights_int8(dev(no.pack_dense_weights(b, 16)))
    got = torch.full((m, n + 16), 7, dtype=torch.int32, device='cuda')
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.unit_dense_u8s8s32(m, n, k, ad.data_ptr(), k + gap, pw.buf.data_ptr(), got.data_ptr(), n + 16, st) == 0
    U.device_status()
    want = (ad[:, :k].double() @ dev(b).double().t()).to(torch.int32)
    assert torch.equal(got[:, :n], want) and bool((got[:, n:] == 7).all())


# (batch, chunks, depth, h, w, c_out, kernel, padding): one and two sub-tiles, padding in no and in every dimension,
# kernels that are flat in one dimension, slices smaller than a tile, a column block that is not full
@pytest.mark.parametrize('n,c,d,h,w,co,k,p', [
    (4, 64, 18, 44, 44, 64, (3, 3, 3), (0, 0, 0)),
    (3, 32, 9, 30, 30, 48, (3, 3, 3), (1, 1, 1)),
    (2, 32, 40, 34, 30, 32, (2, 3, 1), (1, 0, 0)),
    (5, 64, 6, 58, 58, 16, (1, 3, 3), (0, 1, 1)),
    (2, 32, 17, 23, 61, 80, (3, 1, 3), (2, 0, 1)),
])
def test_conv3d_windows_over_the_whole_batch(U, n, c, d, h, w, co, k, p):
    from oracle import c_oracle
    rng = np.random.default_rng(n + c + d + h + co)
    x = rng.integers(0, 256, (n, c // 16, d, h, w, 16), dtype=np.uint8)
    wt = rng.integers(-128, 128, (co // 16, c // 16) + k + (4, 16, 4), dtype=np.int8)
    b = rng.integers(-2 ** 15, 2 ** 15, co, dtype=np.int32)
    ref = c_oracle.conv3d_u8s8(x, wt, (1, 1, 1), p, bias=b)
    xd, wd, bd = dev(x), dev(wt), dev(b)
    got, names = launched(lambda: U.conv3d_NCDHWc_int8(xd, wd, stride=1, padding=p, bias=bd))
    U.device_status()
    assert any('A_CONV_WIN' in v for v in names), names
    assert np.array_equal(got.cpu().numpy(), ref)
    gotq = U.conv3d_NCDHWc_int8(xd, wd, stride=1, padding=p, bias=bd, requant_shift=10)
    assert np.array_equal(gotq.cpu().numpy(), np.clip((ref.astype(np.int64) + 512) >> 10, 0, 255).astype(np.uint8))
    U.device_status()


def test_conv3d_window_with_a_residual(U):
    """Through the C ABI: the Python operator has no residual in three dimensions."""
    import ctypes
    from oracle import c_oracle
    from unit_b200 import _lib
    L = _lib.lib()
    n, c, d, h, w, co = 3, 64, 14, 44, 44, 48
    rng = np.random.default_rng(5)
    x = rng.integers(0, 256, (n, c // 16, d, h, w, 16), dtype=np.uint8)
    wt = rng.integers(-128, 128, (co // 16, c // 16, 3, 3, 3, 4, 16, 4), dtype=np.int8)
    b = rng.integers(-2 ** 15, 2 ** 15, co, dtype=np.int32)
    acc = c_oracle.conv3d_u8s8(x, wt, (1, 1, 1), (1, 1, 1), bias=b)
    r = rng.integers(0, 256, acc.shape, dtype=np.uint8)
    xd, bd, rd = dev(x), dev(b), dev(r)
    pw = U.pack_conv3d_weights_int8(dev(wt), 1)
    got = torch.empty(acc.shape, dtype=torch.uint8, device='cuda')
    desc = _lib.Conv3dDesc(n, c, d, h, w, co, 3, 3, 3, 1, 1, 1, 1, 1, 1)
    epi = _lib.Epilogue(bd.data_ptr(), 1, 10, 1, rd.data_ptr(), 0)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc, names = launched(lambda: L.unit_conv3d_int8_ncdhwc(ctypes.byref(desc), xd.data_ptr(), pw.buf.data_ptr(), ctypes.byref(epi),
                                                           got.data_ptr(), st))
    assert rc == 0 and all('A_CONV_WIN, EPI_RES_NCHWC' in v for v in names), (rc, names)
    U.device_status()
    want = np.clip(((acc.astype(np.int64) + 512) >> 10) + r, 0, 255).astype(np.uint8)
    assert np.array_equal(got.cpu().numpy(), want)


# every form of the final pack: the shorter one (8), any other while bias and rounding constant fit the bias step (18
# at most), a dot product that scales the residual (up to 15); the general loop above those; with one and two sub-tiles
# per tile, a ragged last column block and sums on both sides of the clamp
@pytest.mark.parametrize('shift', [1, 7, 8, 9, 15, 16, 17, 18, 19, 20, 23])
@pytest.mark.parametrize('n,c,h,co', [(9, 32, 23, 48), (32, 64, 28, 272)])
def test_requantising_drains_at_every_shift(U, n, c, h, co, shift):
    from oracle import c_oracle
    rng = np.random.default_rng(n + shift)
    x = rng.integers(0, 256, (n, c // 16, h, h, 16), dtype=np.uint8)
    w = rng.integers(-128, 128, (co // 16, c // 16, 1, 1, 4, 16, 4), dtype=np.int8)
    b = rng.integers(-2 ** 15, 2 ** 15, co, dtype=np.int32)
    r = rng.integers(0, 256, (n, co // 16, h, h, 16), dtype=np.uint8)
    for res in (None, r):
        want = c_oracle.conv2d_i8_ex(x, w, (1, 1), (0, 0), bias=b, requant_shift=shift, residual=res)
        got = U.conv2d_NCHWc_int8(dev(x), dev(w), bias=dev(b), out_dtype='uint8', requant_shift=shift,
                                  residual=None if res is None else dev(res))
        U.device_status()
        assert np.array_equal(got.cpu().numpy(), want)


# grids smaller than the GPU: column blocks cut into narrow tiles (blocks of 144, 192, 208 and 256 columns, the last
# one not full), with and without a split of the reduction, for every way the A operand arrives
@pytest.mark.parametrize('m,n,k', [(1, 272, 256), (128, 3072, 768), (33, 208, 3072), (130, 1008, 1040), (500, 192, 4096), (300, 2064, 96)])
def test_narrow_tiles_dense(U, m, n, k):
    dense_case(U, m, n, k)
    gemm_case(U, m, n, k)


@pytest.mark.parametrize('n,c,h,w,co,k,s', [
    (1, 256, 14, 14, 208, 3, 1),    # gather
    (1, 512, 7, 7, 2048, 1, 1),     # gather, a short reduction for its width
    (2, 192, 17, 17, 192, 7, 1),    # boxes, odd rows
    (1, 288, 35, 35, 384, 3, 2),    # im2col copies
    (1, 256, 28, 28, 272, 3, 2),    # pixel pairs
])
def test_narrow_tiles_conv(U, n, c, h, w, co, k, s):
    from oracle import c_oracle
    rng = np.random.default_rng(n + c + h + co)
    p = k // 2
    x = rng.integers(0, 256, (n, c // 16, h, w, 16), dtype=np.uint8)
    wt = rng.integers(-128, 128, (co // 16, c // 16, k, k, 4, 16, 4), dtype=np.int8)
    b = rng.integers(-2 ** 15, 2 ** 15, co, dtype=np.int32)
    oh, ow = (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1
    r = rng.integers(0, 256, (n, co // 16, oh, ow, 16), dtype=np.uint8)
    xd, wd, bd = dev(x), dev(wt), dev(b)
    for opt in ({}, {'bias': b}, {'bias': b, 'mul': 11}, {'bias': b, 'requant_shift': 10}, {'bias': b, 'requant_shift': 8, 'residual': r}):
        want = c_oracle.conv2d_i8_ex(x, wt, (s, s), (p, p), **opt)
        kw = {key: dev(v) if isinstance(v, np.ndarray) else v for key, v in opt.items()}
        if 'requant_shift' in opt:
            kw['out_dtype'] = 'uint8'
        got = U.conv2d_NCHWc_int8(xd, wd, stride=s, padding=p, **kw)
        U.device_status()
        assert np.array_equal(got.cpu().numpy(), want), opt


@pytest.mark.parametrize('m,n,k', [(128, 3072, 768), (4096, 1024, 512)])   # narrow tiles, whole column blocks
def test_trace_marks_the_weight_copies(U, m, n, k):
    from unit_b200 import _lib
    L = _lib.lib()
    a = torch.randint(0, 256, (m, k), dtype=torch.uint8, device='cuda')
    pw = U.pack_dense_weights_int8(torch.randint(-128, 128, (n // 16, k // 4, 16, 4), dtype=torch.int8, device='cuda'))
    U.dense_dotprod(a, pw)
    trace = torch.zeros((4, 16), dtype=torch.int64, device='cuda')
    torch.cuda.synchronize()
    try:
        assert L.unit_trace_attach(trace.data_ptr(), 4) == 0
        U.dense_dotprod(a, pw)
        torch.cuda.synchronize()
    finally:
        assert L.unit_trace_attach(None, 0) == 0
    U.device_status()
    row = trace[0].cpu().tolist()
    assert row[2] > 0 and row[1] > 0, row


@pytest.mark.parametrize('batch', [1, 16])
def test_shared_plans_take_fewer_blocks_and_give_the_same_results(U, batch):
    """Launches that run beside others: SM time counts, so a small grid is cut less than for its own latency."""
    from unit_b200 import resnet50 as R
    alone, shared = {}, {}
    for i, l in enumerate(R.LAYERS):
        if l.c_block != 16:
            continue
        x, w, b = (dev(a) for a in R.make_layer_inputs(l, i, batch))
        pw = U.pack_conv_weights_int8(w, l.stride, l.pad)
        opt = dict(stride=l.stride, padding=l.pad, bias=b, out_dtype='uint8')
        plans = [U.conv2d_NCHWc_int8_plan(x, pw, shared=s, **opt) for s in (False, True)]
        assert torch.equal(plans[0].run(), plans[1].run()), l.name
        alone[l.name], shared[l.name] = plans[0].ctas * l.count, plans[1].ctas * l.count
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        assert 1 <= plans[1].ctas <= plans[0].ctas <= sms, l.name
    U.device_status()
    # per layer the time of a block grows as their number falls, but by less than the number does
    assert sum(shared.values()) < 0.9 * sum(alone.values()), (alone, shared)


@pytest.mark.parametrize('n,c,h,co,k,small', [(1, 256, 14, 256, 1, True), (8, 256, 14, 256, 1, True), (8, 512, 7, 512, 3, True),
                                              (64, 256, 14, 512, 1, False), (64, 64, 56, 64, 1, False)])
def test_tuner_finds_the_grids_that_the_library_cuts_itself(U, n, c, h, co, k, small):
    from unit_b200 import tune
    x = torch.zeros((n, c // 16, h, h, 16), dtype=torch.uint8, device='cuda')
    w = torch.zeros((co // 16, c // 16, k, k, 4, 16, 4), dtype=torch.int8, device='cuda')
    assert tune.one_tile_per_sm(x, w, (1, 1), k // 2) == small
