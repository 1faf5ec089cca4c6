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
    b = rng.integers(-128, 128, (k, n), dtype=np.int8)
    got, names = launched(lambda: U.dense_dotprod(dev(a), dev(no.pack_dense_weights(b, 16))))
    U.device_status()
    # (float64 holds these integer sums exactly: |sum| <= 255 * 128 * k < 2^53)
    want = (dev(a).double() @ dev(b).double()).to(torch.int32)
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
