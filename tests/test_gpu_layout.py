"""NCHW <-> channel blocks over the sizes where the tiles can go wrong: units smaller than a tile (grouped), larger
than one (cut into pixel spans), odd row lengths, a partly filled last channel block, misaligned tensors."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import np_oracle as no

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('cb', [4, 16])
@pytest.mark.parametrize('dtype', [torch.uint8, torch.float16, torch.int32])
@pytest.mark.parametrize('n,c,h,w', [
    (1, 1, 1, 1), (3, 3, 7, 7), (2, 16, 35, 35), (5, 33, 14, 14), (2, 20, 17, 13), (1, 3, 299, 299), (2, 48, 56, 56),
    (1, 5, 1, 5003), (130, 64, 7, 7), (1, 17, 63, 65), (7, 256, 5, 3),
])
def test_pack_and_unpack(n, c, h, w, dtype, cb):
    import unit_b200 as U
    g = torch.Generator(device='cuda').manual_seed(n * 7 + c)
    bits = {torch.uint8: torch.uint8, torch.float16: torch.int16, torch.int32: torch.int32}[dtype]
    info = torch.iinfo(bits)
    x = torch.randint(info.min, info.max, (n, c, h, w), dtype=bits, device='cuda', generator=g)
    y = U.pack_data_nchwc(x.view(dtype) if dtype != bits else x, cb)
    assert np.array_equal((y.view(bits) if dtype != bits else y).cpu().numpy(), no.pack_nchw_to_nchwc(x.cpu().numpy(), cb))
    back = U.unpack_data_nchwc(y, c)
    assert torch.equal(back.view(bits) if dtype != bits else back, x)


@pytest.mark.parametrize('hw', [(7, 7), (37, 41), (64, 64)])
@pytest.mark.parametrize('shift', [1, 4, 9])
def test_misaligned_tensors_and_no_writes_outside(hw, shift):
    """Pointers that are not 16-byte aligned, through the C ABI; the bytes around the result stay as they were."""
    from unit_b200 import _lib
    L = _lib.lib()
    n, c, cb = 2, 19, 16
    size, blocked = n * c * hw[0] * hw[1], n * 2 * hw[0] * hw[1] * cb
    g = torch.Generator(device='cuda').manual_seed(3)
    src = torch.randint(0, 256, (size + 64,), dtype=torch.uint8, device='cuda', generator=g)
    dst = torch.full((blocked + 64,), 7, dtype=torch.uint8, device='cuda')
    back = torch.full((size + 64,), 9, dtype=torch.uint8, device='cuda')
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    at = lambda t: ctypes.c_void_p(t.data_ptr() + shift)
    assert L.unit_pack_data_nchw_to_nchwc(at(src), at(dst), n, c, hw[0], hw[1], cb, 1, st) == 0
    assert L.unit_unpack_data_nchwc_to_nchw(at(dst), at(back), n, c, hw[0], hw[1], cb, 1, st) == 0
    torch.cuda.synchronize()
    x = src[shift:shift + size].cpu().numpy().reshape(n, c, *hw)
    assert np.array_equal(dst[shift:shift + blocked].cpu().numpy(), no.pack_nchw_to_nchwc(x, cb).reshape(-1))
    assert torch.equal(back[shift:shift + size], src[shift:shift + size])
    for t, k, v in ((dst, blocked, 7), (back, size, 9)):
        assert bool((t[:shift] == v).all()) and bool((t[shift + k:] == v).all())


def test_more_channel_blocks_than_one_launch_numbers():
    """Above 2^30 channel blocks a transform goes in two halves.  (Four channels of one pixel: both layouts are the
    same bytes.)"""
    import unit_b200 as U
    n = 2 ** 30 + 5
    if torch.cuda.mem_get_info()[0] < 16 * 2 ** 30:
        pytest.skip('needs 16 GB')
    x = torch.empty((n, 4, 1, 1), dtype=torch.uint8, device='cuda')
    x.view(-1).view(torch.int32).copy_(torch.arange(n, dtype=torch.int32, device='cuda'))
    y = U.pack_data_nchwc(x, 4)
    assert y.shape == (n, 1, 1, 1, 4) and torch.equal(y.view(-1).view(torch.int32), x.view(-1).view(torch.int32))
    back = U.unpack_data_nchwc(y)
    assert torch.equal(back.view(-1).view(torch.int32), x.view(-1).view(torch.int32))
    del x, y, back
    torch.cuda.empty_cache()
