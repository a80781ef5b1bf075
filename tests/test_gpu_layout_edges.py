"""Image-layout and gap kernels at their tile edges and alignments, against plain indexing.

Both only move values, so results are bit-equal: images that start on a 16-byte boundary and
off it (1 to 3 floats) take different load widths, and sinogram counts below, at and past a
32-wide tile leave different remainders."""
import ctypes

import pytest
import torch

from nipet_b200 import _lib, geometry

pytestmark = pytest.mark.gpu

COLS, Z = 320 * 320, 127


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _s():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _bits(t):
    return t.contiguous().view(torch.uint8)


@pytest.mark.parametrize('nimg', [1, 2, 3])
@pytest.mark.parametrize('off', [0, 1, 2, 3])
def test_col128_round_trip(nimg, off):
    lib = _lib.load()
    n = nimg * COLS * Z
    g = torch.Generator(device='cuda').manual_seed(nimg * 7 + off)
    im = torch.randn(n + 4, device='cuda', generator=g)[off:off + n]
    im[::1001] = float('nan')
    im[5::1003] = float('inf')
    want = torch.zeros(nimg, COLS, 128, device='cuda')
    v = im.view(nimg, COLS, Z)
    want[..., :64] = v[..., 0::2]
    want[..., 64:127] = v[..., 1::2]
    got = torch.full_like(want, -1.)
    _lib.check(lib.nb_im_to_col128(_p(got), _p(im), nimg, _s()))
    assert torch.equal(_bits(got), _bits(want))

    buf = torch.full((n + 8,), -7., device='cuda')
    _lib.check(lib.nb_col128_to_im(_p(buf[off:]), _p(got), nimg, _s()))
    assert torch.equal(_bits(buf[off:off + n]), _bits(im))
    assert bool((buf[:off] == -7.).all()) and bool((buf[off + n:] == -7.).all())


@pytest.mark.parametrize('nsn', [1, 2, 31, 32, 33, 64, 837])
def test_gaps(nsn):
    lib = _lib.load()
    tx = geometry.get_mmrparams()['txLUT']
    idx = torch.as_tensor(tx['aw2ali'].astype('int64'), device='cuda')
    aw = idx.to(torch.int32)
    g = torch.Generator(device='cuda').manual_seed(nsn)
    # odd offsets too: neither array has to start on a 16-byte boundary
    full = torch.rand(nsn * 252 * 344 + 1, device='cuda', generator=g)[1:].view(nsn, -1)
    want = full[:, idx].T.contiguous()
    got = torch.full((want.numel() + 1,), -1., device='cuda')[1:].view_as(want)
    _lib.check(lib.nb_remgaps(_p(got), _p(full), nsn, _p(aw), _s()))
    assert torch.equal(got, want)

    u = (full * 60000).to(torch.int32).to(torch.int16).contiguous()
    gu = torch.full(want.shape, -1, device='cuda', dtype=torch.int16)
    _lib.check(lib.nb_remgaps_u16(_p(gu), _p(u), nsn, _p(aw), _s()))
    assert torch.equal(gu, u[:, idx].T)

    back = torch.zeros_like(full)
    back[:, idx] = want.T
    out = torch.full_like(full, -1.)
    _lib.check(lib.nb_putgaps(_p(out), _p(got), nsn, _p(aw), _s()))
    assert torch.equal(out, back)
