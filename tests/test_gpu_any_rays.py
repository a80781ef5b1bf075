"""Axial LUTs whose rays are not the mMR's ring pairs (rings moved, or off by a rounding): the
projections run step by step instead of by crossing schedules, with the same results.  Against
the FP64 oracle on the same LUTs: 1e-6 relative L2 (float32 walks of ~270 steps)."""
import numpy as np
import pytest
import torch

from nipet_b200 import _lib, diffprj, geometry, petprj
from nipet_b200.device import Geometry, RingSet, dev_ptr, get_geometry, stream_ptr
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def env():
    p = geometry.get_mmrparams()
    rng = p['axLUT']['li2rng']
    moved = {'shift': (rng + np.float32(0.05)).astype(np.float32),
             'ulp': np.nextafter(rng, np.float32(99), dtype=np.float32)}
    ps = {k: dict(p, axLUT=dict(p['axLUT'], li2rng=v)) for k, v in moved.items()}
    subs = np.array([0, 254, 14216, 24839, 42285, 50001, 68515], np.int32)
    return {'p': p, 'ps': ps, 'orc': {k: O.Oracle(q) for k, q in ps.items()}, 'subs': subs}


def _rel(got, want):
    return np.linalg.norm(got - want) / np.linalg.norm(want)


def _image(seed):
    im = np.random.default_rng(seed).uniform(0.0, 1.0, (320, 320, 127)).astype(np.float32) ** 4
    im[:, :, 40:47] = 0
    return im


@pytest.mark.parametrize('how', ['shift', 'ulp'])
@pytest.mark.parametrize('span', [11, 1])
def test_any_rays_projections(env, how, span):
    p, orc, subs = env['ps'][how], env['orc'][how], env['subs']
    nsn = 4084 if span == 1 else 837
    Cnt = dict(p['Cnt'], SPN=span)
    im = _image(span)
    for att in (0, 1):
        x = im * np.float32(0.05) if att else im
        out = torch.empty((subs.size, nsn), device='cuda')
        petprj.fprj(out, torch.from_numpy(x).cuda(), p['txLUT'], p['axLUT'], subs, Cnt, att)
        want = orc.fprj(x, subs, att=att, span=span)
        assert _rel(out.cpu().numpy(), want) <= 1e-6
        assert not out.cpu().numpy()[want == 0].any()
    si = np.random.default_rng(2).exponential(1.0, (subs.size, nsn)).astype(np.float32)
    b = torch.empty((320, 320, 127), device='cuda')
    petprj.bprj(b, torch.from_numpy(si).cuda(), p['txLUT'], p['axLUT'], subs, Cnt)
    want = orc.bprj(si, subs, span=span)
    assert _rel(b.cpu().numpy(), want) <= 1e-6 and not b.cpu().numpy()[want == 0].any()
    prj = diffprj.MMRProjector(p, span=span, subs=subs)
    ims = np.stack([_image(i) for i in range(3)])
    got = prj.project(torch.from_numpy(ims).cuda()).cpu().numpy()
    sis = np.stack([si, 2 * si, si[::-1]])
    back = prj.backproject(torch.from_numpy(sis).cuda()).cpu().numpy()
    prj.check()
    for i in range(3):
        assert _rel(got[i], orc.fprj(ims[i], subs, span=span)) <= 1e-6
        assert _rel(back[i], orc.bprj(sis[i], subs, span=span)) <= 1e-6


@pytest.mark.parametrize('span,bs', [(11, 2), (1, 4)])
def test_any_rays_fused(env, span, bs):
    p, orc, subs, nimg = env['ps']['shift'], env['orc']['shift'], env['subs'], 3
    nsn = 4084 if span == 1 else 837
    dev = torch.device('cuda')
    g, lib, st = get_geometry(p['txLUT'], p['axLUT'], dev), _lib.load(), stream_ptr(dev)
    r = np.random.default_rng(bs)
    ims = np.stack([_image(i) + np.float32(0.1) for i in range(nimg)])
    y = np.zeros((nimg, 68516, nsn), np.uint16)
    y[:, subs] = r.poisson(3.0, (nimg, subs.size, nsn))
    rs = np.zeros((68516, nsn), np.float32)
    rs[subs] = r.uniform(0.1, 2.0, (subs.size, nsn))
    d = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
    x, d_y, d_rs, d_subs = d(ims), d(y), d(rs), d(subs)
    one, n = torch.ones(nimg, device=dev), 320 * 320 * 128
    sens, msk = torch.ones(n, device=dev), torch.ones(n, device=dev, dtype=torch.uint8)
    xb = torch.empty(-(-nimg // bs) * bs * n, device=dev)
    bb = torch.zeros_like(xb)
    _lib.check(lib.nb_to_batch(dev_ptr(xb), dev_ptr(x), nimg, bs, st))
    _lib.check(lib.nb_osem_batch_subset(g.handle, dev_ptr(xb), dev_ptr(bb), dev_ptr(sens),
                                        dev_ptr(msk), dev_ptr(d_y), dev_ptr(d_rs), dev_ptr(one),
                                        nimg, bs, 0, span, dev_ptr(d_subs), subs.size, st))
    out = torch.empty_like(x)
    _lib.check(lib.nb_from_batch(dev_ptr(out), dev_ptr(xb), nimg, bs, st))
    g.check()
    for i in range(nimg):
        e = orc.fprj(ims[i], subs, span=span) + rs[subs].astype(np.float64)
        want = ims[i] * orc.bprj((y[i, subs] / e).astype(np.float32), subs, span=span)
        assert _rel(out[i].cpu().numpy(), want) <= 4e-6


def test_any_rays_reduced_range(env):
    """A ring range of such a geometry against the mMR's own (positions a rounding apart)."""
    p, q, subs, rs, re = env['p'], env['ps']['ulp'], env['subs'], 20, 33
    Cnt = dict(p['Cnt'], SPN=1, RNG_STRT=rs, RNG_END=re)
    ax = geometry.axial_lut(Cnt)
    ax2 = dict(ax, li2rng=np.nextafter(ax['li2rng'], np.float32(99), dtype=np.float32))
    dev, lib = torch.device('cuda', 0), _lib.load()
    nz, d_subs = 2 * (re - rs) - 1, torch.from_numpy(subs).cuda()
    im = torch.from_numpy(np.ascontiguousarray(_image(1)[:, :, 2 * rs:2 * rs + nz])).cuda()
    res = []
    for params, lut in ((p, ax), (q, ax2)):
        g = Geometry(params['txLUT'], params['axLUT'], dev)
        rr = RingSet(g, rs, re, lut)
        s = torch.empty((subs.size, rr.nsino), device=dev)
        b = torch.empty_like(im)
        _lib.check(lib.nb_fprj_rings(g.handle, rr.handle, dev_ptr(s), dev_ptr(im), dev_ptr(d_subs),
                                     subs.size, 0, stream_ptr(dev)))
        _lib.check(lib.nb_bprj_rings(g.handle, rr.handle, dev_ptr(b), dev_ptr(s), dev_ptr(d_subs),
                                     subs.size, stream_ptr(dev)))
        g.check()
        res.append((s.cpu().numpy(), b.cpu().numpy()))
        rr.close()
        g.close()
    assert _rel(res[1][0], res[0][0]) <= 1e-5 and _rel(res[1][1], res[0][1]) <= 1e-5


def test_ring_positions_outside_the_fov_are_refused(env):
    p = env['p']
    far = (p['axLUT']['li2rng'] + np.float32(5.0)).astype(np.float32)
    with pytest.raises(_lib.NBError, match='leave the axial FOV'):
        Geometry(p['txLUT'], dict(p['axLUT'], li2rng=far), torch.device('cuda', 0))
