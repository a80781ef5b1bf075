"""The projector kernel at the sizes where its chunks, schedules and fixed-point scales can go
wrong, against the FP64 oracle.

Bars: forward, a ray's fraction terms are float32 (relative 2^-24 each, up to ~35 of them and
one conversion per chunk) and its integer part is good to 2^-29 of its chunk's integral, so
1e-6 relative L2 per projection, 1e-5 per bin, and exact zeros where the oracle has zeros; backward, values are rounded by up to 2^-23 of the LOR's largest: 1e-6."""
import numpy as np
import pytest
import torch

from nipet_b200 import _lib, diffprj, geometry, petprj
from nipet_b200.device import dev_ptr, get_geometry, stream_ptr
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def env():
    p = geometry.get_mmrparams()
    tt, _ = O.siddon_tables(p['txLUT'])
    n = tt.reshape(-1, 10)[:, 9].astype(int) - 3       # steps of each LOR
    order = np.argsort(n, kind='stable')
    pick = [order[0], order[-1],                       # shortest and longest walk
            24839,                                     # a ray reaches the plane above the image
            254, 48, 47,                               # second crossings taken a step late
            42285]                                     # a walk starting on a plane boundary
    for ch in (16, 24, 32, 64, 128):                   # chunk edges: 1, ch - 1 or 0 steps left
        for rest in (0, 1, ch - 1):
            m = np.flatnonzero((n % ch == rest) & (n > ch))
            pick += [m[m.size // 3], m[m.size // 2]]
    subs = np.unique(np.asarray(pick)).astype(np.int32)
    return {'p': p, 'orc': O.Oracle(p), 'subs': subs}


def _cnt(env, span):
    return dict(env['p']['Cnt'], SPN=span)


def _image(seed):
    """Positive with empty planes and columns, values over four decades."""
    r = np.random.default_rng(seed)
    im = r.uniform(0.0, 1.0, (320, 320, 127)).astype(np.float32) ** 8
    im[:, :, 40:47] = 0
    im[100:130, 90:200] = 0
    return im


def _check_fwd(got, want, peak):
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
    big = want >= 1e-3 * want.max()
    assert (np.abs(got - want)[big] / want[big]).max() <= 1e-5
    # every bin, with a sliver of a step besides (test_walk_weak_planes)
    assert (np.abs(got - want) <= 1e-5 * want + 0.3 * 2.0 ** -25 * peak).all()
    assert not got[want == 0].any()


@pytest.mark.parametrize('span', [11, 1])
@pytest.mark.parametrize('nimg', [1, 2, 3, 4])
def test_walk_edges(env, span, nimg):
    p, orc, subs = env['p'], env['orc'], env['subs']
    prj = diffprj.MMRProjector(p, span=span, subs=subs)
    ims = np.stack([_image(7 * nimg + i) * 10.0 ** (-2 * i) for i in range(nimg)])
    got = prj.project(torch.from_numpy(ims).cuda()).cpu().numpy().astype(np.float64)
    r = np.random.default_rng(nimg)
    si = r.exponential(1.0, got.shape).astype(np.float32) * 10.0 ** (2 * np.arange(nimg))[:, None, None]
    si = si.astype(np.float32)
    si[:, 3] = 0
    back = prj.backproject(torch.from_numpy(si).cuda()).cpu().numpy().astype(np.float64)
    prj.check()
    for i in range(nimg):
        _check_fwd(got[i], orc.fprj(ims[i], subs, span=span), ims[i].max())
        want = orc.bprj(si[i], subs, span=span)
        assert np.linalg.norm(back[i] - want) <= 1e-6 * np.linalg.norm(want)
        assert not back[i][want == 0].any()


@pytest.mark.parametrize('value', [np.inf, -np.inf, np.nan, 1e35])
def test_walk_non_finite_voxel(env, value):
    """A voxel without a fixed-point scale reaches the rays that meet it and no others."""
    p, subs, Cnt = env['p'], env['subs'], _cnt(env, 1)
    im = _image(1)
    vox = (160, 150, 63)
    im[vox] = 0
    one = np.zeros_like(im)
    one[vox] = 1
    run = lambda x: _project(p, Cnt, x, subs)  # noqa: E731
    ref, hit = run(im), run(one) != 0
    im[vox] = value
    got = run(im)
    assert hit.any() and np.allclose(got[~hit], ref[~hit], rtol=1e-5, atol=1e-6 * ref.max())
    if np.isfinite(value):
        assert (got[hit] > 1e28).all()
    else:
        assert not np.isfinite(got[hit]).any()


def _project(p, Cnt, im, subs):
    out = torch.zeros((subs.size, 4084 if Cnt['SPN'] == 1 else 837), device='cuda')
    petprj.fprj(out, torch.from_numpy(im).cuda(), p['txLUT'], p['axLUT'], subs, Cnt, 0)
    return out.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize('scale', [1e-30, 1e-15, 1e20])
def test_walk_scales(env, scale):
    """Results scale with their inputs, also where values are near the ends of float32."""
    p, orc, subs, Cnt = env['p'], env['orc'], env['subs'], _cnt(env, 11)
    im = _image(2)
    want = orc.fprj(im, subs)
    got = _project(p, Cnt, im * np.float32(scale), subs) / scale
    assert np.linalg.norm(got - want) <= 2e-6 * np.linalg.norm(want)
    si = np.random.default_rng(3).exponential(1.0, (subs.size, 837)).astype(np.float32)
    b = torch.zeros((320, 320, 127), device='cuda')
    petprj.bprj(b, torch.from_numpy(si * np.float32(scale)).cuda(), p['txLUT'], p['axLUT'], subs, Cnt)
    want = orc.bprj(si, subs)
    got = b.cpu().numpy().astype(np.float64) / scale
    assert np.linalg.norm(got - want) <= 2e-6 * np.linalg.norm(want)


def _ray_bin(p, d, r0, up):
    """Span-1 sinogram of the ray of rings r0, r0 + d (up: towards the higher ring)."""
    rno = p['axLUT']['li2rno'].astype(int)
    li = int(np.flatnonzero((rno.min(1) == r0) & (rno.max(1) == r0 + d))[0])
    return int(p['axLUT']['li2sn1'][li, 0 if up else 1])


def _line(orc, lor, sino):
    """1 in the voxels that one ray of one LOR meets."""
    si = np.zeros((1, 4084), np.float32)
    si[0, sino] = 1
    return (orc.bprj(si, np.array([lor], np.int32), span=1) > 0).astype(np.float32)


@pytest.fixture(scope='module')
def lines(env):
    """LORs and, per ring difference, an image of one-voxel lines along one ray of each."""
    r = np.random.default_rng(11)
    subs = np.sort(r.choice(68516, 40, replace=False)).astype(np.int32)
    ims = []
    for d in (30, 45, 60):
        im = np.zeros((320, 320, 127), np.float32)
        for i, lor in enumerate(subs):
            im = np.maximum(im, _line(env['orc'], lor, _ray_bin(env['p'], d, i % (64 - d), i & 1)))
        ims.append(im)
    return subs, ims


@pytest.mark.parametrize('kind', ['alone', 'background', 'signed'])
@pytest.mark.parametrize('nimg', [1, 2, 4])
def test_walk_ray_outruns_planes(env, lines, nimg, kind):
    """A ray that changes planes can collect more from a chunk than any plane holds: thin lines
    along rays.  Bar per bin: 1e-5 of the integral of |value| (float32 conversions and fractions)
    and 1e-6 of the largest (the scale of a LOR's fixed-point sums)."""
    subs, ims = lines
    ims = [{'alone': x, 'background': 1 + 50 * x, 'signed': 8 * x - 0.5}[kind] for x in ims]
    ims = [ims[i % 3] for i in range(max(nimg, 3))][:max(nimg, 3)]
    prj = diffprj.MMRProjector(env['p'], span=1, subs=subs)
    for a in range(0, len(ims), nimg):
        part = ims[a:a + nimg]
        x = torch.from_numpy(np.stack(part).astype(np.float32)).cuda()
        got = prj.project(x).cpu().numpy().astype(np.float64)
        prj.check()
        for g, im in zip(got, part):
            want = env['orc'].fprj(im, subs, span=1)
            size = env['orc'].fprj(np.abs(im), subs, span=1)
            assert (np.abs(g - want) <= 1e-5 * size + 1e-6 * size.max()).all()


def _errors(env, im, subs, nimg, slack):
    """Bins of nimg copies of an image against the oracle: 1e-5 of each, and `slack` besides."""
    prj = diffprj.MMRProjector(env['p'], span=1, subs=subs)
    got = prj.project(torch.from_numpy(np.stack([im] * nimg)).cuda()).cpu().numpy()
    prj.check()
    want = env['orc'].fprj(im, subs, span=1)
    for g in got.astype(np.float64):
        bad = np.abs(g - want) > 1e-5 * want + slack
        assert not bad.any(), (bad.sum(), (np.abs(g - want)[bad] / want[bad]).max())


@pytest.mark.parametrize('ratio', [1e3, 1e4, 1e5, 1e6, 1e8])
@pytest.mark.parametrize('nimg', [1, 2, 4])
def test_walk_weak_planes(env, nimg, ratio):
    """Every bin of a positive image, however much hotter neighbouring planes are.  A crossing's
    fraction of its step (0.3 cm at the most) is good to 2^-25, so rays that meet a hot plane,
    perhaps with a sliver of a step, have that much of its value besides."""
    im = np.random.default_rng(5).uniform(0.5, 1.5, (320, 320, 127)).astype(np.float32)
    im[:, :, 20:60:4] *= np.float32(ratio)
    im[:, :, 90:] /= np.float32(ratio)
    subs = env['subs']
    hot = env['orc'].fprj((im >= ratio / 2).astype(np.float32), subs, span=1) > 0
    _errors(env, im, subs, nimg, hot * (0.3 * 2.0 ** -25 * im.max()))


@pytest.mark.parametrize('seed', [0, 1, 2])
@pytest.mark.parametrize('nimg', [1, 2, 4])
def test_walk_planes_of_all_scales(env, nimg, seed):
    """Planes of random levels over twelve decades, alone and in blocks, with voxel noise: most
    rays are weak against some plane of their LOR, many of them against a chunk's first pass."""
    r = np.random.default_rng(seed)
    level = 10.0 ** r.uniform(-12, 0, 127)
    if seed:
        level[:40], level[90:] = 10.0 ** r.uniform(-12, -3), 10.0 ** r.uniform(-12, -3)
    im = (r.uniform(0.5, 1.5, (320, 320, 127)) * level).astype(np.float32)
    rno = env['p']['axLUT']['li2rno'].astype(int)
    slack = np.zeros(4084)
    for li, (r0, r1) in enumerate(zip(rno.min(1), rno.max(1))):
        top = level[max(0, 2 * r0 - 1):2 * r1 + 2].max()   # of the planes between the rings
        slack[env['p']['axLUT']['li2sn1'][li]] = 1.5 * top * 0.3 * 2.0 ** -25
    _errors(env, im, env['subs'], nimg, slack)


@pytest.mark.parametrize('ratio', [100, 300, 700, 2000, 10000])
def test_walk_equal_weak_values(env, ratio):
    """Equal weak values on LORs of equal steps (along the grid and its diagonals), whose rounding
    errors would add up."""
    s2c, crs = env['p']['txLUT']['s2c'].astype(int), env['p']['txLUT']['crs'].astype(float)
    x, y = 0.5 * (crs[:, 0] + crs[:, 2]), 0.5 * (crs[:, 1] + crs[:, 3])
    dx, dy = np.abs(x[s2c[:, 0]] - x[s2c[:, 1]]), np.abs(y[s2c[:, 0]] - y[s2c[:, 1]])
    near = [np.argsort(v, kind='stable')[:200:20] for v in (dx, dy, np.abs(dx - dy))]
    subs = np.unique(np.concatenate(near)).astype(np.int32)
    im = np.full((320, 320, 127), 1.0 / ratio, np.float32)
    im[:, :, 50:70] = 1.0
    hot = env['orc'].fprj((im == 1).astype(np.float32), subs, span=1) > 0
    for nimg in (1, 2, 4):
        _errors(env, im, subs, nimg, hot * (0.3 * 2.0 ** -25))


@pytest.mark.parametrize('value', [1e6, 1e9, 1e12])
@pytest.mark.parametrize('nimg', [1, 2, 4])
def test_walk_hot_voxel(env, nimg, value):
    """A hot voxel leaves the rays that miss it, and those that only pass its plane, alone."""
    im = np.random.default_rng(6).uniform(0.5, 1.5, (320, 320, 127)).astype(np.float32)
    im[:, :, 100:] *= 1e-3
    for vox in ((160, 150, 63), (161, 150, 20), (159, 210, 100)):
        im[vox] = value
    subs = env['subs']
    hot = env['orc'].fprj((im == np.float32(value)).astype(np.float32), subs, span=1) > 0
    _errors(env, im, subs, nimg, hot * (0.3 * 2.0 ** -25 * value))


@pytest.mark.parametrize('nimg', [1, 2, 4])
def test_walk_clipped_voxels(env, lines, nimg):
    """Bins that clip a voxel or two, to 1e-5 of their own value."""
    subs, ims = lines
    _errors(env, ims[1], subs, nimg, 0.0)


@pytest.mark.parametrize('value', [1e-20, 1e-33])
@pytest.mark.parametrize('nimg', [1, 2, 4])
def test_walk_faint_background(env, nimg, value):
    """Values far below 2^-60 beside ordinary ones, and on their own."""
    r = np.random.default_rng(8)
    im = (r.uniform(0.5, 1.5, (320, 320, 127)) * value).astype(np.float32)
    im[140:180, 140:180, 50:70] += r.uniform(0.5, 1.5, (40, 40, 20)).astype(np.float32)
    _errors(env, im, env['subs'], nimg, 0.0)


def test_walk_pairs_with_own_crossings(env):
    """LORs on which a first or last plane boundary of some ring pairs rounds to the next one, so
    that they cross planes at other floats than the rest of their difference.  Bar: each ray's
    value is rounded by up to 2^-23 of the largest, and a voxel's rays and its float32 sum, 2e-6."""
    p, orc = env['p'], env['orc']
    r = np.random.default_rng(4)
    for lor in (11712, 13025, 14216, 17924, 32699, 35929, 45722, 53209, 64252):
        sub = np.array([lor], np.int32)
        si = r.exponential(1.0, (1, 4084)).astype(np.float32)
        b = torch.zeros((320, 320, 127), device='cuda')
        petprj.bprj(b, torch.from_numpy(si).cuda(), p['txLUT'], p['axLUT'], sub, _cnt(env, 1))
        want = orc.bprj(si, sub, span=1)
        assert np.abs(b.cpu().numpy() - want).max() <= 2e-6 * want.max(), lor


@pytest.mark.parametrize('bad', [np.inf, np.nan])
@pytest.mark.parametrize('nimg', [1, 2, 4])
def test_walk_non_finite_bin(env, nimg, bad):
    """A value that is not finite reaches the voxels of its ray, in its image, and no others."""
    p, orc, subs = env['p'], env['orc'], env['subs']
    row, o = 5, _ray_bin(p, 20, 11, True)
    prj = diffprj.MMRProjector(p, span=1, subs=subs)
    si = np.random.default_rng(nimg).exponential(1.0, (nimg, subs.size, 4084)).astype(np.float32)
    si[:, row, o] = 0
    run = lambda x: prj.backproject(torch.from_numpy(x).cuda()).cpu().numpy().astype(np.float64)  # noqa: E731
    ref = run(si)
    hit = _line(orc, subs[row], o) > 0
    si[nimg - 1, row, o] = bad
    got = run(si)
    prj.check()
    assert hit.any() and not np.isfinite(got[-1][hit]).any()
    for i in range(nimg):
        keep = ~hit if i == nimg - 1 else np.ones_like(hit)
        assert np.linalg.norm((got[i] - ref[i])[keep]) <= 1e-6 * np.linalg.norm(ref[i])
        assert not got[i][keep & (ref[i] == 0)].any()


def test_walk_fused_non_finite_ratio(env):
    """The same for a ratio of the fused sub-iteration (NaN randoms of one bin)."""
    p, orc, subs = env['p'], env['orc'], env['subs']
    dev = torch.device('cuda')
    g, lib, st = get_geometry(p['txLUT'], p['axLUT'], dev), _lib.load(), stream_ptr(dev)
    row, o = 7, _ray_bin(p, 33, 20, False)
    hit = _line(orc, subs[row], o) > 0
    y = torch.ones((1, 68516, 4084), device=dev, dtype=torch.int16).view(torch.uint16)
    rs = torch.ones((68516, 4084), device=dev)
    rs[int(subs[row]), o] = float('nan')
    d_subs, one = torch.from_numpy(subs).to(dev), torch.ones(1, device=dev)
    n = 320 * 320 * 128
    x, b, sens = torch.ones(n, device=dev), torch.zeros(n, device=dev), torch.ones(n, device=dev)
    _lib.check(lib.nb_osem_batch_subset(g.handle, dev_ptr(x), dev_ptr(b), dev_ptr(sens),
                                        dev_ptr(sens.to(torch.uint8)), dev_ptr(y), dev_ptr(rs),
                                        dev_ptr(one), 1, 1, 0, 1, dev_ptr(d_subs), subs.size, st))
    out = torch.empty((320, 320, 127), device=dev)
    _lib.check(lib.nb_from_batch(dev_ptr(out), dev_ptr(x), 1, 1, st))
    g.check()
    out = out.cpu().numpy()
    assert np.isnan(out[hit]).all() and np.isfinite(out[~hit]).all()


@pytest.mark.parametrize('span', [11, 1])
@pytest.mark.parametrize('bs,nimg', [(1, 1), (1, 2), (2, 1), (2, 3), (4, 3), (4, 5)])
def test_walk_fused_edges(env, span, bs, nimg):
    """One fused sub-iteration over the edge LORs, images not a multiple of the width and count
    levels decades apart, against the oracle's projections.  Bar: two projections' 1e-6 each and
    the float32 ratio and update, 4e-6 relative L2."""
    p, orc, subs = env['p'], env['orc'], env['subs']
    nsn = 4084 if span == 1 else 837
    dev = torch.device('cuda')
    g, lib, st = get_geometry(p['txLUT'], p['axLUT'], dev), _lib.load(), stream_ptr(dev)
    r = np.random.default_rng(10 * bs + nimg)
    ims = np.stack([_image(3 * bs + i) + np.float32(1e-3) for i in range(nimg)])
    ims *= (10.0 ** (-np.arange(nimg)))[:, None, None, None].astype(np.float32)
    y = np.zeros((nimg, 68516, nsn), np.uint16)
    y[:, subs] = r.poisson(3.0, (nimg, subs.size, nsn))
    rs = np.zeros((68516, nsn), np.float32)
    rs[subs] = r.uniform(0.1, 2.0, (subs.size, nsn))
    rs[subs[2]] = 0
    rscale = r.uniform(0.5, 2.0, nimg).astype(np.float32)
    groups = -(-nimg // bs)
    d = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
    x, d_y, d_rs, d_sc, d_subs = d(ims), d(y), d(rs), d(rscale), d(subs)
    sens = torch.full((320 * 320 * 128,), 2.0, device=dev)
    msk = torch.ones(320 * 320 * 128, device=dev, dtype=torch.uint8)
    xb = torch.empty(groups * bs * 320 * 320 * 128, device=dev)
    bb = torch.empty_like(xb)
    _lib.check(lib.nb_to_batch(dev_ptr(xb), dev_ptr(x), nimg, bs, st))
    _lib.check(lib.nb_osem_batch_subset(g.handle, dev_ptr(xb), dev_ptr(bb.zero_()), dev_ptr(sens),
                                        dev_ptr(msk), dev_ptr(d_y), dev_ptr(d_rs), dev_ptr(d_sc),
                                        nimg, bs, 0, span, dev_ptr(d_subs), subs.size, st))
    out = torch.empty_like(x)
    _lib.check(lib.nb_from_batch(dev_ptr(out), dev_ptr(xb), nimg, bs, st))
    g.check()
    for i in range(nimg):
        e = orc.fprj(ims[i], subs, span=span) + rscale[i] * rs[subs].astype(np.float64)
        q = np.where(np.abs(e) < 1e-6, 0.0, y[i, subs] / np.where(e == 0, 1, e))
        want = ims[i] * orc.bprj(q.astype(np.float32), subs, span=span) / 2.0
        got = out[i].cpu().numpy().astype(np.float64)
        assert np.linalg.norm(got - want) <= 4e-6 * np.linalg.norm(want)
