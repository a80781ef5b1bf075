"""The work users have this framework do, as timed cases.

Each case is one pass through the public entry points a program calls: projections of a
few LORs, of one OSEM subset and of the whole sinogram; one OSEM iteration through the
drop-in, batched over replicates and over dynamic frames; one step of the differentiable
projector; list-mode histograms from a short frame to a long one and with bootstrap
replicates; and one frame from list mode to image.

Inputs come from a seed alone: an emission image of ellipsoids with noise, water
attenuation, log-normal crystal efficiencies, and Poisson prompts whose mean is the
phantom's line integrals in closed form (chords of ellipsoids), so that no projector of
the package shapes them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nipet_b200 import batch, diffprj, geometry, mmr_lmproc, mmrhist, mmrrec, petprj

NAW, NRAYS = 68516, 4084
NSN = {1: 4084, 11: 837}
IMG = (320, 320, 127)
VOXY, VOXZ, RING = float(np.float32(0.208626)), 0.203125, 0.40625
FOV2 = 890.0
_CACHE: dict = {}


def _dev():
    return torch.device('cuda', 0)


def _params():
    if 'params' not in _CACHE:
        _CACHE['params'] = geometry.get_mmrparams()
    return _CACHE['params']


def listed():
    return [
        # a quick look at a few lines of response: launch and host latency
        {'name': 'fprj_s11_few', 'kind': 'fprj', 'span': 11, 'nlor': 33, 'att': 0},
        # the forward half of one OSEM subset
        {'name': 'fprj_s11_subset', 'kind': 'fprj', 'span': 11, 'nlor': 4894, 'att': 0},
        # attenuation factors of a study, once per mu-map
        {'name': 'att_s11_full', 'kind': 'fprj', 'span': 11, 'nlor': NAW, 'att': 1},
        # back projection of an odd set of lines at the finest axial sampling
        {'name': 'bprj_s1_ragged', 'kind': 'bprj', 'span': 1, 'nlor': 5003},
        # one iteration of the drop-in: 14 subsets
        {'name': 'osem_s11', 'kind': 'osem', 'span': 11, 'psf': 0.0},
        # one iteration of bootstrap replicates, a count the batch width does not divide
        {'name': 'batch_s11_9', 'kind': 'batch', 'span': 11, 'nimg': 9},
        # one iteration of dynamic frames at very different count levels
        {'name': 'dynamic_s1_4', 'kind': 'batch', 'span': 1, 'nimg': 4},
        # one gradient step of a learned reconstruction: forward, loss, backward
        {'name': 'diff_s11_8', 'kind': 'diff', 'span': 11, 'nimg': 8, 'nlor': NAW},
        # a gating window or motion frame: a short stretch of list mode, planned and counted
        {'name': 'hist_s11_short', 'kind': 'hist', 'span': 11, 'words': 300_001, 'nrep': 1},
        # a static scan at the finest axial sampling
        {'name': 'hist_s1_long', 'kind': 'hist', 'span': 1, 'words': 100_000_000, 'nrep': 1},
        # bootstrap replicates of one scan
        {'name': 'hist_s11_boot', 'kind': 'hist', 'span': 11, 'words': 20_000_000, 'nrep': 10},
        # one frame from list mode to image, with resolution modelling
        {'name': 'chain_s11_psf', 'kind': 'chain', 'span': 11, 'words': 30_000_000, 'psf': 4.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['fprj', 'bprj', 'fprj', 'bprj', 'osem', 'batch', 'batch', 'diff', 'hist',
                       'hist', 'chain'])
    span = rng.choice([11, 11, 1])
    if kind == 'fprj':
        return {'kind': kind, 'span': span, 'nlor': _log(rng, 1, NAW), 'att': rng.randint(0, 1)}
    if kind == 'bprj':
        return {'kind': kind, 'span': span, 'nlor': _log(rng, 1, NAW)}
    if kind == 'osem':
        return {'kind': kind, 'span': 11, 'psf': rng.choice([0.0, rng.uniform(2.0, 6.0)])}
    if kind == 'batch':
        return {'kind': kind, 'span': span, 'nimg': rng.randint(1, 9 if span == 11 else 4)}
    if kind == 'diff':
        return {'kind': kind, 'span': 11, 'nimg': rng.randint(1, 8), 'nlor': _log(rng, 40, NAW)}
    if kind == 'hist':
        nrep = rng.choice([1, 1, rng.randint(2, 10)])
        top = 100_000_000 if nrep == 1 else 20_000_000
        return {'kind': kind, 'span': span if nrep == 1 else 11, 'words': _log(rng, 20_000, top),
                'nrep': nrep}
    return {'kind': kind, 'span': 11, 'words': _log(rng, 1_000_000, 30_000_000),
            'psf': rng.choice([0.0, rng.uniform(2.0, 6.0)])}


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _ellipsoids(seed):
    """(centre, radii, activity) of a head and hot and cold regions in it, cm."""
    r = np.random.default_rng(seed)
    out = [((0.0, 0.0, 0.0), (7.2, 9.2, 8.5), 1.0), ((0.0, 0.5, 0.3), (6.3, 8.1, 7.5), 2.2),
           ((0.0, 0.5, 0.3), (5.4, 6.9, 6.6), -1.9)]
    for _ in range(5):
        rad = r.uniform(0.5, 1.5)
        c = (r.uniform(-3.5, 3.5), r.uniform(-5, 5), r.uniform(-4.5, 4.5))
        out.append((c, (rad, rad, rad), r.uniform(2.0, 7.0)))
    return out


def _image(seed, noise=0.15):
    """Emission image (y, x, z) as an OSEM iterate looks: structure plus voxel noise."""
    dev = _dev()
    g = torch.Generator(device=dev).manual_seed(seed)
    x = (torch.arange(320, device=dev) - 159.5) * VOXY
    y = (159.5 - torch.arange(320, device=dev)) * VOXY
    z = (torch.arange(127, device=dev) - 63.0) * VOXZ
    im = torch.zeros(IMG, device=dev)
    for c, r, a in _ellipsoids(seed):
        q = (((y[:, None, None] - c[1]) / r[1]) ** 2 + ((x[None, :, None] - c[0]) / r[0]) ** 2
             + ((z[None, None, :] - c[2]) / r[2]) ** 2)
        im += a * (q <= 1)
    return im * (1 + noise * torch.randn(IMG, generator=g, device=dev)).clamp_(min=0.0)


def _mumap():
    """Water, 0.096 per cm."""
    dev = _dev()
    x = (torch.arange(320, device=dev) - 159.5) * VOXY
    y = (159.5 - torch.arange(320, device=dev)) * VOXY
    z = (torch.arange(127, device=dev) - 63.0) * VOXZ
    q = ((y[:, None, None] / 9.6) ** 2 + (x[None, :, None] / 7.6) ** 2
         + (z[None, None, :] / 9.0) ** 2)
    return 0.096 * (q <= 1).float()


def _chords(span, lors, shapes):
    """Sum over `shapes` of activity x chord length (cm) for every LOR and sinogram."""
    p, dev = _params(), _dev()
    crs = torch.from_numpy(p['txLUT']['crs']).to(dev)
    s2c = torch.from_numpy(p['txLUT']['s2c'].astype(np.int64)).to(dev)
    s2c = s2c if lors is None else s2c[lors]
    cx, cy = 0.5 * (crs[:, 0] + crs[:, 2]), 0.5 * (crs[:, 1] + crs[:, 3])
    rno = torch.from_numpy(p['axLUT']['sn1_rno'].astype(np.int64)).to(dev)
    zz = (rno.float() - 31.5) * RING
    if span == 11:
        s11 = torch.from_numpy(p['axLUT']['sn1_sn11'].astype(np.int64)).to(dev)
        m = torch.zeros((837, 2), device=dev).index_add_(0, s11, zz)
        zz = m / torch.bincount(s11, minlength=837)[:, None]
    x0, x1, y0, y1 = cx[s2c[:, 0]], cx[s2c[:, 1]], cy[s2c[:, 0]], cy[s2c[:, 1]]
    dz = zz[:, 1] - zz[:, 0]
    length = torch.sqrt(((x1 - x0) ** 2 + (y1 - y0) ** 2)[:, None] + dz[None, :] ** 2)
    out = torch.zeros_like(length)
    for c, r, a in shapes:
        A = (((x1 - x0) / r[0]) ** 2 + ((y1 - y0) / r[1]) ** 2)[:, None] + (dz / r[2]) ** 2
        B = ((x1 - x0) * (x0 - c[0]) / r[0] ** 2 + (y1 - y0) * (y0 - c[1]) / r[1] ** 2)[:, None] \
            + dz * (zz[:, 0] - c[2]) / r[2] ** 2
        C = (((x0 - c[0]) / r[0]) ** 2 + ((y0 - c[1]) / r[1]) ** 2)[:, None] \
            + ((zz[:, 0] - c[2]) / r[2]) ** 2 - 1
        out += a * 2 * torch.sqrt((B * B - A * C).clamp_(min=0)) / A * length
    return out.clamp_(min=0)


def _scan(span, seed):
    """Noise-free trues, attenuation and normalisation of a scan; the same phantom for all
    seeds (kept), efficiencies from the seed."""
    if ('scan', span) not in _CACHE:
        trues = _chords(span, None, _ellipsoids(0))
        asng = torch.exp(-0.096 * _chords(span, None, [((0, 0, 0), (7.6, 9.6, 9.0), 1.0)]))
        _CACHE['scan', span] = trues, asng
    trues, asng = _CACHE['scan', span]
    dev, p = _dev(), _params()
    g = torch.Generator(device=dev).manual_seed(1000 + seed)
    eff = torch.exp(0.05 * torch.randn((64, 504), generator=g, device=dev))
    s2c = torch.from_numpy(p['txLUT']['s2c'].astype(np.int64)).to(dev)
    rno = torch.from_numpy(p['axLUT']['sn1_rno'].astype(np.int64)).to(dev)
    if span == 11:   # the ring pair nearest the middle of a sinogram stands for it
        s11 = p['axLUT']['sn1_sn11']
        first = np.array([np.flatnonzero(s11 == i)[np.sum(s11 == i) // 2] for i in range(837)]) \
            if 'mid11' not in _CACHE else _CACHE['mid11']
        _CACHE['mid11'] = first
        rno = rno[torch.from_numpy(first).to(dev)]
    nsng = eff[rno[:, 0]][:, s2c[:, 0]] * eff[rno[:, 1]][:, s2c[:, 1]]
    return trues, asng, nsng.t().contiguous()


def _prompts(mean_trues, counts, g):
    """uint16 Poisson prompts of `counts` in all, a fifth of them flat randoms; the randoms
    per bin."""
    r = 0.2 * counts / mean_trues.numel()
    m = mean_trues * (0.8 * counts / mean_trues.sum(dtype=torch.float64).item()) + r
    return torch.poisson(m, generator=g).clamp_(max=65535).to(torch.int32).to(torch.uint16), r


def _lors(n, seed):
    r = np.random.default_rng(seed)
    return None if n == NAW else np.sort(r.choice(NAW, n, replace=False)).astype(np.int32)


def _words(n, seed, seconds):
    """int32 list-mode words on the device: `n` events (addresses from the attenuated
    phantom, a fifth of them delayeds spread evenly) with a time tag every millisecond."""
    dev, p = _dev(), _params()
    if 'cdf' not in _CACHE:
        trues = _chords(1, None, _ellipsoids(0))
        trues *= torch.exp(-0.096 * _chords(1, None, [((0, 0, 0), (7.6, 9.6, 9.0), 1.0)]))
        rows = trues.sum(1, dtype=torch.float64).cumsum(0)
        _CACHE['cdf'] = rows / rows[-1], torch.cumsum(trues, 1, dtype=torch.float32)
        live = np.flatnonzero(p['txLUT']['msino'].T.reshape(-1) > 0).astype(np.int64)
        _CACHE['live'] = torch.from_numpy(live).to(dev)
    rows, cum = _CACHE['cdf']
    live = _CACHE['live']
    g = torch.Generator(device=dev).manual_seed(seed)
    n_del = n // 5
    rand = lambda k, dt=torch.float32: torch.rand(k, generator=g, device=dev, dtype=dt)  # noqa: E731
    aw = torch.searchsorted(rows, rand(n - n_del, torch.float64)).clamp_(max=NAW - 1)
    u = rand(n - n_del)
    lo = torch.zeros_like(aw)          # bisection of each LOR's own cumulative row
    for step in (2048, 1024, 512, 256, 128, 64, 32, 16, 8, 4, 2, 1):
        t = (lo + step).clamp_(max=4083)
        lo = torch.where(cum[aw, t - 1] <= u * cum[aw, 4083], t, lo)
    pr = (lo * 86688 + live[aw]) | (1 << 30)
    ri = lambda hi: torch.randint(0, hi, (n_del,), generator=g, device=dev)  # noqa: E731
    words = torch.cat([pr, ri(4084) * 86688 + live[ri(live.numel())]])
    ticks = torch.randint(0, seconds * 1000, (n,), generator=g, device=dev)
    ticks, order = torch.sort(ticks, stable=True)   # a random time each: prompts and delayeds mix
    words = words[order]
    counts = torch.bincount(ticks, minlength=seconds * 1000)
    k = torch.arange(seconds * 1000, device=dev)
    out = torch.empty(n + seconds * 1000, device=dev, dtype=torch.int32)
    out[k + torch.cumsum(counts, 0) - counts] = (k + 1000 - 2 ** 31).to(torch.int32)
    out[torch.arange(n, device=dev) + ticks + 1] = words.to(torch.int32)
    return out


def _seconds(words):
    return int(min(600, max(2, words // 150_000)))


def _cnt(**kw):
    return dict(_params()['Cnt'], DEVID=0, **kw)


def prepare(case, seed):
    dev, p, kind, span = _dev(), _params(), case['kind'], case['span']
    s = {'kind': kind, 'span': span, 'Cnt': _cnt(SPN=span), 'tx': p['txLUT'], 'ax': p['axLUT']}
    g = torch.Generator(device=dev).manual_seed(seed)
    if kind == 'fprj':
        subs = _lors(case['nlor'], seed)
        s['subs'] = np.array([-1], np.int32) if subs is None else subs
        s['att'] = case['att']
        s['im'] = 0.096 * (_image(seed) > 0.5).float() if case['att'] else _image(seed)
        s['out'] = torch.zeros((case['nlor'], NSN[span]), device=dev)
    elif kind == 'bprj':
        subs = _lors(case['nlor'], seed)
        s['subs'] = np.array([-1], np.int32) if subs is None else subs
        # a ratio sinogram: about one, noisier where the phantom's shadow ends
        s['sino'] = torch.empty((case['nlor'], NSN[span]), device=dev).exponential_(1.0, generator=g)
        s['out'] = torch.zeros(IMG, device=dev)
    elif kind == 'osem':
        trues, asng, nsng = _scan(span, seed)
        s['psng'], r = _prompts(trues * asng * nsng, 3e7, g)
        s['asng'], s['nsng'] = asng, nsng
        s['rsng'] = torch.full_like(asng, r)
        s['ssng'] = torch.zeros_like(asng)
        s['subs'] = mmrrec.subset_table(p)
        s['krnl'] = mmrrec.psf_config(case['psf'] or None, s['Cnt'])
        an, sens = asng * nsng, torch.zeros((14,) + IMG, device=dev)
        for i in range(14):
            sub = s['subs'][i, 1:]
            petprj.bprj(sens[i], an[torch.from_numpy(sub).to(dev).long()].contiguous(), s['tx'],
                        s['ax'], sub, s['Cnt'])
        s['sens'] = sens
        s['msk'] = torch.from_numpy(geometry.get_cylinder(s['Cnt'], rad=29., gpu_dim=True)).to(
            dev, torch.float32)
        s['img'] = torch.ones(IMG, device=dev)
    elif kind == 'batch':
        trues, asng, nsng = _scan(span, seed)
        an = asng * nsng
        n = case['nimg']
        # replicates of a scan; frames from a short early one to a long late one
        counts = [3e7 if i % 8 != 5 else 3e6 for i in range(n)] if span == 11 else \
            list(np.geomspace(2e5, 5e7, n + 1)[1:])
        psng = torch.empty((n, NAW, NSN[span]), device=dev, dtype=torch.uint16)
        mean, rs = trues * an, []
        for i in range(n):
            psng[i], r = _prompts(mean, counts[i], g)
            rs.append(r)
        inv = torch.where(an.abs() < 1e-6, torch.zeros_like(an), 1.0 / an)
        s['rec'] = batch.BatchRecon(p, psng, inv, an, rscale=np.asarray(rs, np.float32),
                                    device=dev, span=span)
        s['rec'].sensitivity()
    elif kind == 'diff':
        lors = _lors(case['nlor'], seed)
        trues, asng, nsng = _scan(span, seed)
        s['prj'] = diffprj.MMRProjector(p, mu=_mumap(), nsng=nsng, span=span, subs=lors, device=dev)
        ti = slice(None) if lors is None else torch.from_numpy(lors).to(dev).long()
        mean = (trues * asng * nsng)[ti]
        s['x'] = torch.stack([_image(seed * 16 + i) for i in range(case['nimg'])])
        s['y'] = torch.stack([torch.poisson(mean + 0.5, generator=g) for _ in range(case['nimg'])])
    elif kind == 'hist':
        s['lm'] = _words(case['words'], seed, _seconds(case['words']))
        s['nrep'], s['seed'] = case['nrep'], seed
        if case['nrep'] > 1:
            s['Cnt'].update(BTP=2, BTPRT=1.0)
        host = s['lm'].cpu().numpy()
        # a frame of a stream is planned by the call itself; of a long stream, histogrammed
        # several times, a program keeps the chunk plan
        s['host'], s['plan'] = (host, None) if case['words'] < 2_000_000 else \
            (None, mmr_lmproc.plan(host))
    else:
        s['lm'] = _words(case['words'], seed, _seconds(case['words']))
        s['plan'] = mmr_lmproc.plan(s['lm'].cpu().numpy())
        s['params'] = dict(p, Cnt=s['Cnt'])
        mu = geometry.convert2e7(_mumap(), s['Cnt']).cpu().numpy()
        s['mu'] = [np.zeros_like(mu), mu]
        r = np.random.default_rng(seed)
        u = lambda lo, hi, shape: r.uniform(lo, hi, size=shape).astype(np.float32)  # noqa: E731
        ceff = u(0.9, 1.1, (64, 504))
        ceff[:, 8::9] = 0.0
        s['norm'] = {'geo': u(0.8, 1.2, (127, 344)), 'cinf': u(0.9, 1.1, (344, 9)), 'ceff': ceff,
                     'axe1': u(0.9, 1.1, 837), 'axf1': u(0.9, 1.1, 4084),
                     'dtp': u(-3e-6, -1e-6, 64), 'dtnp': u(1e-7, 4e-7, 64)}
        s['psf'] = case['psf'] or None
    return s


def run(s):
    kind = s['kind']
    if kind == 'fprj':
        petprj.fprj(s['out'], s['im'], s['tx'], s['ax'], s['subs'], s['Cnt'], s['att'])
        return s['out']
    if kind == 'bprj':
        petprj.bprj(s['out'], s['sino'], s['tx'], s['ax'], s['subs'], s['Cnt'])
        return s['out']
    if kind == 'osem':
        img = s['img'].clone()
        petprj.osem(img, s['psng'], s['rsng'], s['ssng'], s['nsng'], s['asng'], s['subs'],
                    s['sens'], s['msk'], s['krnl'], s['tx'], s['ax'], s['Cnt'])
        return img
    if kind == 'batch':
        s['rec'].init_images()
        s['rec'].iteration()
        return s['rec'].images()
    if kind == 'diff':
        x = s['x'].detach().requires_grad_(True)
        nll = diffprj.poisson_nll(s['prj'](x) + 0.5, s['y'])
        (grad,) = torch.autograd.grad(nll, x)
        return {'nll': nll.detach(), 'grad': grad}
    if kind == 'hist':
        r = mmr_lmproc.hist_stream(s['lm'], s['tx'], s['ax'], s['Cnt'], nrep=s['nrep'],
                                   seed=s['seed'], lm_host=s['host'], pl=s['plan'])
        whole = ('psn', 'dsn', 'ssr', 'phc', 'dhc', 'pvs', 'fan', 'bck')
        views = {torch.uint16: torch.int16, torch.uint32: torch.int32}
        out = {k: r[k].view(views[r[k].dtype]) for k in whole}
        return dict(out, mss=r['mss'], psum=r['psum'], dsum=r['dsum'])
    hst = mmrhist.hist_device(s['lm'], s['params'], pl=s['plan'])
    rec = mmrrec.osemone({}, s['mu'], hst, s['params'], recmod=1, itr=1, psf=s['psf'],
                         normcomp=s['norm'])
    return {'im': rec.im, 'psino': hst['psino'].view(torch.int16)}


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def work(case):
    """Bytes: every input read and every output written once.  Flops: per LOR the weighted
    running sums of its columns (290 steps x 127 planes on average), and per ray one
    interpolation at each of its ~35 axial crossings."""
    kind, span = case['kind'], case['span']
    im = 4 * 320 * 320 * 127
    lor = 2 * 290 * 127 + 4 * 35 * NRAYS
    nsn = NSN[span]
    if kind in ('fprj', 'bprj'):
        return {'bytes': im + 4 * case['nlor'] * nsn, 'flops': case['nlor'] * lor}
    if kind == 'osem':
        return {'bytes': NAW * nsn * (2 + 4 * 4) + im * (14 + 3), 'flops': 2 * NAW * lor}
    if kind == 'batch':
        n = case['nimg']
        return {'bytes': n * (NAW * nsn * 2 + im * 2) + NAW * nsn * 4 + 14 * im,
                'flops': 2 * n * NAW * lor}
    if kind == 'diff':
        n, rows = case['nimg'], case['nlor'] * nsn * 4
        return {'bytes': n * (2 * im + rows) + rows + im, 'flops': (2 * n + 2) * case['nlor'] * lor}
    out = 354_033_792 if span == 1 else 72_557_856
    words = case['words'] + 1000 * _seconds(case['words'])
    if kind == 'hist':
        return {'bytes': 4 * words + case['nrep'] * 4 * (out + 127 * 86688), 'flops': words}
    return {'bytes': 4 * words + 4 * out + NAW * nsn * 4 * 4 + im * 17,
            'flops': words + 4 * NAW * lor}


def tolerance(case):
    return 'exact' if case['kind'] == 'hist' else TOL[case['kind']]


# Histograms are counts.  A projection or gradient is 32-bit sums of some 300 terms along
# walks whose steps are fixed by 32-bit tables: run twice, with its sums in another order,
# it differs by 1e-9 to 1e-7, and at single bins (a few terms of 300 left after rounding) by
# more.  OSEM multiplies 14 such updates into the image (3e-7 run to run): the package's
# bar against its 64-bit oracle.
TOL = {'fprj': {'rel': 1e-5}, 'bprj': {'rel': 1e-5}, 'diff': {'rel': 1e-5},
       'osem': {'rel': 1e-4}, 'batch': {'rel': 1e-4}, 'chain': {'rel': 1e-4}}


# ---------------------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------------------
def _axial():
    """Per oblique ring pair (difference d, lower ring r): index tables of its axial plane
    crossings.  A ray between ring centres 2 r + 1/2 and 2 (r + d) + 1/2 (voxels) crosses 2 d
    planes at the fractions (k + 1/2) / (2 d) of its way."""
    if 'axial' not in _CACHE:
        p, dev = _params(), _dev()
        rno = p['axLUT']['li2rno'].astype(np.int64)
        ob = rno[64:]
        d = np.arange(1, 61)
        first = np.concatenate([[0], np.cumsum(2 * d)])       # first crossing of a difference
        frac = np.concatenate([(np.arange(2 * k) + 0.5) / (2 * k) for k in d])
        diff = ob[:, 1] - ob[:, 0]
        assert (diff > 0).all() and diff.max() <= 60
        ray = np.repeat(np.arange(len(ob)), 2 * diff)
        k = np.concatenate([np.arange(2 * q) for q in diff])
        ent = first[diff - 1][ray] + k
        up, down = 2 * ob[ray, 0] + 1 + k, 2 * ob[ray, 1] - k
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        _CACHE['axial'] = {'frac': t(frac), 'ray': t(ray), 'ent': t(ent), 'up': t(up),
                           'down': t(down), 'r0': t(ob[:, 0]), 'r1': t(ob[:, 1]),
                           'az': t(diff * RING)}
    return _CACHE['axial']


def _rays64(x, lors):
    """Line integrals [len(lors), 4084] (direct planes, upward, downward rays) of x
    [102400, 127] float64.  The walk runs between the first and the last grid line inside
    the field of view; per plane the running integral C over the transaxial steps, and at
    every axial crossing the difference of the two planes' running integrals."""
    p, dev, ax = _params(), _dev(), _axial()
    crs = torch.from_numpy(p['txLUT']['crs']).to(dev).double()
    c = torch.from_numpy(p['txLUT']['s2c'].astype(np.int64)).to(dev)[lors]
    cx, cy = 0.5 * (crs[:, 0] + crs[:, 2]), 0.5 * (crs[:, 1] + crs[:, 3])
    px, py = cx[c[:, 0]], cy[c[:, 0]]
    ux, uy = cx[c[:, 1]] - px, cy[c[:, 1]] - py
    atn = torch.sqrt(ux * ux + uy * uy)
    ux, uy = ux / atn, uy / atn
    b = px * ux + py * uy
    half = torch.sqrt((b * b - px * px - py * py + FOV2).clamp(min=0))
    grid = (torch.arange(321, device=dev) - 160).double() * VOXY
    t = torch.cat([(grid - px[:, None]) / ux[:, None], (grid - py[:, None]) / uy[:, None]], 1)
    inside = (t >= (-b - half)[:, None]) & (t <= (-b + half)[:, None])
    t = torch.where(inside, t, torch.full_like(t, math.inf)).sort(1).values
    m = int(inside.sum(1).max())
    n = inside.sum(1, keepdim=True)
    t = torch.minimum(t[:, :m], torch.gather(t, 1, n - 1))
    lt, mid = t[:, 1:] - t[:, :-1], 0.5 * (t[:, 1:] + t[:, :-1])
    u = torch.floor((px[:, None] + mid * ux[:, None]) / VOXY).long() + 160
    v = 160 - torch.ceil((py[:, None] + mid * uy[:, None]) / VOXY).long()
    C = torch.cumsum(x[v * 320 + u] * lt[:, :, None], 1)
    C = torch.nn.functional.pad(C, (0, 1, 1, 0))                 # plane 127 and step 0: nothing
    end = C[:, -1]
    D = (torch.nn.functional.pad(C, (1, 0))[:, :, :128] - C).reshape(len(c), -1)
    tk = ax['frac'][None, :] * atn[:, None]
    i = (torch.searchsorted(t.contiguous(), tk) - 1).clamp(0, m - 2)
    f = ((tk - torch.gather(t, 1, i)) / torch.gather(lt, 1, i).clamp(min=1e-30)).clamp(0, 1)
    i, f = i[:, ax['ent']] * 128, f[:, ax['ent']]
    out = [end[:, 0:127:2]]
    for plane, last, sign in ((ax['up'], 2 * ax['r1'], 1.0), (ax['down'], 2 * ax['r0'], -1.0)):
        a = torch.gather(D, 1, i + plane)
        a = a + f * (torch.gather(D, 1, i + plane + 128) - a)
        s = torch.zeros((len(c), last.numel()), device=dev, dtype=torch.float64)
        s = sign * s.index_add(1, ax['ray'], a) + end[:, last]
        out.append(s * torch.sqrt(1 + (ax['az'] / atn[:, None]) ** 2))
    return torch.cat(out, 1)


def _sino64(x, lors, span, att):
    p, dev = _params(), _dev()
    r = _rays64(x, lors)
    key = 'li2sn' if span == 11 else 'li2sn1'
    to = p['axLUT'][key].astype(np.int64)
    to = torch.from_numpy(np.concatenate([to[:64, 0], to[64:, 0], to[64:, 1]])).to(dev)
    if att:
        r = torch.exp(-r)
        if span == 11:
            r = r / torch.bincount(to, minlength=837)[to]
    return torch.zeros((r.shape[0], NSN[span]), device=dev, dtype=torch.float64).index_add(1, to, r)


def exact(case, seed):
    """64-bit values where they take seconds: projections and gradients of a subset."""
    kind, span = case['kind'], case['span']
    lines = case.get('nlor', NAW) * case.get('nimg', 1)
    if kind not in ('fprj', 'bprj', 'diff') or lines > (6000 if kind == 'fprj' else 5100):
        return None
    s = prepare(case, seed)
    lors = torch.from_numpy(_lors(case['nlor'], seed)).to(_dev()).long()
    parts = [slice(a, a + 32) for a in range(0, lors.numel(), 32)]
    if kind == 'fprj':
        x = s['im'].double().reshape(-1, 127)
        return torch.cat([_sino64(x, lors[q], span, case['att']) for q in parts])

    def adjoint(x, of):
        """Gradient of sum(of) over the parts; of(x, part) a scalar."""
        x = x.clone().requires_grad_(True)
        total = 0.0
        for q in parts:
            v = of(x, q)
            v.backward()
            total += float(v.detach())
        return total, x.grad.reshape(IMG)

    if kind == 'bprj':
        x = torch.zeros((320 * 320, 127), device=_dev(), dtype=torch.float64)
        return adjoint(x, lambda x, q: (_sino64(x, lors[q], span, 0) * s['sino'][q]).sum())[1]
    mu = _mumap().double().reshape(-1, 127)
    nsng = s['prj'].nsng[lors].double()
    w = torch.cat([_sino64(mu, lors[q], span, 1) for q in parts]) * nsng
    nll, grad = 0.0, []
    for b in range(case['nimg']):
        y = s['y'][b].double()

        def loss(x, q):
            yb = _sino64(x, lors[q], span, 0) * w[q] + 0.5
            return (yb - torch.xlogy(y[q], yb)).sum()
        v, gr = adjoint(s['x'][b].double().reshape(-1, 127), loss)
        nll, grad = nll + v, grad + [gr]
    return {'nll': torch.tensor(nll, dtype=torch.float64), 'grad': torch.stack(grad)}
