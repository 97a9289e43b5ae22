"""The workloads this framework's speed is judged on: what a user's program has the engine do, through its public
entry points, over the sizes it is used at.

Families (the key 'family' of a case):
  matvec       one Gram mat-vec S e over the modes of a fit (operator.Plan.apply): circular pball lattices and interval
               (slits x sinc) lattices; the step every solver, certificate and gradient repeats
  sweep        BLMLBinnedBatch: a cut-off sweep's fits in lockstep, cold (the real start, then L-BFGS) or one round of a
               certified sweep (rank-K L-BFGS from given starts, then the certificate of every fit)
  fit          BLMLBinned: one complex two-mode fit (signal and background pball), the single-fit drop-in
  rows         local_gpu.rows_dev: pair sums over occupied lattice bins, values or values and derivatives
  points       BLMLQuick.predict: the fitted density at off-lattice points (exact kernels per point and bin)
  predict      BLMLBinned.predict: the same for a periodic band (plane-wave sums over its spectrum)
  net_predict  WarmStartNet.predict: the learned start's network on a batch of lattices
  net_train    one training step of that network: forward, loss, backward, Adam

The solvers are capped at a fixed, small number of iterations: the same work on any input, and few enough that rounding
(which a non-convex ascent amplifies from step to step) leaves the results comparable. Sides, cut-offs,
counts, ranks, lattices and batch sizes are those of blml_b200.workloads, of the benchmark's rows and of the tests;
`draw` spreads over the same ranges, sides off the FFT lengths included."""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'band-limited-ml_b200'))

SIDES = (64, 96, 128, 192, 256, 384)          # the cut-off sweep's lattice sides


# ---------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest mat-vec: one mode on the sweep's smallest lattice, where launches and latency count
        dict(name='matvec_pball_64', family='matvec', kernel='pball', m1=64, m2=64, fc=0.2, modes=1, f32=False),
        # a certified fit at its last ranks on the largest lattice
        dict(name='matvec_pball_384_k8', family='matvec', kernel='pball', m1=384, m2=384, fc=0.33, modes=8, f32=False),
        # a non-periodic kernel on a ragged lattice (the two-slit fits): restricted transforms
        dict(name='matvec_slits_200x150', family='matvec', kernel='slits', m1=200, m2=150, fc=0.25, modes=2, f32=False),
        # a cold cut-off sweep: the real start and the first L-BFGS steps of 64 uneven lattices
        dict(name='sweep_cold_64', family='sweep', fits=64, layout=1, rank=1, iters=4, cold=True, f32=False),
        # one round of a certified sweep at rank 4: L-BFGS from given starts, then every fit's certificate
        dict(name='sweep_round_rank4', family='sweep', fits=64, layout=2, rank=4, iters=12, cold=False, f32=False),
        # the single-fit drop-in on the 256 x 256 signal-plus-background workload
        dict(name='fit_256_two_modes', family='fit', m1=256, m2=256, fc=0.33, iters=6, f32=False),
        # 5-D occupied bins in the point fits' default precision (float32 tables): every bin against every bin
        dict(name='rows_5d_f32', family='rows', bins=24000, dims=5, grad=False, f32=True),
        # a mixed kernel with derivative rows (an fc step of a fused fit): periodic, slit and sinc columns, float64
        dict(name='rows_grad_3d', family='rows', bins=9000, dims=3, grad=True, f32=False),
        # density of a point fit (a sinc and a periodic column) at off-lattice points
        dict(name='points_quick_20k', family='points', points=30000, queries=20000),
        # density of a binned periodic fit at off-lattice points
        dict(name='predict_pball_256', family='predict', m1=256, m2=256, fc=0.33, queries=50000),
        # the learned start's network, one batch of 128 x 128 lattices
        dict(name='net_predict_16x128', family='net_predict', batch=16, m1=128, m2=128),
        # a training step on the same batch
        dict(name='net_train_16x128', family='net_train', batch=16, m1=128, m2=128),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _fft_side(rng, lo, hi):
    """A side with an FFT route: 2^a 3^b in [lo, hi]."""
    sides = sorted(2 ** a * 3 ** b for a in range(1, 13) for b in range(5) if lo <= 2 ** a * 3 ** b <= hi)
    return rng.choice(sides)


def draw(rng):
    fam = rng.choice(('matvec', 'matvec', 'matvec', 'sweep', 'sweep', 'fit', 'rows', 'rows', 'points', 'predict',
                      'net_predict', 'net_train'))
    fc = round(_log(rng, 0.05, 0.45), 4)
    if fam == 'matvec':
        kernel = rng.choice(('pball', 'pball', 'slits'))
        if kernel == 'pball' and rng.random() < 0.75:
            m1, m2 = _fft_side(rng, 48, 512), _fft_side(rng, 48, 512)
        else:                                    # sides off the FFT lengths (51 x 51 windows and the like)
            m1, m2 = int(_log(rng, 40, 260)), int(_log(rng, 40, 260))
        return dict(family='matvec', kernel=kernel, m1=m1, m2=m2, fc=fc, modes=rng.randint(1, 8),
                    f32=rng.random() < 0.4)
    if fam == 'sweep':
        cold = rng.random() < 0.5
        return dict(family='sweep', fits=int(_log(rng, 4, 48)), layout=rng.randrange(1000),
                    rank=1 if cold else rng.randint(2, 4), iters=rng.randint(2, 4) if cold else rng.randint(6, 12),
                    cold=cold, f32=False)
    if fam == 'fit':
        return dict(family='fit', m1=_fft_side(rng, 48, 384), m2=_fft_side(rng, 48, 384), fc=max(fc, 0.1),
                    iters=rng.randint(3, 6), f32=False)
    if fam == 'rows':
        return dict(family='rows', bins=int(_log(rng, 500, 24000)), dims=rng.randint(2, 5),
                    grad=rng.random() < 0.3, f32=rng.random() < 0.5)
    if fam == 'points':
        return dict(family='points', points=int(_log(rng, 2000, 30000)), queries=int(_log(rng, 200, 20000)))
    if fam == 'predict':
        return dict(family='predict', m1=_fft_side(rng, 48, 384), m2=_fft_side(rng, 48, 384), fc=fc,
                    queries=int(_log(rng, 500, 60000)))
    # the network: sides are multiples of 8; training takes whole batches
    return dict(family=fam, batch=rng.choice((8, 16)) if fam == 'net_train' else rng.randint(1, 16),
                m1=8 * rng.randint(6, 16), m2=8 * rng.randint(6, 16))


# --------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _disks(shape, fc, g):
    """The unit-norm amplitude of workloads.two_disk_field: two displaced disks in the band, a random relative phase."""
    k1 = torch.fft.fftfreq(shape[0], device='cuda', dtype=torch.float64)[:, None]
    k2 = torch.fft.fftfreq(shape[1], device='cuda', dtype=torch.float64)[None, :]
    r = fc / 4
    ph = 2 * math.pi * torch.rand((), generator=g, device='cuda', dtype=torch.float64)
    a = (((k1 - r) ** 2 + k2 ** 2) <= r * r).to(torch.complex128)
    a = a + torch.polar(torch.ones_like(ph), ph) * (((k1 + r) ** 2 + k2 ** 2) <= r * r)
    h = torch.fft.ifft2(a)
    return h / h.abs().square().sum().sqrt()


def _counts(shape, fc, N, g):
    h = _disks(shape, fc, g)
    p = 0.95 * h.abs().square() + 0.05 / (shape[0] * shape[1])
    return torch.poisson(N * p, generator=g)


def _coefs(shape, fc, N, modes, cplx, g):
    """Coefficients as a fit's iterate has them: sqrt(counts) on the occupied bins with smooth-ish phases, each further
    mode weaker, zero elsewhere."""
    w = _counts(shape, fc, N, g)
    amp = w.sqrt() * (0.5 ** torch.arange(modes, device='cuda', dtype=torch.float64))[:, None, None]
    z = 0.5 * torch.randn((modes,) + tuple(shape), generator=g, device='cuda', dtype=torch.float64)
    return w, (torch.polar(amp, z) if cplx else amp * z.sign())


def _modes(kernel, shape, fc):
    from blml_b200 import workloads
    return workloads.pball_modes(shape, fc) if kernel == 'pball' else workloads.slits_modes(shape, fc)


def _layout(case):
    """The sweep's lattices, cut-offs and photon counts (they belong to the case; the seed draws the photons)."""
    r = random.Random(case['layout'])
    return [((r.choice(SIDES), r.choice(SIDES)), round(0.05 * 9 ** (r.randrange(16) / 15), 6), 10 ** r.uniform(4, 6))
            for _ in range(case['fits'])]


# --- pair rows: kinds, cut-offs, derivative entries and bins
_STEPS = {2: 512, 3: 128, 4: 64, 5: 64}       # lattice steps per unit length


def _rows_kernel(case):
    d = case['dims']
    if not case['grad']:
        return ['sinc'] * d, [6.4] * d, [None] * d, []
    kinds = ['sinc', 'slits:0.5', 'dirichlet', 'sinc', 'dirichlet'][:d]
    return kinds, [6.4, 8.0, 10.0, 5.0, 7.0][:d], [1.0 if k == 'dirichlet' else None for k in kinds], \
        [(0, 'fc'), (1, 'fc'), (0, 'shift')]


def _bins(case, seed):
    """`bins` occupied bins (n, d) of a Gaussian mixture in the unit cube, and their counts (host)."""
    rng = np.random.default_rng(seed)
    n, d, m = case['bins'], case['dims'], _STEPS[case['dims']]
    means = rng.uniform(0.25, 0.75, (8, d)); sds = rng.uniform(0.05, 0.1, (8, d))
    X = np.zeros((0, d), np.int64)
    while True:                                  # points until n bins are occupied
        c = rng.integers(0, 8, n)
        X = np.r_[X, np.rint(m * np.clip(means[c] + sds[c] * rng.standard_normal((n, d)), 0.0, 1 - 1 / m)).astype(np.int64)]
        Z, w = np.unique(X, axis=0, return_counts=True)
        if len(Z) >= n:
            keep = np.sort(rng.permutation(len(Z))[:n])
            return Z[keep], w[keep].astype(np.float64)


def _point_data(case, seed):
    rng = np.random.default_rng(seed)

    def blobs(n):
        a = rng.uniform(size=n) < 0.6
        X = np.where(a[:, None], rng.normal([0.35, 0.4], 0.08, (n, 2)), rng.normal([0.7, 0.75], 0.05, (n, 2)))
        X[:, 1] = np.mod(X[:, 1], 1.0)
        return X
    return blobs(case['points']), blobs(case['queries'])


_POINT_FC = (3.0, 4.0)


def _net_inputs(case, seed):
    """The network's inputs (workloads.warm_start_set's ranges, pball fits) and targets, on the device."""
    g = _gen(seed)
    r = random.Random(seed)
    shape = (case['m1'], case['m2'])
    x = torch.zeros((case['batch'],) + shape + (8,), device='cuda')
    t = torch.zeros((case['batch'],) + shape + (2,), device='cuda')
    for s in range(case['batch']):
        fc, N = r.uniform(0.1, 0.4), 10 ** r.uniform(4, 6)
        h = _disks(shape, fc, g)
        c = torch.poisson(N * (0.95 * h.abs().square() + 0.05 / (shape[0] * shape[1])), generator=g)
        x[s, :, :, 0] = torch.log1p(c) / 8.0
        x[s, :, :, 1] = 4.0 * fc
        x[s, :, :, 2] = 1.0
        x[s, :, :, 4] = torch.log10(c.sum()) / 6.0
        t[s] = torch.view_as_real(h.to(torch.complex64)) * math.sqrt(shape[0] * shape[1])
    return x.to(torch.bfloat16), t


# -------------------------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    fam = case['family']
    st = dict(case=case)
    if fam == 'matvec':
        from blml_b200 import _lib
        from blml_b200.operator import Plan, mode_transform, pad_rule
        from blml_b200.spec import parse_modes
        shape = (case['m1'], case['m2'])
        specs, _ = parse_modes(_modes(case['kernel'], shape, case['fc']), 2)
        h = np.ones(2)
        freqs, W = mode_transform(specs[0], shape, h, pad_rule(shape, h, specs))
        st['plan'] = Plan(freqs, W, shape, _lib.F32 if case['f32'] else _lib.F64)
        _, e = _coefs(shape, case['fc'], 1e5, case['modes'], True, _gen(seed))
        st['x'] = e.to(torch.complex64 if case['f32'] else torch.complex128).contiguous()
        st['y'] = torch.empty_like(st['x'])
    elif fam == 'sweep':
        g = _gen(seed)
        lay = _layout(case)
        st['modes'] = [_modes('pball', s, fc) * case['rank'] for s, fc, _ in lay]
        if case['cold']:
            st['counts'] = [_counts(s, fc, N, g) for s, fc, N in lay]
            st['init'] = None
        else:
            both = [_coefs(s, fc, N, case['rank'], True, g) for s, fc, N in lay]
            st['counts'] = [w for w, _ in both]
            st['init'] = [e for _, e in both]
    elif fam == 'fit':
        from blml_b200 import workloads
        shape = (case['m1'], case['m2'])
        st['counts'] = _counts(shape, case['fc'], 1e6, _gen(seed))
        st['modes'] = workloads.pball_modes(shape, case['fc'], bg_fc=3.0 / max(shape))
    elif fam == 'rows':
        from blml_b200.local_gpu import ProductKernel, rank_coords
        kinds, fc, per, want = _rows_kernel(case)
        Z, w = _bins(case, seed)
        st['tab'] = ProductKernel(kinds, per).tables(fc, per, [1.0 / _STEPS[case['dims']]] * case['dims'], Z, want=want)
        st['Z'] = torch.as_tensor(rank_coords(Z, st['tab'])).cuda()
        st['w'] = torch.as_tensor(np.sqrt(w)).cuda()
    elif fam == 'points':
        from blml_b200 import make_modes
        from blml_b200.quick import BLMLQuick
        X, st['Xq'] = _point_data(case, seed)
        modes = make_modes(list(_POINT_FC), ['sinc', 'dirichlet'], periods=[None, 1.0])
        st['fit'] = BLMLQuick(dtype=np.float64, max_sweeps=0).fit(X, modes)
    elif fam == 'predict':
        from blml_b200 import workloads
        from blml_b200.binned import BLMLBinned
        shape = (case['m1'], case['m2'])
        counts = _counts(shape, case['fc'], 1e5, _gen(seed))
        st['fit'] = BLMLBinned(solver='lbfgs', max_sweeps=0).fit(counts, workloads.pball_modes(shape, case['fc']),
                                                                complex_g=True)
        st['Xq'] = np.random.default_rng(seed).uniform(0, 1, (case['queries'], 2)) * np.array(shape)
    else:
        from blml_b200.warmstart import WarmStartNet
        st['net'] = WarmStartNet(seed=seed)
        st['x'], st['t'] = _net_inputs(case, seed)
    return st


# ------------------------------------------------------------------------------------------------------------ run
def run(st):
    case = st['case']
    fam = case['family']
    if fam == 'matvec':
        st['plan'].apply(st['x'], st['y'], case['modes'], True, torch.cuda.current_stream().cuda_stream)
        return st['y']
    if fam == 'sweep':
        from blml_b200.sweep import BLMLBinnedBatch
        b = BLMLBinnedBatch(tol=1e-6, max_sweeps=case['iters'], dtype=np.float32 if case['f32'] else np.float64)
        fits = b.fit(st['counts'], st['modes'], init=st['init'])
        out = dict(e=b.E_t, Se=b.U_t, density=b.dens_t, loglik=np.array([r.loglik_ for r in fits]))
        if not case['cold']:
            out['certificate'] = b.certificate()
        return out
    if fam == 'fit':
        from blml_b200.binned import BLMLBinned
        m = BLMLBinned(tol=1e-6, solver='lbfgs', max_sweeps=case['iters'],
                       dtype=np.float32 if case['f32'] else np.float64).fit(st['counts'], st['modes'], complex_g=True)
        return dict(e=m.e_hat_t_, Se=m.Se_t_, density=m.density_t_, loglik=m.loglik_)
    if fam == 'rows':
        from blml_b200.local_gpu import rows_dev
        s, ds = rows_dev(st['Z'], st['Z'], st['w'], st['tab'], grad=case['grad'], f32=case['f32'])
        return (s, ds) if case['grad'] else s
    if fam in ('points', 'predict'):
        return st['fit'].predict(st['Xq'])
    net = st['net']
    if fam == 'net_predict':
        return net.predict(st['x'], batch=16)
    u = net.forward(st['x'], case['batch'], case['m1'], case['m2'])
    loss, du = net.loss(u, st['t'])
    net.backward(du)
    net.adam(1e-3)
    # the gradients and the updated weights, each as one vector in the network's parameter order
    return dict(u=u, loss=loss, grads=torch.cat([v.reshape(-1) for v in net.g.values()]),
                params=torch.cat([v.reshape(-1) for v in net.p.values()]))


# ----------------------------------------------------------------------------------------------------------- work
_CONVS = [(8, 32, 1), (32, 32, 1), (32, 64, 4), (64, 64, 4), (64, 128, 16), (128, 128, 16), (128, 256, 64),
          (256, 256, 64), (384, 128, 16), (128, 128, 16), (192, 64, 4), (64, 64, 4), (96, 32, 1), (32, 32, 1)]


def _fft_flops(m1, m2):
    return 2 * 5.0 * m1 * m2 * math.log2(m1 * m2)


def work(case):
    fam = case['family']
    if fam == 'matvec':
        B, esz = case['m1'] * case['m2'], 8 if case['f32'] else 16
        if case['kernel'] == 'pball':
            flops = case['modes'] * _fft_flops(case['m1'], case['m2'])
        else:                                    # the band's degrees of freedom along each axis
            h1, h2 = case['fc'] * case['m1'] / 2 + 1, case['fc'] * case['m2'] + 1
            flops = case['modes'] * 16.0 * (B * h2 + case['m1'] * h1 * h2)
        return dict(bytes=2.0 * case['modes'] * B * esz, flops=flops)
    if fam in ('sweep', 'fit'):
        lay = _layout(case) if fam == 'sweep' else [((case['m1'], case['m2']), case['fc'], 0)]
        K = case['rank'] if fam == 'sweep' else 2
        esz = 8 if case['f32'] else 16
        tot = sum(a * b for (a, b), _, _ in lay) * K * esz
        it = case['iters']
        # an iteration reads the stored pairs (20 at most) and reads and writes the iterate, field and gradient
        vecs = sum(2 * min(i, 20) + 6 for i in range(it))
        flops = sum(2 * it * K * _fft_flops(a, b) for (a, b), _, _ in lay)
        if fam == 'fit' or case['cold']:         # the real start's iterations: half the bytes, up to 5 pairs
            vecs += 0.5 * sum(2 * min(i, 5) + 6 for i in range(it))
            flops += sum(2 * it * K * _fft_flops(a, b) for (a, b), _, _ in lay)
        return dict(bytes=float(tot) * vecs, flops=flops)
    if fam == 'rows':
        n = case['bins']
        d, q = case['dims'], 3 if case['grad'] else 0
        return dict(bytes=n * (16.0 * d + 16 + 8 * q), flops=float(n) * n * (d + 1 + 2 * q))
    if fam == 'points':
        n = 0.6 * case['points']
        return dict(bytes=24.0 * (n + case['queries']), flops=n * case['queries'] * 2 * 12.0)
    if fam == 'predict':
        q = math.pi / 4 * case['fc'] ** 2 * case['m1'] * case['m2']
        return dict(bytes=24.0 * case['queries'] + 16.0 * q, flops=8.0 * q * case['queries'])
    P = case['batch'] * case['m1'] * case['m2']
    flops = sum(18.0 * ci * co * P / s for ci, co, s in _CONVS)
    acts = sum(2.0 * (ci + co) * P / s for ci, co, s in _CONVS)
    weights = sum(9.0 * ci * co for ci, co, _ in _CONVS)
    if fam == 'net_predict':
        return dict(bytes=acts + 2 * weights + 8.0 * P, flops=flops)
    # backward: the activations again, their gradients written and read, two products; Adam on weights and moments
    return dict(bytes=4 * acts + 30 * weights, flops=3 * flops)


# ---------------------------------------------------------------------------------------------------------- exact
def _pball_mask(shape, fc):
    k1 = torch.fft.fftfreq(shape[0], 1.0 / shape[0], dtype=torch.float64, device='cuda')[:, None] / shape[0]
    k2 = torch.fft.fftfreq(shape[1], 1.0 / shape[1], dtype=torch.float64, device='cuda')[None, :] / shape[1]
    R = fc / 2
    return ((k1 ** 2 + k2 ** 2) <= R * R * (1 + 1e-9) + 1e-12).to(torch.float64)


def _sinc(f, t):
    return f * torch.sinc(f * t)


def _kernel_1d(kind, f, t, P=None):
    """A column's kernel at differences t, and its derivatives by log fc and by a shift."""
    if kind == 'dirichlet':
        M = 2 * math.floor(f * P / 2 + 1e-9) + 1
        u = torch.remainder(t.abs(), P)
        u = torch.minimum(u, P - u)
        near = u < 1e-10
        v = torch.sin(math.pi * M * u / P) / torch.sin(math.pi * torch.where(near, 0.5 * P, u) / P)
        return torch.where(near, M, v) / P, None, None
    v, dl = _sinc(f, t), f * torch.cos(math.pi * f * t)
    small = (math.pi * f * t).abs() < 1e-4
    ts = torch.where(small, 1.0, t)
    ds = torch.where(small, -f * (math.pi * f) ** 2 * t / 3.0,
                     (math.pi * f * t * torch.cos(math.pi * f * t) - torch.sin(math.pi * f * t)) / (math.pi * ts * ts))
    if kind.startswith('slits'):
        fi = (1.0 - float(kind.split(':')[1])) * f
        v, dl, ds = v - _sinc(fi, t), dl - fi * torch.cos(math.pi * fi * t), None
    return v, dl, ds


def _exact_matvec(case, seed):
    shape = (case['m1'], case['m2'])
    _, e = _coefs(shape, case['fc'], 1e5, case['modes'], True, _gen(seed))
    if case['f32']:
        e = e.to(torch.complex64).to(torch.complex128)
    if case['kernel'] == 'pball':
        return torch.fft.ifft2(_pball_mask(shape, case['fc']) * torch.fft.fft2(e))
    t1, t2 = (torch.arange(m, device='cuda', dtype=torch.float64) for m in shape)
    k1 = _kernel_1d('slits:0.5', case['fc'], t1[:, None] - t1[None, :])[0].to(torch.complex128)
    k2 = _kernel_1d('sinc', case['fc'], t2[:, None] - t2[None, :])[0].to(torch.complex128)
    return k1 @ e @ k2


def _exact_rows(case, seed):
    kinds, fc, per, want = _rows_kernel(case)
    Z, w = _bins(case, seed)
    Z, w = torch.as_tensor(Z).cuda(), torch.as_tensor(np.sqrt(w)).cuda()
    s = torch.zeros(len(Z), dtype=torch.float64, device='cuda')
    ds = torch.zeros((len(Z), max(len(want), 1)), dtype=torch.float64, device='cuda')
    for i in range(0, len(Z), 1000):
        v = [_kernel_1d(kd, fc[k], (Z[i:i + 1000, None, k] - Z[None, :, k]).to(torch.float64) / _STEPS[case['dims']], per[k])
             for k, kd in enumerate(kinds)]
        prod = lambda vs: math.prod(vs[1:], start=vs[0])  # noqa: E731
        s[i:i + 1000] = prod([x[0] for x in v]) @ w
        for q, (u, p) in enumerate(want):
            ds[i:i + 1000, q] = prod([x[1 if p == 'fc' else 2] if k == u else x[0] for k, x in enumerate(v)]) @ w
    return (s, ds) if case['grad'] else s


def _exact_points(case, seed):
    X, Xq = _point_data(case, seed)
    n, fc = float(len(X)), np.array(_POINT_FC)
    h = 0.1 * n ** -0.25 / fc
    h[1] = 1.0 / max(8, math.ceil(1.0 / h[1] - 1e-9))
    Zx = np.round(X[:, 0] / h[0]) * h[0]
    Zy = np.mod(np.round(np.mod(X[:, 1], 1.0) / h[1]) * h[1], 1.0)
    Z, w = np.unique(np.stack([Zx, Zy], 1) + 0.0, axis=0, return_counts=True)
    Z, w, Xq = (torch.as_tensor(a, dtype=torch.float64).cuda() for a in (Z, w, Xq))

    def gram(A, v):
        out = torch.empty(len(A), dtype=torch.float64, device='cuda')
        for i in range(0, len(A), 500):
            t = A[i:i + 500, None] - Z[None]
            out[i:i + 500] = (_kernel_1d('sinc', fc[0], t[..., 0])[0] *
                              _kernel_1d('dirichlet', fc[1], t[..., 1], 1.0)[0]) @ v
        return out
    k0 = fc[0] * (2 * math.floor(fc[1] / 2 + 1e-9) + 1)
    e = (n * w / k0).sqrt()
    e = e * (n / (e @ gram(Z, e)).sqrt())
    return ((gram(Xq, e) / n) ** 2).cpu().numpy()


def _exact_predict(case, seed):
    shape = (case['m1'], case['m2'])
    w = _counts(shape, case['fc'], 1e5, _gen(seed))
    n = float(w.sum())
    mask = _pball_mask(shape, case['fc'])
    S = lambda e: torch.fft.ifft2(mask * torch.fft.fft2(e))  # noqa: E731
    dot = lambda a, b: float((a.conj() * b).real.sum())  # noqa: E731
    unit = lambda e, u: n / math.sqrt(dot(e, u))  # noqa: E731
    e = (n * w / (float(mask.sum()) / (shape[0] * shape[1]))).sqrt().to(torch.complex128)
    e = e * unit(e, S(e))                            # the real start, uniterated
    z = torch.as_tensor(np.random.default_rng(0).standard_normal(shape)).cuda()
    e = e * torch.polar(torch.ones_like(z), 0.1 * z)
    u = S(e)
    e, u = e * unit(e, u), u * unit(e, u)
    like = lambda a, b: float(torch.where(w > 0, w * b.abs().square().log(), 0.0).sum()) - n * math.log(dot(a, b))  # noqa: E731
    ec = torch.where(w > 0, dot(e, u) / n * w / u.abs().square() * u, 0.0)
    uc = S(ec)
    if like(ec, uc) >= like(e, u) - 1e-9 * n:        # the canonical form
        e, u = ec, uc
    e = e * unit(e, u)
    C = mask * torch.fft.fft2(e) / (shape[0] * shape[1])
    Xq = torch.as_tensor(np.random.default_rng(seed).uniform(0, 1, (case['queries'], 2)) * np.array(shape)).cuda()
    k1, k2 = (torch.fft.fftfreq(m, 1.0 / m, dtype=torch.float64, device='cuda') for m in shape)
    C = C[mask.any(1)][:, mask.any(0)]
    k1, k2 = k1[mask.any(1)], k2[mask.any(0)]
    out = []
    for x in Xq.split(4096):
        p1, p2 = (torch.polar(torch.ones_like(a), 2 * math.pi * (a - a.round()))
                  for a in (x[:, :1] * k1 / shape[0], x[:, 1:] * k2 / shape[1]))
        out.append(((p1 @ C) * p2).sum(1) / n)
    return torch.cat(out).abs().square().cpu().numpy()


def _exact_net(case, seed):
    import torch.nn.functional as F
    from blml_b200 import warmstart
    x, t = _net_inputs(case, seed)
    P = {k: torch.as_tensor(np.asarray(v, np.float32)).cuda().double().requires_grad_(case['family'] == 'net_train')
         for k, v in warmstart.init_params(seed).items()}

    def conv(name, a):
        wt = P[name + '.w']
        return F.relu(F.conv2d(a, wt.view(wt.shape[0], 3, 3, -1).permute(0, 3, 1, 2), P[name + '.b'], padding=1))
    up = lambda a: F.interpolate(a, scale_factor=2, mode='nearest')  # noqa: E731
    s1 = conv('enc1b', conv('enc1a', x.double().permute(0, 3, 1, 2)))
    s2 = conv('enc2b', conv('enc2a', F.avg_pool2d(s1, 2)))
    s3 = conv('enc3b', conv('enc3a', F.avg_pool2d(s2, 2)))
    b = conv('bot2', conv('bot1', F.avg_pool2d(s3, 2)))
    d3 = conv('dec3b', conv('dec3a', torch.cat([up(b), s3], 1)))
    d2 = conv('dec2b', conv('dec2a', torch.cat([up(d3), s2], 1)))
    d1 = conv('dec1b', conv('dec1a', torch.cat([up(d2), s1], 1)))
    u = (torch.einsum('oc,nchw->nhwo', P['head.w'], d1) + P['head.b']).contiguous()
    HW = case['m1'] * case['m2']
    if case['family'] == 'net_predict':
        return (torch.view_as_complex(u) / math.sqrt(HW)).detach()
    uc, tc = torch.view_as_complex(u).flatten(1), torch.view_as_complex(t.double()).flatten(1)
    tt = tc.abs().square().sum(1)
    m = torch.maximum((tc.conj() * uc).sum(1).abs(), (tc * uc).sum(1).abs())
    loss = (uc.abs().square().sum(1) + tt - 2 * m) / tt
    loss.mean().backward()
    grads = torch.cat([v.grad.reshape(-1) for v in P.values()])
    # Adam's first step is close to the sign of the gradient: no useful 64-bit value for the weights
    return dict(u=u.detach(), loss=loss.detach(), grads=grads, params=None)


def exact(case, seed):
    fam = case['family']
    if fam in ('sweep', 'fit'):
        return None          # iterated solvers: a whole fit in plain 64-bit code takes minutes
    return dict(matvec=_exact_matvec, rows=_exact_rows, points=_exact_points, predict=_exact_predict,
                net_predict=_exact_net, net_train=_exact_net)[fam](case, seed)
