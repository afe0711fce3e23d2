"""Performance cases of binder_b200: the calls a registration program makes, through
`binder_b200._core`, over the sizes it makes them at.

Kinds of case
  register   a whole registration from host arrays (the shape of FastRegistration.run): a new
             Registration, the MI likelihood, the prior, EM, optionally topology correction, and
             the field and theta read back
  em         EM on a registration that the program keeps (restarted from its starting positions),
             with the SSD or the two-channel MI filter likelihood
  batch      many registrations of uneven sizes run as one RegistrationBatch
  sample     the Gibbs sampler, one chain or a batch of chains, every sampling switch on
  prior      the prior transformation: one smoothing and a few prior samples
  topology   topology correction of a field that folds in some thousands of voxels

Images are random ellipsoid phantoms (blur, noise), the moving one warped by a smooth random field
and passed through a monotone intensity curve, both binned between robust percentiles, as in this
repository's benchmark.  Everything is made on the GPU from the seed; host arrays that a program
would pass again and again are page-locked, as in the benchmark's end-to-end step.
"""
import math

import numpy as np
import torch

from binder_b200 import _core

ALPHA = 2.0
GAMMA = 1e-6  # per voxel: run_BINDER's default smoothness, scaled by the number of voxels
NEVER = -1e300  # convergence threshold that never fires: every pass does the same work
SIGMA2 = 9.0 / (8.0 * math.pi)
MOST_VOXELS = 160 * 192 * 160


def listed():
    return [
        # one 2D slice pair, the plain 2D benchmark configuration
        dict(name="register_2d_128x128", kind="register", nx=128, ny=128, nz=1, bins=32, iters=50,
             topology=True),
        # the smallest real volume of this repository's tests, and a pyramid's coarsest level:
        # launches and latency count
        dict(name="register_22x24x24", kind="register", nx=22, ny=24, nz=24, bins=64, iters=30,
             topology=True),
        # a cropped or coarse volume, as the learned initialiser's training registers by thousands
        dict(name="register_64x64x64", kind="register", nx=64, ny=64, nz=64, bins=64, iters=50,
             topology=False),
        # a 2 mm brain volume: every side odd, rows that are not 16-byte aligned
        dict(name="register_91x109x91", kind="register", nx=91, ny=109, nz=91, bins=64, iters=25,
             topology=False),
        # the 3D benchmark: a 1 mm brain volume, 50 iterations and topology correction
        dict(name="register_160x192x160", kind="register", nx=160, ny=192, nz=160, bins=64,
             iters=50, topology=True),
        # same-modality registration
        dict(name="em_ssd_96x96x96", kind="em", nx=96, ny=96, nz=96, bins=64, iters=20,
             likelihood="ssd"),
        # two feature channels with the MI filter likelihood
        dict(name="em_mi_filter_64x64x64", kind="em", nx=64, ny=64, nz=64, bins=48, iters=10,
             likelihood="mi_filter"),
        # a served batch of uneven pairs
        dict(name="batch_12_uneven", kind="batch", pairs=12, low=32, high=112, shapes=4242,
             bins=64, iters=20),
        # uncertainty of one registration: a single chain
        dict(name="sample_64x64x64_1", kind="sample", nx=64, ny=64, nz=64, bins=64, chains=1,
             burn=4, samples=16),
        # the sampling benchmark: 32 chains of a 96^3 pair in one batch
        dict(name="sample_96x96x96_32", kind="sample", nx=96, ny=96, nz=96, bins=64, chains=32,
             burn=2, samples=10),
        # a smoothing and eight samples of the deformation prior
        dict(name="prior_96x96x96_8", kind="prior", nx=96, ny=96, nz=96, samples=8),
        # the benchmark's folding field
        dict(name="topology_160x192x160", kind="topology", nx=160, ny=192, nz=160, rms=0.8,
             spacing=3.0),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _sides(rng, low, high, most):
    """three sides in [low, high], none far from the others, `most` voxels at most"""
    while True:
        c = _log_uniform(rng, low, high)
        s = [max(low, min(high, int(round(c * rng.uniform(0.8, 1.2))))) for _ in range(3)]
        if s[0] * s[1] * s[2] <= most:
            return s


def draw(rng):
    kind = rng.choice(["register", "register", "register", "register_2d", "em", "batch", "sample",
                       "sample_chains", "prior", "topology"])
    if kind == "register_2d":
        return dict(kind="register", nx=_log_uniform(rng, 32, 256), ny=_log_uniform(rng, 32, 256),
                    nz=1, bins=rng.randint(16, 64), iters=rng.randint(10, 50),
                    topology=rng.random() < 0.5)
    if kind == "register":
        x, y, z = _sides(rng, 20, 192, MOST_VOXELS)
        return dict(kind="register", nx=x, ny=y, nz=z, bins=rng.randint(24, 64),
                    iters=rng.randint(10, 40), topology=rng.random() < 0.3)
    if kind == "em":
        x, y, z = _sides(rng, 24, 96, 96 ** 3)
        return dict(kind="em", nx=x, ny=y, nz=z, bins=rng.randint(24, 64),
                    iters=rng.randint(5, 20), likelihood=rng.choice(["ssd", "mi_filter"]))
    if kind == "batch":
        return dict(kind="batch", pairs=rng.randint(4, 16), low=32, high=rng.randint(48, 112),
                    shapes=rng.randint(1, 1 << 30), bins=rng.randint(32, 64),
                    iters=rng.randint(10, 20))
    if kind == "sample":
        x, y, z = _sides(rng, 24, 112, 112 ** 3)
        return dict(kind="sample", nx=x, ny=y, nz=z, bins=rng.randint(32, 64), chains=1, burn=2,
                    samples=rng.randint(8, 24))
    if kind == "sample_chains":
        x, y, z = _sides(rng, 24, 96, 96 ** 3)
        return dict(kind="sample", nx=x, ny=y, nz=z, bins=rng.randint(32, 64),
                    chains=rng.randint(2, 32), burn=2, samples=rng.randint(4, 10))
    if kind == "prior":
        x, y, z = _sides(rng, 24, 128, 128 ** 3)
        return dict(kind="prior", nx=x, ny=y, nz=z, samples=rng.randint(1, 8))
    x, y, z = _sides(rng, 32, 160, 160 ** 3)
    return dict(kind="topology", nx=x, ny=y, nz=z, rms=0.8, spacing=3.0)


# ---- inputs ---------------------------------------------------------------------------------
def _dct_matrix(n):
    """orthonormal DCT-II, rows are outputs (FP64, on the GPU)"""
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    m = torch.cos(math.pi * (2 * k[None, :] + 1) * k[:, None] / (2 * n)) * math.sqrt(2.0 / n)
    m[0] *= math.sqrt(0.5)
    return m


def _eigenvalues(shape):
    """the second-order prior's eigenvalue of every DCT coefficient (FP64, on the GPU)"""
    out = torch.zeros((), dtype=torch.float64, device="cuda")
    for a, n in enumerate(shape):
        k = torch.arange(n, dtype=torch.float64, device="cuda")
        side = [1] * len(shape)
        side[a] = n
        out = out + (2.0 - 2.0 * torch.cos(math.pi * k / n)).reshape(side)
    return out ** 2


def _transform(f, inverse=False):
    """separable orthonormal DCT over all axes of f"""
    for a in range(f.dim()):
        m = _dct_matrix(f.shape[a])
        f = torch.movedim(torch.tensordot(m.T if inverse else m, f, dims=([1], [a])), 0, a)
    return f


def _smooth_field(shape, rms, spacing, gen):
    filt = 1.0 / (1.0 + (spacing / math.pi) ** 4 * _eigenvalues(shape))
    comps = [_transform(torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
                        * filt, inverse=True) for _ in shape]
    f = torch.stack(comps, -1)
    return f * (rms / f.square().sum(-1).mean().sqrt())


def _grid(shape):
    return torch.stack(torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float64)
                                        for n in shape], indexing="ij"), -1)


def _blur(img, sigma):
    r = int(4 * sigma + 0.5)
    t = torch.arange(-r, r + 1, device="cuda", dtype=torch.float32)
    w = torch.exp(-0.5 * (t / sigma) ** 2)
    w /= w.sum()
    for a in range(img.dim()):
        n = img.shape[a]
        at = torch.arange(n, device="cuda")
        img = sum(w[q] * img.index_select(a, (at + q - r).clamp(0, n - 1))
                  for q in range(2 * r + 1))
    return img


def _binned(img, bins):
    """floor bins between the 1% and 99% points, clamped (int32)"""
    flat = img.flatten()
    some = flat[:: max(1, flat.numel() // 1_000_000)].sort().values
    lo = some[int(0.01 * (some.numel() - 1))]
    hi = some[int(0.99 * (some.numel() - 1))]
    b = torch.floor((img - lo) / ((hi - lo) / (bins - 1)))
    return b.clamp(0, bins - 1).to(torch.int32)


def _pair(shape, bins, gen, moving_rms=None):
    """(fixed bins u, moving bins v) of one phantom pair, int32 on the GPU"""
    nd = len(shape)
    grid = _grid(shape).float()
    img = torch.zeros(shape, device="cuda")
    side = min(shape)
    for _ in range(12 if nd == 2 else 40):
        c = torch.rand(nd, generator=gen, device="cuda") * torch.tensor(shape, device="cuda")
        a = 0.03 * side + torch.rand(nd, generator=gen, device="cuda") * 0.28 * side
        val = torch.rand((), generator=gen, device="cuda")
        img += val * (((grid - c) / a).square().sum(-1) <= 1.0)
    img = _blur(img, 1.5 if nd == 2 else 1.0)
    img = img + 0.02 * torch.randn(shape, generator=gen, device="cuda")
    rms = moving_rms if moving_rms else (2.0 if nd == 2 else min(3.0, 0.04 * side))
    at = grid + _smooth_field(shape, rms, 8.0 if nd == 2 else 5.0, gen).float()
    size = torch.tensor(shape, device="cuda", dtype=torch.float32)
    norm = (2.0 * at / (size - 1).clamp(min=1.0) - 1.0).flip(-1)
    warped = torch.nn.functional.grid_sample(img[None, None], norm[None], mode="bilinear",
                                             padding_mode="border", align_corners=True)[0, 0]
    w = (warped - warped.min()) / (warped.max() - warped.min())
    p = 0.6 + 1.2 * torch.rand((), generator=gen, device="cuda")
    return _binned(img, bins), _binned(w ** p, bins)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)


def _host(t):
    return t.contiguous().cpu().pin_memory().numpy()


def _shape(case):
    return (case["nx"], case["ny"]) if case["nz"] == 1 else (case["nx"], case["ny"], case["nz"])


def _batch_shapes(case):
    r = np.random.default_rng(case["shapes"])
    return [tuple(int(v) for v in r.integers(case["low"], case["high"] + 1, 3))
            for _ in range(case["pairs"])]


def _inputs(shape, bins, gen):
    """the host arrays of one MI registration"""
    u, v = _pair(shape, bins, gen)
    return dict(shape=shape, bins=bins, grid=_host(_grid(shape).float()),
                D=_host(_eigenvalues(shape).float()), u=_host(u), v=_host(v),
                theta=np.full((bins, bins), 1.0 / bins, np.float32),
                nzv=float((u != 0).sum()), gamma=GAMMA * float(np.prod(shape)))


def _registration(h):
    dims = h["shape"] if len(h["shape"]) == 3 else h["shape"] + (1,)
    reg = _core.Registration(h.get("start", h["grid"]), 1, h["grid"], h["grid"], *dims, *dims, 3,
                             h["nzv"])
    reg.setNonLinearTransformation(h["gamma"], h["gamma"], h["gamma"], 1, 1, 1, 1, 1, 1, h["D"])
    return reg


def _mi_registration(h):
    reg = _registration(h)
    reg.setMILikelihood(ALPHA, h["theta"], h["bins"], h["bins"], 1, h["v"], h["u"])
    return reg


def _filter_inputs(h, gen):
    """two interleaved channels: the pair's bins and those of a second contrast"""
    u, v = _pair(h["shape"], h["bins"], gen)
    h["uf"] = np.stack([h["u"].ravel(), u.cpu().numpy().ravel()], -1).astype(np.int32).ravel()
    h["vf"] = np.stack([h["v"].ravel(), v.cpu().numpy().ravel()], -1).astype(np.int32).ravel()
    th = 0.5 + torch.rand((2, h["bins"], h["bins"]), generator=gen, device="cuda")
    h["thetaf"] = (th / th.sum(-1, keepdim=True)).cpu().numpy()
    return h


def prepare(case, seed):
    gen, kind = _generator(seed), case["kind"]
    if kind == "batch":
        regs = [_mi_registration(_inputs(s, case["bins"], gen)) for s in _batch_shapes(case)]
        return dict(case=case, regs=regs, batch=_core.RegistrationBatch(regs))
    shape = _shape(case)
    if kind == "topology":
        f = _grid(shape) + _smooth_field(shape, case["rms"], case["spacing"], gen)
        return dict(case=case, field=f.cpu().numpy())
    if kind == "prior":
        D = _eigenvalues(shape).float().cpu().numpy()
        g = 1e-3 * float(np.prod(shape)) / 64 ** 3
        field = _smooth_field(shape, 1.0, 2.0, gen).float().cpu().numpy()
        nlt = _core.NonLinearTransformation(g, g, g, 1, 1, 1, 1, 1, 1, D, *shape, 1,
                                            math.sqrt(SIGMA2), 1.0)
        return dict(case=case, nlt=nlt, field=field, gamma=g, D=D)
    h = _inputs(shape, case["bins"], gen)
    if kind == "register":
        return dict(case=case, inputs=h)
    if kind == "em":
        if case["likelihood"] == "ssd":
            # same contrast: the fixed image's bins against themselves, warped
            h["v"] = np.ascontiguousarray(np.roll(h["u"], (1, -1, 1), (0, 1, 2)))
            reg = _registration(h)
            reg.setSSDLikelihood(h["bins"], 1, 9.0, 1, 1.0, 0.0, h["v"], h["u"], 1.0, 1.0)
        else:
            _filter_inputs(h, gen)
            reg = _registration(h)
            reg.setMILikelihoodFilter(ALPHA, h["thetaf"], 1, h["vf"], h["uf"], h["bins"],
                                      h["bins"], 2)
        return dict(case=case, reg=reg, inputs=h)
    # the sampler starts from a registration's result: its positions and theta
    reg = _mi_registration(h)
    reg.EM(10, NEVER, 1, 0)
    h["start"] = reg.get_final_locations_as_numpy_array()
    h["theta"] = reg.get_likelihood_parameters().reshape(h["bins"], h["bins"])
    return dict(case=case, reg=_mi_registration(h), seed=int(seed))


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "register":
        reg = _mi_registration(state["inputs"])
        its = reg.EM(case["iters"], NEVER, 1, 0)
        if case["topology"]:
            reg.correct_topology(0.01, 100.0, 10, 10, [1.0, 1.0, 1.0])
        return dict(positions=reg.get_final_locations_as_numpy_array(),
                    theta=reg.get_likelihood_parameters(), iterations=its)
    if kind == "em":
        reg = state["reg"]
        reg.reset()
        its = reg.EM(case["iters"], NEVER, 1, 0)
        out = dict(positions=reg.get_final_locations_as_numpy_array(),
                   theta=reg.get_likelihood_parameters(), iterations=its)
        if case["likelihood"] == "ssd":
            out["sigma_sq"] = reg.ssd_parameters()["sigma_sq"]
        return out
    if kind == "batch":
        for r in state["regs"]:
            r.reset()
        its = state["batch"].EM(case["iters"], NEVER, 1)
        return dict(positions=[r.get_final_locations_as_numpy_array() for r in state["regs"]],
                    theta=[r.get_likelihood_parameters() for r in state["regs"]], iterations=its)
    if kind == "sample":
        reg = state["reg"]
        if case["chains"] == 1:
            reg.reset()
            mean, cov = reg.sampler(state["seed"], case["burn"], case["samples"], 1, 1, 1, 1, 1)
        else:
            mean, cov = reg.sampler_chains(state["seed"], case["chains"], case["burn"],
                                           case["samples"], 1, 1, 1, 1, 1, per_chain=False)
        return dict(mean=mean, cov=cov)
    if kind == "prior":
        cost, smooth = state["nlt"].smooth_deformation(state["field"])
        samples = state["nlt"].sampleDeformationField(state["field"], case["samples"])
        return dict(cost=cost, smooth=smooth, samples=samples)
    tc = _core.topology_correction_3D()
    return tc.correct_topology(state["field"], 0.01, 100.0, 10, 10, 1, [1.0, 1.0, 1.0],
                               case["nx"], case["ny"], case["nz"])


# ---- what a pass cannot do without ----------------------------------------------------------
def _em_work(shape, bins, iters, channels=1):
    """an EM iteration reads the positions and bins and writes the positions; the posterior and
    its moments are some 10 operations per neighbour, the prior six FFT-like passes"""
    V, N = float(np.prod(shape)), len(shape)
    per = V * (4 * N + 4 * N + 2 * channels)
    logs = sum(math.log2(max(n, 2)) for n in shape)
    flops = V * (4 ** N) * (8 + 2 * channels) + 2 * N * V * 2.5 * logs
    return per * iters, flops * iters


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [_em_work(s, case["bins"], case["iters"]) for s in _batch_shapes(case)]
        return dict(bytes=sum(b for b, _ in w), flops=sum(f for _, f in w))
    shape = _shape(case)
    V, N = float(np.prod(shape)), len(shape)
    if kind in ("register", "em"):
        b, f = _em_work(shape, case["bins"], case["iters"],
                        2 if case.get("likelihood") == "mi_filter" else 1)
        return dict(bytes=b + V * (8 * N + 12), flops=f)
    if kind == "sample":
        sweeps = (case["burn"] + case["samples"]) * case["chains"]
        b, f = _em_work(shape, case["bins"], sweeps)
        moments = 8 * (N + N * N) * V
        return dict(bytes=b + moments, flops=f + 30.0 * V * case["samples"] * case["chains"])
    if kind == "prior":
        logs = sum(math.log2(n) for n in shape)
        calls = 1 + case["samples"]
        return dict(bytes=V * (4 * N * (1 + calls) + 4), flops=calls * 2 * N * V * 2.5 * logs)
    return dict(bytes=V * 16 * N, flops=V * 8 * 14.0)


# ---- the same in 64 bits --------------------------------------------------------------------
def _spline(t):
    e = 1.0 - t
    return [e ** 3 / 6.0, 2.0 / 3.0 - t ** 2 + 0.5 * t ** 3, 2.0 / 3.0 - e ** 2 + 0.5 * e ** 3,
            t ** 3 / 6.0]


class _Exact:
    """EM of one registration in FP64: posterior over the 4^N nearest nodes (a node outside the
    moving image has bin 0), the likelihood's update from the soft joint histogram, and the DCT
    prior's smoothing of the posterior mean positions."""

    def __init__(self, h, u, v, log_table):
        self.shape, self.nd, self.bins = h["shape"], len(h["shape"]), h["bins"]
        self.V = int(np.prod(self.shape))
        self.x = _grid(self.shape).reshape(self.V, self.nd)
        self.pos = self.x.clone()
        D = torch.from_numpy(np.asarray(h["D"])).cuda().double()
        self.filt = 1.0 / (1.0 + h["gamma"] * SIGMA2 * D)
        self.u = [t.reshape(-1).long() for t in u]
        pad = 3
        self.vpad = []
        for t in v:
            p = torch.zeros([n + 2 * pad for n in self.shape], dtype=torch.int64, device="cuda")
            p[tuple(slice(pad, pad + n) for n in self.shape)] = t.reshape(self.shape).long()
            self.vpad.append(p)
        self.pad = pad
        self.log_table = log_table  # log-space weights (the SSD likelihood)

    def _terms(self, base, w):
        """(offsets, spline weight, per-channel node bins) of every neighbour"""
        lo = -self.pad
        idx = [[(base[:, a] + o).clamp(lo, self.shape[a] + self.pad - 1) + self.pad
                for o in range(-1, 3)] for a in range(self.nd)]
        for q in np.ndindex(*([4] * self.nd)):
            at = tuple(idx[a][q[a]] for a in range(self.nd))
            b = w[0][q[0]]
            for a in range(1, self.nd):
                b = b * w[a][q[a]]
            yield [o - 1 for o in q], b, [p[at] for p in self.vpad]

    def step(self, tables):
        """one E-step and M-step; tables: per channel [K, L] likelihoods (log ones if log_table).
        Returns the joint histograms."""
        base = torch.floor(self.pos)
        frac = self.pos - base
        base = base.long()
        w = [_spline(frac[:, a]) for a in range(self.nd)]
        flat = [t.reshape(-1) for t in tables]
        L = self.bins

        def weight(b, ks):
            if self.log_table:
                return b, flat[0][ks[0] * L + self.u[0]]
            for t, k, u in zip(flat, ks, self.u):
                b = b * t[k * L + u]
            return b, None

        top = None
        if self.log_table:
            top = torch.full((self.V,), -math.inf, dtype=torch.float64, device="cuda")
            for _, b, ks in self._terms(base, w):
                top = torch.maximum(top, weight(b, ks)[1])

        def mass(b, ks):
            b, lg = weight(b, ks)
            return b * torch.exp(lg - top) if lg is not None else b

        S = torch.zeros(self.V, dtype=torch.float64, device="cuda")
        mom = torch.zeros((self.nd, self.V), dtype=torch.float64, device="cuda")
        for off, b, ks in self._terms(base, w):
            m = mass(b, ks)
            S += m
            for a in range(self.nd):
                if off[a]:
                    mom[a] += off[a] * m
        copies = 64
        spread = (torch.arange(self.V, device="cuda") % copies) * (L * L)
        hist = [torch.zeros(copies * L * L, dtype=torch.float64, device="cuda") for _ in flat]
        for _, b, ks in self._terms(base, w):
            p = mass(b, ks) / S
            for hh, k, u in zip(hist, ks, self.u):
                hh.index_add_(0, spread + k * L + u, p)
        dream = base.double() + (mom / S).T
        r = dream - self.x
        for a in range(self.nd):
            c = _transform(r[:, a].reshape(self.shape)) * self.filt
            self.pos[:, a] = self.x[:, a] + _transform(c, inverse=True).reshape(-1)
        return [hh.reshape(copies, L, L).sum(0) for hh in hist]


def _exact_mi(h, iters, u, v, theta):
    e = _Exact(h, u, v, False)
    for _ in range(iters):
        theta = [(hh + ALPHA - 1.0) / (hh + ALPHA - 1.0).sum(1, keepdim=True)
                 for hh in e.step(theta)]
    return e.pos, torch.stack(theta)


def _exact_ssd(h, iters, u, v):
    e = _Exact(h, [u], [v], True)
    k = torch.arange(h["bins"], dtype=torch.float64, device="cuda")
    s2, scale, shift = 9.0, 1.0, 0.0
    for _ in range(iters):
        table = -(k[None, :] - shift - scale * k[:, None]) ** 2 / (2.0 * s2)
        hh = e.step([table])[0]
        G, S1, S2 = hh.sum(1), (hh * k).sum(1), (hh * k * k).sum(1)
        a00, a01, a11 = float(G.sum()), float((G * k).sum()), float((G * k * k).sum())
        b0, b1 = float(S1.sum()), float((S1 * k).sum())
        det = a00 * a11 - a01 * a01
        shift, scale = (b0 * a11 - a01 * b1) / det, (a00 * b1 - a01 * b0) / det
        t = shift + scale * k
        s2 = (float((S2 - 2.0 * S1 * t + G * t * t).sum()) + 1.0) / (a00 + 1.0)
    return e.pos, torch.tensor([scale, shift], dtype=torch.float64), s2


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sample", "topology"):
        return None  # draws, and a sequential limiter: held to the bound of their type
    gen = _generator(seed)
    if kind == "batch":
        pos, theta = [], []
        for s in _batch_shapes(case):
            h = _inputs(s, case["bins"], gen)
            p, t = _exact_mi(h, case["iters"], [torch.from_numpy(h["u"]).cuda()],
                             [torch.from_numpy(h["v"]).cuda()],
                             [torch.from_numpy(h["theta"]).cuda().double()])
            pos.append(p.reshape(*s, 3))
            theta.append(t.reshape(-1))
        return dict(positions=pos, theta=theta, iterations=None)
    shape = _shape(case)
    if kind == "prior":
        s = prepare(case, seed)
        f = torch.from_numpy(s["field"]).cuda().double()
        D = torch.from_numpy(s["D"]).cuda().double()
        out, cost = torch.empty_like(f), 0.0
        for a in range(len(shape)):
            c = _transform(f[..., a]) / (1.0 + s["gamma"] * SIGMA2 * D)
            cost += 0.5 * s["gamma"] * float((D * c * c).sum())
            out[..., a] = _transform(c, inverse=True)
        return dict(cost=cost, smooth=out, samples=None)
    h = _inputs(shape, case["bins"], gen)
    if kind == "register" and float(np.prod(shape)) * case["iters"] > 1e8:
        return None  # more than about 20 seconds of FP64
    if kind == "em" and case["likelihood"] == "ssd":
        v = np.ascontiguousarray(np.roll(h["u"], (1, -1, 1), (0, 1, 2)))
        p, t, s2 = _exact_ssd(h, case["iters"], torch.from_numpy(h["u"]).cuda(),
                              torch.from_numpy(v).cuda())
        return dict(positions=p.reshape(*shape, 3), theta=t, iterations=None, sigma_sq=s2)
    if kind == "em":
        _filter_inputs(h, gen)
        V = int(np.prod(shape))
        uf, vf = torch.from_numpy(h["uf"]).cuda(), torch.from_numpy(h["vf"]).cuda()
        # channel m of voxel (node) i is read at [i + m]
        p, t = _exact_mi(h, case["iters"], [uf[m:m + V] for m in range(2)],
                         [vf[m:m + V] for m in range(2)],
                         [torch.from_numpy(x).cuda().double() for x in h["thetaf"]])
    else:
        p, t = _exact_mi(h, case["iters"], [torch.from_numpy(h["u"]).cuda()],
                         [torch.from_numpy(h["v"]).cuda()],
                         [torch.from_numpy(h["theta"]).cuda().double()])
    # a corrected field has no plain FP64 counterpart; theta does
    return dict(positions=None if case.get("topology") else p.reshape(*shape, len(shape)),
                theta=t.reshape(-1), iterations=None)
