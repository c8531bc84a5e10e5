"""Performance cases: what users of the framework have it do, through its
public entry points, with the bytes and operations each pass cannot do
without and a plain float64 PyTorch value of every computed output.

Kinds of case (``case["kind"]``):

* ``ops``: the forward operator and its adjoint, the two callables a
  reconstruction loop of one's own is built from.
* ``tv``: the Chambolle TV denoiser with the long inner loops of the legacy
  drivers (30 steps) or the short ones of the plug-and-play loops (5).
* ``driver``: the reference-facing ``gap_denoise`` with the ground truth at
  hand, as the reference's scripts call it (per-iteration PSNR, per-frame
  PSNR and SSIM).
* ``solver``: a device-resident reconstruction (GAP or ADMM, binary or
  grayscale coded aperture, scikit-image or MATLAB-default TV).
* ``cassi``: spectral reconstruction behind one dispersed aperture.
* ``batch``: many uneven measurements solved together.
* ``unrolled``: forward and backward of the differentiable unrolled solver,
  the training step of a learned mask.
* ``metrics``: per-frame PSNR and SSIM of a reconstruction.
* ``cnn``: one denoiser call of the plug-and-play CNN stage.
"""
import math

import torch
import torch.nn.functional as F

import sci_algorithms_gb300 as sci

EPS_TV = 2e-4  # the TV stop tolerance every driver passes on


def listed():
    return [
        # the smallest calls: A and At on the reference's benchmark size
        # (256 x 256 x 8), where launches and host work are everything
        dict(name="ops_256x256x8", kind="ops", H=256, W=256, B=8),
        # the legacy drivers' 30-step TV, on odd frame sizes (a crop)
        dict(name="tv30_517x643x10", kind="tv", H=517, W=643, B=10, steps=30, weight=0.1),
        # the reference demo's reconstruction: 40 GAP iterations of a 256 x
        # 256 x 8 block with the ground truth tracked
        dict(name="gap_driver_256x256x8", kind="driver", H=256, W=256, B=8, iters=40),
        # the headline reconstruction: annealed weights, binary mask, 60 iterations
        dict(name="gap_2048x2048x24", kind="solver", proj="gap", tvm="tv_chambolle", gray=False,
             H=2048, W=2048, B=24, iters=60),
        # ADMM on an ordinary camera crop, the reference's 50 iterations
        dict(name="admm_512x512x10", kind="solver", proj="admm", tvm="tv_chambolle", gray=False,
             H=512, W=512, B=10, iters=50),
        # a calibrated (grayscale) aperture at HD with the MATLAB twin's default TV
        dict(name="clip_gray_1080x1920x8", kind="solver", proj="gap", tvm="ATV_ClipA", gray=True,
             H=1080, W=1920, B=8, iters=40),
        # spectral imaging, 28 bands
        dict(name="cassi_256x256x28", kind="cassi", H=256, W=256, B=28, iters=80),
        # bulk solve of uneven measurements
        dict(name="batch16_uneven", kind="batch", n=16, most=512, shapes=3, iters=50),
        # one training step of a learned aperture: 16 scenes, 20 unrolled iterations
        dict(name="unrolled_16x256x256x8", kind="unrolled", N=16, H=256, W=256, B=8, K=20),
        # quality of a full-size reconstruction
        dict(name="metrics_2048x2048x8", kind="metrics", H=2048, W=2048, B=8),
        # the CNN stage at the reference's benchmark size, default precision
        dict(name="ffdnet_256x256x8", kind="cnn", net="ffdnet", H=256, W=256, B=8,
             precision="tf32"),
        # the CNN stage at a large size, bfloat16 tensor cores
        dict(name="fastdvdnet_1024x1024x8", kind="cnn", net="fastdvdnet", H=1024, W=1024, B=8,
             precision="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, most, B):
    """H, W over [lo, hi] (any residue), B H W at most `most`."""
    while True:
        H, W = _log(rng, lo, hi), _log(rng, lo, hi)
        if rng.random() < 0.5:  # sensor-like widths
            W = max(lo, W // 8 * 8)
        if H * W * B <= most:
            return H, W


def draw(rng):
    kind = rng.choice(["ops", "tv", "driver", "solver", "solver", "cassi", "batch", "unrolled",
                       "metrics", "cnn"])
    B = rng.randint(4, 24)
    if kind == "ops":
        H, W = _size(rng, 64, 2048, 1 << 26, B)
        return dict(kind=kind, H=H, W=W, B=B)
    if kind == "tv":
        H, W = _size(rng, 64, 2048, 1 << 26, B)
        return dict(kind=kind, H=H, W=W, B=B, steps=rng.choice([5, 10, 20, 30, 50]),
                    weight=round(rng.uniform(0.05, 0.3), 3))
    if kind == "driver":
        H, W = _size(rng, 64, 1024, 1 << 23, B)
        return dict(kind=kind, H=H, W=W, B=B, iters=rng.randint(20, 50))
    if kind == "solver":
        H, W = _size(rng, 128, 2048, 1 << 26, B)
        return dict(kind=kind, proj=rng.choice(["gap", "gap", "admm"]),
                    tvm=rng.choice(["tv_chambolle", "tv_chambolle", "ATV_ClipA"]),
                    gray=rng.random() < 0.3, H=H, W=W, B=B, iters=rng.randint(20, 60))
    if kind == "cassi":
        B = rng.randint(16, 31)
        H, W = _size(rng, 128, 512, 1 << 22, B)
        return dict(kind=kind, H=H, W=W, B=B, iters=rng.randint(40, 80))
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(4, 16), most=rng.choice([256, 512]),
                    shapes=rng.randrange(1 << 20), iters=rng.randint(20, 50))
    if kind == "unrolled":
        H, W = _size(rng, 64, 256, 1 << 19, 8)
        return dict(kind=kind, N=rng.randint(2, 16), H=H, W=W, B=8, K=rng.randint(5, 20))
    if kind == "metrics":
        H, W = _size(rng, 64, 2048, 1 << 25, B)
        return dict(kind=kind, H=H, W=W, B=B)
    B = rng.randint(4, 10)
    net = rng.choice(["ffdnet", "fastdvdnet"])
    H, W = _size(rng, 128, 1024, 1 << 23, B)
    return dict(kind=kind, net=net, H=H, W=W, B=B, precision=rng.choice(["tf32", "bf16"]))


# ------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * (salt + 1) + int(seed))


def _scene(H, W, B, seed):
    """A smooth moving scene in [0, 1], B x H x W: plane waves and drifting
    Gaussian blobs, like the package's own synthetic videos."""
    g = torch.Generator().manual_seed(int(seed))
    r = torch.rand(11, 6, generator=g, dtype=torch.float64).tolist()
    y = torch.arange(H, device="cuda", dtype=torch.float32).view(1, H, 1)
    x = torch.arange(W, device="cuda", dtype=torch.float32).view(1, 1, W)
    t = torch.arange(B, device="cuda", dtype=torch.float32).view(B, 1, 1)
    out = torch.zeros(B, H, W, device="cuda")
    for a in r[:6]:
        k = 2 * math.pi * (2 + 14 * a[0]) / max(H, W)
        th = math.pi * a[1]
        out += (0.2 + 0.8 * a[3]) * torch.cos(
            k * math.cos(th) * x + k * math.sin(th) * y + 2 * math.pi * a[2]
            + (0.6 * a[4] - 0.3) * t)
    for a in r[6:]:
        s = 8 + 12 * a[0]
        cy, cx = (0.15 + 0.7 * a[1]) * H, (0.15 + 0.7 * a[2]) * W
        v, th = 2 + 2 * a[3], 2 * math.pi * a[4]
        out += (0.6 + a[5]) * torch.exp(
            -0.5 * (((y - cy - v * math.sin(th) * t) / s) ** 2
                    + ((x - cx - v * math.cos(th) * t) / s) ** 2))
    out -= out.min()
    return out / out.max()


def _mask(H, W, B, seed, gray=False, p=0.5):
    """Coded aperture: Bernoulli, or calibrated gray values of one."""
    m = (torch.rand(B, H, W, device="cuda", generator=_gen(seed, 1)) < p).float()
    if gray:
        m = m * 0.8 + 0.05 + 0.1 * torch.rand(B, H, W, device="cuda", generator=_gen(seed, 2))
    return m


def _measure(scene, mask, seed, noise=0.01):
    y = (scene * mask).sum(0)
    return y + noise * y.max() * torch.randn(y.shape, device="cuda", generator=_gen(seed, 3))


def _last(t):
    """The reference's frames-last view of a planar stack, without a copy."""
    return t.permute(1, 2, 0)


def _weights(case):
    """Annealed TV weights, 0.2 to 0.05."""
    n = case["iters"]
    return [0.2 * (0.25 ** (k / max(1, n - 1))) for k in range(n)]


def _video(case, seed):
    H, W, B = case["H"], case["W"], case["B"]
    scene = _scene(H, W, B, seed)
    mask = _mask(H, W, B, seed, case.get("gray", False))
    return scene, mask, _measure(scene, mask, seed)


def _spectral(case, seed):
    """A cube of smooth spectra, one Bernoulli aperture, the dispersed
    measurement (2 pixels per band)."""
    H, W, L = case["H"], case["W"], case["B"]
    cube = _scene(H, W, L, seed)
    ap = _mask(H, W, 1, seed)[0]
    y = torch.zeros(H, W + 2 * (L - 1), device="cuda")
    for b in range(L):
        y[:, 2 * b:2 * b + W] += ap * cube[b]
    return cube, ap, y


def _batch_shapes(case):
    """(S, S, B, p) of each measurement, from the case alone."""
    g = torch.Generator().manual_seed(case["shapes"])
    sizes = [s for s in (128, 256, 512, 1024) if s <= case["most"]]
    out = []
    for _ in range(case["n"]):
        i, b = (int(torch.randint(k, (1,), generator=g)) for k in (len(sizes), 4))
        out.append((sizes[i], sizes[i], (8, 16, 24, 32)[b],
                    0.3 + 0.4 * float(torch.rand(1, generator=g))))
    return out


def _batch(case, seed):
    out = []
    for i, (H, W, B, p) in enumerate(_batch_shapes(case)):
        s = 64 * int(seed) + i
        mask = _mask(H, W, B, s, p=p)
        out.append((mask, _measure(_scene(H, W, B, s), mask, s, noise=0.0)))
    return out


def _training(case, seed):
    N, H, W, B = case["N"], case["H"], case["W"], case["B"]
    x = torch.stack([_scene(H, W, B, 64 * int(seed) + i) for i in range(N)])
    logits = torch.randn(B, H, W, device="cuda", generator=_gen(seed, 4))
    lambdas = torch.full((case["K"],), 0.1, device="cuda")
    return logits, lambdas, x


def _noisy(case, seed, level):
    t = _scene(case["H"], case["W"], case["B"], seed)
    return t, t + level * torch.randn(t.shape, device="cuda", generator=_gen(seed, 5))


_DEN = {"in0": (2, 90, 3), "in1": (90, 32, 1), "d0a": (32, 64, 1), "d0b": (64, 64, 1),
        "d0c": (64, 64, 1), "d1a": (64, 128, 1), "d1b": (128, 128, 1), "d1c": (128, 128, 1),
        "u2a": (128, 128, 1), "u2b": (128, 128, 1), "u2c": (128, 256, 1), "u1a": (64, 64, 1),
        "u1b": (64, 64, 1), "u1c": (64, 128, 1), "o0": (32, 32, 1), "o1": (32, 1, 1)}
_NO_BN = ("u2c", "u1c", "o1")


def _net_weights(net, seed):
    """Seeded parameters (the trained checkpoints are not in the tree):
    variance-preserving convolutions, batch norm statistics near 1, a weak
    last layer so that the estimated noise stays small."""
    g = torch.Generator().manual_seed(7 + int(seed))
    sd = {}

    def conv(name, cin, cout, gain=1.4):
        sd[name + ".weight"] = torch.randn(cout, cin, 3, 3, generator=g) * gain / math.sqrt(9 * cin)

    def norm(name, c):
        sd[name + ".weight"] = 0.9 + 0.2 * torch.rand(c, generator=g)
        sd[name + ".bias"] = 0.05 * torch.randn(c, generator=g)
        sd[name + ".running_mean"] = 0.05 * torch.randn(c, generator=g)
        sd[name + ".running_var"] = 0.8 + 0.4 * torch.rand(c, generator=g)
        sd[name + ".num_batches_tracked"] = torch.tensor(1)

    if net == "ffdnet":
        for i in range(15):
            conv("convs.%d" % i, 5 if i == 0 else 64, 4 if i == 14 else 64, 0.2 if i == 14 else 1.4)
            if 0 < i < 14:
                norm("norms.%d" % (i - 1), 64)
        return sd
    for blk in ("temp1", "temp2"):
        for name, (cin, cout, _) in _DEN.items():
            conv("%s.conv.%s" % (blk, name), cin, cout, 0.2 if name == "o1" else 1.4)
            if name not in _NO_BN:
                norm("%s.bn.%s" % (blk, name), cout)
    return sd


_SIGMA = 25 / 255


# ----------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "ops":
        scene, mask, _ = _video(case, seed)
        st.update(ops=sci.make_ops(_last(mask)), x=_last(scene))
    elif kind == "tv":
        st.update(f=_last(_noisy(case, seed, 0.1)[1]))
    elif kind == "driver":
        scene, mask, y = _video(case, seed)
        A, At = sci.make_ops(_last(mask))
        st.update(A=A, At=At, y=y, phisum=_guard(mask.sum(0)), orig=_last(scene))
    elif kind == "solver":
        _, mask, y = _video(case, seed)
        st.update(y=y, solver=sci.Solver(
            sci.MaskOperator(_last(mask)), case["proj"], iters=case["iters"],
            tv_weight=_weights(case) if case["tvm"] == "tv_chambolle" else 0.02,
            tvm=case["tvm"], accelerate=True, gamma=0.01))
    elif kind == "cassi":
        _, ap, y = _spectral(case, seed)
        st.update(y=y, solver=sci.CassiSolver(sci.CassiOperator(ap, case["B"], 2), case["iters"]))
    elif kind == "batch":
        items = _batch(case, seed)
        st.update(solver=sci.BatchSolver([y for _, y in items], [_last(m) for m, _ in items],
                                         iters=case["iters"]))
    elif kind == "unrolled":
        logits, lambdas, x = _training(case, seed)
        st.update(logits=logits.requires_grad_(), lambdas=lambdas.requires_grad_(), x=x,
                  ws=sci.unrolled_workspace(*x.shape, K=case["K"]))
    elif kind == "metrics":
        orig, x = _noisy(case, seed, 0.03)
        st.update(orig=orig, x=x)
    else:
        ff = case["net"] == "ffdnet"
        net = sci.FFDNet(1) if ff else sci.FastDVDnet(5, 1)
        net.load_state_dict(_net_weights(case["net"], seed))
        st.update(net=net.to(_dev()).eval(), v=_last(_noisy(case, seed, _SIGMA)[1]))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "ops":
        A, At = st["ops"]
        y = A(st["x"])
        return y, At(y)
    if kind == "tv":
        return sci.denoise_tv_chambolle(st["f"], case["weight"], n_iter_max=case["steps"],
                                        multichannel=True)
    if kind == "driver":
        x, psnr, ssim, psnr_all = sci.gap_denoise(
            st["y"], st["phisum"], st["A"], st["At"], _lambda=1, accelerate=True,
            iter_max=case["iters"], tv_weight=0.1, tv_iter_max=5, X_orig=st["orig"])
        return dict(x=x, psnr=torch.tensor(psnr), ssim=torch.tensor(ssim),
                    psnr_all=torch.tensor(psnr_all))
    if kind in ("solver", "cassi"):
        return st["solver"].run(st["y"])
    if kind == "batch":
        return list(st["solver"].run())
    if kind == "unrolled":
        loss = sci.unrolled_loss(st["logits"], st["lambdas"], st["x"], K=case["K"], ws=st["ws"])
        return loss.detach(), torch.autograd.grad(loss, (st["logits"], st["lambdas"]))
    if kind == "metrics":
        psnr, ssim = sci.metrics.frame_psnr_ssim(st["orig"], st["x"])
        return torch.tensor(psnr), torch.tensor(ssim)
    if case["net"] == "ffdnet":
        return sci.ffdnet_vdenoiser(st["v"], _SIGMA, model=st["net"], precision=case["precision"])
    return sci.fastdvdnet_denoiser(st["v"], _SIGMA, model=st["net"], gray=True,
                                   precision=case["precision"])


# -------------------------------------------------------------------- work
_UPDATE = 22  # operations of one TV dual update of a pixel
_FIRST = 8    # of the projection of a pixel


def work(case):
    """Inputs read once, outputs written once; operations of the method."""
    kind = case["kind"]
    if kind == "batch":
        n = sum(h * w * b for h, w, b, _ in _batch_shapes(case))
        hw = sum(h * w for h, w, _, _ in _batch_shapes(case))
        return dict(bytes=4 * n + 8 * hw, flops=case["iters"] * n * (4 * _UPDATE + _FIRST))
    H, W, B = case["H"], case["W"], case["B"]
    hw, n = H * W, H * W * B
    if kind == "ops":
        return dict(bytes=12 * n + 4 * hw, flops=3 * n)
    if kind == "tv":
        return dict(bytes=8 * n, flops=(case["steps"] - 1) * n * _UPDATE)
    if kind == "metrics":
        return dict(bytes=8 * n, flops=40 * n)
    if kind == "driver":
        return dict(bytes=8 * n + 12 * hw,
                    flops=case["iters"] * n * (4 * _UPDATE + _FIRST + 3) + 40 * n)
    if kind == "solver":
        mask = 4 * n if case["gray"] else 4 * hw
        return dict(bytes=4 * n + 8 * hw + mask, flops=case["iters"] * n * (4 * _UPDATE + _FIRST))
    if kind == "cassi":
        wd = W + 2 * (B - 1)
        return dict(bytes=4 * n + 4 * hw + 8 * H * wd,
                    flops=case["iters"] * n * (4 * _UPDATE + _FIRST))
    if kind == "unrolled":
        N, K = case["N"], case["K"]
        return dict(bytes=4 * N * n + 8 * n, flops=3 * K * N * n * (4 * _UPDATE + _FIRST))
    if case["net"] == "ffdnet":
        h, w = (H + 1) // 2, (W + 1) // 2
        macs = h * w * 9 * (5 * 64 + 13 * 64 * 64 + 64 * 4)
        weights = 9 * (5 * 64 + 13 * 64 * 64 + 64 * 4)
    else:
        level = dict(in0=1, in1=1, d0a=4, d0b=4, d0c=4, d1a=16, d1b=16, d1c=16, u2a=16, u2b=16,
                     u2c=16, u1a=4, u1b=4, u1c=4, o0=1, o1=1)
        macs = sum(2 * 9 * a * c * hw / level[k] for k, (a, c, _) in _DEN.items())
        weights = sum(2 * 9 * a * c for a, c, _ in _DEN.values())
    return dict(bytes=8 * n + 4 * weights, flops=2 * macs * B)


# ------------------------------------------------- the same in 64 bits
def _grad64(u):
    r, c = torch.zeros_like(u), torch.zeros_like(u)
    r[..., :-1, :] = u[..., 1:, :] - u[..., :-1, :]
    c[..., :-1] = u[..., 1:] - u[..., :-1]
    return r, c


def _div64(pr, pc):
    d = pr + pc
    d[..., 1:, :] -= pr[..., :-1, :]
    d[..., 1:] -= pc[..., :-1]
    return d


def _tv64(f, weight, steps, eps=EPS_TV):
    """Chambolle's iteration per frame with its energy stop test."""
    pr, pc = torch.zeros_like(f), torch.zeros_like(f)
    res = f.clone()
    live = torch.ones(f.shape[0], dtype=torch.bool, device=f.device)
    first = prev = None
    size = f.shape[1] * f.shape[2]
    for i in range(steps):
        d = -_div64(pr, pc)
        out = f + d
        res[live] = out[live]
        gr, gc = _grad64(out)
        norm = torch.sqrt(gr * gr + gc * gc)
        e = ((d * d).sum((1, 2)) + weight * norm.sum((1, 2))) / size
        norm.mul_(0.25 / weight).add_(1)
        pr.sub_(gr, alpha=0.25).div_(norm)
        pc.sub_(gc, alpha=0.25).div_(norm)
        if i == 0:
            first = e
        else:
            live = live & ~((prev - e).abs() < eps * first)
            if not bool(live.any()):
                break
        prev = e
    return res


def _clip64(f, lam, steps=5):
    """The MATLAB twin's default denoiser: clipped dual steps, both
    directions averaged."""
    zh = torch.zeros_like(f)
    zv = torch.zeros_like(f)
    for _ in range(steps):  # z: forward differences, zero on the last column / row
        dh, dv = zh.clone(), zv.clone()
        dh[..., 1:] -= zh[..., :-1]
        dv[..., 1:, :] -= zv[..., :-1, :]
        u = f + 0.5 * (dh + dv)
        gr, gc = _grad64(u)
        zh = (zh + gc / 5).clamp_(-lam / 2, lam / 2)
        zv = (zv + gr / 5).clamp_(-lam / 2, lam / 2)
    return u


def _loop64(y, A, At, ps, proj, weights, tv, orig=None):
    x = At(y)
    track = []

    def psnr(x):
        if orig is not None:
            track.append(float(-10 * torch.log10(((x - orig) ** 2).mean())))

    if proj == "gap":
        y1 = torch.zeros_like(y)
        for w in weights:
            yb = A(x)
            y1 += y - yb
            x = tv(x + At((y1 - yb) / ps), w)
            psnr(x)
        return x, track
    theta, b = x, torch.zeros_like(x)
    for w in weights:
        t = theta + b
        x = t + At((y - A(t)) / (ps + 0.01))
        v = x - b
        theta = tv(v, w)
        b = theta - v
        psnr(x)
    return x, track


def _guard(ps):
    return torch.where(ps == 0, torch.ones_like(ps), ps)


def _video64(case, mask, y, proj, weights, tv, orig=None):
    phi = mask.double()
    return _loop64(y.double(), lambda x: (x * phi).sum(0), lambda r: r * phi, _guard(phi.sum(0)),
                   proj, weights, tv, orig)


def _quality64(orig, x):
    """Per-frame PSNR and SSIM (7 x 7 uniform windows, sample covariance)."""
    orig, x = orig.double(), x.double()
    psnr = -10 * torch.log10(((orig - x) ** 2).mean((1, 2)))
    a, b = orig[:, None], x[:, None]

    def mean(t):
        return F.avg_pool2d(t, 7, 1)

    ua, ub = mean(a), mean(b)
    k = 49 / 48
    va, vb, vab = (k * (mean(p * q) - u * v) for p, q, u, v in
                   ((a, a, ua, ua), (b, b, ub, ub), (a, b, ua, ub)))
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    s = ((2 * ua * ub + c1) * (2 * vab + c2)) / ((ua * ua + ub * ub + c1) * (va + vb + c2))
    return psnr.float(), s.mean((1, 2, 3)).float()


def _conv64(x, w, stride=1, groups=1):
    """3 x 3 convolution as a float64 matrix product over row strips."""
    if groups > 1:
        return torch.cat([_conv64(a, b, stride) for a, b in
                          zip(x.chunk(groups, 1), w.chunk(groups, 0))], 1)
    n, c, H, W = x.shape
    wf = w.double().reshape(w.shape[0], -1)
    out = []
    for i in range(n):
        cols = F.unfold(x[i:i + 1], 3, padding=1, stride=stride)
        out.append((wf @ cols[0]).view(1, -1, (H - 1) // stride + 1, (W - 1) // stride + 1))
    return torch.cat(out)


def _ffdnet64(sd, v):
    n, H, W = v.shape
    x = F.pixel_unshuffle(F.pad(v[:, None], (0, W % 2, 0, H % 2), mode="replicate"), 2)
    h = torch.cat([torch.full_like(x[:, :1], float(torch.tensor(_SIGMA))), x], 1)
    for i in range(15):
        h = _conv64(h, sd["convs.%d.weight" % i])
        if 0 < i < 14:
            h = _norm64(sd, "norms.%d" % (i - 1), h)
        if i < 14:
            h = h.relu_()
    return v - F.pixel_shuffle(h, 2)[:, 0, :H, :W]


def _norm64(sd, name, h):
    p = {k: sd["%s.%s" % (name, k)].double() for k in ("weight", "bias", "running_mean",
                                                      "running_var")}
    s = p["weight"] / torch.sqrt(p["running_var"] + 1e-5)
    return h * s[:, None, None] + (p["bias"] - p["running_mean"] * s)[:, None, None]


def _den64(sd, blk, f0, f1, f2, sigma):
    def c(name, h, stride=1, groups=1):
        h = _conv64(h, sd["%s.conv.%s.weight" % (blk, name)], stride, groups)
        return h if name in _NO_BN else _norm64(sd, "%s.bn.%s" % (blk, name), h).relu_()

    m = torch.full_like(f0, sigma)
    x0 = c("in1", c("in0", torch.stack([f0, m, f1, m, f2, m])[None], groups=3))
    x1 = c("d0c", c("d0b", c("d0a", x0, 2)))
    x2 = c("d1c", c("d1b", c("d1a", x1, 2)))
    x1 = x1 + F.pixel_shuffle(c("u2c", c("u2b", c("u2a", x2))), 2)
    x0 = x0 + F.pixel_shuffle(c("u1c", c("u1b", c("u1a", x1))), 2)
    return f1 - c("o1", c("o0", x0))[0, 0]


def _fastdvdnet64(sd, v):
    n, H, W = v.shape
    x = F.pad(v[:, None], (0, -W % 4, 0, -H % 4), mode="reflect")[:, 0]
    s = float(torch.tensor(_SIGMA))
    for blk in ("temp1", "temp2"):
        x = torch.stack([_den64(sd, blk, x[g - 1], x[g], x[(g + 1) % n], s) for g in range(n)])
    return x[:, :H, :W]


def _unrolled64(case, logits, lambdas, x_true):
    logits = logits.double().requires_grad_()
    lambdas = lambdas.double().requires_grad_()
    total, count = 0.0, x_true.numel()
    gl, gk = torch.zeros_like(logits), torch.zeros_like(lambdas)
    for part in x_true.split(2):  # scenes share the mask: their gradients add up
        xt = part.double()
        phi = torch.sigmoid(logits)
        ps = phi.sum(0)
        y = (xt * phi).sum(1)
        x = phi * (y / ps).unsqueeze(1)
        y1 = torch.zeros_like(y)
        for k in range(case["K"]):
            yb = (x * phi).sum(1)
            y1 = y1 + (y - yb)
            f = x + lambdas[k] * (phi * ((y1 - yb) / ps).unsqueeze(1))
            pr = pc = torch.zeros_like(f)
            x = f
            for _ in range(4):
                gr = F.pad(x[..., 1:, :] - x[..., :-1, :], (0, 0, 0, 1))
                gc = F.pad(x[..., 1:] - x[..., :-1], (0, 1))
                s = gr * gr + gc * gc
                pos = s > 0
                den = 1 + 2.5 * torch.where(pos, torch.sqrt(torch.where(pos, s, 1.0)), 0.0)
                pr, pc = (pr - 0.25 * gr) / den, (pc - 0.25 * gc) / den
                x = f - (pr + pc - F.pad(pr[..., :-1, :], (0, 0, 1, 0))
                         - F.pad(pc[..., :-1], (1, 0)))
        loss = ((x - xt) ** 2).sum() / count
        a, b = torch.autograd.grad(loss, (logits, lambdas))
        total += float(loss)
        gl += a
        gk += b
    return torch.tensor(total, dtype=torch.float64), (gl, gk)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ops":
        scene, mask, _ = _video(case, seed)
        y = (scene.double() * mask.double()).sum(0)
        return y, _last(mask.double() * y)
    if kind == "tv":
        return _last(_tv64(_noisy(case, seed, 0.1)[1].double(), case["weight"], case["steps"]))
    if kind == "driver":
        scene, mask, y = _video(case, seed)
        x, track = _video64(case, mask, y, "gap", [0.1] * case["iters"],
                            lambda v, w: _tv64(v, w, 5), scene.double())
        psnr, ssim = _quality64(scene, x)
        return dict(x=_last(x), psnr=psnr, ssim=ssim, psnr_all=torch.tensor(track))
    if kind == "solver":
        _, mask, y = _video(case, seed)
        if case["tvm"] == "tv_chambolle":
            return _video64(case, mask, y, case["proj"], _weights(case),
                            lambda v, w: _tv64(v, w, 5))[0]
        return _video64(case, mask, y, case["proj"], [0.02] * case["iters"], _clip64)[0]
    if kind == "cassi":
        _, ap, y = _spectral(case, seed)
        ap, L, W = ap.double(), case["B"], case["W"]

        def A(x):
            out = torch.zeros(y.shape, dtype=torch.float64, device="cuda")
            for b in range(L):
                out[:, 2 * b:2 * b + W] += ap * x[b]
            return out

        def At(r):
            return torch.stack([ap * r[:, 2 * b:2 * b + W] for b in range(L)])

        ps = _guard(A(ap.expand(L, -1, -1)))
        return _loop64(y.double(), A, At, ps, "gap", [0.1] * case["iters"],
                       lambda v, w: _tv64(v, w, 5))[0]
    if kind == "batch":
        out = []
        for mask, y in _batch(case, seed):
            phi = mask.double()
            ps = _guard(phi.sum(0))
            x, y1, yd = phi * (y.double() / ps), torch.zeros_like(ps), y.double()
            for _ in range(case["iters"]):
                yb = (x * phi).sum(0)
                y1 += yd - yb
                x = _tv64(x + phi * ((y1 - yb) / ps), 0.1, 5)
            out.append(x)
        return out
    if kind == "unrolled":
        return _unrolled64(case, *_training(case, seed))
    if kind == "metrics":
        return _quality64(*_noisy(case, seed, 0.03))
    if work(case)["flops"] > 8e12:  # float64 convolutions of more would take too long
        return None
    sd = {k: v.cuda() for k, v in _net_weights(case["net"], seed).items()}
    v = _noisy(case, seed, _SIGMA)[1].double()
    return _last((_ffdnet64 if case["net"] == "ffdnet" else _fastdvdnet64)(sd, v))
