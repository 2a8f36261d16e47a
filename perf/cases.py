"""Performance cases: the solves and the other calls a user of this package makes.

listed() gives the standing cases, draw(rng) another one of the same ranges,
prepare(case, seed) what a program holds before the call (host arrays, a plan,
a network), run(state) one pass through the public entry points with its
outputs, work(case) the bytes and operations a pass cannot do without, and
exact(case, seed) the outputs in 64 bits from plain torch: the NUFFT as the
exact Fourier sum, and the MFISTA loop (c/mfista_nufft_lib.c:660-744), the FGP
prox (c/mfista_TV_lib.c:189-384), the leave-one-out error (c/looe_lib.c) and
the U-Net's gradients restated here.

Solves run a fixed number of iterations (no stopping rule), so that a pass is
the same work on every input.  Images of the reduced-precision forms are kept
as float32, as image files hold them; images of the FP64 forms as float64.
"""
import math
import os

import numpy as np
import torch

os.environ.setdefault("MFISTA_QUIET", "1")  # the drop-in calls print a banner otherwise

import sparseimaging_b200 as si  # noqa: E402
from sparseimaging_b200 import synth, warmstart  # noqa: E402

DEV = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
PRECISION = {"fp64": si.FP64, "fp32": si.FP32, "bf16x6": si.BF16X6, "bf16x3": si.BF16X3}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the drop-in entry on the reference's smallest configuration: 64 x 64,
        # 8 stations x 72 hour angles; one problem, every launch counts
        dict(name="dropin 64", kind="dropin", n=64, m=2016, iters=100),
        # one problem in the precision form: what is left of a lambda grid when
        # its last problem is still running
        dict(name="grid fp32 128 b1", kind="grid", n=128, m=8100, b=1, iters=20, precision="fp32"),
        # the headline workload of the benchmark: 64 lambda pairs on one uv coverage
        dict(name="grid fp32 128 b64", kind="grid", n=128, m=8100, b=64, iters=12, precision="fp32"),
        # a lambda grid in the default precision, sizes that are multiples of nothing
        dict(name="grid fp64 100 b11", kind="grid", n=100, m=2987, b=11, iters=40, precision="fp64"),
        # training targets of the 256 x 256 warm start: 64 problems of one coverage in FP64
        dict(name="grid fp64 256 b64", kind="grid", n=256, m=19998, b=64, iters=6, precision="fp64"),
        # a movie as one problem, uneven frames, the whole call from host arrays
        dict(name="movie fp64 128 t16", kind="movie", n=128, m_lo=800, m_hi=12000, frames=16, iters=40,
             precision="fp64"),
        # the gridded variant with TV (FGP 50), one problem
        dict(name="fft tv fp64 128 b1", kind="fft", n=128, cells=3000, b=1, iters=30, fgp=50, precision="fp64"),
        # a lambda grid of it in the precision form, an odd size and count
        dict(name="fft tv fp32 96 b13", kind="fft", n=96, cells=1701, b=13, iters=16, fgp=50, precision="fp32"),
        # the dense DFT lambda grid in FP64, and a smaller ragged one in the split
        # BF16 form on the tensor cores; the matrix comes from the host on every call
        dict(name="dft fp64 64 b64", kind="dft", n=64, m=8000, b=64, iters=16, precision="fp64"),
        dict(name="dft bf16x6 50 b27", kind="dft", n=50, m=3002, b=27, iters=16, precision="bf16x6"),
        # choosing lambda: leave-one-out error of three of its solutions
        dict(name="looe 64", kind="looe", n=64, m=8000, b=3, active=1261),
        # one gradient of the warm start's training at its larger size
        dict(name="unet grad 256 b8", kind="unet", n=256, b=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi, step=2):
    """An image side whose FFT lengths have small prime factors only."""
    while True:
        n = max(lo, _log(rng, lo, hi) // step * step)
        r = n
        for f in (2, 3, 5, 7, 11, 13):
            while r % f == 0:
                r //= f
        if r == 1:
            return n


def draw(rng):
    kind = rng.choice(["dropin", "grid", "grid", "grid", "movie", "fft", "fft", "dft", "looe", "unet"])
    if kind == "dropin":
        return dict(kind=kind, n=_side(rng, 32, 200), m=_log(rng, 300, 15000), iters=rng.randint(20, 60))
    if kind == "grid":
        precision = rng.choice(["fp32", "fp64"])
        n = _side(rng, 32, 256 if precision == "fp64" else 160)
        return dict(kind=kind, n=n, m=_log(rng, 500, 20000 if n > 64 else 6000), b=_log(rng, 1, 64),
                    iters=rng.randint(4, 6) if n > 160 else rng.randint(8, 16), precision=precision)
    if kind == "movie":
        lo = _log(rng, 300, 1500)
        return dict(kind=kind, n=_side(rng, 48, 128), m_lo=lo, m_hi=_log(rng, 4 * lo, 12000), frames=rng.randint(3, 16),
                    iters=rng.randint(8, 16), precision=rng.choice(["fp32", "fp64"]))
    if kind == "fft":
        n = _side(rng, 32, 160, 4)
        return dict(kind=kind, n=n, cells=max(64, int(n * n * rng.uniform(0.08, 0.25))), b=_log(rng, 1, 24),
                    iters=rng.randint(8, 16), fgp=rng.randint(30, 100), precision=rng.choice(["fp32", "fp64"]))
    if kind == "dft":
        return dict(kind=kind, n=rng.randint(32, 64), m=2 * _log(rng, 500, 4000), b=_log(rng, 1, 64),
                    iters=rng.randint(4, 8), precision=rng.choice(["fp64", "bf16x6", "bf16x3"]))
    if kind == "looe":
        n = rng.randint(32, 64)
        return dict(kind=kind, n=n, m=2 * _log(rng, 1500, 4000), b=rng.randint(1, 3),
                    active=_log(rng, 60, min(1300, n * n // 2)))
    return dict(kind=kind, n=8 * _log(rng, 4, 32), b=rng.randint(1, 8))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a), device=DEV).to(dtype)


def _phases(u, v, n):
    """exp(+i u (i - n/2)), exp(+i v (j - n/2)): the exact Fourier sum's factors."""
    k = torch.arange(n, device=DEV, dtype=torch.float64) - n // 2
    return torch.exp(1j * torch.outer(_t(u), k)), torch.exp(1j * torch.outer(_t(v), k))


def _fourier(x, ex, ey):
    return ((ex @ x.to(torch.complex128)) * ey).sum(1)


def _fourier_adj(r, ex, ey):
    return (ex.conj().transpose(0, 1) @ (r[:, None] * ey.conj())).real


def _coverage(rng, n, m):
    """m points of an Earth-rotation coverage, in baseline order."""
    stations = int(min(12, max(5, round(math.sqrt(m) / 9))))
    pairs = stations * (stations - 1) // 2
    u, v = synth.earth_rotation_uv(stations, -(-m // pairs), None, rng=rng)
    u, v = synth.scale_uv_to_radians(u, v, n, synth.safe_kmax(n))
    keep = np.sort(rng.choice(u.size, m, replace=False))
    return np.ascontiguousarray(u[keep]), np.ascontiguousarray(v[keep])


def _sky(rng, n):
    return synth.sky_blobs_ring(n, None, ring_radius=12.0 * n / 64.0, ring_width=2.0 * n / 64.0, rng=rng)


def _observe(rng, sky, u, v, noise):
    """Noisy visibilities of a sky: (vis_r, vis_i, vis_std)."""
    vis = _fourier(_t(sky), *_phases(u, v, sky.shape[0])).cpu().numpy()
    s = noise * np.abs(vis).max()
    vis = vis + s * (rng.standard_normal(vis.size) + 1j * rng.standard_normal(vis.size))
    return vis.real.copy(), vis.imag.copy(), np.full(vis.size, s)


def _largest(op, adj, shape, rng, steps=12):
    """Power iteration for the largest eigenvalue of adj(op(.)): the starting step size."""
    x = _t(rng.standard_normal(shape))
    lam = 1.0
    for _ in range(steps):
        x = x / torch.linalg.norm(x)
        y = adj(op(x))
        lam = float((x * y).sum())
        x = y
    return lam


def _pairs(top, b, tv=False):
    """b lambda pairs over 1e-4 .. 1 of the gradient's largest value at zero."""
    if b == 1:
        return [(1e-2 * top, 1e-3 * top if not tv else 1e-2 * top)]
    side = math.ceil(math.sqrt(b))
    one = np.logspace(-4, 0, side) * top
    two = np.logspace(-4, 0, -(-b // side)) * top
    return [(float(p), float(q)) for p in one for q in two][:b]


def _problems(pairs, c, iters, tv=False):
    key = "lambda_tv" if tv else "lambda_tsv"
    return [{"lambda_l1": p, key: q, "cinit": c, "maxiter": iters, "nonneg_flag": 1} for p, q in pairs]


def _nufft_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    u, v = _coverage(rng, n, case["m"])
    vr, vi, vs = _observe(rng, _sky(rng, n), u, v, 0.01)
    ex, ey = _phases(u, v, n)
    w2 = _t(1 / vs ** 2)
    top = float(_fourier_adj(_t(vr + 1j * vi, torch.complex128) * w2, ex, ey).abs().max())
    c = _largest(lambda x: _fourier(x, ex, ey) * w2, lambda r: _fourier_adj(r, ex, ey), (n, n), rng)
    return dict(geo=(u, v, vr, vi, vs), top=top, c=c)


def _movie_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n, parts, c, tops = case["n"], [], 0.0, []
    for f in range(case["frames"]):
        m = int(rng.integers(case["m_lo"], case["m_hi"] + 1))
        u, v = _coverage(rng, n, m)
        vr, vi, vs = _observe(rng, synth.sky_movie_frame(n, f, seed=seed % 9973, ring_radius=24.0 * n / 128.0), u, v, 0.02)
        ex, ey = _phases(u, v, n)
        w2 = _t(1 / vs ** 2)
        tops.append(float(_fourier_adj(_t(vr + 1j * vi, torch.complex128) * w2, ex, ey).abs().max()))
        c = max(c, _largest(lambda x: _fourier(x, ex, ey) * w2, lambda r: _fourier_adj(r, ex, ey), (n, n), rng, 8))
        parts.append((u, v, vr, vi, vs))
    off = np.concatenate([[0], np.cumsum([p[0].size for p in parts])]).astype(np.int32)
    lam = 1e-2 * float(np.median(tops))
    t = np.cumsum(rng.uniform(0.5, 1.5, case["frames"]))
    return dict(geo=tuple(np.concatenate([p[k] for p in parts]) for k in range(5)), off=off, lam=lam, c=c, t=t)


def _fft_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n, half = case["n"], case["cells"]
    a, b = np.meshgrid(np.arange(-n // 2 + 1, n // 2), np.arange(0, n // 2), indexing="ij")
    r = np.hypot(a, b)
    ok = (r >= 0.03 * n) & (r <= 0.47 * n) & ~((b == 0) & (a <= 0))
    cells = np.stack([a[ok], b[ok]], 1)
    cells = cells[rng.choice(len(cells), min(half, len(cells)), replace=False)]
    half = len(cells)
    F = np.fft.fft2(_sky(rng, n)) / n
    ua = np.concatenate([cells[:, 0] % n, -cells[:, 0] % n]).astype(np.int32)
    va = np.concatenate([cells[:, 1] % n, -cells[:, 1] % n]).astype(np.int32)
    y = F[ua[:half], va[:half]]
    s = 0.01 * np.abs(y).max()
    y = y + s * (rng.standard_normal(half) + 1j * rng.standard_normal(half))
    y = np.concatenate([y, y.conj()])
    top = float(np.abs(np.fft.ifft2(_on_grid(ua, va, y / s ** 2, n)).real).max() * n / 2)
    return dict(data=(ua, va, y.real.copy(), y.imag.copy(), np.full(2 * half, s)), top=top, c=0.5 / s ** 2)


def _on_grid(ua, va, y, n):
    g = np.zeros((n, n), y.dtype)
    g[ua, va] = y
    return g


def _dft_inputs(case, seed):
    """The stacked real matrix [Re; Im] / sigma, column-major in pinned host memory."""
    rng = np.random.default_rng(seed)
    n, m = case["n"], case["m"] // 2
    u, v = _coverage(rng, n, m)
    ex, ey = _phases(u, v, n)
    sky = _sky(rng, n)
    vis = _fourier(_t(sky), ex, ey)
    s = 0.01 * float(vis.abs().max())
    noise = rng.standard_normal(2 * m)
    y = torch.cat([vis.real, vis.imag]) / s + _t(noise)
    At = torch.empty((n * n, 2 * m), device=DEV, dtype=torch.float64)  # A's columns, one after another
    for j in range(n):  # column i n + j of A is ex[:, i] ey[:, j]
        p = ex * ey[:, j:j + 1]
        At[j::n, :m] = p.real.transpose(0, 1) / s
        At[j::n, m:] = p.imag.transpose(0, 1) / s
    host = torch.empty((n * n, 2 * m), dtype=torch.float64, pin_memory=DEV.type == "cuda")
    host.copy_(At)
    top = float((At @ y).abs().max())
    c = _largest(lambda x: x @ At, lambda r: At @ r, (n * n,), rng)
    return dict(A=host.numpy().T, y=y.cpu().numpy(), top=top, c=c, sky=sky, At=At)


def _looe_inputs(case, seed):
    d = _dft_inputs(case, seed)
    rng = np.random.default_rng(seed + 1)
    n2 = case["n"] ** 2
    X = np.zeros((case["b"], n2))
    for k in range(case["b"]):  # the sky's brightest pixels, a different count for every solution
        count = max(8, int(case["active"] * (1 - 0.1 * k)))
        keep = np.argsort(d["sky"].reshape(-1) + 1e-6 * rng.random(n2))[-count:]
        X[k, keep] = d["sky"].reshape(-1)[keep] * (1 + 0.02 * rng.standard_normal(count)) + 1e-9
    # a diagonal of the size of a tenth to a hundredth of A's squared columns
    lam = float((d["At"][0] ** 2).sum()) * np.logspace(-2, -1, max(2, case["b"]))[:case["b"]]
    return dict(A=d["A"], y=d["y"], X=X, lam=lam)


def _unet_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n, b = case["n"], case["b"]
    x, t = np.zeros((b, 2, n, n), np.float32), np.zeros((b, n, n), np.float32)
    for k in range(b):
        sky = _sky(rng, n)
        beam = np.abs(np.fft.fft2((rng.random((n, n)) < 0.1).astype(float)))
        beam = np.fft.fftshift(beam / beam.max())
        dirty = np.fft.ifft2(np.fft.fft2(sky) * np.fft.fft2(np.fft.ifftshift(beam))).real
        x[k] = [dirty / dirty.max(), beam]
        t[k] = sky / dirty.max()
    p = np.zeros(0, np.float32)
    for co, ci in _unet_shapes():
        p = np.concatenate([p, (rng.standard_normal(co * ci * 9) * math.sqrt(2.0 / (9 * ci))).astype(np.float32),
                            (0.02 * rng.standard_normal(co)).astype(np.float32)])
    p = np.concatenate([p, (0.35 * rng.standard_normal(16)).astype(np.float32), np.float32([0.01])])
    return dict(x=x, t=t, p=p)


_INPUTS = dict(dropin=_nufft_inputs, grid=_nufft_inputs, movie=_movie_inputs, fft=_fft_inputs, dft=_dft_inputs,
               looe=_looe_inputs, unet=_unet_inputs)


def prepare(case, seed):
    d = _INPUTS[case["kind"]](case, seed)
    d["case"] = case
    d.pop("At", None)
    if case["kind"] == "grid":
        # a program that solves on one coverage keeps its plan
        d["plan"] = si.Plan(*d["geo"], case["n"], case["n"], case["b"], precision=PRECISION[case["precision"]])
        d["problems"] = _problems(_pairs(d["top"], case["b"]), d["c"], case["iters"])
    elif case["kind"] in ("fft", "dft"):
        tv = case["kind"] == "fft"
        d["problems"] = _problems(_pairs(d["top"], case["b"], tv), d["c"], case["iters"], tv)
    elif case["kind"] == "unet":
        d["net"] = warmstart.UNet(case["n"], case["n"], case["b"])
        d["net"].set_params(d["p"])
    return d


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _solved(X, results, precision):
    dt = np.float64 if precision == "fp64" else np.float32
    return dict(x=X.astype(dt, copy=False), iters=np.array([r["ITER"] for r in results]),
                cost=np.array([r["finalcost"] for r in results], dt), chi2=np.array([r["sq_error"] for r in results], dt))


def run(s):
    case = s["case"]
    kind, n = case["kind"], case["n"]
    if kind == "dropin":
        (l1, ltsv), = _pairs(s["top"], 1)
        x, r = si.imaging_core_nufft(*s["geo"], n, n, case["iters"], 0.0, l1, 0.0, ltsv, s["c"])
        return _solved(x, [r], "fp64")
    if kind == "grid":
        s["plan"].set_problems(s["problems"], 0.0)
        s["plan"].run()
        return _solved(*s["plan"].fetch(), case["precision"])
    if kind == "movie":
        X, r, temporal = si.nufft_movie(*s["geo"], s["off"], n, n, s["lam"], 1e-3 * s["lam"], 5 * s["lam"], s["c"],
                                        case["iters"], 0.0, t_list=s["t"], precision=PRECISION[case["precision"]])
        return dict(_solved(X, r, case["precision"]), temporal=np.array([temporal], X.dtype if case["precision"] == "fp64" else np.float32))
    if kind == "fft":
        return _solved(*si.fft_batch(*s["data"], n, n, s["problems"], 0.0, precision=PRECISION[case["precision"]],
                                     fgp_iter=case["fgp"]), case["precision"])
    if kind == "dft":
        return _solved(*si.dft_batch(s["y"], s["A"], n, n, s["problems"], 0.0, precision=PRECISION[case["precision"]]),
                       case["precision"])
    if kind == "looe":
        mean, std, positive = si.dft_looe(s["y"], s["A"], s["X"], n, lambda_tsv=s["lam"])
        return dict(mean=mean, std=std, positive=positive)
    loss, grad = s["net"].grad(s["x"], s["t"])
    return dict(loss=np.float32(loss), grad=grad)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _nufft_flops(n, m):
    """One application: a 24 x 24 tap sum of complex cells per point and the padded FFT."""
    return 4.0 * 576 * m + 2.5 * 4 * n * n * math.log2(4 * n * n)


def work(case):
    k, n = case["kind"], case["n"]
    if k in ("dropin", "grid"):
        b = case.get("b", 1)  # an iteration: one forward and one adjoint at least
        return dict(bytes=40.0 * case["m"] + 8.0 * b * n * n, flops=2.0 * b * case["iters"] * _nufft_flops(n, case["m"]))
    if k == "movie":
        m, t = 0.5 * (case["m_lo"] + case["m_hi"]), case["frames"]
        return dict(bytes=t * (40.0 * m + 8.0 * n * n), flops=2.0 * t * case["iters"] * _nufft_flops(n, m))
    if k == "fft":  # two FFTs and one prox of `fgp` stencil sweeps (about 25 operations a pixel) an iteration
        per = 2 * 2.5 * n * n * math.log2(n * n) + 25.0 * case["fgp"] * n * n
        return dict(bytes=64.0 * case["cells"] + 8.0 * case["b"] * n * n, flops=case["b"] * case["iters"] * per)
    if k == "dft":
        a = float(case["m"]) * n * n
        return dict(bytes=8 * a + 8.0 * case["b"] * n * n, flops=4.0 * a * case["b"] * case["iters"])
    if k == "looe":  # A_S^T A_S (half of it), the factor, and the triangular solve, per solution
        s = sum(2.0 * case["m"] * (c := max(8, int(case["active"] * (1 - 0.1 * j)))) ** 2 + c ** 3 / 3 for j in range(case["b"]))
        return dict(bytes=8.0 * case["m"] * n * n, flops=s)
    macs, shapes = 0, _unet_shapes()
    for (co, ci), level in zip(shapes, _LEVEL):
        macs += co * ci * 9 * (n >> level) ** 2
    return dict(bytes=12.0 * case["b"] * n * n + 8.0 * sum(9 * co * ci for co, ci in shapes), flops=6.0 * case["b"] * macs)


# ---------------------------------------------------------------------------
# the outputs in 64 bits
# ---------------------------------------------------------------------------

def _tsv(x):
    return float((x[..., 1:, :] - x[..., :-1, :]).square().sum() + (x[..., :, 1:] - x[..., :, :-1]).square().sum())


def _tsv_grad(x):
    g = torch.zeros_like(x)
    for dim in (-1, -2):
        d = 2 * x.diff(dim=dim)
        k = x.shape[dim] - 1
        g.narrow(dim, 0, k).sub_(d)
        g.narrow(dim, 1, k).add_(d)
    return g


def _tv(x):
    a, b = x[:, 1:] - x[:, :-1], x[1:] - x[:-1]
    return float(torch.sqrt(a[:-1].square() + b[:, :-1].square()).sum() + a[-1].abs().sum() + b[:, -1].abs().sum())


def _fgp(b, lam, iters):
    """argmin |x - b|^2 / 2 + lam TV(x), x >= 0, by `iters` FGP steps."""
    n0, n1 = b.shape
    p = b.new_zeros(n0, n1 - 1)  # along the rows
    q = b.new_zeros(n0 - 1, n1)
    r, s, t = p, q, 1.0

    def x_of(p, q):
        v = b.new_zeros(n0, n1)
        v[:, :-1] += p
        v[:, 1:] -= p
        v[:-1] += q
        v[1:] -= q
        return (b - lam * v).clamp(min=0)

    for _ in range(iters):
        x = x_of(r, s)
        rp, sq = r + (x[:, :-1] - x[:, 1:]) / (8 * lam), s + (x[:-1] - x[1:]) / (8 * lam)
        size_p, size_q = rp.abs(), sq.abs()
        both = torch.sqrt(rp[:-1].square() + sq[:, :-1].square())
        size_p[:-1] = both
        size_q[:, :-1] = both
        p1, q1 = rp / size_p.clamp(min=1), sq / size_q.clamp(min=1)
        t1 = (1 + math.sqrt(1 + 4 * t * t)) / 2
        r, s = p1 + (t - 1) / t1 * (p1 - p), q1 + (t - 1) / t1 * (q1 - q)
        p, q, t = p1, q1, t1
    return x_of(p, q)


def _mfista(data, x0, l1, c, iters, smooth=None, tv=None, zero_stop=True):
    """The MFISTA loop: data(x) gives (F, -gradient of F or None), smooth(x) the
    same of a smooth regulariser, tv (lambda, FGP steps) the TV form."""
    def cost(x):
        f = data(x, False)[0]
        return f + (smooth(x, False)[0] if smooth else 0.0)

    def rest(x):
        return l1 * float(x.abs().sum()) + (tv[0] * _tv(x) if tv else 0.0)

    x = z = x0
    now, mu, done = cost(x) + rest(x), 1.0, iters
    for it in range(iters):
        f, g = data(z, True)
        if smooth:
            f2, g2 = smooth(z, True)
            f, g = f + f2, g + g2
        for _ in range(iters):
            b = z + g / c - (l1 / c)
            new = _fgp(b, tv[0] / c, tv[1]) if tv else b.clamp(min=0)
            d = new - z
            fn = cost(new)
            if fn <= f - float((g * d).sum()) + 0.5 * c * float((d * d).sum()):
                break
            c *= 1.1
        c /= 1.1
        mu1 = (1 + math.sqrt(1 + 4 * mu * mu)) / 2
        fn += rest(new)
        if fn < now:
            now = fn
            z = x * ((1 - mu) / mu1) + new * (1 + (mu - 1) / mu1)
            x = new
        else:
            z = x * (1 - mu / mu1) + new * (mu / mu1)
            if zero_stop and it > 1 and not bool(x.any()):
                done = it + 1
                break
        mu = mu1
    return x, done


def _nufft_data(u, v, vr, vi, vs, n):
    ex, ey = _phases(u, v, n)
    vis, w = _t(vr + 1j * vi, torch.complex128), _t(1 / vs)

    def data(x, grad):
        r = (vis - _fourier(x, ex, ey)) * w
        return 0.5 * float(r.abs().square().sum()), _fourier_adj(r * w, ex, ey) if grad else None
    return data


def _smooth(lam):
    return lambda x, grad: (lam * _tsv(x), -lam * _tsv_grad(x) if grad else None)


def _answer(X, costs, chi2, **more):
    return dict(x=X.reshape(X.shape[0], -1).cpu().numpy(), iters=None, cost=np.array(costs), chi2=np.array(chi2), **more)


def _solve_all(data, pairs, case, c, n, tv=None):
    """Every problem of a batch: images, objectives and chi^2 at the end."""
    X, costs, chi2 = [], [], []
    for l1, l2 in pairs:
        smooth = None if tv else _smooth(l2)
        x, _ = _mfista(data, torch.zeros(n, n, device=DEV, dtype=torch.float64), l1, c, case["iters"], smooth,
                       (l2, tv) if tv else None)
        f = data(x, False)[0]
        X.append(x)
        chi2.append(2 * f)
        costs.append(f + l1 * float(x.abs().sum()) + l2 * (_tv(x) if tv else _tsv(x)))
    return torch.stack(X), costs, chi2


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    d = _INPUTS[kind](case, seed)
    if kind in ("dropin", "grid"):
        if case.get("b", 1) * case["iters"] * case["m"] * n * n > 1e12:  # about 10 seconds
            return None
        X, costs, chi2 = _solve_all(_nufft_data(*d["geo"], n), _pairs(d["top"], case.get("b", 1)), case, d["c"], n)
        got = _answer(X, costs, chi2)
        return got if kind == "grid" else dict(got, x=got["x"][0])
    if kind == "movie":
        return _exact_movie(case, d)
    if kind == "fft":
        if case["b"] * case["iters"] * case["fgp"] > 12000:  # FGP steps are many small launches here
            return None
        ua, va, yr, yi, sd = d["data"]
        mask, y = _t(_on_grid(ua, va, 1 / sd, n)), _t(_on_grid(ua, va, (yr + 1j * yi) / sd, n), torch.complex128)

        def data(x, grad):
            r = y - mask * torch.fft.fft2(x) / n
            return 0.25 * float(r.abs().square().sum()), torch.fft.ifft2(r * mask).real * (n / 2) if grad else None
        return _answer(*_solve_all(data, _pairs(d["top"], case["b"], True), case, d["c"], n, tv=case["fgp"]))
    At = d.get("At")
    if At is None and kind != "unet":
        At = _t(np.ascontiguousarray(d["A"].T))
    if kind == "dft":
        y = _t(d["y"])

        def data(x, grad):
            r = y - x.reshape(-1) @ At
            return 0.5 * float((r * r).sum()), (At @ r).reshape(n, n) if grad else None
        return _answer(*_solve_all(data, _pairs(d["top"], case["b"]), case, d["c"], n))
    if kind == "looe":
        return _exact_looe(case, d, At)
    return _exact_unet(case, d)


def _exact_movie(case, d):
    n, off = case["n"], d["off"]
    if case["iters"] * n * n * float(off[-1]) > 2e11:
        return None
    frames = [_nufft_data(*(a[off[k]:off[k + 1]] for a in d["geo"]), n) for k in range(case["frames"])]
    wt = _t(1 / np.diff(d["t"]))[:, None, None]
    lam, lt = d["lam"], 5 * d["lam"]

    def pairs(x):
        return float(((x[:-1] - x[1:]).square() * wt).sum())

    def data(x, grad):
        got = [f(x[k], grad) for k, f in enumerate(frames)]
        return sum(g[0] for g in got), torch.stack([g[1] for g in got]) if grad else None

    def smooth(x, grad):
        g = None
        if grad:
            g = -1e-3 * lam * _tsv_grad(x)
            e = 2 * lt * (x[:-1] - x[1:]) * wt
            g[:-1] -= e
            g[1:] += e
        return 1e-3 * lam * _tsv(x) + lt * pairs(x), g

    x, _ = _mfista(data, torch.zeros(case["frames"], n, n, device=DEV, dtype=torch.float64), lam, d["c"], case["iters"],
                   smooth, zero_stop=False)
    chi2 = [2 * f(x[k], False)[0] for k, f in enumerate(frames)]
    costs = [0.5 * s + lam * float(x[k].abs().sum()) + 1e-3 * lam * _tsv(x[k]) for k, s in enumerate(chi2)]
    return _answer(x, costs, chi2, temporal=np.array([lt * pairs(x)]))


def _exact_looe(case, d, At):
    n, y, mean, std = case["n"], _t(d["y"]), [], []
    for x, lam in zip(d["X"], d["lam"]):
        S = np.nonzero(x)[0]
        Z = At[torch.as_tensor(S, device=DEV)]
        edge = [int(0 < k % n < n - 1) + int(0 < k // n < n - 1) for k in S]
        H = Z @ Z.transpose(0, 1) + torch.diag(_t([4.0 + 2 * e for e in edge]) * lam)
        lev = torch.linalg.solve_triangular(torch.linalg.cholesky(H), Z, upper=False).square().sum(0)
        t = (y - _t(x[S]) @ Z) / (1 - lev)
        s = 0.5 * t * t
        m = s.numel()
        mean.append(float(s.mean()))
        std.append(math.sqrt(float(s.square().sum()) / (m - 1) - mean[-1] ** 2 * m / (m - 1)))
    return dict(mean=np.array(mean), std=np.array(std), positive=None)


# the U-Net's convolutions in parameter order: (output, input) channels and level
_LEVEL = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 2, 1, 1, 1, 0, 0, 0]


def _unet_shapes():
    return [(16, 2), (16, 16), (32, 16), (32, 32), (64, 32), (64, 64), (128, 64), (128, 128), (64, 128), (64, 128),
            (64, 64), (32, 64), (32, 64), (32, 32), (16, 32), (16, 32), (16, 16)]


def _exact_unet(case, d):
    """Weights act through their BF16 rounding, which passes gradients on."""
    import torch.nn.functional as F
    full = _t(d["p"], torch.float32)
    weights, biases, at = [], [], 0
    for co, ci in _unet_shapes():
        k = co * ci * 9
        weights.append(full[at:at + k].bfloat16().double().reshape(co, ci, 3, 3).requires_grad_())
        biases.append(full[at + k:at + k + co].double().requires_grad_())
        at += k + co
    head = full[at:at + 16].bfloat16().double().requires_grad_()
    last = full[at + 16:].double().requires_grad_()
    conv = iter(zip(weights, biases))

    def c(x):
        w, b = next(conv)
        return F.relu(F.conv2d(x, w, b, padding=1))

    def up(x):
        return x.repeat_interleave(2, 2).repeat_interleave(2, 3)

    with torch.backends.cudnn.flags(enabled=False):
        x = _t(d["x"])
        e1 = c(c(x))
        e2 = c(c(F.max_pool2d(e1, 2)))
        e3 = c(c(F.max_pool2d(e2, 2)))
        v = c(c(F.max_pool2d(e3, 2)))
        for skip in (e3, e2, e1):
            v = c(up(v))
            v = c(c(torch.cat([v, skip], 1)))
        out = (v * head[None, :, None, None]).sum(1) + last
        loss = (out - _t(d["t"])).square().mean()
        loss.backward()
    grad = [g.grad.reshape(-1) for pair in zip(weights, biases) for g in pair] + [head.grad, last.grad]
    return dict(loss=float(loss.detach()), grad=torch.cat(grad).cpu().numpy())
