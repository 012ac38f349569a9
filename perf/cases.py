"""Timing cases of the forward transform and its neighbours, through the public entry points.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare``
makes what a user's program holds before the call (inputs and the plan it keeps), ``run`` is
one call, ``work`` the bytes and operations one call cannot do without, and ``exact`` the
result from the definition in 64-bit torch, without this package.

Kinds of call:

* ``call``   ``DirectSHT.__call__`` on CUDA tensors (polar points rotated);
* ``host``   the same on numpy arrays, as the reference is called (copies included);
* ``basic``  ``DirectSHT.basic_sht`` on an equatorial band;
* ``maps``   ``DirectSHT.call_maps``: several weight maps on one point set;
* ``batch``  ``DirectSHT.call_batch``: point sets of different sizes on one plan;
* ``mask``   ``MaskDeconvolution`` (the mode-coupling matrix) and ``DirectSHT.alm2cl``.
"""
import math

import numpy as np
import torch

from directsht_b200 import DirectSHT, MaskDeconvolution

XMAX = 0.75  # the constructor's default


def listed():
    return [
        # A quick look at a handful of objects: latency and launches count.
        dict(name="call_small", kind="call", precision="fp64", Nl=64, Nx=128, N=1000, sky="full", wt="ones"),
        # Full-sky catalogue at the default level, few points per spline bin.
        dict(name="call_fullsky", kind="call", precision="fp64", Nl=256, Nx=512, N=100_000, sky="full", wt="ones"),
        # A galaxy catalogue over a survey footprint, sizes that are no powers of two.
        dict(name="call_catalogue", kind="call", precision="fp64", Nl=500, Nx=1000, N=530_000, sky="survey",
             wt="lognormal"),
        # A dense survey (data or its randoms) at the default level.
        dict(name="call_survey", kind="call", precision="fp64", Nl=1024, Nx=2048, N=10_000_000, sky="survey",
             wt="lognormal"),
        # numpy arrays in, numpy alm out, as a program written for the reference calls it.
        dict(name="host_randoms", kind="host", precision="fp64", Nl=564, Nx=1000, N=1_390_001, sky="survey",
             wt="ones"),
        # Signed weights (an overdensity) on an equatorial band; Nx odd.
        dict(name="basic_band", kind="basic", precision="fp64", Nl=385, Nx=769, N=60_001, sky="band", wt="normal"),
        # Data, randoms and two systematics maps on one point set at the default level.
        dict(name="maps_fp64", kind="maps", precision="fp64", Nl=512, Nx=1024, N=400_000, sky="full", wt="normal",
             maps=4, wt32=False),
        # The mixed level: the dense survey, one transform at a time.
        dict(name="mixed_survey", kind="call", precision="mixed", Nl=1024, Nx=2048, N=10_000_000, sky="survey",
             wt="lognormal"),
        # The mixed level: float32 weight maps sharing a full-sky point set.
        dict(name="mixed_maps", kind="maps", precision="mixed", Nl=1024, Nx=2048, N=2_000_000, sky="full",
             wt="near_one", maps=8, wt32=True),
        # The mixed level: an uneven batch of mocks on one plan.
        dict(name="mixed_batch", kind="batch", precision="mixed", Nl=512, Nx=1024, N=1_000_000, sky="full",
             wt="uniform", sets=8),
        # High l on compact tables: a cap-shaped footprint.
        dict(name="mixed_high_l", kind="call", precision="mixed", Nl=1500, Nx=3000, N=4_000_000, sky="cap",
             wt="uniform", compact=True),
        # Mode-coupling matrix of a mask and the pseudo-spectra of a few alm vectors.
        dict(name="mask_coupling", kind="mask", Nl=1000, maps=4),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "call", "host", "basic", "maps", "batch", "mask"])
    if kind == "mask":
        return dict(kind="mask", Nl=_log_uniform(rng, 100, 1000), maps=rng.randint(1, 8))
    Nl = _log_uniform(rng, 48, 1024)
    Nx = max(16, min(2048, int(Nl * rng.uniform(1.7, 2.1))))
    if rng.random() < 0.7:
        Nx += Nx & 1
    case = dict(kind=kind, precision=rng.choice(["fp64", "fp64", "mixed", "mixed", "mixed_f64_tables"]), Nl=Nl, Nx=Nx,
                N=_log_uniform(rng, 1000, 6_000_000), sky=rng.choice(["full", "survey", "cap"]),
                wt=rng.choice(["ones", "lognormal", "uniform", "normal", "near_one"]))
    if kind == "basic":
        case["sky"] = "band"
    if kind == "host":
        case["N"] = min(case["N"], 1_390_001)
    if kind == "maps":
        case.update(maps=rng.randint(2, 8), wt32=rng.random() < 0.5, N=max(1000, case["N"] // 8))
    if kind == "batch":
        case.update(sets=rng.randint(2, 8), N=max(2000, case["N"] // 6))
    return case


# -- inputs ---------------------------------------------------------------------------------
def _points(sky, N, gen):
    """theta, phi (float64, CUDA) of N points: the whole sky, a survey footprint with polar and
    equatorial parts, a cap of half-angle 0.9 around theta = 1, or a band clear of the poles."""
    def u(lo, hi):
        return lo + (hi - lo) * torch.rand(N, generator=gen, device="cuda", dtype=torch.float64)

    if sky == "full":
        return torch.arccos(u(-1.0, 1.0)), u(0.0, 2 * math.pi)
    if sky == "survey":
        return torch.arccos(u(math.cos(1.2), math.cos(0.3))), u(0.0, 1.5 * math.pi)
    if sky == "band":
        return torch.arccos(u(-0.7, 0.74)), u(0.0, 2 * math.pi)
    cd, az = u(math.cos(0.9), 1.0), u(0.0, 2 * math.pi)
    sd = torch.sqrt(1.0 - cd * cd)
    c, s = math.cos(1.0), math.sin(1.0)
    x, y, z = c * sd * torch.cos(az) + s * cd, sd * torch.sin(az), c * cd - s * sd * torch.cos(az)
    return torch.arccos(z.clamp(-1.0, 1.0)), torch.remainder(torch.atan2(y, x), 2 * math.pi)


def _weights(wt, shape, gen, dtype=torch.float64):
    def normal():
        return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)

    if wt == "ones":
        w = torch.ones(shape, device="cuda", dtype=torch.float64)
    elif wt == "lognormal":
        w = torch.exp(0.5 * normal())
    elif wt == "uniform":
        w = 0.5 + torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)
    elif wt == "near_one":
        w = 1.0 + 0.3 * normal()
    else:
        w = normal()
    return w.to(dtype)


def _inputs(case, seed):
    """The case's arrays from the seed alone (CUDA tensors)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "mask":
        Nl = case["Nl"]
        ell = torch.arange(2 * Nl - 1, dtype=torch.float64, device="cuda")
        power = torch.rand(2 * Nl - 1, generator=gen, device="cuda", dtype=torch.float64) + 0.5
        window = (power / (1.0 + (ell / 30.0) ** 2)).cpu().numpy()
        alm = torch.randn((case["maps"], Nl * (Nl + 1) // 2, 2), generator=gen, device="cuda", dtype=torch.float64)
        return dict(window=window, alm=torch.view_as_complex(alm))
    if kind == "batch":
        # sizes spread over two decades up to N, the largest first
        sizes = [max(1, int(case["N"] * 10 ** (-2.0 * i / max(1, case["sets"] - 1)))) for i in range(case["sets"])]
        return dict(sets=[(*_points(case["sky"], n, gen), _weights(case["wt"], (n,), gen)) for n in sizes])
    t, p = _points(case["sky"], case["N"], gen)
    shape = (case["maps"], case["N"]) if kind == "maps" else (case["N"],)
    w = _weights(case["wt"], shape, gen, torch.float32 if case.get("wt32") else torch.float64)
    return dict(t=t, p=p, w=w)


def prepare(case, seed):
    state = dict(_inputs(case, seed), case=case)
    if case["kind"] == "mask":
        state["plan"] = DirectSHT(case["Nl"], 2)  # alm2cl needs the order alone
        return state
    state["plan"] = DirectSHT(case["Nl"], case["Nx"], precision=case["precision"],
                              compact_tables=case.get("compact", False))
    if case["kind"] == "host":
        state.update(t=state["t"].cpu().numpy(), p=state["p"].cpu().numpy(), w=state["w"].cpu().numpy())
    return state


def run(state):
    kind, plan = state["case"]["kind"], state["plan"]
    if kind in ("call", "host"):
        return plan(state["t"], state["p"], state["w"])
    if kind == "basic":
        return plan.basic_sht(state["t"], state["p"], state["w"], verbose=False)
    if kind == "maps":
        return plan.call_maps(state["t"], state["p"], state["w"])
    if kind == "batch":
        return plan.call_batch(state["sets"])
    return dict(M=MaskDeconvolution(state["case"]["Nl"], state["window"], verbose=False).Mll,
                cl=plan.alm2cl(state["alm"]))


def work(case):
    """Bytes: the points and weights once, the alm once, and one stored 8-byte value of the Ylm
    table per (l, m, node) (dYlm/dx follows from two rows of it).  Operations: the table product
    (Y and dY with two halves of a complex fold), twelve-cell spreads of four Hermite weights per
    point, the circle transforms, and the rotation's products."""
    Nl = case["Nl"]
    nlm = Nl * (Nl + 1) // 2
    if case["kind"] == "mask":
        return {"bytes": 8.0 * Nl * Nl + 8.0 * 2 * Nl + case["maps"] * (16.0 * nlm + 8.0 * Nl),
                "flops": 10.0 * Nl ** 3 / 3 + 4.0 * case["maps"] * nlm}
    Nx = case["Nx"]
    maps = case.get("maps", case.get("sets", 1))
    if case["kind"] == "batch":
        points = sum(max(1, int(case["N"] * 10 ** (-2.0 * i / max(1, maps - 1)))) for i in range(maps))
        inputs, sums = 24.0 * points, points
    else:
        inputs, sums = case["N"] * (16.0 + (4.0 if case.get("wt32") else 8.0) * maps), case["N"] * maps
    n = 4.0 * 2 ** math.ceil(math.log2(max(Nl, 2)))
    sets = 2 if case["sky"] == "band" else 4
    nodes = min(sets * Nx, 2 * max(1, case["N"])) * maps
    return {"bytes": inputs + 8.0 * nlm * Nx + 16.0 * nlm * maps,
            "flops": 16.0 * nlm * Nx * maps + 96.0 * sums + 5.0 * n * math.log2(n) * nodes
            + (0.0 if case["sky"] == "band" else 4.0 * Nl ** 3 / 3 * maps)}


# -- the definition in 64 bits --------------------------------------------------------------
def _bins(x, node_x):
    j = torch.bucketize(x, node_x, right=True) - 1
    return j.clamp(0, len(node_x) - 2)


def _fold(x, phi, w, Nl, node_x):
    """Node sums of points with cos(theta) = x (sign included): A, B of shape (maps, 2, Nl, Nx),
    complex, the second axis the parity of l - m; B goes with dY/dx.  phi is multiplied by m in
    two exact parts, so that large m lose nothing."""
    maps, Nx, dev = w.shape[0], len(node_x), x.device
    dx = float(node_x[1] - node_x[0])
    A = torch.zeros((maps, 2, Nl, Nx), dtype=torch.complex128, device=dev)
    B = torch.zeros_like(A)
    hi = (phi * 2.0 ** 26).round() / 2.0 ** 26
    lo = phi - hi
    for sign in (1, -1):
        pick = (x >= 0) if sign > 0 else (x < 0)
        if not bool(pick.any()):
            continue
        ax, wp, h, r = x[pick].abs(), w[:, pick], hi[pick], lo[pick]
        j = _bins(ax, node_x)
        order = torch.argsort(j)
        j, ax, wp, h, r = j[order], ax[order], wp[:, order], h[order], r[order]
        t = (ax - node_x[j]) / dx
        g = torch.stack([(2 * t + 1) * (1 - t) ** 2, t * (1 - t) ** 2, t * t * (3 - 2 * t), t * t * (t - 1)])
        # points padded to rows of at most `width` points of one bin
        count = torch.bincount(j, minlength=Nx - 1)
        width = int(min(max(int(count.max()), 1), max(16, 2 * len(j) // max(1, int((count > 0).sum())))))
        rows_of = (count + width - 1) // width
        first = torch.cumsum(rows_of, 0) - rows_of
        rank = torch.arange(len(j), device=dev) - (torch.cumsum(count, 0) - count)[j]
        row, col = first[j] + rank // width, rank % width
        rows = int(rows_of.sum())
        row_bin = torch.repeat_interleave(torch.arange(Nx - 1, device=dev), rows_of)
        pad_h = torch.zeros((rows, width), dtype=torch.float64, device=dev)
        pad_r = torch.zeros_like(pad_h)
        pad_g = torch.zeros((rows, 4 * maps, width), dtype=torch.float64, device=dev)
        pad_h[row, col], pad_r[row, col] = h, r
        for k in range(4):
            for q in range(maps):
                pad_g[row, 4 * q + k, col] = g[k] * wp[q]
        step = max(1, int(1.2e8 // (rows * width)))
        for m0 in range(0, Nl, step):
            m = torch.arange(m0, min(m0 + step, Nl), device=dev, dtype=torch.float64)
            a, b = pad_h[:, :, None] * m, pad_r[:, :, None] * m
            ca, sa, cb, sb = torch.cos(a), torch.sin(a), torch.cos(b), torch.sin(b)
            v = torch.complex(torch.bmm(pad_g, ca * cb - sa * sb), -torch.bmm(pad_g, sa * cb + ca * sb))
            del a, b, ca, sa, cb, sb
            s = torch.zeros((Nx - 1, 4 * maps, len(m)), dtype=torch.complex128, device=dev)
            s = s.index_add_(0, row_bin, v).reshape(Nx - 1, maps, 4, len(m)).permute(1, 2, 3, 0)
            for par in range(2):
                f = 1.0 if sign > 0 or par == 0 else -1.0
                block = slice(m0, m0 + len(m))
                A[:, par, block, :-1] += f * s[:, 0]
                A[:, par, block, 1:] += f * s[:, 2]
                B[:, par, block, :-1] += f * dx * s[:, 1]
                B[:, par, block, 1:] += f * dx * s[:, 3]
    return A, B


def _contract(folds, Nl, node_x):
    """alm (maps, Nlm) of each (A, B) in folds: rows l of Y and dY/dx for all m at once, by the
    recurrences in l."""
    dev, x = node_x.device, node_x
    m = torch.arange(Nl, device=dev, dtype=torch.float64)[:, None]
    om = 1 - x * x
    sx = torch.sqrt(om)
    diag = torch.ones((Nl, len(x)), dtype=torch.float64, device=dev)
    for k in range(1, Nl):
        diag[k] = -math.sqrt(1.0 - 1.0 / (2 * k)) * sx * diag[k - 1]
    y1 = torch.zeros_like(diag)  # row l - 1 of every m
    y2 = torch.zeros_like(diag)
    out = [torch.zeros((A.shape[0], Nl * (Nl + 1) // 2), dtype=torch.complex128, device=dev) for A, _ in folds]
    mi = torch.arange(Nl, device=dev)
    start = mi * (2 * Nl - 1 - mi) // 2
    for l in range(Nl):
        n = l + 1  # columns m = 0 .. l
        mm = m[:n]
        y = torch.zeros_like(diag)
        if l >= 2:
            k = l - 1
            f2 = torch.sqrt((l - mm[:k] - 1) / (l + mm[:k] - 1))
            q = torch.sqrt((l - mm[:k]) / (l + mm[:k])) / (l - mm[:k])
            y[:k] = ((2 * l - 1) * x * y1[:k] - (l + mm[:k] - 1) * y2[:k] * f2) * q
        if l >= 1:
            y[l - 1] = math.sqrt(2.0 * (l - 1) + 1.0) * x * y1[l - 1]
        y[l] = diag[l]
        dy = (torch.sqrt((l - mm) * (l + mm)) * y1[:n] - l * x * y[:n]) / om
        nrm = math.sqrt((2 * l + 1) / (4 * math.pi))
        par = (l - mi[:n]) % 2
        for o, (A, B) in zip(out, folds):
            for c in range(A.shape[0]):
                a, b = A[c, par, mi[:n]], B[c, par, mi[:n]]
                o[c, start[:n] + l] = torch.complex((y[:n] * a.real + dy * b.real).sum(1),
                                                    (y[:n] * a.imag + dy * b.imag).sum(1)) * nrm
        y2, y1 = y1, y
    return out


def _rotate_back(alm, Nl):
    """alm (maps, Nlm) of points rotated by 90 degrees about y, in the original frame: Wigner
    d^l(pi/2) by the downward recursion in the first index, all l and m at once, values kept as
    (number, binary exponent) pairs."""
    dev, maps = alm.device, alm.shape[0]
    mant, expo = np.zeros((Nl, Nl)), np.zeros((Nl, Nl), dtype=np.int64)
    for l in range(Nl):  # d_{l,m}: a running product of ratios from m = l down
        k = np.arange(l, 0, -1, dtype=np.longdouble)
        col = np.cumprod(np.concatenate([[np.longdouble(1.0)], -np.sqrt((l + k) / (l - k + 1))]))
        f, e = np.frexp(col[::-1])
        mant[l, :l + 1], expo[l, :l + 1] = f.astype(np.float64), e - l
    c, E = torch.from_numpy(mant).to(dev), torch.from_numpy(expo).to(dev)
    nxt = torch.zeros_like(c)
    ll = torch.arange(Nl, device=dev, dtype=torch.float64)[:, None]
    mm = torch.arange(Nl, device=dev, dtype=torch.float64)[None, :]
    valid = mm <= ll
    li = torch.arange(Nl, device=dev)[:, None]
    re = torch.zeros((maps, Nl, Nl), dtype=torch.float64, device=dev)
    im = torch.zeros_like(re)
    even_m = (torch.arange(Nl, device=dev)[None, :] % 2) == 0
    for step in range(Nl):  # row k = l - step of every l
        k = ll - step
        live = k >= 0
        ki = (li - step).clamp(min=0)[:, 0]
        idx = ki * (2 * Nl - 1 - ki) // 2 + li[:, 0]
        a = alm[:, idx]
        scale = torch.where(ki > 0, 2.0, 1.0)
        term = torch.where(live & valid, c, torch.zeros_like(c))
        # l + m + k even: real part; l + k has the parity of step
        to_re = even_m if step % 2 == 0 else ~even_m
        re += torch.where(to_re, term, 0.0) * (a.real * scale)[:, :, None]
        im += torch.where(to_re, 0.0, term) * (a.imag * torch.where(ki > 0, 2.0, 0.0))[:, :, None]
        up = torch.sqrt(((ll - k) * (ll + k + 1)).clamp(min=0.0))
        down = torch.sqrt(((ll + k) * (ll - k + 1)).clamp(min=1.0))
        c, nxt = torch.where(k > 0, (2 * mm * c - up * nxt) / down, 0.0), c  # no rows below k = 0
        big = c.abs() > 2.0 ** 200
        f = torch.where(big, torch.full_like(c, 2.0 ** -200), torch.ones_like(c))
        c, nxt, re, im = c * f, nxt * f, re * f, im * f
        E = E + torch.where(big, 200, 0)
    scale = torch.where(E > -1000, torch.exp2(E.clamp(min=-1000, max=1000).double()), torch.zeros_like(c))
    out = torch.zeros_like(alm)
    lv, mv = torch.nonzero(valid, as_tuple=True)
    out[:, mv * (2 * Nl - 1 - mv) // 2 + lv] = torch.complex((re * scale)[:, lv, mv], (im * scale)[:, lv, mv])
    return out


def _exact_alm(t, p, w, Nl, Nx):
    node_x = torch.arange(Nx, dtype=torch.float64, device=t.device) * (XMAX / float(Nx - 1))
    c = torch.cos(t)
    equ = c.abs() < XMAX
    pol = ~equ
    folds = [_fold(c[equ], p[equ], w[:, equ], Nl, node_x)]
    if bool(pol.any()):
        st = torch.sin(t[pol])
        z = -st * torch.cos(p[pol])
        folds.append(_fold(z, torch.atan2(st * torch.sin(p[pol]), c[pol]), w[:, pol], Nl, node_x))
    alms = _contract(folds, Nl, node_x)
    return alms[0] + _rotate_back(alms[1], Nl) if len(alms) > 1 else alms[0]


def _exact_mask(state):
    """The matrix from 3j symbols of binomials, (l1 l2 l3; 000)^2 = q(g-l1) q(g-l2) q(g-l3) /
    (q(g) (2g+1)) with q(n) = C(2n, n) / 4^n, one diagonal l1 - l2 at a time."""
    W, Nl = state["window"], state["case"]["Nl"]
    n = np.arange(1, 2 * Nl + 1, dtype=np.longdouble)
    q = np.concatenate([[np.longdouble(1.0)], np.cumprod((2 * n - 1) / (2 * n))]).astype(np.float64)
    dev = state["alm"].device
    q, W = torch.from_numpy(q).to(dev), torch.from_numpy(W).to(dev)
    M = torch.zeros((Nl, Nl), dtype=torch.float64, device=dev)
    for d in range(Nl):
        b = torch.arange(Nl - d, device=dev)[:, None]      # the smaller l
        i = torch.arange(Nl - d, device=dev)[None, :]      # l3 = d + 2 i, g = b + d + i
        ok = i <= b
        l3, g = (d + 2 * i), (b + d + i).clamp(max=2 * Nl - 1)
        term = q[i] * q[(d + i)] * q[(b - i).clamp(min=0)] / (q[g] * (2 * g + 1)) * ((2 * l3 + 1) * W[l3])
        s = torch.where(ok, term, torch.zeros_like(term)).sum(1) / (4 * math.pi)
        lo = torch.arange(Nl - d, device=dev)
        M[lo, lo + d] = s * (2 * (lo + d) + 1)
        M[lo + d, lo] = s * (2 * lo + 1)
    alm = state["alm"]
    cl = torch.zeros((alm.shape[0], Nl), dtype=torch.float64, device=dev)
    for l in range(Nl):
        m = torch.arange(l + 1, device=dev)
        a = alm[:, m * (2 * Nl - 1 - m) // 2 + l]
        power = a.real ** 2 + a.imag ** 2
        cl[:, l] = (a[:, 0].real ** 2 + 2 * power[:, 1:].sum(1)) / (2 * l + 1)
    return dict(M=M.cpu().numpy(), cl=cl)


def exact(case, seed):
    state = dict(_inputs(case, seed), case=case)
    if case["kind"] == "mask":
        return _exact_mask(state)
    Nl, Nx = case["Nl"], case["Nx"]
    if case["kind"] == "batch":
        return [_exact_alm(t, p, w[None, :], Nl, Nx)[0] for t, p, w in state["sets"]]
    w = state["w"].double()
    alm = _exact_alm(state["t"], state["p"], w if w.dim() == 2 else w[None, :], Nl, Nx)
    if case["kind"] == "maps":
        return alm
    return alm[0].cpu().numpy() if case["kind"] == "host" else alm[0]
