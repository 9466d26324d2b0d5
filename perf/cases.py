"""Performance cases: the calls that a program makes to phase-link SLC stacks.

Each case is one call of a public entry point (phase_link, sequential, nmap,
integrate_ps) on CUDA tensors, on scenes of the coherence and amplitude model
of fringe_gb300/synth.py, drawn on the GPU from the seed alone.  Sizes,
windows, depths and options are those of the test suite, the benchmark and
the module scripts' defaults, with ragged ones among them.
"""
import math

import numpy as np
import torch

import fringe_gb300
from fringe_gb300 import synth
from fringe_gb300.sequential import ministack_plan
from fringe_gb300.sequential import sequential as run_sequential

DEV = "cuda:0"
CELL = 18                       # Voronoi cell size in pixels
NCLASS = 8                      # amplitude classes


def _link(name, scene, rows, cols, nbands, ny, nx, method="MLE", semantics="evd", precision="fp32", mini=1, bw=-1,
          min_neighbors=2):
    c = dict(kind="link", scene=scene, rows=rows, cols=cols, nbands=nbands, ny=ny, nx=nx, method=method,
             semantics=semantics, precision=precision, mini=mini, bw=bw, min_neighbors=min_neighbors)
    return dict(c, name=name) if name else c


def _nmap(name, rows, cols, nbands, ny, nx, method, prob=0.05):
    c = dict(kind="nmap", rows=rows, cols=cols, nbands=nbands, ny=ny, nx=nx, method=method, prob=prob)
    return dict(c, name=name) if name else c


def _merge(name, rows, cols, nbands, master=0):
    c = dict(kind="merge", rows=rows, cols=cols, nbands=nbands, master=master)
    return dict(c, name=name) if name else c


def _seq(name, rows, cols, nbands, ny, nx, mini_size, precision):
    c = dict(kind="sequential", rows=rows, cols=cols, nbands=nbands, ny=ny, nx=nx, mini_size=mini_size,
             precision=precision)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a preview tile at the module's default 11 x 11 window: launches and latency
        _link("evd_tile64_n10", "uniform", 64, 64, 10, 5, 5, "EVD"),
        # the small scene of the module's own test size: 200 x 200, 10 dates, every window bit set
        _link("mle_uniform200_n10", "uniform", 200, 200, 10, 5, 5),
        # one frame of the usual wide-area run: 30 dates, 11 x 21 window, tensor-core form
        _link("mle_2048_n30_mixed", "voronoi", 2048, 2048, 30, 5, 10, precision="mixed"),
        # the same work in the default (plain FP32) form, a quarter frame
        _link("mle_1024_n30_fp32", "voronoi", 1024, 1024, 30, 5, 10),
        # third ministack of a sequential run, ragged frame: two compressed SLCs and 13 dates
        _link("mle_ragged_n15_mixed", "voronoi", 1023, 777, 15, 5, 10, precision="mixed", mini=3),
        # two years of data at once, decorrelated pixels among them (ill-conditioned coherence)
        _link("mle_illcond_n64_mixed", "illcond", 384, 320, 64, 5, 10, precision="mixed"),
        # the phase_link module (MLE where |C| is invertible), tall window, odd sizes
        _link("plink_ragged_n23_mixed", "voronoi", 333, 517, 23, 7, 3, semantics="phase_link", precision="mixed",
              min_neighbors=5),
        # short-baseline subset of a long stack, plain form
        _link("stbas_n45_fp32", "voronoi", 256, 384, 45, 5, 10, "STBAS", bw=10),
        # the whole sequential estimator: four ministacks of 10 dates, datum, adjustment
        _seq("sequential_40x10_mixed", 384, 512, 40, 5, 10, 10, "mixed"),
        # the SHP map that every run starts from, both tests
        _nmap("nmap_ks2_2048_n30", 2048, 2048, 30, 5, 10, "KS2"),
        _nmap("nmap_ad2_ragged_n17", 701, 1023, 17, 5, 5, "AD2"),
        # the PS/DS merge behind the linked frame
        _merge("merge_2048_n30", 2048, 2048, 30),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, px_max):
    """rows, cols of a frame of 1,000 .. px_max pixels"""
    px = _log_size(rng, 1000, max(px_max, 2000))
    rows = max(8, int(round(math.sqrt(px) * math.exp(rng.uniform(-0.6, 0.6)))))
    return rows, max(8, px // rows)


def draw(rng):
    kind = rng.choice(["link"] * 6 + ["nmap"] * 3 + ["merge", "sequential"])
    if kind == "link":
        n = rng.choice([_log_size(rng, 4, 64), rng.randint(8, 32)])
        precision = rng.choice(["fp32", "mixed"])
        method = rng.choice(["MLE", "MLE", "EVD", "STBAS"]) if n >= 6 else "MLE"
        semantics = "phase_link" if method == "MLE" and rng.random() < 0.25 else "evd"
        scene = rng.choice(["voronoi", "voronoi", "uniform", "illcond"])
        # a frame costs at most what the largest listed one does
        px = 2048 * 2048 * min(1.0, (30.0 / n) ** 4) * (0.4 if precision == "fp32" else 0.9)
        if scene == "illcond":
            px *= 0.6
        rows, cols = _dims(rng, int(px))
        ny, nx = rng.choice([(5, 5), (5, 10), (3, 5), (7, 3), (rng.randint(2, 8), rng.randint(2, 10))])
        return _link(None, scene, rows, cols, n, ny, nx, method, semantics, precision,
                     mini=rng.choice([1, 1, 1, min(n, rng.randint(1, 4))]),
                     bw=rng.randint(2, n - 2) if method == "STBAS" else -1, min_neighbors=rng.choice([2, 5]))
    if kind == "nmap":
        n = _log_size(rng, 8, 64)            # below 8 dates neither test rejects a pair at 0.01
        px = 2048 * 2048 * min(1.0, 30.0 / n)
        rows, cols = _dims(rng, int(px))
        ny, nx = rng.choice([(5, 5), (5, 10), (rng.randint(1, 6), rng.randint(1, 10))])
        return _nmap(None, rows, cols, n, ny, nx, rng.choice(["KS2", "AD2"]), rng.choice([0.05, 0.05, 0.01, 0.1]))
    if kind == "merge":
        n = _log_size(rng, 4, 64)
        rows, cols = _dims(rng, 2048 * 2048)
        return _merge(None, rows, cols, n, rng.choice([0, rng.randrange(n)]))
    rows, cols = _dims(rng, 600 * 600)
    return _seq(None, rows, cols, rng.randint(12, 48), rng.choice([3, 5]), rng.choice([5, 10]), rng.choice([8, 10, 12]),
                rng.choice(["fp32", "mixed"]))


# ---- inputs ------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _classes(rows, cols, g):
    """Class map of Voronoi cells: one random site per CELL x CELL square, a
    pixel takes the class of the nearest site of the 5 x 5 squares around it."""
    gy, gx = rows // CELL + 5, cols // CELL + 5
    sy = (torch.rand((gy, gx), generator=g, device=DEV) + torch.arange(-2, gy - 2, device=DEV)[:, None]) * CELL
    sx = (torch.rand((gy, gx), generator=g, device=DEV) + torch.arange(-2, gx - 2, device=DEV)[None, :]) * CELL
    cls = torch.randint(0, NCLASS, (gy, gx), generator=g, device=DEV, dtype=torch.int32)
    yy = torch.arange(rows, device=DEV)
    xx = torch.arange(cols, device=DEV)
    by, bx = yy // CELL, xx // CELL
    best = torch.full((rows, cols), float("inf"), device=DEV)
    out = torch.zeros((rows, cols), dtype=torch.int32, device=DEV)
    for dy in range(5):
        for dx in range(5):
            iy, ix = (by + dy)[:, None], (bx + dx)[None, :]
            d = (sy[iy, ix] - yy[:, None]) ** 2 + (sx[iy, ix] - xx[None, :]) ** 2
            near = d < best
            best = torch.where(near, d, best)
            out = torch.where(near, cls[iy, ix], out)
    return out


def _bitmap(rows, cols, ny, nx, classes):
    """SHP bitmask (Ulongmask layout): same-class neighbours, or every bit."""
    if classes is None:
        return torch.from_numpy(synth.nmap_all_ones(1, 1, ny, nx).view(np.int32)).to(DEV).expand(rows, cols, -1).contiguous()
    out = torch.zeros((rows, cols, synth.nulong_for(ny, nx)), dtype=torch.int32, device=DEV)
    for f in range((2 * ny + 1) * (2 * nx + 1)):
        ii, jj = f // (2 * nx + 1) - ny, f % (2 * nx + 1) - nx
        r0, r1, c0, c1 = max(0, -ii), min(rows, rows - ii), max(0, -jj), min(cols, cols - jj)
        if r0 >= r1 or c0 >= c1:
            continue
        same = classes[r0:r1, c0:c1] == classes[r0 + ii:r1 + ii, c0 + jj:c1 + jj]
        bit = (1 << (f % 32)) - (1 << 32 if f % 32 == 31 else 0)
        out[r0:r1, c0:c1, f // 32] |= same.to(torch.int32) * bit
    return out


def _stack(scene, rows, cols, nbands, g, classes):
    """complex64 [nbands, rows, cols]: circular Gaussian samples coloured by
    the temporal coherence of the scene, a deformation ramp, class amplitudes."""
    npx = rows * cols
    z = torch.randn((nbands, npx, 2), generator=g, device=DEV)
    z = torch.view_as_complex(z)
    if scene == "illcond":
        # per-pixel coherence: gamma0 in [0.05, 0.9], a tenth without a floor
        q0 = torch.randint(13, 231, (npx,), generator=g, device=DEV)
        qi = torch.where(torch.rand((npx,), generator=g, device=DEV) < 0.1, 0, 51)
        key = q0 * 64 + torch.minimum(qi, q0)
        order = torch.argsort(key)
        keys, counts = torch.unique_consecutive(key[order], return_counts=True)
        x, at = torch.empty_like(z), 0
        for k, m in zip(keys.tolist(), counts.tolist()):
            sel = order[at:at + m]
            at += m
            root = synth.eig_sqrt(synth.coherence_matrix(nbands, k // 64 / 256.0, k % 64 / 256.0))
            x[:, sel] = torch.from_numpy(root.astype(np.complex64)).to(DEV) @ z[:, sel]
    else:
        root = synth.eig_sqrt(synth.coherence_matrix(nbands))
        x = torch.from_numpy(root.astype(np.complex64)).to(DEV) @ z
    del z
    ramp = 0.03 * 0.5 * (torch.linspace(0, 1, rows, device=DEV)[:, None] + torch.linspace(0, 1, cols, device=DEV)[None, :])
    ramp = (2.0 * math.pi / synth.WAVELENGTH_M * 12.0 / synth.DAYS_PER_YEAR) * ramp.reshape(-1)
    amp = torch.ones(npx, device=DEV) if classes is None else 1.0 + 0.5 * classes.reshape(-1).to(torch.float32)
    for k in range(nbands):
        x[k] *= torch.polar(amp, ramp * k)
    return x.reshape(nbands, rows, cols)


def prepare(case, seed):
    g = _generator(seed)
    rows, cols, n = case["rows"], case["cols"], case["nbands"]
    s = {"case": case}
    if case["kind"] == "merge":
        s["slc"] = _stack("uniform", rows, cols, n, g, None)
        ph = torch.rand((n, rows, cols), generator=g, device=DEV) * (2 * math.pi)
        s["ds"] = torch.polar(torch.ones_like(ph), ph)
        s["tcorr"] = torch.rand((rows, cols), generator=g, device=DEV)
        # the PS map: a tenth of the pixels, in patches along the rows
        s["ps"] = (torch.rand((rows, (cols + 3) // 4), generator=g, device=DEV) < 0.1).to(torch.uint8)
        s["ps"] = s["ps"].repeat_interleave(4, dim=1)[:, :cols].contiguous()
        return s
    classes = None if case.get("scene") == "uniform" else _classes(rows, cols, g)
    s["stack"] = _stack(case.get("scene", "voronoi"), rows, cols, n, g, classes)
    if case["kind"] != "nmap":
        s["nmap"] = _bitmap(rows, cols, case["ny"], case["nx"], classes)
    return s


def run(state):
    c = state["case"]
    if c["kind"] == "merge":
        return fringe_gb300.integrate_ps(state["ds"], state["slc"], state["tcorr"], state["ps"], master=c["master"])
    half = (c["ny"], c["nx"])
    if c["kind"] == "nmap":
        return fringe_gb300.nmap(state["stack"], half, prob=c["prob"], method=c["method"])
    if c["kind"] == "sequential":
        return run_sequential(state["stack"], state["nmap"], half, mini_stack_size=c["mini_size"],
                              precision=c["precision"])
    return fringe_gb300.phase_link(state["stack"], state["nmap"], half, method=c["method"], semantics=c["semantics"],
                                   mini_stack_count=c["mini"], band_width=c["bw"], min_neighbors=c["min_neighbors"],
                                   precision=c["precision"], want_status=True)


# ---- what a pass cannot do without -----------------------------------------------
def _link_work(px, n, ny, nx, voronoi, method):
    k = (2 * ny + 1) * (2 * nx + 1)
    shp = k * (0.65 if voronoi else 0.95)
    # the coherence sums; for MLE two complex Cholesky factorisations, a real
    # inverse and three pairs of triangular solves; else ten products C x
    solve = (2 * 4.0 / 3.0 + 1.0) * n ** 3 + 3 * 8.0 * n * n if method == "MLE" else 10 * 8.0 * n * n
    return {"bytes": px * (16.0 * n + 4 * synth.nulong_for(ny, nx) + 16), "flops": px * (4.0 * n * (n + 1) * shp + solve)}


def work(case):
    px, n = float(case["rows"] * case["cols"]), case["nbands"]
    if case["kind"] == "merge":
        return {"bytes": px * (8.0 * n + 8.0 * (n - 1) + 9), "flops": px * 8.0 * n}
    ny, nx = case["ny"], case["nx"]
    if case["kind"] == "nmap":
        # each pair of the half window is compared once: two sorted samples
        pairs = ((2 * ny + 1) * (2 * nx + 1) - 1) / 2
        return {"bytes": px * (8.0 * n + 4 * synth.nulong_for(ny, nx) + 4), "flops": px * pairs * 2 * n}
    if case["kind"] == "sequential":
        total = {"bytes": px * 24.0 * n, "flops": px * 8.0 * n}
        plan = ministack_plan(n, case["mini_size"])
        for depth in [count - 1 + end - start for count, start, end in plan] + [len(plan)]:
            for k, v in _link_work(px, depth, ny, nx, True, "MLE").items():
                total[k] += v
        return total
    return _link_work(px, n, ny, nx, case["scene"] != "uniform", case["method"])


# ---- the same outputs in 64 bits ------------------------------------------------
def _dominant(a):
    """Eigenvector of the largest eigenvalue of Hermitian matrices, by
    repeated squaring (power 2^11)."""
    a = a / torch.linalg.matrix_norm(a)[:, None, None]
    for _ in range(11):
        a = a @ a
        a = a / torch.linalg.matrix_norm(a)[:, None, None]
    best = torch.diagonal(a, dim1=1, dim2=2).real.argmax(dim=1)
    return torch.gather(a, 2, best[:, None, None].expand(-1, a.shape[1], 1))[:, :, 0]


def _unit(z):
    m = z.abs()
    return torch.where(m > 0, z / torch.where(m > 0, m, 1.0), 1.0 + 0j)


def _link64(stack, bits, ny, nx, method, semantics, mini, bw, min_neighbors):
    n, rows, cols = stack.shape
    wx = 2 * nx + 1
    pad = torch.zeros((n, rows + 2 * ny, cols + 2 * nx), dtype=torch.complex128, device=DEV)
    pad[:, ny:ny + rows, nx:nx + cols] = stack
    inside = torch.zeros((rows + 2 * ny, cols + 2 * nx), dtype=torch.bool, device=DEV)
    inside[ny:ny + rows, nx:nx + cols] = True
    phase = torch.zeros((n, rows, cols), dtype=torch.complex128, device=DEV)
    tcorr = torch.zeros((rows, cols), dtype=torch.float64, device=DEV)
    comp = torch.zeros((rows, cols), dtype=torch.complex128, device=DEV)
    plink = semantics == "phase_link"
    eye = torch.eye(n, dtype=torch.complex128, device=DEV)
    step = max(1, int(4e9 / (16.0 * n * n * cols)))
    for r0 in range(0, rows, step):
        r1 = min(rows, r0 + step)
        px = (r1 - r0) * cols
        gram = torch.zeros((px, n, n), dtype=torch.complex128, device=DEV)
        count = torch.zeros(px, dtype=torch.int32, device=DEV)
        for f in range((2 * ny + 1) * wx):
            ii, jj = f // wx, f % wx
            on = ((bits[r0:r1, :, f // 32] >> (f % 32)) & 1).bool() & inside[r0 + ii:r1 + ii, jj:jj + cols]
            x = (pad[:, r0 + ii:r1 + ii, jj:jj + cols] * on).reshape(n, px).T
            gram.addcmul_(x[:, :, None], x[:, None, :].conj())
            count += on.reshape(-1)
        centre = ny * wx + nx
        use = ((bits[r0:r1, :, centre // 32] >> (centre % 32)) & 1).bool().reshape(-1)
        use &= count >= (min_neighbors if plink else 2)
        p = torch.diagonal(gram, dim1=1, dim2=2).real
        coh = gram / torch.sqrt(p[:, :, None] * p[:, None, :])
        del gram
        # a date without power in the window: the first eigen call fails
        code = torch.zeros(px, dtype=torch.float64, device=DEV)
        code[~(coh.abs() < math.inf).all(dim=2).all(dim=1)] = -1.0 if plink or method == "MLE" else -6.0
        coh = torch.where((use & (code == 0))[:, None, None], coh, eye)
        if method == "MLE":
            mag = coh.abs() + 0j
            shift = 0.0 if plink else 1e-6
            fine = torch.linalg.cholesky_ex(mag - shift * eye)[1] == 0
            if not plink:
                code[~fine] = -4.0
                code[torch.linalg.cholesky_ex(coh - 1e-6 * eye)[1] != 0] = -2.0
            fine &= code == 0
            m = torch.linalg.inv(torch.where(fine[:, None, None], mag, eye)).real * coh
            m = torch.linalg.inv(torch.where(fine[:, None, None], m, eye))
            z = _dominant(torch.where(fine[:, None, None], m, coh))
            del mag, m
        else:
            if method == "STBAS":
                k = torch.arange(n, device=DEV)
                coh = coh * ((k[:, None] - k[None, :]).abs() <= bw)
            z = _dominant(coh)
        ph = _unit(z)
        ph = ph * ph[:, mini - 1:mini].conj()
        x = stack[:, r0:r1].reshape(n, px).T.to(torch.complex128)
        cs = (x[:, mini - 1:] * ph[:, mini - 1:].conj()).sum(dim=1) / (n - mini + 1)
        k = torch.arange(n, device=DEV)
        pairs = (k[None, :] > k[:, None]) & (k[None, :] - k[:, None] <= (bw if method == "STBAS" else n))
        tc = (_unit(coh) * ph[:, None, :] * ph[:, :, None].conj() * pairs).sum(dim=(1, 2)).abs() / pairs.sum()
        good = use & (code == 0)
        phase[:, r0:r1] = torch.where(good[:, None], ph, 0).T.reshape(n, r1 - r0, cols)
        comp[r0:r1] = torch.where(good, cs, 0).reshape(r1 - r0, cols)
        tcorr[r0:r1] = torch.where(good, tc, torch.where(use, code, 0.0)).reshape(r1 - r0, cols)
    return {"phase": phase, "tcorr": tcorr, "comp": comp}


def exact(case, seed):
    if case["kind"] == "nmap":
        return None                                  # whole numbers
    n, px = case["nbands"], case["rows"] * case["cols"]
    if case["kind"] == "merge":
        s = prepare(case, seed)
        m = case["master"]
        out = torch.empty((max(n - 1, 0),) + tuple(s["tcorr"].shape), dtype=torch.complex128, device=DEV)
        ds0, slc0 = s["ds"][m].to(torch.complex128).conj(), s["slc"][m].to(torch.complex128).conj()
        for q, j in enumerate(j for j in range(n) if j != m):
            out[q] = torch.where(s["ps"] == 1, _unit(s["slc"][j] * slc0), s["ds"][j] * ds0)
        return {"ifg": out, "tcorr": torch.where(s["ps"] == 1, 0.95, s["tcorr"].double())}
    if case["kind"] == "sequential":
        if px > 250_000:
            return None
        s = prepare(case, seed)
        args = (case["ny"], case["nx"], "MLE", "evd")
        comps, minis = [], []
        for count, i0, i1 in ministack_plan(n, case["mini_size"]):
            own = s["stack"][i0:i1].to(torch.complex128)
            ms = torch.cat([torch.stack(comps), own]) if comps else own
            minis.append(_link64(ms, s["nmap"], *args, count, -1, 5))
            comps.append(minis[-1]["comp"])
        comps = torch.stack(comps)
        datum = _link64(comps, s["nmap"], *args, 1, -1, 5)
        adjusted = torch.cat([m["phase"][-(i1 - i0):] * datum["phase"][k]
                              for k, ((_, i0, i1), m) in enumerate(zip(ministack_plan(n, case["mini_size"]), minis))])
        return {"ministacks": minis, "compressed": comps, "datum": datum, "adjusted": adjusted}
    taps = (2 * case["ny"] + 1) * (2 * case["nx"] + 1)
    if px * (2e2 * n ** 3 + 40.0 * n * n * taps) > 1.2e13:
        return None                                  # over the time it may take
    s = prepare(case, seed)
    return _link64(s["stack"], s["nmap"], case["ny"], case["nx"], case["method"], case["semantics"], case["mini"],
                   case["bw"], case["min_neighbors"])
