"""The work that a program using this framework gives it, as timed cases.

Every case goes through the Python mirror of the C ABI (``cosmicatlas_b200.api``)
with particles and meshes resident on the GPU, as a calibration loop keeps
them between its iterations, and with the process's one default context.

* ``job``      one mesh job (``Context.job``): particles -> mesh -> FFT -> P(k)
               and, on request, the T-web of the same mesh.
* ``batch``    many small jobs of one shape in one call (``Context.batch``).
* ``density``  mass assignment alone (``Context.assign``), any box-shaped mesh.
* ``fft``      r2c of a mesh and c2r of its spectrum.
* ``cwc``      the T-web of a mesh: labels, eigenvalue planes and counts.
* ``konvolve`` a BAM kernel update and the convolution of a mesh with it.

``draw`` gives further cases of the same six kinds.
"""
import math

import numpy as np
import torch

from cosmicatlas_b200 import _lib, synth
from cosmicatlas_b200 import api as cam

_SCHEME = {"ngp": cam.NGP, "cic": cam.CIC, "tsc": cam.TSC}
_PREC = {"f32": cam.F32, "f64": cam.F64}
_METHOD = {"fft": _lib.TWEB_FFT, "fd": _lib.TWEB_FD}
_DEV = "cuda"


def listed():
    return [
        # One calibration mesh at a time: the smallest job BAM issues, where
        # launches and the one host round trip are most of the time.
        dict(name="calib64_job", kind="job", n=64, np=262_144, box=500.0, scheme="cic", weights=False, prec="f32",
             nbins=32, tweb="", R=0.0, lth=0.0, source="clumps", sigma=2.5),
        # The calibration batch: independent 64^3 jobs with P(k) and T-web
        # label counts, packed into one call.
        dict(name="calib64_batch", kind="batch", n=64, np=262_144, jobs=64, box=500.0, scheme="cic", nbins=32,
             tweb="fft", R=8.0, lth=0.0, sigma=2.5),
        # The plain small configuration: double precision mesh, P(k), T-web.
        dict(name="plain128_f64", kind="job", n=128, np=2_000_000, box=1000.0, scheme="cic", weights=False,
             prec="f64", nbins=64, tweb="fft", R=8.0, lth=0.0, source="clumps", sigma=2.0),
        # The assignment-scheme sweep: 16.8 M halo-weighted particles onto
        # 256^3, one job per scheme.
        dict(name="sweep256_ngp", kind="job", n=256, np=16_777_216, box=1000.0, scheme="ngp", weights=True,
             prec="f32", nbins=128, tweb="", R=0.0, lth=0.0, source="clumps", sigma=1.5),
        dict(name="sweep256_cic", kind="job", n=256, np=16_777_216, box=1000.0, scheme="cic", weights=True,
             prec="f32", nbins=128, tweb="", R=0.0, lth=0.0, source="clumps", sigma=1.5),
        dict(name="sweep256_tsc", kind="job", n=256, np=16_777_216, box=1000.0, scheme="tsc", weights=True,
             prec="f32", nbins=128, tweb="", R=0.0, lth=0.0, source="clumps", sigma=1.5),
        # getDensity_* on its own, as catalogue builders call it: a mesh with
        # three different, odd sides and a ragged particle count.
        dict(name="density_ragged", kind="density", n1=243, n2=150, n3=101, np=5_000_011, box=750.0, scheme="tsc",
             weights=False, prec="f32", sigma=1.5),
        # One full-size iteration: CIC, P(k) and the smoothed T-web at 512^3.
        dict(name="single512", kind="job", n=512, np=134_217_728, box=1000.0, scheme="cic", weights=False,
             prec="f32", nbins=256, tweb="fft", R=3.90625, lth=0.0, source="clumps", sigma=1.5),
        # The largest job: a Zel'dovich-displaced 768^3 lattice (particles in
        # lattice order, as initial-condition generators and snapshots keep
        # them), TSC, P(k) and T-web.
        dict(name="large768", kind="job", n=768, np=452_984_832, box=1500.0, scheme="tsc", weights=False, prec="f32",
             nbins=256, tweb="fft", R=3.0, lth=0.1, source="lattice", sigma=0.0),
        # Both FFT directions at a size with a factor 3.
        dict(name="fft384_roundtrip", kind="fft", n=384, prec="f32"),
        # Cwclass::get_CWC on a mesh with the reference's default
        # finite-difference tensor: labels and eigenvalues for the bias bins.
        dict(name="cwc256_fd", kind="cwc", n=256, box=1000.0, prec="f32", tweb="fd", R=4.0, lth=0.0),
        # BAM's GetKernel update followed by Konvolve.
        dict(name="konvolve256", kind="konvolve", n=256, box=1000.0, prec="f32", nbins=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["job", "job", "job", "batch", "density", "density", "fft", "cwc", "konvolve"])
    if kind == "job":
        n = rng.choice([32, 64, 96, 128, 144, 192, 256, 288, 384, 512])
        prec = "f64" if n <= 256 and rng.random() < 0.2 else "f32"
        return dict(kind="job", n=n, np=_log_int(rng, 1e5, 1.3e8 if n >= 256 else 5e7),
                    box=round(rng.uniform(250.0, 2000.0), 1), scheme=rng.choice(["ngp", "cic", "tsc"]),
                    weights=rng.random() < 0.4, prec=prec, nbins=rng.choice([n // 2, n // 3, n // 4]),
                    tweb=rng.choice(["", "", "fft", "fd"]), R=round(rng.uniform(0.0, 8.0), 2),
                    lth=rng.choice([0.0, 0.1, 0.2]), source="clumps", sigma=round(rng.uniform(1.0, 4.0), 2))
    if kind == "batch":
        n = rng.choice([32, 48, 64, 96, 128])
        return dict(kind="batch", n=n, np=_log_int(rng, 3e4, 6e5), jobs=rng.randint(5, 72),
                    box=round(rng.uniform(250.0, 1000.0), 1), scheme=rng.choice(["ngp", "cic", "tsc"]), nbins=n // 2,
                    tweb=rng.choice(["", "fft"]), R=round(rng.uniform(2.0, 8.0), 2), lth=0.0,
                    sigma=round(rng.uniform(1.0, 4.0), 2))
    if kind == "density":
        return dict(kind="density", n1=_log_int(rng, 33, 400), n2=_log_int(rng, 33, 400), n3=_log_int(rng, 33, 400),
                    np=_log_int(rng, 1e5, 5e7), box=round(rng.uniform(250.0, 2000.0), 1),
                    scheme=rng.choice(["ngp", "cic", "tsc"]), weights=rng.random() < 0.5,
                    prec=rng.choice(["f32", "f32", "f64"]), sigma=round(rng.uniform(1.0, 4.0), 2))
    sizes = [24, 32, 48, 54, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384]
    n = rng.choice(sizes)
    prec = "f64" if n <= 256 and rng.random() < 0.25 else "f32"
    if kind == "fft":
        return dict(kind="fft", n=rng.choice(sizes + [432, 486, 512, 576, 648]) if prec == "f32" else n, prec=prec)
    box = round(rng.uniform(250.0, 2000.0), 1)
    if kind == "cwc":
        return dict(kind="cwc", n=n, box=box, prec=prec, tweb=rng.choice(["fft", "fd"]),
                    R=round(rng.uniform(0.0, 8.0), 2), lth=rng.choice([0.0, 0.1, 0.2]))
    return dict(kind="konvolve", n=n, box=box, prec=prec, nbins=n // 2)


# ---------------------------------------------------------------- inputs

def _particles(case, seed, npart):
    box = case["box"]
    if case.get("source") == "lattice":
        x, y, z, _ = synth.zeldovich_lattice(case["n"], box, seed=seed, device=_DEV)
    else:
        x, y, z = synth.clumped_torch(npart, box, max(64, npart // 84), case["sigma"], 0.8, seed, _DEV)
    w = None
    if case.get("weights"):
        # halo-like masses: log10 M ~ N(12.5, 0.5) within [11, 15]
        g = torch.Generator(device=_DEV).manual_seed(seed + 1_000_003)
        lg = 12.5 + 0.5 * torch.randn(npart, generator=g, device=_DEV, dtype=torch.float64)
        lg = torch.where((lg < 11.0) | (lg > 15.0), torch.full_like(lg, 12.5), lg)
        w = torch.pow(10.0, lg).to(torch.float32)
    return x, y, z, w


def _mesh(n, box, prec, seed):
    """A lognormal density of mean about 1 with a power-law spectrum."""
    g = torch.Generator(device=_DEV).manual_seed(seed)
    f = torch.fft.rfftn(torch.randn((n, n, n), generator=g, device=_DEV, dtype=torch.float64))
    k = torch.sqrt(_k2(n)) * (2.0 * math.pi / box)
    f *= torch.where(k > 0, k.clamp_min(1e-30) ** -0.75 * torch.exp(-0.5 * (k / 0.5) ** 2), torch.zeros_like(k))
    d = torch.fft.irfftn(f, s=(n, n, n))
    d = torch.exp(d / d.std() - 0.5)
    return d.to(torch.float64 if prec == "f64" else torch.float32).contiguous()


def _axis(n):
    i = torch.arange(n, device=_DEV, dtype=torch.float64)
    return torch.where(i <= n // 2, i, i - n)


def _k2(n):
    f, h = _axis(n), torch.arange(n // 2 + 1, device=_DEV, dtype=torch.float64)
    return f[:, None, None] ** 2 + f[None, :, None] ** 2 + h[None, None, :] ** 2


def _tweb_opts(case, input_type=_lib.INPUT_DENSITY):
    return cam.Context.tweb_opts(case["R"], case["lth"], 1e-5, input_type, _METHOD[case["tweb"]])


def _pk_opts(case):
    return cam.Context.pk_opts(_SCHEME[case["scheme"]], nbins=case["nbins"], ndel=_ndel(case))


def _ndel(case):
    return case["n"] / 2 / case["nbins"]


def prepare(case, seed):
    state = dict(case=case, ctx=cam.default_context())
    kind = case["kind"]
    if kind in ("job", "density"):
        state["parts"] = _particles(case, seed, case["np"])
        sides = (case["n1"], case["n2"], case["n3"]) if kind == "density" else case["n"]
        state["grid"] = cam.make_grid(sides, case["box"])
    elif kind == "batch":
        state["grid"] = cam.make_grid(case["n"], case["box"])
        state["parts"] = [_particles(case, seed * 1009 + k, case["np"]) for k in range(case["jobs"])]
    else:
        state["mesh"] = _mesh(case["n"], case["box"] if "box" in case else 1000.0, case["prec"], seed)
        if kind == "konvolve":
            n = case["n"]
            state["kernel"] = torch.ones((n, n, n // 2 + 1), device=_DEV, dtype=state["mesh"].dtype)
            state["ratio"] = 0.5 + np.random.default_rng(seed).random(case["nbins"])
    torch.cuda.synchronize()  # the context launches on its own stream
    return state


# ---------------------------------------------------------------- the calls

def _job_outputs(r, prec):
    # BAM keeps P(k) in its real_prec vectors: the mesh's precision
    real = np.float64 if prec == "f64" else np.float32
    out = {"n_in": r["assign"].n_in, "n_lost": r["assign"].n_lost, "sum_mesh": r["assign"].sum_mesh}
    if r["pk"] is not None:
        out.update(pk=r["pk"].pk.astype(real), modes=r["pk"].modes, kvector=r["pk"].kvector,
                   shot_noise=r["pk"].shot_noise, normal=r["pk"].normal)
    if r["tweb"] is not None:
        out.update(counts=r["tweb"].counts, ties=r["tweb"].ties, mean=r["tweb"].mean)
    return out


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "job":
        x, y, z, w = state["parts"]
        r = ctx.job(x, y, z, w, grid=state["grid"], scheme=_SCHEME[case["scheme"]], precision=_PREC[case["prec"]],
                    pk=_pk_opts(case), tweb=_tweb_opts(case) if case["tweb"] else None)
        return _job_outputs(r, case["prec"])
    if kind == "batch":
        jobs = [cam.JobSpec(x, y, z, w, grid=state["grid"], scheme=_SCHEME[case["scheme"]], pk=_pk_opts(case),
                            tweb=_tweb_opts(case) if case["tweb"] else None) for x, y, z, w in state["parts"]]
        rs = [_job_outputs(r, "f32") for r in ctx.batch(jobs)]
        return {k: np.stack([np.asarray(r[k]) for r in rs]) for k in rs[0] if k not in ("shot_noise", "normal")} | {
            "shot_noise": np.array([r["shot_noise"] for r in rs]), "normal": np.array([r["normal"] for r in rs])}
    if kind == "density":
        x, y, z, w = state["parts"]
        r = ctx.assign(x, y, z, w, state["grid"], _SCHEME[case["scheme"]], _PREC[case["prec"]])
        return {"mesh": r.mesh, "n_in": r.n_in, "n_lost": r.n_lost, "sum_mesh": r.sum_mesh}
    if kind == "fft":
        spec = ctx.fft_r2c(state["mesh"])
        return {"spec": spec, "back": ctx.fft_c2r(spec)}
    if kind == "cwc":
        r = ctx.tweb(state["mesh"], case["box"], _tweb_opts(case), want_lambdas=True)
        return {"labels": r.labels, "lambdas": r.lambdas, "counts": r.counts, "ties": r.ties, "mean": r.mean}
    # the kernel is set to the ratio of the spectra in each bin (GetKernel
    # without rejection), so a repeated pass gives the same kernel
    binned, modes = ctx.bam_kernel_update(state["kernel"], case["box"], state["ratio"], _lib.KERNEL_SET)
    real = np.float64 if case["prec"] == "f64" else np.float32
    return {"out": ctx.konvolve(state["mesh"], case["box"], state["kernel"]), "kernel": state["kernel"],
            "binned": binned.astype(real), "modes": modes}


# ---------------------------------------------------------------- work

_STENCIL = {"ngp": 1, "cic": 8, "tsc": 27}


def _fft_flops(n):
    return 2.5 * n ** 3 * 3 * math.log2(n)


def work(case):
    kind = case["kind"]
    es = 8 if case.get("prec") == "f64" else 4
    if kind in ("job", "batch"):
        n, npart, jobs = case["n"], case["np"], case.get("jobs", 1)
        # particles in; the mesh and its spectrum stay on the device, but a
        # mesh is needed before its mean, its FFT before P(k): one write and
        # one read each
        by = npart * (16 if case.get("weights") else 12) + 2 * es * n ** 3
        fl = npart * _STENCIL[case["scheme"]] * 4 + _fft_flops(n)
        if case["tweb"]:
            by += 2 * es * n ** 3
            fl += 6 * _fft_flops(n) + 60 * n ** 3
        return {"bytes": jobs * by, "flops": jobs * fl}
    if kind == "density":
        cells = case["n1"] * case["n2"] * case["n3"]
        return {"bytes": case["np"] * (16 if case["weights"] else 12) + es * cells,
                "flops": case["np"] * _STENCIL[case["scheme"]] * 4}
    n = case["n"]
    if kind == "fft":
        return {"bytes": 4 * es * n ** 3, "flops": 2 * _fft_flops(n)}
    if kind == "cwc":
        return {"bytes": n ** 3 * (es + 1 + 12), "flops": 7 * _fft_flops(n) + 100 * n ** 3}
    half = n * n * (n // 2 + 1)
    return {"bytes": 2 * es * n ** 3 + 2 * es * half, "flops": 2 * _fft_flops(n) + 4 * half}


# ---------------------------------------------------------------- 64 bits

def _axis_weights(pos, scheme, d, n):
    """[(cell index, weight)] along one axis in FP64; NGP cells by the
    reference's float32 arithmetic."""
    if scheme == "ngp":
        c = torch.floor(pos / torch.tensor(d, dtype=torch.float32, device=pos.device)).to(torch.int64)
        return [(torch.remainder(c, n), None)]
    u = pos.double() / d
    if scheme == "cic":
        c = torch.floor(u - 0.5)
        t = u - 0.5 - c
        ws = [(0, 1.0 - t), (1, t)]
    else:
        c = torch.floor(u)
        t = u - 0.5 - c
        ws = [(-1, 0.5 * (0.5 - t) ** 2), (0, 0.75 - t * t), (1, 0.5 * (0.5 + t) ** 2)]
    c = c.to(torch.int64)
    return [(torch.remainder(c + o, n), w) for o, w in ws]


def _exact_mesh(parts, scheme, sides, box):
    mesh = torch.zeros(sides[0] * sides[1] * sides[2], dtype=torch.float64, device=_DEV)
    d = [float(np.float32(np.float32(box) / np.float32(s))) for s in sides]
    npart = parts[0].numel()
    for a in range(0, npart, 1 << 24):
        b = min(npart, a + (1 << 24))
        ax = [_axis_weights(parts[k][a:b], scheme, d[k], sides[k]) for k in range(3)]
        wt = parts[3][a:b].double() if parts[3] is not None else torch.ones(b - a, dtype=torch.float64, device=_DEV)
        for ci, wi in ax[0]:
            for cj, wj in ax[1]:
                row = (ci * sides[1] + cj) * sides[2]
                wij = wt if wi is None else wt * wi * wj
                for ck, wk in ax[2]:
                    mesh.index_add_(0, row + ck, wij if wk is None else wij * wk)
    return mesh.reshape(sides)


def _sq(p, s):
    s2 = s * s
    return torch.ones_like(s) if p == 0 else 1 - 2 / 3 * s2 if p == 1 else 1 - s2 + 2 / 15 * s2 * s2


def _exact_pk(mesh, case):
    n, h, p = case["n"], case["n"] // 2, {"ngp": 0, "cic": 1, "tsc": 2}[case["scheme"]]
    nb, ndel, box = case["nbins"], _ndel(case), float(np.float32(case["box"]))
    nobj = float(mesh.sum())
    f = torch.fft.rfftn(mesh - nobj / n ** 3)
    ang = math.pi * _axis(n).abs() / n
    iw = torch.where(ang > 0, (torch.sin(ang) / ang.clamp_min(1e-30)), torch.ones_like(ang)) ** (-2 * (p + 1))
    sn = _sq(p, torch.sin(ang)) * iw
    edges = torch.tensor([(b * ndel) ** 2 for b in range(nb + 1)], dtype=torch.float64, device=_DEV)
    fa, fc = _axis(n), torch.arange(h + 1, device=_DEV, dtype=torch.float64)
    raw, shot, cnt = (torch.zeros(nb, dtype=torch.float64, device=_DEV) for _ in range(3))
    j = torch.arange(n, device=_DEV)
    for i in range(n):
        if i == h:
            continue
        q = fa[i] ** 2 + fa[:, None] ** 2 + fc[None, :] ** 2
        b = torch.searchsorted(edges, q, right=True) - 1
        seen = (b >= 0) & (b < nb) & (j != h)[:, None]
        zero = (j <= h) & ~((j == 0) & (i == 0 or i > h))  # k = 0: one of each conjugate pair
        seen[:, 0] &= zero
        b = b.clamp(0, nb - 1)
        m = seen.to(torch.float64)
        w = iw[i] * iw[:, None] * iw[None, :h + 1] * m
        s = sn[i] * sn[:, None] * sn[None, :h + 1] * m
        pw = f[i].real ** 2 + f[i].imag ** 2
        raw.index_add_(0, b.reshape(-1), (pw * w).reshape(-1))
        shot.index_add_(0, b.reshape(-1), s.reshape(-1))
        cnt.index_add_(0, b.reshape(-1), m.reshape(-1))
    vol = box ** 3
    normal, noise = nobj * nobj / vol, vol / nobj
    md = cnt.clamp_min(1.0)
    pk = torch.where(cnt > 0, raw / (md * normal) - noise * shot / md, torch.zeros_like(raw))
    kv = 2.0 * math.pi / box * (np.arange(nb) + 0.5) * ndel
    return {"pk": pk.cpu().numpy(), "kvector": kv, "sum_mesh": nobj, "shot_noise": noise, "normal": normal}


def _eigenvalues(xx, yy, zz, xy, xz, yz):
    """Descending eigenvalues of symmetric 3x3 matrices (Smith 1961), FP64."""
    q = (xx + yy + zz) / 3
    a, b, c = xx - q, yy - q, zz - q
    pp = torch.sqrt((a * a + b * b + c * c + 2 * (xy * xy + xz * xz + yz * yz)) / 6).clamp_min(1e-300)
    det = a * (b * c - yz * yz) - xy * (xy * c - yz * xz) + xz * (xy * yz - b * xz)
    phi = torch.acos((det / (2 * pp ** 3)).clamp(-1.0, 1.0)) / 3
    l1 = q + 2 * pp * torch.cos(phi)
    l3 = q + 2 * pp * torch.cos(phi + 2 * math.pi / 3)
    return torch.stack([l1, 3 * q - l1 - l3, l3])


def _exact_lambdas(mesh, case):
    n, box = case["n"], float(np.float32(case["box"]))
    kf = 2.0 * math.pi / box
    mean = float(mesh.mean())
    k2 = _k2(n)
    f = torch.fft.rfftn(mesh / mean - 1.0) * torch.exp(-0.5 * k2 * (kf * float(np.float32(case["R"]))) ** 2)
    f = torch.where(k2 > 0, f / k2.clamp_min(1.0), torch.zeros_like(f))
    del k2
    if case["tweb"] == "fd":  # multiplier of the 4th-order centred difference
        t = 2 * math.pi * _axis(n) / n
        s = n * (8 * torch.sin(t) - torch.sin(2 * t)) / (12 * math.pi)
        s[n // 2] = 0.0
    else:
        s = _axis(n)
    ks = (s[:, None, None], s[None, :, None], s[None, None, :n // 2 + 1])
    t = [torch.fft.irfftn(f * ks[a] * ks[b], s=(n, n, n)) for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    return _eigenvalues(*t), mean


def _kernel_bins(case):
    """Bin of every half-complex element by GetKernel's real_prec arithmetic
    (products left to right, every step rounded)."""
    n = case["n"]
    real = torch.float64 if case["prec"] == "f64" else torch.float32
    dk0 = 2.0 * math.pi / float(np.float32(case["box"]))
    width = math.sqrt(dk0 * dk0 + dk0 * dk0 + dk0 * dk0) / math.sqrt(3.0)
    dk, width = (torch.tensor(v, dtype=torch.float64, device=_DEV).to(real) for v in (dk0, width))
    f, g = _axis(n).to(real), torch.arange(n // 2 + 1, device=_DEV).to(real)
    f2, g2 = f * dk * f * dk, g * dk * g * dk
    k = torch.sqrt((f2[:, None, None] + f2[None, :, None]) + g2[None, None, :])
    return torch.floor(k / width).to(torch.int64)


def exact(case, seed):
    kind = case["kind"]
    if kind == "job":
        parts = _particles(case, seed, case["np"])
        n = case["n"]
        mesh = _exact_mesh(parts, case["scheme"], (n, n, n), case["box"])
        del parts
        out = {"n_in": None, "n_lost": None, "modes": None} | _exact_pk(mesh, case)
        if case["tweb"]:
            out.update(counts=None, ties=None, mean=float(mesh.mean()))
        return out
    if kind == "batch":
        n, rs = case["n"], []
        for k in range(case["jobs"]):
            mesh = _exact_mesh(_particles(case, seed * 1009 + k, case["np"]), case["scheme"], (n, n, n), case["box"])
            rs.append(_exact_pk(mesh, case) | {"mean": float(mesh.mean())})
        out = {k: np.stack([np.asarray(r[k]) for r in rs]) for k in rs[0] if case["tweb"] or k != "mean"}
        return out | {"n_in": None, "n_lost": None, "modes": None}
    if kind == "density":
        sides = (case["n1"], case["n2"], case["n3"])
        mesh = _exact_mesh(_particles(case, seed, case["np"]), case["scheme"], sides, case["box"])
        return {"mesh": mesh, "n_in": None, "n_lost": None, "sum_mesh": float(mesh.sum())}
    mesh = _mesh(case["n"], case["box"] if "box" in case else 1000.0, case["prec"], seed).double()
    if kind == "fft":
        return {"spec": torch.fft.rfftn(mesh), "back": mesh}
    if kind == "cwc":
        lam, mean = _exact_lambdas(mesh, case)
        return {"labels": None, "lambdas": lam, "counts": None, "ties": None, "mean": mean}
    n, nb = case["n"], case["nbins"]
    bins = _kernel_bins(case)
    ratio = torch.from_numpy(0.5 + np.random.default_rng(seed).random(nb)).to(_DEV)
    kernel = torch.where(bins < nb, ratio[bins.clamp_max(nb - 1)], torch.ones((), dtype=torch.float64, device=_DEV))
    out = torch.fft.irfftn(torch.fft.rfftn(mesh) * kernel, s=(n, n, n)) * (2.0 * float(kernel.sum()) / n ** 3)
    binned = ratio.cpu().numpy().copy()
    binned[0] = binned[1:5].mean()
    return {"out": out, "kernel": kernel, "binned": binned, "modes": None}
