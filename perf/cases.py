"""The workloads whose speed and results are tracked, each one pass through the public entry points.

listed()   the fixed cases; draw() gives more of the same ranges
prepare()  what a refinement program holds before the call: particles on the device (made from the
           seed), and the context with its references, sampling and trained network, which a program
           configures once and uses for every batch (kept here for the case last prepared)
run()      the pass itself, device buffers in and out where the entry point takes them
work()     the bytes and operations that the pass cannot do without
exact()    the same outputs from plain torch in 64 bits

Kinds: "estep" (expectation of one batch of particles, on device buffers), "train" and "grad" (the
proposal network), "prep" (image preparation), "mstep" (symmetrisation, FSC, SSNR and the map).
The references are sums of seeded Gaussian blobs, whose Fourier transforms are known in closed form.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

DEV = "cuda"
PAD = 2
C128, F64, F32 = torch.complex128, torch.float64, torch.float32


def package():
    """The repository's package (its folder's name is no Python identifier)."""
    if "t2relion_b200" not in sys.modules:
        root = os.path.join(os.getcwd(), "t2-relion_b200")
        spec = importlib.util.spec_from_file_location("t2relion_b200", os.path.join(root, "__init__.py"),
                                                      submodule_search_locations=[root])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["t2relion_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["t2relion_b200"]


def device_view(ptr, n):
    return importlib.import_module(package().__name__ + ".parallel").device_view(ptr, n, torch.cuda.current_device())


# ------------------------------------------------------------------------------------ the cases
def estep(name, **kw):
    c = dict(name=name, kind="estep", dim=3, box=128, r=40, apix=1.3, order=3, psi=7.5, ovs=1, range=5, step=1.0,
             classes=1, n=64, mode="split", chunk=0, scale=0, nomask=0, snr=0.03, blobs=40)
    c.update(kw)
    return c


def listed():
    return [
        # one particle of a small 3D refinement: what a call costs when nothing fills the device
        estep("refine_one", box=64, r=16, apix=2.0, order=2, ovs=0, range=3, n=1, mode="plain", snr=0.05),
        # an odd-sized batch, two classes, unmasked images and scale correction, plain FP32
        estep("refine_ragged", box=100, r=37, apix=1.7, order=2, classes=2, range=4, n=37, mode="plain", scale=1,
              nomask=1, snr=0.05),
        # the full coarse pass of the box-128 refinement (fine pass at HEALPix order 4), split-BF16
        estep("refine_dense"),
        # the same refinement with learned proposals, the mode a refinement of many particles runs in
        estep("refine_learned", n=500, mode="learned", snr=0.1),
        # 2D classification: 50 references of 100 x 100
        estep("class2d", dim=2, box=100, r=50, apix=2.0, order=0, psi=6.0, classes=50, n=500, snr=0.05, blobs=12),
        # 3D classification of large boxes: projections made chunk by chunk inside each batch
        estep("class3d_large", box=256, r=100, apix=0.85, order=3, classes=2, range=4, n=32, chunk=16384, snr=0.02,
              blobs=60),
        # training of the proposal network on the box-128 references, as before each iteration
        dict(name="train", kind="train", box=128, r=40, apix=1.3, order=3, psi=7.5, range=5, n_train=16384, batch=256,
             n_posterior=512, n_val=256, snr=0.03),
        # one minibatch of that training, forward and backward, at a coarser sampling
        dict(name="train_grad", kind="grad", box=64, r=16, order=2, psi=7.5, n=256),
        # image preparation before the E-step: box 128 with noise background, one call of 1024 particles
        dict(name="prep_box128", kind="prep", box=128, window=80, n=1024, zero_mask=0, apix=1.3),
        # the same for a box whose transforms don't fit in shared memory, average background
        dict(name="prep_box256", kind="prep", box=256, window=200, n=160, zero_mask=1, apix=0.85),
        # end of an iteration: two half grids -> FSC, SSNR and a map (the default reconstruction)
        dict(name="mstep_box128", kind="mstep", box=128, r=64, group="C1", gridding=0),
        # the same for an icosahedral particle with the gridding iterations
        dict(name="mstep_icos_gridding", kind="mstep", box=128, r=64, group="I", gridding=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["estep", "estep", "estep", "class2d", "large", "learned", "train", "grad", "prep", "prep", "mstep"])
    box = 2 * rng.randint(24, 64)
    r = rng.randint(max(12, box // 5), box // 2 - 2)
    if kind == "estep":
        mode = rng.choice(["plain", "split", "split"])
        order = rng.choice([1, 2] if mode == "plain" else [1, 2, 3])
        return dict(kind="estep", dim=3, box=box, r=min(r, 40), apix=round(rng.uniform(1.0, 3.0), 2), order=order,
                    psi=rng.choice([15.0, 7.5]), ovs=rng.choice([0, 1, 1]), range=rng.choice([2, 3, 4, 5]), step=1.0,
                    classes=rng.choice([1, 1, 2, 3]) if order < 3 else 1, n=_log(rng, 1, 64), mode=mode, chunk=0,
                    scale=rng.randint(0, 1), nomask=rng.randint(0, 1), snr=round(rng.uniform(0.03, 0.08), 3), blobs=40)
    if kind == "class2d":
        return dict(kind="estep", dim=2, box=box, r=box // 2, apix=2.0, order=0, psi=rng.choice([5.0, 6.0, 9.0]),
                    ovs=1, range=rng.choice([3, 4, 5]), step=1.0, classes=rng.randint(4, 50), n=_log(rng, 16, 400),
                    mode="split", chunk=0, scale=0, nomask=rng.randint(0, 1), snr=round(rng.uniform(0.05, 0.1), 3),
                    blobs=12)
    if kind == "large":
        box = 2 * rng.randint(64, 112)
        return dict(kind="estep", dim=3, box=box, r=rng.randint(32, box // 2 - 8), apix=1.0, order=2, psi=7.5, ovs=1,
                    range=rng.choice([3, 4]), step=1.0, classes=rng.randint(1, 3), n=_log(rng, 4, 48), mode="split",
                    chunk=rng.choice([1000, 2048, 4096]), scale=0, nomask=0, snr=0.03, blobs=40)
    if kind == "learned":
        return dict(kind="estep", dim=3, box=128, r=40, apix=1.3, order=rng.choice([2, 3]), psi=7.5, ovs=1,
                    range=rng.choice([4, 5]), step=1.0, classes=1, n=50 * rng.randint(1, 9), mode="learned", chunk=0,
                    scale=rng.randint(0, 1), nomask=0, snr=0.1, blobs=40)
    if kind == "train":
        return dict(kind="train", box=64, r=rng.randint(14, 24), apix=2.0, order=2, psi=7.5, range=3,
                    n_train=512 * rng.randint(4, 16), batch=rng.choice([64, 128, 256]), n_posterior=128, n_val=128,
                    snr=0.05)
    if kind == "grad":
        return dict(kind="grad", box=64, r=16, order=rng.choice([1, 2]), psi=7.5, n=_log(rng, 8, 400))
    if kind == "prep":
        box = rng.choice([60, 64, 72, 80, 90, 96, 100, 108, 120, 128, 144, 150, 160, 180, 192, 216, 240, 270, 300, 320])
        return dict(kind="prep", box=box, window=2 * rng.randint(box // 5, box // 2 - 1),
                    n=max(1, min(_log(rng, 4, 1000), (1024 * 128 * 128) // (box * box))), zero_mask=rng.randint(0, 1),
                    apix=1.3)
    box = rng.choice([48, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120])
    return dict(kind="mstep", box=box, r=box // 2 - rng.randint(0, 4), group=rng.choice(["C1", "C4", "D7", "O", "I"]),
                gridding=rng.choice([0, 0, 10]))


# ---------------------------------------------------------------------------------- references
def blob_set(box, k, dim, seed):
    g = np.random.default_rng(seed)
    return dict(c=torch.tensor(g.uniform(-0.3 * box, 0.3 * box, (k, dim)), device=DEV),
                s=torch.tensor(g.uniform(2.0, 5.0, k), device=DEV), a=torch.tensor(g.uniform(0.5, 1.5, k), device=DEV))


def blob_fourier(b, box, *k):
    """The blobs' Fourier transform / box^dim at frequencies k (one tensor for each axis)."""
    dim = b["c"].shape[1]
    k2 = sum(x * x for x in k)
    out = torch.zeros(k2.shape, dtype=C128, device=DEV)
    for c, s, a in zip(b["c"], b["s"], b["a"]):
        amp = a * (2 * math.pi) ** (dim / 2) * s ** dim / box ** dim * torch.exp(-2 * math.pi ** 2 * s * s * k2 / box ** 2)
        out += torch.polar(amp, -2 * math.pi / box * sum(ci * x for ci, x in zip(c, k)))
    return out


def pad_size(r):
    return 2 * (PAD * r + 1) + 1


def reference(case, iclass):
    return blob_set(case["box"], case.get("blobs", 40), case.get("dim", 3), 100 + iclass)


def fourier_map(b, case):
    """The padded half-complex map of the Projector layout, complex64, zero beyond r * PAD."""
    ps, r = pad_size(case["r"]), case["r"]
    ax = torch.arange(-(ps // 2), ps // 2 + 1, device=DEV, dtype=F64)
    x = torch.arange(ps // 2 + 1, device=DEV, dtype=F64)
    if case.get("dim", 3) == 2:
        ky, kx = torch.meshgrid(ax, x, indexing="ij")
        f = blob_fourier(b, case["box"], kx / PAD, ky / PAD)
        return torch.where(kx * kx + ky * ky <= (r * PAD) ** 2, f, 0).to(torch.complex64)
    out = torch.zeros((ps, ps, ps // 2 + 1), dtype=torch.complex64, device=DEV)
    ky, kx = torch.meshgrid(ax, x, indexing="ij")
    for i, kz in enumerate(ax):
        f = blob_fourier(b, case["box"], kx / PAD, ky / PAD, (kz / PAD).expand_as(kx))
        out[i] = torch.where(kx * kx + ky * ky + kz * kz <= (r * PAD) ** 2, f, 0).to(torch.complex64)
    return out


def window(s):
    xh = s // 2 + 1
    i = torch.arange(s, device=DEV)
    ky = torch.where(i < xh, i, i - s)[:, None].expand(s, xh).reshape(-1).to(F64)
    kx = torch.arange(xh, device=DEV)[None, :].expand(s, xh).reshape(-1).to(F64)
    return ky, kx


def rings(s):
    """Ring of each window pixel, -1 outside the resolution mask."""
    ky, kx = window(s)
    ires = torch.round(torch.sqrt(ky * ky + kx * kx)).long()
    return torch.where((ires < s // 2 + 1) & ~((kx == 0) & (ky < 0)), ires, -1)


def ctf_image(du, dv, ang, box, apix, s):
    """CTF of 300 kV, Cs 2.7 mm, 10 % amplitude contrast on the window, n x P."""
    ky, kx = window(s)
    lam = 12.2643247 / math.sqrt(300e3 * (1 + 300e3 * 0.978466e-6))
    k1, k2, k3 = math.pi * lam, math.pi / 2 * 2.7e7 * lam ** 3, math.atan(0.1 / math.sqrt(0.99))
    c, sn = torch.cos(ang), torch.sin(ang)
    axx, axy, ayy = -du * c * c - dv * sn * sn, (dv - du) * c * sn, -du * sn * sn - dv * c * c
    x, y = kx / (box * apix), ky / (box * apix)
    u2 = x * x + y * y
    g = k1 * (axx[:, None] * x * x + 2 * axy[:, None] * x * y + ayy[:, None] * y * y) + k2 * u2 * u2 - k3
    v = -torch.sin(g)
    return torch.where(v.abs() < 1e-8, torch.where(v >= 0, 1e-8, -1e-8), v)


def euler(rot, tilt, psi):
    ca, cb, cg, sa, sb, sg = (f(t) for f in (torch.cos, torch.sin) for t in (rot, tilt, psi))
    cc, cs, sc, ss = cb * ca, cb * sa, sb * ca, sb * sa
    return torch.stack([cg * cc - sg * sa, cg * cs + sg * ca, -cg * sb, -sg * cc - cg * sa, -sg * cs + cg * ca, sg * sb,
                        sc, ss, cb], -1).reshape(-1, 3, 3)


def signal(case, g, n):
    """Noise-free particles (CTF, shift and true pose drawn from g): n x P complex128, CTF n x P."""
    s, box = 2 * case["r"], case["box"]
    ky, kx = window(s)
    u = torch.rand((n, 8), generator=g, device=DEV, dtype=F64)
    three = case.get("dim", 3) == 3
    zero = torch.zeros(n, device=DEV, dtype=F64)
    A = euler((2 * u[:, 0] - 1) * math.pi if three else zero, torch.acos(2 * u[:, 1] - 1) if three else zero,
              u[:, 2] * 2 * math.pi)
    K = case.get("classes", 1)
    cls = torch.randint(0, K, (n,), generator=g, device=DEV)
    inside = kx * kx + ky * ky <= case["r"] ** 2
    f = torch.zeros((n, ky.numel()), dtype=C128, device=DEV)
    for k in range(K):
        m = (cls == k).nonzero()[:, 0]
        if m.numel():
            q = [A[m, 0, j, None] * kx + A[m, 1, j, None] * ky for j in range(3 if three else 2)]
            f[m] = torch.where(inside, blob_fourier(reference(case, k), box, *q), 0)
    du = 10000 + 20000 * u[:, 3]
    ctf = ctf_image(du, du - 1000 * u[:, 4], u[:, 5] * math.pi, box, case["apix"], s)
    sh = (2 * u[:, 6:8] - 1) * case["range"]
    return f * ctf * torch.polar(torch.ones_like(ctf), 2 * math.pi / box * (sh[:, :1] * kx + sh[:, 1:] * ky)), ctf


def noise_level(case):
    """Variance of each noise component: the signal's mean power over the window / (2 snr)."""
    g = torch.Generator(device=DEV).manual_seed(7)
    sig, _ = signal(case, g, 64)
    return float((sig[:, rings(2 * case["r"]) > 0].abs() ** 2).mean() / (2 * case["snr"]))


def particles(case, seed, sigma2):
    g = torch.Generator(device=DEV).manual_seed(seed)
    n, s, box = case["n"], 2 * case["r"], case["box"]
    sig, ctf = signal(case, g, n)
    noise = torch.randn((2, n, sig.shape[1], 2), generator=g, device=DEV, dtype=F64) * math.sqrt(sigma2)
    f = sig + torch.view_as_complex(noise[0])
    out = dict(fimg=f.to(torch.complex64), ctf=ctf.to(F32))
    # the unmasked image: the same particle with the noise of the solvent around it
    out["nomask"] = (f + 0.5 * torch.view_as_complex(noise[1])).to(torch.complex64) if case["nomask"] else None
    ok = rings(s) > 0
    out["minv"] = torch.where(ok, 1 / sigma2, 0.0).to(F32).expand(n, -1).contiguous()
    nhr = max(0, int(math.pi / 2 * ((box // 2) ** 2 - (s // 2) ** 2)))
    scal = torch.zeros((n, 8), dtype=F64, device=DEV)
    scal[:, 0] = 1 / sigma2
    scal[:, 1] = 2 * sigma2 * (nhr + math.sqrt(nhr) * torch.randn(n, generator=g, device=DEV, dtype=F64)) if nhr else 0
    scal[:, 6] = 1 + (0.05 * torch.randn(n, generator=g, device=DEV, dtype=F64) if case["scale"] else 0)
    out["scal"] = scal
    return out


# ------------------------------------------------------------------------------------- context
class Context:
    """The E-step context of a case, with what a program configures once."""

    def __init__(self, case):
        t2b = package()
        self.key = {k: v for k, v in case.items() if k not in ("name", "n")}
        self.max_n = case.get("n", 256)
        self.case = case
        kind = case["kind"]
        self.es = t2b.EStep()
        self.stream = torch.cuda.Stream()
        if kind == "prep":
            self.configure_prep(case)
            return
        if kind == "mstep":
            for k in range(2):
                self.es.init_backprojector(k, 3, pad_size(case["r"]), case["r"], PAD)
            self.grids = self.views(2)
            return
        full = dict(estep("", dim=3, ovs=0, classes=1, range=3, step=1.0, apix=2.0, snr=0.05), **case)
        dim, K = full["dim"], full["classes"]
        s, box = 2 * full["r"], full["box"]
        self.samp = t2b.sampling(dim, full["order"], full["psi"], full["ovs"], full["range"], full["step"], full["apix"])
        self.maps = []
        for k in range(K):
            m = fourier_map(reference(full, k), full)
            self.es.set_projector(k, m.cpu().numpy(), dim, full["r"], PAD)
            self.es.init_backprojector(k, dim, pad_size(box // 2), box // 2, PAD)
        self.sigma2 = noise_level(full) if kind != "grad" else 1.0
        nd = self.samp["n_dir"]
        half = box // 2 + 1
        self.dvp = np.where(np.arange(half) < full["r"] // 2, 10.0, 1.0)[None].repeat(K, 0) if full["scale"] else None
        self.es.configure(ori_size=box, current_size=s, ref_dim=dim, nr_classes=K, samp=self.samp,
                          pdf_direction=np.full((K, nd), 1.0 / (K * nd)), pdf_class=np.full(K, 1.0 / K),
                          sigma2_offset=(full["range"] * full["apix"]) ** 2, pixel_size=full["apix"],
                          adaptive_fraction=0.999, adaptive_oversampling=full["ovs"],
                          diff2_mode=t2b.DIFF2_PLAIN_FP32 if full["mode"] == "plain" else t2b.DIFF2_SPLIT_BF16,
                          max_batch=self.max_n, data_vs_prior=self.dvp, orientation_chunk=full["chunk"])
        self.minv = np.where(rings(s).cpu().numpy() > 0, 1 / self.sigma2, 0).astype(np.float32)
        if full["mode"] == "learned":
            # a short training on the same kind of particles; an audited particle in fifty
            self.es.train_proposals(self.minv, n_train=40960, n_posterior=2048, n_val=0, epochs=2, seed=11,
                                    max_shift=full["range"])
            self.es.enable_proposals(64, 1024, 50, 0.999)
        self.grids = self.views(K)

    def configure_prep(self, case):
        N = case["box"]
        r = np.arange(N // 2 + 1)
        self.sigma2 = 0.5 / N ** 2 * (1 + 4 * np.exp(-r / 6.0))
        self.es.configure_prep(image_size=N, current_size=case["window"], max_batch=case["n"], sigma2_noise=self.sigma2,
                               pixel_size=case["apix"], mask_radius=0.4 * N, zero_mask=case["zero_mask"], random_seed=3,
                               do_norm_correction=1, avg_norm_correction=0.9)

    def views(self, K):
        nvox = int(np.prod(self.es._grid_shape))
        out = []
        for k in range(K):
            d, w = self.es.backprojector_device_ptrs(k)
            out.append((device_view(d, 2 * nvox), device_view(w, nvox)))
        return out

    def close(self):
        torch.cuda.synchronize()
        self.grids = None
        self.es.close()


_kept = []


def context(case):
    key = {k: v for k, v in case.items() if k not in ("name", "n")}
    if not (_kept and _kept[0].key == key and case.get("n", 256) == _kept[0].max_n):
        while _kept:
            _kept.pop().close()
        torch.cuda.empty_cache()
        _kept.append(Context(case))
    return _kept[0]


def results(case, samp):
    n, K, half = case["n"], case["classes"], case["box"] // 2 + 1
    z = lambda *s, dt=F64: torch.zeros(s, dtype=dt, device=DEV)  # noqa: E731
    return dict(min_diff2=z(n), sum_weight=z(n), sig_weight=z(n), coarse_sum_weight=z(n), coarse_sig_weight=z(n),
                nr_sign=z(n, dt=torch.int64), n_coarse_sig=z(n, dt=torch.int64), pmax=z(n), pose=z(n, 5, dt=torch.int32),
                wsum_norm=z(n), sumw=z(n), wsum_sigma2_offset=z(n), wsum_sigma2=z(n, half), wsum_pdf_class=z(n, K),
                wsum_pdf_dir=z(n, K * samp["n_dir"]), status=z(n, dt=torch.int32), audit_mass=z(n),
                learned=z(n, dt=torch.int32), wsum_scale_xa=z(n), wsum_scale_aa=z(n))


def prepare(case, seed):
    ctx = context(case)
    st = dict(case=case, ctx=ctx)
    kind = case["kind"]
    if kind == "estep":
        p = particles(case, seed, ctx.sigma2)
        st.update(p, out=results(case, ctx.samp))
        st["ptr"] = {k: None if v is None else ctypes.c_void_p(v.data_ptr()) for k, v in p.items()}
        st["optr"] = {k: ctypes.c_void_p(v.data_ptr()) for k, v in st["out"].items()}
    elif kind == "train":
        st["seed"] = seed
    elif kind == "grad":
        st.update(grad_inputs(case, seed, ctx.samp["n_dir"] * ctx.samp["n_psi"]))
        ctx.es.proposal_params(set_to=grad_params(ctx.samp["n_dir"] * ctx.samp["n_psi"]))
    elif kind == "prep":
        st.update(prep_inputs(case, seed))
        n, P = case["n"], case["window"] * (case["window"] // 2 + 1)
        st["out"] = dict(fimg=torch.zeros((n, P), dtype=torch.complex64, device=DEV),
                         fimg_nomask=torch.zeros((n, P), dtype=torch.complex64, device=DEV),
                         ctf=torch.zeros((n, P), device=DEV), minvsigma2=torch.zeros((n, P), device=DEV),
                         scalars=torch.zeros((n, 8), dtype=F64, device=DEV),
                         power=torch.zeros((n, case["box"] // 2 + 1), dtype=F64, device=DEV))
        st["optr"] = {k: ctypes.c_void_p(v.data_ptr()) for k, v in st["out"].items()}
    elif kind == "mstep":
        st["grid"] = half_grids(case, seed)
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------------------- run
def run(st):
    case, ctx = st["case"], st["ctx"]
    return globals()["run_" + case["kind"]](st, case, ctx, ctx.es)


def run_estep(st, case, ctx, es):
    # a batch of its own iteration: the grids start at zero
    with torch.cuda.stream(ctx.stream):
        torch._foreach_zero_([v for g in ctx.grids for v in g])
        p = st["ptr"]
        es.expectation_device(case["n"], p["fimg"], p["ctf"], p["minv"], p["scal"], st["optr"],
                              stream=ctx.stream.cuda_stream, fimg_nomask_ptr=p["nomask"])
        if len(ctx.grids) > 4:
            data, weight = torch.cat([g[0] for g in ctx.grids]), torch.cat([g[1] for g in ctx.grids])
        else:
            data, weight = [g[0] for g in ctx.grids], [g[1] for g in ctx.grids]
        # numbers of significant samples go on as numbers: the sample at the threshold is rounding's choice
        count = {k: st["out"][k].to(F64) for k in ("nr_sign", "n_coarse_sig")}
    return dict(st["out"], **count, grid_data=data, grid_weight=weight)


def run_train(st, case, ctx, es):
    rep = es.train_proposals(ctx.minv, n_train=case["n_train"], n_posterior=case["n_posterior"], n_val=case["n_val"],
                             epochs=1, batch=case["batch"], rescore=0, seed=st["seed"], max_shift=case["range"])
    return dict(loss=np.array(rep["loss"]), mass=np.array([rep["val_mass_init"], rep["val_mass_trained"]]),
                params=es.proposal_params())


def run_grad(st, case, ctx, es):
    loss, g = es.proposal_grad(st["imgs"], st["tgt_oc"], st["tgt_w"])
    return dict(loss=loss, grad=g)


def run_prep(st, case, ctx, es):
    es.prepare_images_device(case["n"], *(ctypes.c_void_p(st[k].data_ptr()) for k in ("images", "params", "part_id")),
                             st["optr"], stream=ctx.stream.cuda_stream)
    return st["out"]


def run_mstep(st, case, ctx, es):
    box = case["box"]
    # the grids as the E-step left them (the symmetries below work in place)
    for g, h in zip(ctx.grids, st["grid"]):
        for v, x in zip(g, h):
            v.copy_(x)
    torch.cuda.current_stream().synchronize()
    for k in range(2):
        es.enforce_hermitian_symmetry(k)
        if case["group"] != "C1":
            es.apply_point_group_symmetry(k, case["group"])
    fsc = es.fsc_halves(0, 1, box)
    tau2, sigma2, dvp, cov = es.update_ssnr(0, box, np.zeros(box // 2 + 1), fsc=fsc)
    vol = es.reconstruct(0, box, tau2=tau2, gridding_iter=case["gridding"], normalise=1000.0 if case["gridding"] else 1.0)
    return dict(fsc=fsc, tau2=tau2, sigma2=sigma2, data_vs_prior=dvp, coverage=cov, map=vol, grid_data=ctx.grids[0][0],
                grid_weight=ctx.grids[0][1])


# --------------------------------------------------------------------------------------- inputs
def grad_inputs(case, seed, KO):
    g = np.random.default_rng(seed)
    n = case["n"]
    imgs = g.standard_normal((2 * n + 8, 256))
    imgs = (imgs / np.sqrt((imgs ** 2).mean(1, keepdims=True))).astype(np.float32)
    # images without an activation at rounding distance of zero: there rounding decides a ReLU's gradient
    zs = forward(grad_weights(KO), torch.tensor(imgs, device=DEV, dtype=F64))[:-1]
    near = torch.stack([(z.abs().flatten(1).amin(1) < 2e-5 * z.std()) for z in zs]).any(0)
    imgs = np.ascontiguousarray(imgs[~near.cpu().numpy()][:n])
    oc = g.integers(0, KO, (n, 9)).astype(np.int32)
    w = g.random((n, 9)) ** 3
    oc[:, 6:] = -1
    w[:, 6:] = 0
    return dict(imgs=imgs, tgt_oc=oc, tgt_w=(w / w.sum(1, keepdims=True)).astype(np.float32))


def grad_layout(KO):
    al = lambda x: (x + 63) // 64 * 64  # noqa: E731
    L, o = {}, 0
    for name, shape in (("wc1", (16, 1, 3, 3)), ("bc1", (16,)), ("wc2", (32, 16, 3, 3)), ("bc2", (32,)), ("b1", (1024,)),
                        ("b2", (1024,)), ("b3", (KO,)), ("w1", (1024, 2048)), ("w2", (1024, 1024)), ("w3", (KO, 1024))):
        L[name] = (o, shape)
        o = al(o + int(np.prod(shape)))
    return L


def grad_params(KO):
    """Weights of a network in training: He-scaled layers, small biases (flat, in the library's layout)."""
    if KO not in _params:
        _params.clear()
        g = np.random.default_rng(5)
        L = grad_layout(KO)
        out = np.zeros(L["w3"][0] + KO * 1024, np.float32)
        for name, (o, shape) in L.items():
            fan = int(np.prod(shape[1:])) if name[0] == "w" else 0
            x = g.standard_normal(int(np.prod(shape)), np.float32) * (math.sqrt(2 / fan) if fan else 0.02)
            out[o:o + x.size] = x
        _params[KO] = out
    return _params[KO]


_params = {}


def grad_weights(KO):
    """The parameters as every pass reads them, rounded to BF16, by layer in 64 bits."""
    th = torch.tensor(grad_params(KO), device=DEV).to(torch.bfloat16).to(F64)
    return {k: th[o:o + int(np.prod(sh))].reshape(sh) for k, (o, sh) in grad_layout(KO).items()}


def forward(p, x):
    """The network's values before each ReLU, and its logits last."""
    conv = torch.nn.functional.conv2d
    z1 = conv(x.reshape(-1, 1, 16, 16), p["wc1"], p["bc1"], padding=1)
    z2 = conv(torch.relu(z1), p["wc2"], p["bc2"], padding=1, stride=2)
    z3 = torch.relu(z2).reshape(-1, 2048) @ p["w1"].T + p["b1"]
    z4 = torch.relu(z3) @ p["w2"].T + p["b2"]
    return z1, z2, z3, z4, torch.relu(z4) @ p["w3"].T + p["b3"]


def prep_inputs(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    n, N = case["n"], case["box"]
    b = blob_set(N, 24, 2, 300)
    ax = torch.arange(N, device=DEV, dtype=F64) - N // 2
    y, x = torch.meshgrid(ax, ax, indexing="ij")
    img = sum(a * torch.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2) / (2 * s * s)) for c, s, a in zip(b["c"], b["s"], b["a"]))
    u = torch.rand((n, 8), generator=g, device=DEV, dtype=F64)
    images = ((0.5 + u[:, 7, None, None]) * img + torch.randn((n, N, N), generator=g, device=DEV)).to(F32)
    par = torch.zeros((n, 12), dtype=F64, device=DEV)
    par[:, 0:2] = (u[:, 0:2] - 0.5) * 12
    par[:, 2:4] = 999.0
    par[:, 4] = 0.8 + 0.4 * u[:, 2]
    par[:, 5] = 10000 + 20000 * u[:, 3]
    par[:, 6] = par[:, 5] - 1000 * u[:, 4]
    par[:, 7] = 180 * u[:, 5]
    par[:, 8] = 20 * u[:, 6]
    par[:, 9] = 1.0
    par[:, 11] = 1.0
    return dict(images=images, params=par, part_id=torch.arange(n, device=DEV) + seed % 100003)


def half_grids(case, seed):
    """Two half-set grids: weights as a few thousand particles leave them (falling as 1 / radius, uneven), data =
    weight x (map + noise)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    ps, box = pad_size(case["r"]), case["box"]
    ax = torch.arange(-(ps // 2), ps // 2 + 1, device=DEV, dtype=F32)
    x = torch.arange(ps // 2 + 1, device=DEV, dtype=F32)
    b = {k: v.to(F32) for k, v in blob_set(box, 40, 3, 100).items()}
    kz, ky, kx = torch.meshgrid(ax, ax, x, indexing="ij")
    r2 = kz * kz + ky * ky + kx * kx
    inside = r2 <= (PAD * case["r"]) ** 2
    f = torch.zeros(r2.shape, dtype=torch.complex64, device=DEV)
    for c, s, a in zip(b["c"], b["s"], b["a"]):
        amp = a * (2 * math.pi) ** 1.5 * s ** 3 / box ** 3 * torch.exp(-2 * math.pi ** 2 * s * s / (box * PAD) ** 2 * r2)
        f += torch.polar(amp, -2 * math.pi / (box * PAD) * (c[0] * kx + c[1] * ky + c[2] * kz))
    noise = float(f[inside].abs().square().mean().sqrt())
    out = []
    for _ in range(2):
        w = torch.where(inside, 3000.0 / (1 + r2.sqrt()) * (0.2 + torch.rand(r2.shape, generator=g, device=DEV)), 0)
        z = torch.view_as_complex(torch.randn((*r2.shape, 2), generator=g, device=DEV) * noise)
        out.append((torch.view_as_real(w * (f + z)).reshape(-1).contiguous(), w.reshape(-1).contiguous()))
    return out


# ---------------------------------------------------------------------------------------- work
def sampling_size(case):
    nd = 12 * 4 ** case["order"] if case.get("dim", 3) == 3 else 1
    rng, st = case["range"], case.get("step", 1.0)
    m = int(math.ceil(rng / st))
    T = sum(1 for i in range(-m, m + 1) for j in range(-m, m + 1) if (i * i + j * j) * st * st < rng * rng + 0.001)
    return nd * int(round(360 / case["psi"])), T


def work(case):
    kind = case["kind"]
    if kind in ("estep", "train"):
        O, T = sampling_size(case)
        s = 2 * case["r"]
        P = s * (s // 2 + 1)
        KO = O * case.get("classes", 1)
        full = 8.0 * KO * T * P            # real operations of one particle's cross terms
    if kind == "estep":
        n, K, dim = case["n"], case["classes"], case["dim"]
        grid = pad_size(case["box"] // 2) ** dim / 2 * 12 * K
        model = pad_size(case["r"]) ** dim / 2 * 8 * K
        by = n * P * (16 + 8 * case["nomask"]) + grid + model
        if case["mode"] == "learned":
            net = 2.0 * (2048 * 1024 + 1024 * 1024 + 1024 * KO)
            return dict(bytes=by + 2 * 1024 * KO, flops=n * (8.0 * 64 * T * P + 8.0 * 1024 * T * 145 + net) + n / 50 * full)
        return dict(bytes=by, flops=n * full)
    if kind == "train":
        net = 2.0 * (2048 * 1024 + 1024 * 1024 + 1024 * KO)
        par = 2048 * 1024 + 1024 * 1024 + 1024 * KO
        steps = case["n_train"] // case["batch"]
        return dict(bytes=steps * par * 26.0, flops=3 * net * case["n_train"] + (case["n_posterior"] + 2 * case["n_val"]) * full)
    if kind == "grad":
        KO = 12 * 4 ** case["order"] * int(round(360 / case["psi"]))
        par = 2048 * 1024 + 1024 * 1024 + 1024 * KO
        return dict(bytes=par * 6.0 + case["n"] * 1096, flops=6.0 * par * case["n"])
    if kind == "prep":
        N, s, n = case["box"], case["window"], case["n"]
        fft = 2.5 * N * N * math.log2(N * N)
        return dict(bytes=n * (4.0 * N * N + 24 * s * (s // 2 + 1)), flops=n * fft * (2 if case["zero_mask"] else 3))
    vox = pad_size(case["r"]) ** 3 / 2
    N, box = 2 * case["box"], case["box"]
    ops = {"C1": 0, "C4": 3, "D7": 13, "O": 23, "I": 59}[case["group"]]
    inside = 4 / 3 * math.pi * (PAD * case["r"]) ** 3 / 2
    fft = 2.5 * N ** 3 * math.log2(N ** 3)
    gfft = 2.5 * pad_size(case["r"]) ** 3 * math.log2(pad_size(case["r"]) ** 3)
    return dict(bytes=2 * vox * 24 + 8 * box ** 3, flops=2 * inside * ops * 70 + fft + 2 * case["gridding"] * gfft)


def tolerance(case):
    kind = case["kind"]
    # estep: diff2 is held in FP32 (a value of 1e4 to 6e-4), so a weight is known to 1e-3 and a significance
    # threshold, one single weight, to the spacing of the weights near it.  train: FP32 gradient atomics and Adam's
    # normalised steps, 64 of them
    return {"estep": {"rel": 0.02, "max": 0.5, "differ": 0.01},
            "train": {"rel": 0.015, "max": 0.3}, "grad": {"rel": 2e-6, "max": 1e-3},
            "prep": {"rel": 1e-6, "max": 5e-5}, "mstep": {"rel": 2e-6, "max": 1e-4}}[kind]


# --------------------------------------------------------------------------------------- exact
def exact(case, seed):
    fn = globals().get("exact_" + case["kind"])
    return fn(case, seed) if fn else None


def slices(m, A, s, r, dim):
    """Trilinear (bilinear) central slices of the padded map for Euler matrices A (m x 9): m x P complex128."""
    ky, kx = window(s)
    A = A.reshape(-1, 3, 3)
    c = m.shape[0] // 2
    x, y, z = ((A[:, 0, j, None] * kx + A[:, 1, j, None] * ky) * PAD for j in range(3))
    neg = x < 0
    sg = torch.where(neg, -1.0, 1.0).to(F64)
    x, y, z = x * sg, y * sg, z * sg
    flat = m.reshape(-1)
    yd, xd = m.shape[-2], m.shape[-1]
    x0, y0 = x.floor(), y.floor()
    fx, fy = x - x0, y - y0
    out = 0
    if dim == 3:
        z0 = z.floor()
        fz = z - z0
    for dz in range(2 if dim == 3 else 1):
        for dy in range(2):
            for dx in range(2):
                idx = (y0.long() + c + dy) * xd + x0.long() + dx
                w = (fx if dx else 1 - fx) * (fy if dy else 1 - fy)
                if dim == 3:
                    idx = idx + (z0.long() + c + dz) * yd * xd
                    w = w * (fz if dz else 1 - fz)
                out = out + w * flat[torch.where((kx * kx + ky * ky <= r * r), idx, 0)]
    out = torch.where(neg, out.conj(), out)
    return torch.where(kx * kx + ky * ky <= r * r, out, 0)


def phases(tr, s, box):
    ky, kx = window(s)
    ang = -2 * math.pi / box * (tr[:, :1] * kx + tr[:, 1:] * ky)
    return torch.polar(torch.ones_like(ang), ang)


def threshold(w, frac):
    """(sum, significance threshold, samples counted) of one particle's weights."""
    v = torch.sort(w[w > 0], descending=True).values
    c = torch.cumsum(v, 0)
    i = int(torch.searchsorted(c, frac * c[-1:], right=True).clamp(max=v.numel() - 1))
    return w.sum(), v[i], i + 1


def exact_estep(case, seed):
    ctx = context(case)
    samp, dim, K, box, n = ctx.samp, case["dim"], case["classes"], case["box"], case["n"]
    s, r, apix = 2 * case["r"], case["r"], case["apix"]
    xh, P = s // 2 + 1, s * (s // 2 + 1)
    O, T = samp["n_dir"] * samp["n_psi"], samp["n_trans"]
    if 16.0 * n * K * O * T > 60e9 or 8.0 * n * K * O * T * P > 60e12:
        return None
    p = particles(case, seed, ctx.sigma2)
    X, ctf, minv, scal = p["fimg"].to(C128), p["ctf"].to(F64), p["minv"].to(F64), p["scal"]
    Xn = X if p["nomask"] is None else p["nomask"].to(C128)
    up = lambda a: torch.tensor(a, device=DEV, dtype=F64)  # noqa: E731
    eul_c, eul_f = up(samp["eul_coarse"]), up(samp["eul_fine"] if case["ovs"] else samp["eul_coarse"])
    tr_c, tr_f = up(samp["trans_px"]), up(samp["trans_px_fine"] if case["ovs"] else samp["trans_px"])
    R, V = (samp["nover_rot"], samp["nover_trans"]) if case["ovs"] else (1, 1)
    maps = [fourier_map(reference(case, k), case).to(C128) for k in range(K)]
    c = ctf * scal[:, 6:7]
    c0 = scal[:, 1] / 2 + 0.5 * (minv * X.abs() ** 2).sum(1)
    ab, abf = phases(tr_c, s, box), phases(tr_f, s, box)
    # coarse pass: c0 + |c P|^2 / 2 - Re (c P) conj(X ab), weighted by Minvsigma2
    Y = torch.view_as_real(((minv * c * X)[:, None] * ab)).reshape(n * T, 2 * P)
    d2 = torch.empty((n, K * O, T), dtype=F64, device=DEV)
    rows = max(16, int(2e6) // P)
    for k in range(K):
        for a in range(0, O, rows):
            F = slices(maps[k], eul_c[a:a + rows], s, r, dim)
            m = F.shape[0]
            cross = (torch.view_as_real(F).reshape(m, 2 * P) @ Y.T).reshape(m, n, T)
            nrm = 0.5 * (F.abs() ** 2) @ (minv * c * c).T
            d2[:, k * O + a:k * O + a + m] = (c0 + nrm)[:, :, None].permute(1, 0, 2) - cross.permute(1, 0, 2)
    del Y
    # priors: uniform over orientations, a Gaussian around the old offset over shifts
    tp = up(samp["trans_prior"])
    off, pri = scal[:, 2:4], scal[:, 4:6]
    s2o = (case["range"] * apix) ** 2
    pt = torch.exp((((off - pri)[:, None] + tp) ** 2).sum(2) * apix ** 2 / (-2 * s2o))
    pt = pt / pt.mean(1, keepdim=True)
    out = {q: torch.zeros(v.shape, dtype=F64, device=DEV) for q, v in results(case, samp).items()
           if v.dtype == F64 and q != "audit_mass"}
    gs = [pad_size(box // 2)] * dim
    gs[-1] = gs[-1] // 2 + 1
    gd = [torch.zeros(2 * int(np.prod(gs)), dtype=F64, device=DEV) for _ in range(K)]
    gw = [torch.zeros(int(np.prod(gs)), dtype=F64, device=DEV) for _ in range(K)]
    ring = rings(s)
    dvp = None if ctx.dvp is None else up(ctx.dvp)
    ky, kx = window(s)
    bp = (kx * kx + ky * ky <= (box // 2) ** 2) & ~((kx == 0) & (ky < 0))
    for b in range(n):
        dd = d2[b] - d2[b].min()
        w = torch.where(dd > 700, 0, pt[b] * torch.exp(-dd))
        sw, sig, _ = threshold(w.reshape(-1), 0.999)
        out["coarse_sum_weight"][b], out["coarse_sig_weight"][b] = sw, sig
        mask = w >= sig
        oc = mask.any(1).nonzero()[:, 0]
        cls = oc // O
        e = (oc % O)[:, None] * R + torch.arange(R, device=DEV)
        F = torch.cat([slices(maps[k], eul_f[e[cls == k].reshape(-1)], s, r, dim) for k in range(K) if (cls == k).any()]) * c[b]
        mk = mask[oc][:, None, :, None].expand(-1, R, -1, V).reshape(oc.numel() * R, T * V)
        ptv = pt[b][:, None].expand(T, V).reshape(-1)
        if case["ovs"]:
            Yb = minv[b] * X[b] * abf
            f2 = c0[b] + 0.5 * (F.abs() ** 2) @ minv[b]
            df = f2[:, None] - torch.view_as_real(F).reshape(-1, 2 * P) @ torch.view_as_real(Yb).reshape(-1, 2 * P).T
            mn = df[mk].min()
            wf = torch.where(mk & (df - mn <= 700), ptv * torch.exp(-(df - mn)), 0)
            fs, fsig, _ = threshold(wf[mk], 0.999)
        else:
            mn, wf, fs, fsig = d2[b].min(), torch.where(mk, w[oc], 0), sw, sig
        out["min_diff2"][b], out["sum_weight"][b], out["sig_weight"][b] = mn, fs, fsig
        W = torch.where(mk & (wf >= fsig), wf, 0) / fs
        out["pmax"][b], out["sumw"][b] = W.max(), W.sum()
        Wr = W.sum(1)
        row_cls = cls.repeat_interleave(R)
        out["wsum_pdf_class"][b].index_add_(0, row_cls, Wr)
        out["wsum_pdf_dir"][b].index_add_(0, row_cls * samp["n_dir"] + ((oc % O) // samp["n_psi"]).repeat_interleave(R), Wr)
        out["wsum_sigma2_offset"][b] = (W.sum(0) * ((pri[b] - off[b] - tr_f) ** 2).sum(1)).sum() * apix ** 2
        use = (Wr > 0).nonzero()[:, 0]
        W, Wr, F, row_cls = W[use], Wr[use], F[use], row_cls[use]
        S = W.to(C128) @ abf
        cross, power = (F * (S * X[b]).conj()).real, Wr[:, None] * F.abs() ** 2
        wd = power.sum(0) - 2 * cross.sum(0) + Wr.sum() * X[b].abs() ** 2
        ok = ring >= 0
        out["wsum_sigma2"][b].index_add_(0, ring[ok], wd[ok])
        out["wsum_norm"][b] = wd[ok].sum()
        if dvp is not None:
            sel = ok & (dvp[0][ring.clamp(min=0)] > 3)
            out["wsum_scale_xa"][b], out["wsum_scale_aa"][b] = cross[:, sel].sum() / scal[b, 6], power[:, sel].sum() / scal[b, 6] ** 2
        mi = minv[b].clone()
        mi[0] = scal[b, 0]
        val, wgt = S * (Xn[b] * c[b] * mi), Wr[:, None] * (c[b] ** 2 * mi)
        A = eul_f[((oc % O)[:, None] * R + torch.arange(R, device=DEV)).reshape(-1)[use]]
        for k in range(K):
            q = row_cls == k
            if q.any():
                backproject(gd[k], gw[k], gs, A[q], val[q][:, bp], wgt[q][:, bp], kx[bp], ky[bp], dim)
    # the thresholds are single weights picked by rank: rounding picks the neighbour, in any precision
    for q in ("sig_weight", "coarse_sig_weight"):
        out[q] = None
    if K > 4:
        gd, gw = torch.cat(gd), torch.cat(gw)
    return dict(out, grid_data=gd, grid_weight=gw)


def backproject(gd, gw, gs, A, val, wgt, kx, ky, dim):
    A = A.reshape(-1, 3, 3)
    step = max(1, int(4e6) // kx.numel())
    for a in range(0, A.shape[0], step):
        x, y, z = ((A[a:a + step, 0, j, None] * kx + A[a:a + step, 1, j, None] * ky) * PAD for j in range(3))
        v, w = val[a:a + step], wgt[a:a + step]
        sg = torch.where(x < 0, -1.0, 1.0).to(F64)
        v = torch.where(x < 0, v.conj(), v)
        x, y, z = x * sg, y * sg, z * sg
        for corner in range(2 ** dim):
            idx, t = 0, w > 0
            f = torch.where(w > 0, 1.0, 0.0).to(F64)
            for axis, (q, size) in enumerate(zip([z, y, x][3 - dim:], gs)):
                bit = corner >> (dim - 1 - axis) & 1
                q0 = q.floor()
                f = f * ((q - q0) if bit else (1 - (q - q0)))
                idx = idx * size + q0.long() + bit + (0 if axis == dim - 1 else size // 2)
            for i, u in ((0, v.real), (1, v.imag)):
                gd.index_add_(0, (2 * idx + i).reshape(-1), (f * u).reshape(-1))
            gw.index_add_(0, idx.reshape(-1), (f * w).reshape(-1))


def exact_grad(case, seed):
    KO = 12 * 4 ** case["order"] * int(round(360 / case["psi"]))
    q = grad_inputs(case, seed, KO)
    L = grad_layout(KO)
    p = {k: v.clone().requires_grad_() for k, v in grad_weights(KO).items()}
    logp = torch.log_softmax(forward(p, torch.tensor(q["imgs"], device=DEV, dtype=F64))[-1], 1)
    oc, w = torch.tensor(q["tgt_oc"], device=DEV).long(), torch.tensor(q["tgt_w"], device=DEV, dtype=F64)
    loss = -(logp.gather(1, oc.clamp(min=0)) * torch.where(oc >= 0, w, 0)).sum(1).mean()
    loss.backward()
    g = torch.zeros(L["w3"][0] + KO * 1024, dtype=F64, device=DEV)
    for k, (o, sh) in L.items():
        g[o:o + int(np.prod(sh))] = p[k].grad.reshape(-1)
    return dict(loss=float(loss), grad=g.detach())


def splitmix(z):
    """The SplitMix64 finaliser on int64 tensors (their bits as unsigned)."""
    i64 = lambda v: v - (1 << 64) if v >> 63 else v  # noqa: E731
    sh = lambda v, k: (v >> k) & ((1 << (64 - k)) - 1)  # noqa: E731
    z = z + i64(0x9E3779B97F4A7C15)
    z = (z ^ sh(z, 30)) * i64(0xBF58476D1CE4E5B9)
    z = (z ^ sh(z, 27)) * i64(0x94D049BB133111EB)
    return z ^ sh(z, 31)


def exact_prep(case, seed):
    q = prep_inputs(case, seed)
    N, s, n = case["box"], case["window"], case["n"]
    h = N // 2 + 1
    par = q["params"]
    r = torch.arange(h, device=DEV, dtype=F64)
    sigma2 = 0.5 / N ** 2 * (1 + 4 * torch.exp(-r / 6.0))
    img = q["images"].to(F64) * (0.9 / par[:, 4])[:, None, None]
    sh = torch.sign(par[:, 0:2]) * torch.floor(par[:, 0:2].abs() + 0.5)
    ax = torch.arange(N, device=DEV)
    ix, iy = (ax - sh[:, i, None].long() for i in (0, 1))
    ok = ((ix >= 0) & (ix < N))[:, None, :] & ((iy >= 0) & (iy < N))[:, :, None]
    img = torch.where(ok, img[torch.arange(n, device=DEV)[:, None, None], iy.clamp(0, N - 1)[:, :, None], ix.clamp(0, N - 1)[:, None, :]], 0)
    ky, kx = window(N)
    ires = torch.round(torch.sqrt(ky * ky + kx * kx)).long().reshape(N, h)
    c = ax.to(F64) - N // 2
    rad = torch.sqrt(c[:, None] ** 2 + c[None, :] ** 2)
    r0, width = 0.4 * N, 5.0
    rc = torch.where(rad < r0, 0.0, torch.where(rad > r0 + width, 1.0, 0.5 + 0.5 * torch.cos(math.pi * (r0 + width - rad) / width)))
    if case["zero_mask"]:
        fill = ((rc * img).sum((1, 2)) / rc.sum())[:, None, None]
    else:
        key = splitmix(q["part_id"] + 3)
        x = splitmix(key[:, None] + torch.arange(N * h, device=DEV)).reshape(n, N, h)
        u1 = (((x >> 40) & 0xFFFFFF).to(F64) + 1) * 2.0 ** -24
        u2 = ((x >> 8) & 0xFFFFFF).to(F64) * 2.0 ** -24
        sd = torch.where(ires < h, sigma2[ires.clamp(max=h - 1)].sqrt(), 0)
        fill = torch.fft.irfft2(torch.polar(torch.sqrt(-2 * torch.log(u1)) * sd, 2 * math.pi * u2), s=(N, N)) * N * N
    masked = (1 - rc) * img + rc * fill
    Fu, F = torch.fft.rfft2(img) / N ** 2, torch.fft.rfft2(masked) / N ** 2
    spec = (ires > 0) & (ires < h) & ~((kx == 0) & (ky < 0)).reshape(N, h)
    a2 = F.abs() ** 2
    power = torch.zeros((n, h), dtype=F64, device=DEV).index_add_(1, ires[spec], a2[:, spec])
    wy, wx = window(s)
    sign = torch.where((torch.arange(s, device=DEV)[:, None] ^ torch.arange(s // 2 + 1, device=DEV)) & 1 == 1, -1.0, 1.0).reshape(-1)
    cut = lambda f: f[:, wy.long() % N, wx.long()] * sign  # noqa: E731
    u2w = (wx * wx + wy * wy) / (N * case["apix"]) ** 2
    ctf = ctf_image(par[:, 5], par[:, 6], par[:, 7] * math.pi / 180, N, case["apix"], s) * torch.exp(-par[:, 8:9] / 4 * u2w)
    ring = rings(s)
    minv = torch.where(ring > 0, 1 / sigma2[ring.clamp(min=0)], 0).expand(n, -1)
    sc = torch.zeros((n, 8), dtype=F64, device=DEV)
    sc[:, 0] = 1 / sigma2[0]
    sc[:, 1] = a2[:, spec & (ires >= s // 2 + 1)].sum(1)
    sc[:, 2:4] = sh
    sc[:, 6] = 1
    return dict(fimg=cut(F), fimg_nomask=cut(Fu), ctf=ctf, minvsigma2=minv, scalars=sc, power=power)


def rotations(group):
    """The rotations of a point group other than the identity, closed under products."""
    def about(axis, fold):
        a = np.array(axis, float) / np.linalg.norm(axis)
        cr = np.array([[0, -a[2], a[1]], [a[2], 0, -a[0]], [-a[1], a[0], 0]])
        t = 2 * math.pi / fold
        return math.cos(t) * np.eye(3) + math.sin(t) * cr + (1 - math.cos(t)) * np.outer(a, a)
    phi = (1 + 5 ** 0.5) / 2
    gen = {"C1": [], "C4": [((0, 0, 1), 4)], "D7": [((0, 0, 1), 7), ((1, 0, 0), 2)],
           "O": [((1, 1, 1), 3), ((0, 0, 1), 4)], "I": [((0, 0, 1), 2), ((1, 0, phi), 5)]}[group]
    found, todo = [np.eye(3)], [np.eye(3)]
    while todo:
        m = todo.pop()
        for g in (about(*q) for q in gen):
            p = m @ g
            if not any(np.abs(p - f).max() < 1e-6 for f in found):
                found.append(p)
                todo.append(p)
    return found[1:]


def exact_mstep(case, seed):
    r, box, ps = case["r"], case["box"], pad_size(case["r"])
    fx, c, xd = ps // 2 + 1, ps // 2, ps // 2 + 1
    ax = torch.arange(-c, c + 1, device=DEV)
    kz, ky, kx = torch.meshgrid(ax, ax, torch.arange(xd, device=DEV), indexing="ij")
    r2 = kz * kz + ky * ky + kx * kx
    halves = []
    for d, w in half_grids(case, seed):
        d = torch.view_as_complex(d.to(F64).reshape(ps, ps, xd, 2)).clone()
        w = w.to(F64).reshape(ps, ps, xd).clone()
        # Friedel pairs of the x = 0 plane summed; the origin, its own partner, is left as it is
        d0, w0 = d[c, c, 0].clone(), w[c, c, 0].clone()
        d[:, :, 0] = d[:, :, 0] + d[:, :, 0].flip(0, 1).conj()
        w[:, :, 0] = w[:, :, 0] + w[:, :, 0].flip(0, 1)
        d[c, c, 0], w[c, c, 0] = d0, w0
        # each step leaves the grid in 32 bits, as the device's grids are
        d, w = d.to(torch.complex64).to(C128), w.to(F32).to(F64)
        ops = rotations(case["group"])
        if ops:
            both = torch.stack([d.real, d.imag, w], -1).reshape(-1, 3)
            ins = (r2 <= (PAD * r) ** 2).reshape(-1).nonzero()[:, 0]
            pos = torch.stack([kx.reshape(-1)[ins], ky.reshape(-1)[ins], kz.reshape(-1)[ins]], -1).to(F64)
            total = both.clone()
            for m in ops:
                q = pos @ torch.tensor(m, device=DEV).T
                neg = q[:, 0] < 0
                q = torch.where(neg[:, None], -q, q)
                q0 = q.floor()
                f = q - q0
                q0 = q0.long()
                v = torch.zeros((ins.numel(), 3), dtype=F64, device=DEV)
                for corner in range(8):
                    b = [corner >> j & 1 for j in range(3)]
                    idx = ((q0[:, 2] + b[2] + c) * ps + q0[:, 1] + b[1] + c) * xd + q0[:, 0] + b[0]
                    wt = 1
                    for j in range(3):
                        wt = wt * (f[:, j] if b[j] else 1 - f[:, j])
                    v += wt[:, None] * both[idx]
                v[:, 1] = torch.where(neg, -v[:, 1], v[:, 1])
                total[ins] += v
            total = total.to(F32).to(F64).reshape(ps, ps, xd, 3)
            d, w = torch.complex(total[..., 0], total[..., 1]), total[..., 2].contiguous()
        halves.append((d, w))
    half = lambda v: torch.sign(v) * torch.floor(v.abs() + 0.5)  # noqa: E731
    # FSC of the down-sampled halves
    ds = 2 * (r + 1) + 1
    dh = ds // 2
    i = [(half(q / PAD).long()) for q in (kz, ky, kx)]
    lin = ((i[0] + dh) * ds + i[1] + dh) * (dh + 1) + i[2]
    avg = []
    for d, w in halves:
        a = torch.zeros((ds * ds * (dh + 1), 3), dtype=F64, device=DEV)
        a.index_add_(0, lin.reshape(-1), torch.stack([d.real, d.imag, w], -1).reshape(-1, 3))
        avg.append(torch.complex(a[:, 0], a[:, 1]) / torch.where(a[:, 2] > 0, a[:, 2], 1.0) * (a[:, 2] > 0))
    a = torch.arange(-dh, dh + 1, device=DEV)
    R = torch.sqrt((a[:, None, None] ** 2 + a[None, :, None] ** 2 + torch.arange(dh + 1, device=DEV) ** 2).to(F64)).reshape(-1)
    m = R <= r
    sh = torch.floor(R[m] + 0.5).long()
    nb = box // 2 + 1
    bins = lambda v, ix=sh, k=nb: torch.zeros(k, dtype=F64, device=DEV).index_add_(0, ix, v)  # noqa: E731
    a1, a2 = avg[0][m], avg[1][m]
    den = bins(a1.abs() ** 2) * bins(a2.abs() ** 2)
    fsc = torch.where(den > 0, bins((a1 * a2.conj()).real) / torch.where(den > 0, den, 1).sqrt(), 0)
    fsc[0] = 1
    # SSNR from the FSC
    d, w = halves[0]
    oc = float(PAD) ** 3
    m = r2 < (PAD * r) ** 2
    rad = torch.sqrt(r2.to(F64))
    ires = torch.floor(rad / PAD + 0.5).long()
    s2, cnt = bins(oc * w[m], ires[m]), bins(torch.ones_like(w[m]), ires[m])
    sigma2 = torch.where(s2 > 1e-10, cnt / torch.where(s2 > 1e-10, s2, 1), 0)
    f = fsc.clamp(min=0.001).clamp(max=0.999)
    dvp = f / (1 - f)
    tau2 = dvp * sigma2
    t = tau2[ires.clamp(max=nb - 1)]
    it = torch.where(t > 0, 1 / (oc * torch.where(t > 0, t, 1)), 1 / (0.001 * w))
    cov = bins((w[m] / it[m] >= 1).to(F64), ires[m])
    cov = torch.where(cnt > 0, cov / cnt.clamp(min=1), cov)
    # the map: MAP term, division (or gridding weights), window, inverse transform, mask, gridding correction
    kp = torch.arange(ps, device=DEV)
    kp = torch.where(kp < fx, kp, kp - ps)
    roll = lambda v: v[kp + c][:, kp + c]  # noqa: E731
    r2f = roll(r2)
    ins = r2f <= (PAD * r) ** 2
    Fd, W = torch.where(ins, roll(d), 0), torch.where(ins, roll(w), 0)
    m = r2f < (PAD * r) ** 2
    it = torch.where(t > 0, 1 / (oc * torch.where(t > 0, t, 1)), torch.where(w > 1e-20, 1 / (0.001 * w), 0))
    W = torch.where(m, W + roll(it), W)
    if case["gridding"]:
        W, Fd = W / 1000.0, Fd / 1000.0
        FN = m.to(F64)
        i = torch.arange(10000, device=DEV, dtype=F64) * (0.5 / 10000)
        u = 2 * math.pi * 3.8 * i
        sq = (225.0 - u * u).abs().sqrt()
        bes = torch.where(u > 15, torch.sin(sq) / sq - torch.cos(sq), torch.cosh(sq) - torch.sinh(sq) / sq) * sq ** -2.0
        kc = torch.arange(ps, device=DEV)
        kc = torch.where(kc < ps // 2, kc, kc - ps).to(F64)
        rv = torch.sqrt(kc[:, None, None] ** 2 + kc[None, :, None] ** 2 + kc[None, None, :] ** 2) / (box * PAD)
        ix = (rv / (0.5 / 10000)).long()
        B = torch.where(ix < 10000, bes[ix.clamp(max=9999)], 0) / bes[0]
        for _ in range(case["gridding"]):
            conv = torch.fft.rfftn(torch.fft.irfftn((FN * W).to(C128), s=(ps, ps, ps)) * B)
            FN = torch.where(m, FN / conv.abs().clamp(min=1e-6), FN)
        Fc = Fd * FN
    else:
        shell = torch.floor(torch.sqrt(r2f.to(F64)) / PAD).long()
        av = bins(W[m], shell[m], r) / (1000 * bins(torch.ones_like(W[m]), shell[m], r))
        W = torch.maximum(W, av[shell.clamp(max=r - 1)])
        Fc = torch.where(W != 0, Fd / torch.where(W != 0, W, 1), Fd)
    N = PAD * box
    h = N // 2 + 1
    G = torch.zeros((N, N, h), dtype=C128, device=DEV)
    if N > ps:
        Fc = torch.where(r2f <= (ps // 2) ** 2, Fc, 0)
    q = min(ps // 2, N // 2)
    at = torch.arange(-q + (N == 2 * q), q + 1, device=DEV)
    xs = torch.arange(min(fx, h), device=DEV)
    G[(at % N)[:, None, None], (at % N)[None, :, None], xs] = Fc[(at % ps)[:, None, None], (at % ps)[None, :, None], xs]
    j = torch.arange(N, device=DEV)
    sg = (j[:, None, None] ^ j[None, :, None] ^ torch.arange(h, device=DEV)) & 1
    vol = torch.fft.irfftn(torch.where(sg == 1, -G, G), s=(N, N, N)) * float(N) ** 3
    o = N // 2 - box // 2
    vol = vol[o:o + box, o:o + box, o:o + box] / (oc * box)
    q = (torch.arange(box, device=DEV) - box // 2).to(F64)
    rr = torch.sqrt(q[:, None, None] ** 2 + q[None, :, None] ** 2 + q[None, None, :] ** 2)
    r0, wd = box / 2.0, 3.0
    rc = torch.where(rr < r0, 0.0, torch.where(rr > r0 + wd, 1.0, 0.5 + 0.5 * torch.cos(math.pi * (r0 + wd - rr) / wd)))
    vol = (1 - rc) * vol + rc * ((rc * vol).sum() / rc.sum())
    vol = vol / torch.sinc(rr / N) ** 2
    return dict(fsc=fsc, tau2=tau2, sigma2=sigma2, data_vs_prior=dvp, coverage=cov, map=vol,
                grid_data=torch.view_as_real(d.resolve_conj()).reshape(-1), grid_weight=w.reshape(-1))
