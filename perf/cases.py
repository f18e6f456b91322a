"""The measured cases: what a user of this package has it do, over the range of sizes in use.

Each case drives one public entry point:

  grid2d   engine.Grid2D.step, the per-step loop behind fdtd2d_core.run_beads: a 2D TE or TM
           grid in the middle of a solve, advanced `steps` steps with the detector boxes (and,
           with window=True, every DFT, flux plane and time average of the last periods)
  grid3d   engine.Grid3D.step + accum_e2, the loop behind fdtd3d_core.run_3d and Solve3D
  solve2d  solver2d.Solve2D: one whole planar solve from its setup arrays to phasor and snapshots
  sweep    batch2d.Sweep: uneven 2D solves advanced together, in each field storage
  beads    fdtd2d_core.run_beads: the whole drop-in call

Inputs are made from the seed: a layered waveguide stack (PMMA core, aqueous, mucin, cornea)
with a bead at a seeded place, graded absorbers, a Gaussian one-way source, and for the grids
waves of the medium's wavelength in every field.  exact() advances the same inputs in float64
with plain torch.
"""
import math

import numpy as np
import torch

F32 = np.float32
C0 = 299792458.0
EPS0 = 8.854187817e-12
MU0 = 4e-7 * math.pi
LAM = 850e-9
F0 = C0 / LAM
OMEGA = 2 * math.pi * F0
NPML = 12


def listed():
    return [
        # the size of a quick look (the tests' 2D grids): a few microns of waveguide, launch by launch
        dict(name="te2d_small", kind="grid2d", pol="s", nx=140, ny=96, steps=240, window=False),
        # the planar benchmark's grid, most of a run_beads call: boxes only, before the DFT windows
        dict(name="te2d_planar", kind="grid2d", pol="s", nx=1600, ny=480, steps=200, window=False),
        # absorbing TM grid of odd sizes inside the last periods, every epilogue on
        dict(name="tm2d_window", kind="grid2d", pol="p", nx=1201, ny=431, steps=100, window=True),
        # a long waveguide (the default run_beads domain is 1 mm): larger than the L2
        dict(name="tm2d_long", kind="grid2d", pol="p", nx=16000, ny=700, steps=20, window=False),
        # the tests' 3D grid
        dict(name="tm3d_small", kind="grid3d", pol="p", nx=64, ny=48, nz=40, steps=64, lossy=True, window=False),
        # the 3D benchmark's grid before its windows: detector boxes every step
        dict(name="tm3d_guide", kind="grid3d", pol="p", nx=480, ny=192, nz=256, steps=24, lossy=True, window=False),
        # lossless TE grid of odd sizes inside the DFT window: phasor volumes, flux planes, averages
        dict(name="te3d_window", kind="grid3d", pol="s", nx=301, ny=141, nz=203, steps=16, lossy=False, window=True),
        # one whole planar solve with snapshots
        dict(name="solve2d_planar", kind="solve2d", pol="s", nx=1600, ny=480, steps=1200),
        # a sweep of 16 uneven solves in each storage and on resident launches
        dict(name="sweep_f32", kind="sweep", count=16, nx=1500, ny=430, steps=1400, storage="f32", resident=False),
        dict(name="sweep_f16", kind="sweep", count=16, nx=1500, ny=430, steps=1400, storage="f16", resident=False),
        dict(name="sweep_resident", kind="sweep", count=16, nx=1500, ny=430, steps=1400, storage="f32", resident=True),
        # the drop-in call a user of the reference makes, no frames written
        dict(name="beads_whole", kind="beads", pol="s", length_um=30.0, dx_nm=40.0),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["grid2d", "grid2d", "grid3d", "grid3d", "solve2d", "sweep"])
    pol = rng.choice(["s", "p"])
    if kind == "grid2d":
        nx, ny = _log(rng, 100, 16000), _log(rng, 80, 700)
        steps = max(8, min(240, int(2.2e8 / (nx * ny))))
        return dict(kind=kind, pol=pol, nx=nx, ny=ny, steps=steps, window=rng.random() < 0.4)
    if kind == "grid3d":
        nx, ny, nz = _log(rng, 48, 480), _log(rng, 40, 192), _log(rng, 40, 256)
        return dict(kind=kind, pol=pol, nx=nx, ny=ny, nz=nz, steps=rng.randint(6, 24), lossy=rng.random() < 0.6,
                    window=rng.random() < 0.4)
    if kind == "solve2d":
        return dict(kind=kind, pol=pol, nx=_log(rng, 200, 1600), ny=rng.randint(96, 480), steps=rng.randint(300, 1200))
    return dict(kind=kind, count=rng.randint(2, 16), nx=_log(rng, 300, 1500), ny=rng.randint(150, 430),
                steps=rng.randint(900, 1400), storage=rng.choice(["f32", "f16", "bf16"]), resident=False)


# ---------------------------------------------------------------------------- inputs
def absorber(n, npml, dx, dt):
    """Graded absorber of one axis: kappa, b, c on the n nodes (e) and n-1 half nodes (h)."""
    eta0 = math.sqrt(MU0 / EPS0)
    smax = -4.0 * math.log(1e-6) / (2.0 * eta0 * npml * dx)
    amax = 2.0 * math.pi * EPS0 * F0 / 10.0
    out = {}
    for tag, pos in (("e", np.arange(n, dtype=np.float64)), ("h", np.arange(n - 1, dtype=np.float64) + 0.5)):
        depth = np.clip(np.maximum(npml - pos, pos - (n - 1 - npml)) / npml, 0.0, 1.0)
        sig, a = smax * depth ** 3, np.where(depth > 0, amax * (1.0 - depth), 0.0)
        b = np.exp(-(sig + a) * dt / EPS0)
        c = np.where(sig + a > 0, sig * (b - 1.0) / np.where(sig + a > 0, sig + a, 1.0), 0.0)
        out["k" + tag], out["b" + tag], out["c" + tag] = np.ones(len(pos), F32), b.astype(F32), c.astype(F32)
    return out


def layers(ny, dx, rng):
    """eps and sigma of the stack over y: air, core at 60 % of the height, absorbing aqueous, mucin, cornea;
    core index and layer thicknesses vary as in a tear-film sweep."""
    y = (np.arange(ny) - 0.6 * ny) * dx * 1e6
    core, aq, mu = rng.uniform(1.47, 1.51), rng.uniform(0.5, 3.0), rng.uniform(0.2, 1.0)
    n = np.where(y > 2.0, 1.0, np.where(y >= 0, core, np.where(y > -aq, 1.333, np.where(y > -aq - mu, 1.34, 1.376))))
    sig = np.where((y < 0) & (y > -aq), OMEGA * EPS0 * 2 * 1.333 * 0.001, 0.0)
    return n ** 2, sig


def line_source(ny, dx, dt):
    y = (np.arange(ny) - 0.6 * ny) * dx * 1e6 - 1.0
    kdx = 2.0 * math.asin(min(1.0, dx / (C0 * dt) * math.sin(math.pi * C0 * dt / LAM)))
    amp = np.exp(-(y / 3.0) ** 2) / (2.0 * math.sin(kdx))
    ph = -0.02 * y ** 2
    return amp, ph, ph + kdx


def setup_2d(pol, nx, ny, seed):
    """Setup arrays of a 2D solve in the shapes of geometry.build_2d (TM: absorbing)."""
    dx = 25e-9
    dt = 0.5 * dx / (C0 * math.sqrt(2))
    rng = np.random.default_rng(seed)
    e1, s1 = layers(ny, dx, rng)
    r, xc, yc = rng.uniform(6, 24), rng.uniform(0.3, 0.8) * nx, 0.6 * ny - rng.uniform(8, 24)
    i0, i1 = max(0, int(xc - r) - 3), min(nx, int(xc + r) + 4)     # the rows of the bead; the others repeat
    d = np.hypot(np.arange(i0, i1)[:, None] - xc, np.arange(ny)[None, :] - yc)
    f = np.clip(r - d + 0.5, 0.0, 1.0)
    stack, bead = (e1[None, :], s1[None, :]), (e1 * (1 - f) + 1.59 ** 2 * f, s1 * (1 - f))

    def rows(fn, n):
        """fn(eps, sig) of the plain stack on every row, of the bead on its own."""
        v = np.repeat(fn(*stack).astype(F32), n, 0)
        b = fn(*bead).astype(F32)
        v[i0:i0 + len(b)] = b
        return v
    g = dict(cx=absorber(nx, NPML, dx, dt), cy=absorber(ny, NPML, dx, dt))
    g["ce_e"], g["ce_h"] = np.ones((nx, ny), F32), rows(lambda e, s: dt / (EPS0 * e * dx), nx)
    a, p1, p2 = line_source(ny, dx, dt)
    if pol == "p":
        mean = dict(x=lambda v: (v[:-1] + v[1:]) / 2 if len(v) > 1 else v, y=lambda v: (v[:, :-1] + v[:, 1:]) / 2)
        for q, m in mean.items():
            loss = lambda e, s: m(s) * dt / (2 * EPS0 * m(e))
            g["ca_" + q] = rows(lambda e, s: dt / (EPS0 * m(e) * dx) / (1 + loss(e, s)), nx - (q == "x"))
            g["da_" + q] = rows(lambda e, s: (1 - loss(e, s)) / (1 + loss(e, s)), nx - (q == "x"))
        a, p1, p2 = ((v[:-1] + v[1:]) / 2 for v in (a, p1, p2))
    g["src"] = dict(ix=NPML + 2, amp=a.astype(F32), ph1=p1.astype(F32), ph2=p2.astype(F32), omega=OMEGA)
    return g, dx, dt


def setup_3d(c, seed):
    """Setup arrays of a 3D solve: E update factors, damping (or None), absorbers, source."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    dx = 30e-9
    dt = 0.5 * dx / (C0 * math.sqrt(3))
    rng = np.random.default_rng(seed)
    e1, s1 = layers(ny, dx, rng)
    r, xc, yc, zc = rng.uniform(6, 12), rng.uniform(0.3, 0.8) * nx, 0.6 * ny - 14, rng.uniform(0.4, 0.6) * nz
    off = dict(x=(0.5, 0, 0), y=(0, 0.5, 0), z=(0, 0, 0.5))
    ce, da = [], []
    for q in "xyz":
        shape = tuple(m - (o > 0) for m, o in zip((nx, ny, nz), off[q]))
        col, scol = ((e1[:-1] + e1[1:]) / 2, (s1[:-1] + s1[1:]) / 2) if q == "y" else (e1, s1)
        w = scol * dt / (2 * EPS0 * col) if c["lossy"] else np.zeros_like(col)
        v = np.empty(shape, F32)
        v[:] = (dt / (EPS0 * col * dx) / (1 + w)).astype(F32)[None, :, None]
        w3 = np.empty(shape, F32)
        w3[:] = ((1 - w) / (1 + w)).astype(F32)[None, :, None]
        lo = [max(0, int(p - r) - 2) for p in (xc, yc, zc)]
        sl = tuple(slice(a, min(m, a + int(2 * r) + 6)) for a, m in zip(lo, shape))
        ax = [np.arange(s.start, s.stop) + o - p for s, o, p in zip(sl, off[q], (xc, yc, zc))]
        d = np.sqrt(ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2)
        f = np.clip(r - d + 0.5, 0.0, 1.0)
        blend = col[None, sl[1], None] * (1 - f) + 1.59 ** 2 * f
        v[sl] = np.where(f > 0, dt / (EPS0 * blend * dx), v[sl])
        w3[sl] = np.where(f > 0, 1.0, w3[sl])
        ce.append(v)
        da.append(w3)
    cpml = [absorber(n, 10, dx, dt) for n in (nx, ny, nz)]
    ny1, nz1 = (ny - 1, nz) if c["pol"] == "p" else (ny, nz - 1)
    a, p1, p2 = line_source(ny1, dx, dt)
    z = (np.arange(nz1) - nz1 / 2) * dx * 1e6
    amp = a[:, None] * np.exp(-(z / 1.5) ** 2)[None, :]
    src = dict(ix=14, amp=amp.astype(F32), ph1=np.repeat(p1[:, None], nz1, 1).astype(F32),
               ph2=np.repeat(p2[:, None], nz1, 1).astype(F32), omega=OMEGA)
    return ce, da if c["lossy"] else None, cpml, src, dx, dt


def waves(shape, seed, scale, device):
    """A field of a solve in progress: plane waves of the medium's wavelength, zero on the outer cells."""
    rng = np.random.default_rng(seed)
    axes = [torch.arange(n, device=device, dtype=torch.float32) for n in shape]
    v = torch.zeros(shape, device=device)
    for _ in range(3):
        k = rng.standard_normal(len(shape))
        k *= 2 * math.pi / rng.uniform(18, 28) / np.linalg.norm(k)
        p = axes[0] * float(k[0])
        for q in range(1, len(shape)):
            p = p[..., None] + axes[q] * float(k[q])
        v += torch.cos(p + float(rng.uniform(0, 6.28)))
    v *= scale / 3
    for q in range(len(shape)):
        v.narrow(q, 0, 1).zero_()
        v.narrow(q, shape[q] - 1, 1).zero_()
    return v


def shapes_2d(pol, nx, ny):
    return (dict(ez=(nx, ny), hx=(nx, ny - 1), hy=(nx - 1, ny)) if pol == "s" else
            dict(ex=(nx - 1, ny), ey=(nx, ny - 1), hz=(nx - 1, ny - 1)))


def shapes_3d(nx, ny, nz):
    return dict(ex=(nx - 1, ny, nz), ey=(nx, ny - 1, nz), ez=(nx, ny, nz - 1),
                hx=(nx, ny - 1, nz - 1), hy=(nx - 1, ny, nz - 1), hz=(nx - 1, ny - 1, nz))


def fields_of(shapes, seed, device):
    return {q: waves(s, 1000 * seed + m, 1.0 if q[0] == "e" else 1 / 376.7, device)
            for m, (q, s) in enumerate(shapes.items())}


N0 = 900  # the first step of the grids: the source has ramped up


def envelope(t):
    return 1 - np.exp(-((np.asarray(t) * math.pi * F0 / 4.0) ** 2))


def boxes_2d(c):
    nx, ny = c["nx"], c["ny"]
    w, lo, hi = max(1, nx // 20), int(0.6 * ny), min(ny, int(0.6 * ny) + 80)
    return [(int(0.1 * nx) + 8, int(0.1 * nx) + 8 + 2 * w, lo, hi), (int(0.9 * nx) - w, int(0.9 * nx) + w, lo, hi)]


def planes_2d(c):
    return {"in": int(0.1 * c["nx"]) + 8, "out": int(0.9 * c["nx"]), "src_up": NPML + 1, "src_dn": NPML + 5}


def boxes_3d(c):
    nx, ny = c["nx"], c["ny"]
    lo, hi = int(0.6 * ny), min(ny, int(0.6 * ny) + 66)
    return [(nx // 5, nx // 5 + min(66, nx // 6), lo, hi, 12, -12), (4 * nx // 5 - 8, 4 * nx // 5 - 8 + min(66, nx // 6), lo, hi, 12, -12)]


def planes_3d(c):
    return {"in": c["nx"] // 5 + 4, "out": 4 * c["nx"] // 5, "src_up": 13, "src_dn": 17}


def sweep_sizes(c):
    """Uneven widths and heights of a sweep around its (nx, ny), polarisations in turn."""
    return [("sp"[q % 2], int(c["nx"] * (0.6 + 0.4 * ((q * 7) % c["count"]) / c["count"])),
             int(c["ny"] * (0.7 + 0.3 * ((q * 5) % c["count"]) / c["count"]))) for q in range(c["count"])]


class Setup:
    """The few numbers of a solve that Sweep and Solve2D read beside the setup arrays (geometry.Spec2D)."""

    def __new__(cls, pol, nx, ny, seed):
        from lens_sensor_b200.geometry import Bead2D, Spec2D, Stack
        st = Stack(1.49, 2.0, [(1.5, complex(1.333, 0.001)), (0.5, 1.34)], 1.376)
        return Spec2D(pol, nx, ny, 25e-9, st, 0.6 * ny * 25e-9, Bead2D(5.0 + seed % 7, 0.8, 1.59), npml=NPML)


# ---------------------------------------------------------------------------- the passes
def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "grid2d":
        from lens_sensor_b200 import engine as E
        geo, dx, dt = setup_2d(c["pol"], c["nx"], c["ny"], seed)
        coef = {q: geo[q] for q in (("ce_e", "ce_h") if c["pol"] == "s" else ("ca_x", "ca_y", "da_x", "da_y"))}
        g = E.Grid2D(c["pol"], c["nx"], c["ny"], dx, dt, coef, geo["cx"], geo["cy"], geo["src"])
        for q, v in fields_of(shapes_2d(c["pol"], c["nx"], c["ny"]), seed, "cuda").items():
            g.view(q).copy_(v)
        n, far = c["steps"], 1 << 28
        on = (N0, N0 + n) if c["window"] else (far, far + 1)
        ep = E.Epi2D(g, boxes=boxes_2d(c), dft=on, dft_ex=c["pol"] == "p", prev=(on[0], on[0] + n // 2),
                     iavg_n0=on[0], planes=planes_2d(c))
        return dict(c, g=g, ep=ep, tab=E.StepTable(N0, n, dt, OMEGA, OMEGA, envelope))
    if kind == "grid3d":
        from lens_sensor_b200 import engine as E
        ce, da, cpml, src, dx, dt = setup_3d(c, seed)
        comp = 1 if c["pol"] == "p" else 2
        g = E.Grid3D(c["nx"], c["ny"], c["nz"], dx, dt, ce, da, cpml, src, src_comp=comp)
        for q, v in fields_of(shapes_3d(c["nx"], c["ny"], c["nz"]), seed, "cuda").items():
            g.view(q).copy_(v)
        n, far = c["steps"], 1 << 28
        on = (N0, N0 + n) if c["window"] else (far, far + 1)
        ep = E.Epi3D(g, boxes=boxes_3d(c), dft=on, comps=(0, 1, 2), planes=planes_3d(c), conv=(c["nz"] // 2, (far, far)),
                     iavg=True)
        return dict(c, g=g, ep=ep, tab=E.StepTable(N0, n, dt, OMEGA, OMEGA, envelope))
    if kind == "solve2d":
        geo, dx, dt = setup_2d(c["pol"], c["nx"], c["ny"], seed)
        return dict(c, geo=geo, spec=Setup(c["pol"], c["nx"], c["ny"], seed))
    if kind == "sweep":
        from lens_sensor_b200 import batch2d as B
        sizes = sweep_sizes(c)
        sw = B.Sweep([Setup(p, nx, ny, seed) for p, nx, ny in sizes], c["steps"], c["storage"], resident=c["resident"],
                     geos=[setup_2d(p, nx, ny, seed + q)[0] for q, (p, nx, ny) in enumerate(sizes)])
        return dict(c, sw=sw)
    rng = np.random.default_rng(seed)
    return dict(c, kw=dict(wg_mat="pmma", bead_mat="polystyrol", bead_d_um=float(rng.uniform(0.5, 1.2)), dx_nm=c["dx_nm"],
                           save_frames=False, n_snapshots=4, wg_thickness_um=2.0, length_um=c["length_um"],
                           bead_x_um=float(rng.uniform(0.4, 0.6) * c["length_um"]), polarization=c["pol"],
                           tear_buffer_um=4.0, t_aqueous_um=float(rng.uniform(1.0, 2.0))))


def run(s):
    kind = s["kind"]
    if kind == "grid2d":
        g, ep = s["g"], s["ep"]
        g.step(s["tab"], N0, s["steps"], ep)
        out = {q: g.view(q) for q in shapes_2d(s["pol"], s["nx"], s["ny"])}
        out["box"] = ep.box_acc
        if s["window"]:
            out.update(dft=ep.phasor(), prev=ep.phasor("prev"), iavg=ep.iavg[:, :s["ny"]],
                       planes=[[a, b] for q in planes_2d(s) for _, a, b in ep.plane_dft(q)])
            if s["pol"] == "p":
                out["dft_ex"] = ep.phasor("dft_ex")
        return out
    if kind == "grid3d":
        g, ep, n = s["g"], s["ep"], s["steps"]
        if s["window"]:      # as run_3d does in the second half: |E|^2 every few steps
            for m in range(0, n, 4):
                g.step(s["tab"], N0 + m, min(4, n - m), ep)
                g.accum_e2(ep.iavg)
        else:
            g.step(s["tab"], N0, n, ep)
        out = {q: g.view(q) for q in g.FIELDS}
        out["box"] = ep.box_acc
        if s["window"]:
            out.update(dft=[ep.phasor(q) for q in range(3)], iavg=ep.iavg[:, :, :s["nz"]],
                       planes=[[a, b] for q in planes_3d(s) for _, a, b in ep.plane_dft(q)])
        return out
    if kind == "solve2d":
        from lens_sensor_b200.solver2d import Solve2D
        v = Solve2D(s["spec"], s["steps"], snap_every=200, geo=s["geo"]).run()
        v.check()
        return dict(phasor=v.phasor(), snaps=v.snaps)
    if kind == "sweep":
        s["sw"].reset()
        s["sw"].run()
        return [q["phasor"] for q in s["sw"].results()]
    from lens_sensor_b200 import fdtd2d_core as D
    r = D.run_beads(**s["kw"])
    return {q: r[q] for q in ("P_in", "P_out", "transmission", "Iavg", "Ecw", "steps_total", "p_in_si", "coupling_efficiency")}


def work(case):
    """Every field, coefficient and result once in and once out, and the updates of every step."""
    c, kind = case, case["kind"]
    if kind == "grid2d":
        n = c["nx"] * c["ny"]
        per = 24 + (8 if c["pol"] == "s" else 16) + ((32 if c["pol"] == "s" else 48) + 8 if c["window"] else 0)
        return {"bytes": per * n, "flops": (18 if c["pol"] == "s" else 20) * n * c["steps"]}
    if kind == "grid3d":
        n = c["nx"] * c["ny"] * c["nz"]
        return {"bytes": (48 + (24 if c["lossy"] else 12) + (56 if c["window"] else 0)) * n,
                "flops": (39 if c["lossy"] else 36) * n * c["steps"]}
    if kind == "solve2d":
        n = c["nx"] * c["ny"]
        return {"bytes": (16 + 16 + 4 * (c["steps"] // 200)) * n, "flops": 18 * n * c["steps"]}
    if kind == "sweep":
        n = sum(nx * ny for _, nx, ny in sweep_sizes(c))
        return {"bytes": (12 + 16) * n, "flops": 19 * n * c["steps"]}
    n = c["length_um"] / c["dx_nm"] * 1e3 * 11.0 / c["dx_nm"] * 1e3
    return {"bytes": 40 * n, "flops": 18 * n * 3.6e3 * c["length_um"] / 30.0}


# ---------------------------------------------------------------------------- float64
class Axis64:
    """One absorber axis in float64 along dimension `dim` of a field."""

    def __init__(self, prof, dim, nd, dev):
        self.p = {}
        for tag in "eh":
            b, cc, k = (np.asarray(prof[q + tag], F32) for q in "bck")
            vals = (np.where(cc != 0, b, 0).astype(F32), cc, (F32(1) / k).astype(F32))
            self.p[tag] = [torch.from_numpy(v.astype(np.float64)).to(dev).reshape([-1 if q == dim else 1 for q in range(nd)])
                           for v in vals]


class Psi:
    """Auxiliary fields of the absorbers, one per (name): psi = b psi + c d."""

    def __init__(self):
        self.v = {}

    def __call__(self, name, prof, sl, d):
        b, c, ik = (q[sl] if sl is not None else q for q in prof)
        old = self.v.get(name)
        new = c * d if old is None else b * old + c * d
        self.v[name] = new
        return new + d * ik


def table64(n0, n, dt):
    """The step table's entries: float32(w t) and the float32 envelope and DFT phases."""
    t = np.arange(n0, n0 + n) * dt
    e = lambda ph: np.stack([np.cos(ph), -np.sin(ph)], 1).astype(F32).astype(np.float64)
    return ((OMEGA * t).astype(F32).astype(np.float64), t, e(OMEGA * t), e(OMEGA * (t - 0.5 * dt)))


def cw_ramp(t, ramp=None):
    st = 4.0 / (2 * math.pi * F0) if ramp is None else ramp / (6.0 * F0)
    return (1 - np.exp(-((t / (2 * st)) ** 2))).astype(F32).astype(np.float64)


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class Grid64:
    """2D solve in float64."""

    def __init__(self, pol, nx, ny, geo, dx, dt):
        dev = self.dev = _dev()
        f64 = lambda a: torch.from_numpy(np.asarray(a, F32).astype(np.float64)).to(dev)
        self.pol, self.nx, self.ny = pol, nx, ny
        self.f = {q: torch.zeros(s, dtype=torch.float64, device=dev) for q, s in shapes_2d(pol, nx, ny).items()}
        self.c = {q: f64(geo[q]) for q in (("ce_e", "ce_h") if pol == "s" else ("ca_x", "ca_y", "da_x", "da_y"))}
        self.x, self.y = Axis64(geo["cx"], 0, 2, dev).p, Axis64(geo["cy"], 1, 2, dev).p
        self.ch = float(F32(dt / (MU0 * dx)))
        self.src = {q: f64(geo["src"][q]) for q in ("amp", "ph1", "ph2")}
        self.ix = int(geo["src"]["ix"])
        self.psi = Psi()

    def step(self, wt, env):
        f, c, ch, P, x, y = self.f, self.c, self.ch, self.psi, self.x, self.y
        mid, top = slice(1, -1), slice(1, -1)
        sx, sy = (mid, slice(None)), (slice(None), top)
        inject = [env * torch.sin(wt + self.src[q]) * self.src["amp"] for q in ("ph1", "ph2")]
        if self.pol == "s":
            ez, hx, hy = f["ez"], f["hx"], f["hy"]
            hx -= ch * P("hxy", y["h"], None, ez[:, 1:] - ez[:, :-1])
            hy += ch * P("hyx", x["h"], None, ez[1:] - ez[:-1])
            dhy, dhx = (hy[1:] - hy[:-1])[:, 1:-1], (hx[:, 1:] - hx[:, :-1])[1:-1]
            ez[1:-1, 1:-1] = (c["ce_e"][1:-1, 1:-1] * ez[1:-1, 1:-1] + c["ce_h"][1:-1, 1:-1] *
                              (P("ezx", x["e"], sx, dhy) - P("ezy", y["e"], sy, dhx)))
            ez[self.ix] += inject[0]
            ez[self.ix + 1] -= inject[1]
            for q in (ez[0], ez[-1], ez[:, 0], ez[:, -1]):
                q.zero_()
            return
        ex, ey, hz = f["ex"], f["ey"], f["hz"]
        hz -= ch * (P("hzx", x["h"], None, ey[1:] - ey[:-1]) - P("hzy", y["h"], None, ex[:, 1:] - ex[:, :-1]))
        ex *= c["da_x"]
        ey *= c["da_y"]
        ex[:, 1:-1] += c["ca_x"][:, 1:-1] * P("exy", y["e"], sy, hz[:, 1:] - hz[:, :-1])
        ey[1:-1] -= c["ca_y"][1:-1] * P("eyx", x["e"], sx, hz[1:] - hz[:-1])
        ey[self.ix] += inject[0]
        ey[self.ix + 1] -= inject[1]
        for q in (ex[:, 0], ex[:, -1], ey[0], ey[-1]):
            q.zero_()

    def nodes(self):
        """(driven field, its intensity, the cross field) on the nodes."""
        if self.pol == "s":
            return self.f["ez"], self.f["ez"] ** 2, None
        ex, ey = self.f["ex"], self.f["ey"]
        f = torch.cat([ey[:, :1], 0.5 * (ey[:, 1:] + ey[:, :-1]), ey[:, -1:]], 1)
        x1 = torch.cat([ex[:1], 0.5 * (ex[1:] + ex[:-1]), ex[-1:]], 0)
        x2 = torch.cat([ex[:1] ** 2, 0.5 * (ex[1:] ** 2 + ex[:-1] ** 2), ex[-1:] ** 2], 0)
        return f, f * f + x2, x1


def _phase(p):
    return complex(float(p[0]), float(p[1]))


def exact_grid2d(c, seed):
    geo, dx, dt = setup_2d(c["pol"], c["nx"], c["ny"], seed)
    g = Grid64(c["pol"], c["nx"], c["ny"], geo, dx, dt)
    for q, v in fields_of(shapes_2d(c["pol"], c["nx"], c["ny"]), seed, g.dev).items():
        g.f[q].copy_(v)
    n = c["steps"]
    wt, t, pe, ph = table64(N0, n, dt)
    env = envelope(t).astype(F32)
    box, dft, prev, dft_ex, iavg = [0.0, 0.0], 0.0, 0.0, 0.0, 0.0
    planes = [[0.0, 0.0] for _ in planes_2d(c)]
    for k in range(n):
        g.step(float(wt[k]), float(env[k]))
        F, I, X = g.nodes()
        for q, (a, b, lo, hi) in enumerate(boxes_2d(c)):
            box[q] = box[q] + I[a:b, lo:hi].sum()
        if not c["window"]:
            continue
        w, v = _phase(pe[k]), _phase(ph[k])
        dft = dft + F * w
        if k < n // 2:
            prev = prev + F * w
        if X is not None:
            dft_ex = dft_ex + X * w
        iavg = iavg + I
        for q, i in enumerate(planes_2d(c).values()):
            e, h = (g.f["ez"], g.f["hy"]) if c["pol"] == "s" else (g.f["ey"], g.f["hz"])
            planes[q][0] = planes[q][0] + e[i][:h.shape[1]] * w if c["pol"] == "p" else planes[q][0] + e[i] * w
            planes[q][1] = planes[q][1] + 0.5 * (h[i - 1] + h[i]) * v
    out = dict(g.f, box=torch.stack(box))
    if c["window"]:
        if c["pol"] == "p":   # the planes hold the Ey grid: its last column has no Hz beside it
            planes = [[a, b] for a, b in planes]
            out["dft_ex"] = dft_ex
        out.update(dft=dft, prev=prev, iavg=iavg, planes=planes)
    return out


def exact_grid3d(c, seed):
    nx, ny, nz, dev = c["nx"], c["ny"], c["nz"], _dev()
    ce, da, cpml, src, dx, dt = setup_3d(c, seed)
    f64 = lambda a: torch.from_numpy(np.asarray(a, F32)).to(dev).double()
    f = {q: v.double() for q, v in fields_of(shapes_3d(nx, ny, nz), seed, dev).items()}
    ce = [f64(v) for v in ce]
    da = [f64(v) for v in da] if da is not None else None
    A = [Axis64(p, q, 3, dev).p for q, p in enumerate(cpml)]
    s = {q: f64(src[q]) for q in ("amp", "ph1", "ph2")}
    ch, P, n = float(F32(dt / (MU0 * dx))), Psi(), c["steps"]
    wt, t, pe, ph = table64(N0, n, dt)
    env = envelope(t).astype(F32)
    ins = [tuple(slice(1, -1) if q == d else slice(None) for q in range(3)) for d in range(3)]
    drv = "ey" if c["pol"] == "p" else "ez"
    box, iavg = [0.0, 0.0], 0.0
    dft = [0.0, 0.0, 0.0]
    planes = [[0.0, 0.0] for _ in range(8)]
    diff = lambda v, d: v.narrow(d, 1, v.shape[d] - 1) - v.narrow(d, 0, v.shape[d] - 1)
    inner = lambda v, *dims: v[tuple(slice(1, -1) if q in dims else slice(None) for q in range(3))]

    def onto(F, shape, d):
        """F^2 moved along dimension d onto the driven component's grid."""
        m = F.shape[d]
        if m == shape[d]:
            return F
        if m == shape[d] + 1:
            return 0.5 * (F.narrow(d, 0, m - 1) + F.narrow(d, 1, m - 1))
        return torch.cat([F.narrow(d, 0, 1), 0.5 * (F.narrow(d, 0, m - 1) + F.narrow(d, 1, m - 1)), F.narrow(d, m - 1, 1)], d)
    for k in range(n):
        for q, (a, da1, b, db) in dict(hx=("ey", 2, "ez", 1), hy=("ez", 0, "ex", 2), hz=("ex", 1, "ey", 0)).items():
            f[q] += ch * (P(q + "a", A[da1]["h"], None, diff(f[a], da1)) - P(q + "b", A[db]["h"], None, diff(f[b], db)))
        for m, (q, a, da1, b, db) in enumerate((("ex", "hz", 1, "hy", 2), ("ey", "hx", 2, "hz", 0), ("ez", "hy", 0, "hx", 1))):
            if da is not None:
                f[q] *= da[m]
            d1, d2 = inner(diff(f[a], da1), db), inner(diff(f[b], db), da1)
            curl = P(q + "a", A[da1]["e"], ins[da1], d1) - P(q + "b", A[db]["e"], ins[db], d2)
            inner(f[q], da1, db).add_(inner(ce[m], da1, db) * curl)
            for d in (da1, db):
                f[q].narrow(d, 0, 1).zero_()
                f[q].narrow(d, f[q].shape[d] - 1, 1).zero_()
        for q, i, sg in (("ph1", src["ix"], 1.0), ("ph2", src["ix"] + 1, -1.0)):
            f[drv][i] += sg * float(env[k]) * torch.sin(float(wt[k]) + s[q]) * s["amp"]
        for q, (a, b, lo, hi, z0, z1) in enumerate(boxes_3d(c)):
            box[q] = box[q] + sum((f[e][a:b, lo:hi, z0:z1] ** 2).sum() for e in ("ex", "ey", "ez"))
        if not c["window"]:
            continue
        w, v = _phase(pe[k]), _phase(ph[k])
        for m, q in enumerate(("ex", "ey", "ez")):
            dft[m] = dft[m] + f[q] * w
        for q, i in enumerate(planes_3d(c).values()):
            for pair, (e, h) in enumerate((("ey", "hz"), ("ez", "hy"))):
                hm = 0.5 * (f[h][i - 1] + f[h][i])
                a = planes[2 * q + pair]
                a[0] = a[0] + f[e][i] * w
                a[1] = a[1] + hm * v
        if (k % 4 == 3) or k == n - 1:
            shape = f[drv].shape
            tot = 0.0
            for q in ("ex", "ey", "ez"):
                F = f[q] ** 2
                for d in range(3):
                    F = onto(F, shape, d)
                tot = tot + F
            iavg = iavg + tot
    out = dict(f, box=torch.stack(box))
    if c["window"]:
        full = torch.zeros((nx, ny, nz), dtype=torch.float64, device=dev)
        full[:iavg.shape[0], :iavg.shape[1], :iavg.shape[2]] = iavg
        out.update(dft=dft, iavg=full, planes=planes)
    return out


def solve64(pol, nx, ny, seed, steps, window, every=0):
    geo, dx, dt = setup_2d(pol, nx, ny, seed)
    g = Grid64(pol, nx, ny, geo, dx, dt)
    wt, t, pe, _ = table64(0, steps, dt)
    env = cw_ramp(t)
    dft, snaps = 0.0, []
    for k in range(steps):
        g.step(float(wt[k]), float(env[k]))
        if k >= steps - window:
            dft = dft + g.nodes()[0] * _phase(pe[k])
        if every and (k + 1) % every == 0:
            snaps.append(g.f["ez" if pol == "s" else "ey"].clone())
    return (2.0 / window) * dft, torch.stack(snaps) if snaps else None


def exact(case, seed):
    c = dict(case)
    period = max(4, int(round((1.0 / F0) / (0.5 * 25e-9 / (C0 * math.sqrt(2))))))
    if c["kind"] == "grid2d":
        return exact_grid2d(c, seed)
    if c["kind"] == "grid3d":
        return exact_grid3d(c, seed)
    if c["kind"] == "solve2d":
        p, s = solve64(c["pol"], c["nx"], c["ny"], seed, c["steps"], min(c["steps"], period), 200)
        return dict(phasor=p, snaps=s)
    if c["kind"] == "sweep":
        return [solve64(p, nx, ny, seed + q, c["steps"], min(c["steps"], 8 * period))[0]
                for q, (p, nx, ny) in enumerate(sweep_sizes(c))]
    return None   # the whole drop-in call builds its own geometry
