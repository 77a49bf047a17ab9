"""The work that programs on this package spend their time in, as timed cases.

Every case goes through the public entry points (``mapp_b200.System`` and
``mapp_b200.Batch``) the way a caller of MAPP's boundary uses them: a minimiser
or MD driver that hands over positions and asks for forces, a clock that asks
for rates, a relaxation, an MD or a clock run that stays on the device, the
training of the learned form.  Positions, concentrations and results live in
torch buffers on the GPU, except where the comment of a case says otherwise.
``exact`` computes the same results in FP64 with plain torch.
"""
from __future__ import annotations

import math
import os
import random
import tempfile

import numpy as np
import torch

import mapp_b200 as mb
from mapp_b200 import fixtures as fx

A_DMD, A_MD = 3.58, 3.615     # lattice constants of the DMD and MD workloads
SKIN = 0.5
R_CRD, A_LO, A_HI, TEMP = 3.0, 20.0, 1000.0, 600.0


def listed():
    return [
        # the smallest calls: a host program's minimiser on a small DMD cell, one
        # accepted line-search step (new x, energy_calc, force_calc) through
        # page-locked host arrays, as the C++ callers of the boundary hold them
        dict(name="linesearch_500", kind="linesearch", style="DMD_I", nx=5, ny=5, nz=5, nt=2, nq=3, sigma=0.03),
        # one MD step of a driver that integrates outside the library: binary EAM, small
        dict(name="eam_force_864", kind="eam", nx=6, ny=6, nz=6, nt=2, sigma=0.05),
        # the same for a large one-species crystal
        dict(name="eam_force_256k", kind="eam", nx=40, ny=40, nz=40, nt=1, sigma=0.05),
        # the Nose-Hoover run of the 4000-atom crystal, on the device
        dict(name="md_nvt_4000", kind="md", nx=10, ny=10, nz=10, nt=1, sigma=0.05, steps=200),
        # the plain FP64 DMD evaluation (new x and c, forces and virial) of the binary system
        dict(name="dmd_force_32k", kind="dmd", style="DMD_I", form="fp64", nx=20, ny=20, nz=20, nt=2, nq=3, sigma=0.02),
        # a list rebuild followed by the forces: three species, a ragged slab, four nodes
        dict(name="relist_10k_3sp", kind="relist", style="DMD", nx=17, ny=14, nz=11, nt=3, nq=4, sigma=0.04),
        # the precision form on the large binary system
        dict(name="dmd_fp32_256k", kind="dmd", style="DMD_I", form="fp32", nx=40, ny=40, nz=40, nt=2, nq=3, sigma=0.02),
        # the learned form (network on the tensor cores, quadrature outside its box)
        dict(name="dmd_learned_32k", kind="dmd", style="DMD_I", form="mlp", nx=20, ny=20, nz=20, nt=2, nq=3, sigma=0.02),
        # a concentration clock's evaluation from outside: c_d_calc and calc_g with its gradient
        dict(name="rates_32k", kind="rates", style="DMD_II", form="fp64", nx=20, ny=20, nz=20, nt=2, nq=3, sigma=0.02),
        # the BDF clock, on the device
        dict(name="clock_bdf_13k", kind="clock", style="DMD_II", nx=15, ny=15, nz=15, nt=2, nq=3, sigma=0.0, steps=10),
        # the batched form: independent cells of uneven size relaxed together
        dict(name="batch_relax_32", kind="batch", form="fp64", ncells=32, lo=500, hi=4000, nt=2, iters=10),
        # the learned form's training: labels, forward, backward and Adam steps
        dict(name="mlp_train_400", kind="train", samples=200_000, steps=400, batch=4096, nt=2, nq=3),
    ]


def _cells(rng, lo, hi):
    """nx, ny, nz of an FCC box of about lo..hi sites (log-uniform), cubic or ragged, every edge at least 4 cells."""
    target = math.exp(rng.uniform(math.log(lo), math.log(hi))) / 4.0
    e = target ** (1.0 / 3.0)
    sx, sy = (1.0, 1.0) if rng.random() < 0.4 else (math.exp(rng.uniform(-0.35, 0.35)), math.exp(rng.uniform(-0.35, 0.35)))
    n = [max(4, round(e * sx)), max(4, round(e * sy)), max(4, round(e / (sx * sy)))]
    while 4 * n[0] * n[1] * n[2] > hi:
        n[n.index(max(n))] -= 1
    return n


def draw(rng):
    kind = rng.choice(["linesearch", "eam", "eam", "md", "dmd", "dmd", "dmd", "relist", "rates", "clock", "batch", "train"])
    case = dict(kind=kind)
    top = dict(linesearch=32000, eam=256000, md=16000, dmd=256000, relist=60000, rates=120000, clock=13500).get(kind)
    if top:
        case["nx"], case["ny"], case["nz"] = _cells(rng, 256, top)
        case["sigma"] = round(rng.uniform(0.0, 0.05), 3)
    if kind == "eam":
        case["nt"] = rng.choice([1, 2])
    elif kind == "md":
        case.update(nt=1, sigma=round(rng.uniform(0.02, 0.05), 3), steps=rng.choice([50, 100, 150]))
    elif kind == "dmd":
        form = rng.choice(["fp64", "fp64", "fp32", "mlp"])
        case.update(style=rng.choice(["DMD_I", "DMD_II", "DMD"]), form=form, nt=rng.choice([1, 2, 2, 3] if form != "mlp" else [1, 2]),
                    nq=rng.choice([3, 3, 3, 2, 4, 5]))
        if case["nt"] == 3 or case["nq"] > 3 or form == "mlp":
            while 4 * case["nx"] * case["ny"] * case["nz"] > 64000:
                case[max(("nx", "ny", "nz"), key=lambda k: case[k])] -= 1
    elif kind in ("linesearch", "relist"):
        case.update(style=rng.choice(["DMD_I", "DMD_II", "DMD"]), nt=rng.choice([1, 2, 3]), nq=rng.choice([3, 3, 4]))
    elif kind == "rates":
        case.update(style=rng.choice(["DMD_I", "DMD_II", "DMD"]), form=rng.choice(["fp64", "fp64", "fp32"]), nt=rng.choice([2, 2, 3]), nq=3)
    elif kind == "clock":
        case.update(style="DMD_II", nt=2, nq=3, sigma=0.0, steps=rng.choice([5, 8, 10]))
    elif kind == "batch":
        case.update(form=rng.choice(["fp64", "fp64", "fp32"]), ncells=rng.choice([6, 12, 20, 28]), lo=500, hi=rng.choice([2000, 4000]), nt=2, iters=rng.choice([6, 8, 10]))
    elif kind == "train":
        case.update(samples=rng.choice([50_000, 120_000]), steps=rng.choice([100, 250]), batch=rng.choice([1024, 2048, 4096]), nt=rng.choice([1, 2]), nq=3)
    return case


# ---- inputs -----------------------------------------------------------------

_DIR = []


def _potential(kind, nt):
    """The potential file of a workload, written once per process."""
    if not _DIR:
        _DIR.append(tempfile.mkdtemp(prefix="mapp_cases_"))
    path = os.path.join(_DIR[0], f"{kind}_{nt}")
    if not os.path.exists(path):
        t = fx.make_tables(fx.ALL_SPECIES[:nt])
        (fx.write_setfl if kind == "setfl" else fx.write_fs)(path, t)
    return path


def _box(case, a):
    return np.array([case["nx"], case["ny"], case["nz"]], dtype=np.float64) * a


def _sites(case, a, seed):
    """Displaced FCC sites as fractions of the box, in [0, 1)."""
    rng = np.random.default_rng([seed, 11])
    x = fx.fcc_box(case["nx"], case["ny"], case["nz"], a)
    x = x + 0.1 * a + rng.uniform(-0.5, 0.5, x.shape) * case["sigma"]
    s = x / _box(case, a)
    return s - np.floor(s)


def _dmd_vectors(n, nt, seed):
    """alpha = 1/w^2 with w ~ U(0.08, 0.15) A per site and species; c_A ~ Beta(2, 2), the rest shared."""
    rng = np.random.default_rng([seed, 12])
    w = rng.uniform(0.08, 0.15, size=(n, nt))
    c = np.ones((n, 1))
    if nt > 1:
        ca = rng.beta(2.0, 2.0, size=n)
        c = np.concatenate([ca[:, None], np.repeat(((1.0 - ca) / (nt - 1))[:, None], nt - 1, axis=1)], axis=1)
    return 1.0 / (w * w), np.ascontiguousarray(c)


def _step(n, seed, size=0.02):
    """One move of every site, well inside the skin."""
    return np.random.default_rng([seed, 13]).normal(0.0, size, size=(n, 3)).clip(-3 * size, 3 * size)


def _system(style, nt, H, stream, **atoms):
    s = mb.System(style)
    s.set_stream(stream.cuda_stream)
    sp = fx.ALL_SPECIES[:nt]
    s.set_types([k.name for k in sp], [k.mass for k in sp])
    s.set_box(np.diag(H))
    s.set_skin(SKIN)
    s.set_atoms(**atoms)
    if style == "EAM":
        s.coef(["ff_coef", "SetFL", _potential("setfl", 1)] if nt == 1 else ["ff_coef", "FS", _potential("fs", nt)])
    return s


def _inputs(case, seed):
    """Host arrays of a case's configuration: box edges, fractional sites of the
    list build, Cartesian sites of the evaluation, and alpha, c or the types."""
    dmd = case["kind"] not in ("eam", "md")
    a = A_DMD if dmd else A_MD
    H, s = _box(case, a), _sites(case, a, seed)
    n = len(s)
    d = dict(H=H, s=s, n=n)
    if dmd:
        d["alpha"], d["c"] = _dmd_vectors(n, case["nt"], seed)
    elif case["nt"] == 1:
        d["type"] = np.zeros(n, dtype=np.int32)
    else:
        d["type"] = np.random.default_rng([seed, 14]).integers(0, case["nt"], size=n).astype(np.int32)
    moves = case["kind"] in ("linesearch", "eam", "dmd")
    d["x"] = s * H + (_step(n, seed) if moves else 0.0)
    return d


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _time_step(cd):
    """A clock's resolved time step: a thousandth of the scale 1 / rms(c_d) on which the concentrations move."""
    return 1e-3 / math.sqrt(float((cd * cd).mean()))


def _batch_shapes(case):
    """nx, ny, nz of a batch's cells: log-uniform site counts, cubic and ragged ones mixed; the same for every seed."""
    rng = random.Random(case["ncells"] * 1009 + case["hi"])
    return [_cells(rng, case["lo"], case["hi"]) for _ in range(case["ncells"])]


def prepare(case, seed):
    kind, st = case["kind"], torch.cuda.Stream()
    p = dict(kind=kind, case=case, stream=st)
    if kind == "batch":
        rng = np.random.default_rng([seed, 15])
        b = mb.System("DMD_I")
        sp = fx.ALL_SPECIES[:case["nt"]]
        b.set_types([k.name for k in sp], [k.mass for k in sp])
        b.set_skin(SKIN)
        b.coef(fx.dmd_coef_args(_potential("fs", case["nt"]), R_CRD, 3, A_LO, A_HI, TEMP))
        B = mb.Batch(b)
        for shape in _batch_shapes(case):
            B.add_cell(fx.make_dmd_cell(*shape, a=A_DMD, sigma=0.03, seed=int(rng.integers(1 << 31)), nt=case["nt"],
                                        mean_cA=float(rng.uniform(0.1, 0.9))))
        B.set_params(5, case["iters"], 1e-5, 1e-8, 60)
        if case["form"] == "fp32":
            B.set_form(mb.MG_FORM_FP32)
        p.update(builder=b, batch=B)
        return p
    if kind == "train":
        s = mb.System("DMD_I")
        s.set_stream(st.cuda_stream)
        sp = fx.ALL_SPECIES[:case["nt"]]
        s.set_types([k.name for k in sp], [k.mass for k in sp])
        s.set_box(np.diag([4 * A_DMD] * 3))
        s.set_skin(SKIN)
        al, c = _dmd_vectors(256, case["nt"], seed)
        s.set_atoms(np.concatenate([fx.fcc_box(4, 4, 4, 0.25), al], axis=1), c=c)
        s.coef(fx.dmd_coef_args(_potential("fs", case["nt"]), R_CRD, case["nq"], A_LO, A_HI, TEMP))
        s.init()
        p.update(system=s, seed=seed)
        return p
    d = _inputs(case, seed)
    n, nt = d["n"], case["nt"]
    if kind in ("eam", "md"):
        s = _system("EAM", nt, d["H"], st, x_frac=d["s"], type=d["type"])
        s.init()
        p.update(system=s, x=_dev(d["x"]), f=torch.empty((n, 3), dtype=torch.float64, device="cuda"))
        if kind == "md":
            p["v"] = np.random.default_rng([seed, 16]).normal(0.0, 1.0, size=(n, 3))
        return p
    s = _system(case["style"], nt, d["H"], st, x_frac=np.concatenate([d["s"], d["alpha"]], axis=1), c=d["c"])
    s.coef(fx.dmd_coef_args(_potential("fs", nt), R_CRD, case["nq"], A_LO, A_HI, TEMP))
    s.init()
    x = np.concatenate([d["x"], d["alpha"]], axis=1)
    p["system"] = s
    if kind == "linesearch":
        p["x"] = torch.from_numpy(x).pin_memory().numpy()
        p["f"] = torch.empty((n, 3 + nt), dtype=torch.float64).pin_memory().numpy()
        return p
    p.update(x=_dev(x), c=_dev(d["c"]), f=torch.empty((n, 3 + nt), dtype=torch.float64, device="cuda"))
    form = case.get("form", "fp64")
    if form == "mlp":
        s.mlp_init(seed=1)
        s.mlp_train(nsamples=100_000, steps=1500, batch=4096, seed=7)
    s.set_form({"fp64": mb.MG_FORM_FP64, "fp32": mb.MG_FORM_FP32, "mlp": mb.MG_FORM_MLP}[form])
    if kind == "rates":
        s.force_calc(1, f=p["f"])
        s.create_2nd_neigh_lst()
        rng = np.random.default_rng([seed, 17])
        p.update(a=_dev(-d["c"] + 1e-3 * rng.normal(size=d["c"].shape)), cd=torch.empty_like(p["c"]), g=torch.empty_like(p["c"]))
        p["alpha"] = _time_step(s.c_d_calc())
    if kind == "clock":
        s.force_calc(1, f=p["f"])
        s.create_2nd_neigh_lst()
        p["dt"] = _time_step(s.c_d_calc())
    return p


# ---- one pass -----------------------------------------------------------------

def run(p):
    kind, case = p["kind"], p["case"]
    if kind == "batch":
        B = p["batch"]
        B.relax()
        res = [B.cell_result(k) for k in range(case["ncells"])]
        x = np.concatenate([r[0] for r in res])
        f = np.concatenate([r[1] for r in res])
        if case["form"] == "fp32":  # the precision form's results carry FP32 precision
            x, f = x.astype(np.float32), f.astype(np.float32)
        return dict(x=x, f=f, iterations=np.array([r[2]["iterations"] for r in res]),
                    evaluations=np.array([r[2]["evaluations"] for r in res]))
    s = p["system"]
    if kind == "train":
        s.mlp_init(seed=1 + p["seed"])
        s.mlp_train(nsamples=case["samples"], steps=case["steps"], batch=case["batch"], seed=7 + p["seed"])
        par, scal = s.mlp_state()
        return dict(par=par, scaling=scal, loss=s.mlp_loss_history(case["steps"]))
    if kind == "md":
        s.update_x(p["x"])
        r = s.md_nh(t_tar=300.0, t_period=10.0, steps=case["steps"], dt=0.0982269, boltz=8.617333e-5, xd=p["v"])
        return dict(x=r["x"], v=r["xd"], energy=r["energy"], virial=r["virial"], ke=r["ke"], rebuilds=r["rebuilds"])
    if kind == "eam":
        s.update_x(p["x"], report=False)
        f, en = s.force_calc(1, f=p["f"])
        return dict(f=f, en=en)
    if kind == "linesearch":
        s.update_x(p["x"], report=False)
        e = s.energy_calc()
        f, en = s.force_calc(1, f=p["f"])
        return dict(f=f, en=en, e=e)
    if kind == "relist":
        s.update_x(p["x"], report=False)
        s.rebuild_list()
        f, en = s.force_calc(1, f=p["f"])
        return dict(f=f, en=en)
    if kind == "dmd":
        s.update_x(p["x"], report=False)
        s.update_c(p["c"])
        f, en = s.force_calc(1, f=p["f"])
        if case["form"] == "fp64":
            return dict(f=f, en=en)
        with torch.cuda.stream(p["stream"]):
            return dict(f=f.float(), en=en)  # forces of FP32 (or network) precision, kept as such
    s.update_c(p["c"])
    if kind == "rates":
        cd = s.c_d_calc(out=p["cd"])
        cost, g = s.calc_g(p["a"], p["alpha"], 0, g=p["g"])
        if case["form"] == "fp32":
            with torch.cuda.stream(p["stream"]):
                return dict(cd=cd.float(), g=g.float())
        return dict(cd=cd, g=g, cost=cost)
    r = s.clock_bdf(case["steps"], max_order=2, initial_del_t=p["dt"])
    return dict(c=r["c"], del_t=r["del_t"], t=r["t"], order=r["order"], n_calc_g=r["n_calc_g"])


# ---- what a pass cannot do without ----------------------------------------------

def _pairs(case, a, cut):
    """Half pairs within `cut` of an FCC crystal of the case's size."""
    n = 4 * case["nx"] * case["ny"] * case["nz"]
    return 0.5 * n * (4.0 / a**3) * (4.0 / 3.0) * math.pi * cut**3


def work(case):
    kind = case["kind"]
    if kind == "train":
        rows = case["steps"] * case["batch"]
        # rows read once (4 inputs, 6 labels of 4 bytes), three GEMM passes of 8 832 multiply-adds
        return dict(bytes=rows * 40.0 + case["samples"] * 40.0, flops=rows * 3 * 2 * 8832.0)
    if kind == "batch":
        n = sum(4 * x * y * z for x, y, z in _batch_shapes(case))
        per = n * 0.5 * (4.0 / A_DMD**3) * (4.0 / 3.0) * math.pi * 5.27**3 * (4 * (10 + 66) + 100)
        return dict(bytes=2.0 * n * 5 * 8 * case["iters"], flops=per * case["iters"])
    n, nt = 4 * case["nx"] * case["ny"] * case["nz"], case["nt"]
    if kind in ("eam", "md"):
        p = _pairs(case, A_MD, 5.0)
        k = case.get("steps", 1)
        return dict(bytes=n * 48.0 * k, flops=p * 70.0 * k)
    p = _pairs(case, A_DMD, 5.27)
    smear = p * (nt * nt * (10 + 22 * case["nq"]) + nt * nt * 25)
    io = n * (2 * (3 + nt) + nt) * 8.0
    if kind == "linesearch":
        return dict(bytes=2 * io, flops=1.6 * smear)
    if kind in ("rates", "clock"):
        # c_d_calc and calc_g: four list passes of a dozen operations per species pair
        k = 1 if kind == "rates" else 7 * case["steps"]
        return dict(bytes=n * nt * 8.0 * 4 * k, flops=p * nt * nt * 60.0 * k)
    return dict(bytes=io, flops=smear)


# ---- the same in FP64 with plain torch -------------------------------------------

_F0 = (1.8, 2.0, 1.9, 1.85)                     # F = -f0 sqrt(rho)
_PHI0 = (0.35, 0.40, 0.38, 0.36)
_RE = (2.556, 2.49, 2.52, 2.54)
_BPHI = (8.0, 8.4, 8.2, 8.1)
_BRHO = (4.0, 4.2, 4.1, 4.05)
_MASS = (63.546, 58.693, 55.845, 58.933)
_RC, _NR, _RHO_MAX = 5.0, 10000, 40.0
_DR, _DRHO = _RC / (_NR - 1), _RHO_MAX / (_NR - 1)


def _spline(y):
    """c0..c3 of every knot: cubic Hermite pieces with finite-difference slopes."""
    s = torch.empty_like(y)
    s[0], s[1] = y[1] - y[0], 0.5 * (y[2] - y[0])
    s[-2], s[-1] = 0.5 * (y[-1] - y[-3]), y[-1] - y[-2]
    s[2:-2] = ((y[:-4] - y[4:]) + 8.0 * (y[3:-1] - y[1:-3])) / 12.0
    c2, c3 = torch.zeros_like(y), torch.zeros_like(y)
    c2[:-1] = 3.0 * (y[1:] - y[:-1]) - 2.0 * s[:-1] - s[1:]
    c3[:-1] = s[:-1] + s[1:] - 2.0 * (y[1:] - y[:-1])
    return torch.stack([y, s, c2, c3], dim=1)


def _tables(nt):
    """rho and r*phi splines of every unordered species pair, F splines (with the quartic term) per species."""
    r = torch.from_numpy(np.arange(_NR, dtype=np.float64) * _DR).cuda()
    t = ((r - 4.5) / 0.5).clamp(0.0, 1.0)
    tap = 1.0 - (10.0 * t**3 - 15.0 * t**4 + 6.0 * t**5)
    rho, phi, emb = {}, {}, []
    for i in range(nt):
        for j in range(i + 1):
            p0 = math.sqrt(_PHI0[i] * _PHI0[j]) if i != j else _PHI0[i]
            re, bp, br = (0.5 * (v[i] + v[j]) for v in (_RE, _BPHI, _BRHO))
            rho[i, j] = rho[j, i] = _spline(torch.exp(-br * (r / re - 1.0)) * tap)
            phi[i, j] = phi[j, i] = _spline(r * (p0 * torch.exp(-bp * (r / re - 1.0)) * tap))
        k = torch.from_numpy(np.arange(_NR, dtype=np.float64) * _DRHO).cuda()
        c = _spline(-_F0[i] * torch.sqrt(k))
        c4 = torch.zeros(_NR, dtype=torch.float64, device="cuda")
        c4[:-1] = (c[1:, 2] - c[:-1, 2]) / 6.0 - 0.5 * c[:-1, 3]
        emb.append(torch.cat([c, c4[:, None]], dim=1))
    return rho, phi, emb


def _knot(x, h):
    p = x / h
    m = p.long().clamp(0, _NR - 2)
    return m, (p - m).clamp(max=1.0)


def _val(tab, m, p):
    c = tab[m]
    return ((c[:, 3] * p + c[:, 2]) * p + c[:, 1]) * p + c[:, 0]


def _der(tab, m, p):
    c = tab[m]
    return ((3.0 * c[:, 3] * p + 2.0 * c[:, 2]) * p + c[:, 1]) / _DR


def _F(tab, e, quartic):
    """F, F', F'' of densities e."""
    m, p = _knot(e, _DRHO)
    c = tab[m]
    c4 = c[:, 4] if quartic else torch.zeros_like(p)
    v = (((c4 * p + c[:, 3]) * p + c[:, 2]) * p + c[:, 1]) * p + c[:, 0]
    d = (((4.0 * c4 * p + 3.0 * c[:, 3]) * p + 2.0 * c[:, 2]) * p + c[:, 1]) / _DRHO
    dd = ((12.0 * c4 * p + 3.0 * c[:, 3]) * p + 2.0 * c[:, 2]) / _DRHO / _DRHO  # the reference's own F'' (3, not 6)
    return v, d, dd


def _list(d, cut):
    """Half list over owned sites and their periodic images, numbered as the
    ghost passes make them: (i, j, root of j, x_i - x_j, rsq) within `cut`."""
    H = torch.from_numpy(d["H"]).cuda()
    s = torch.from_numpy(d["s"]).cuda()
    n = d["n"]
    sh = ((cut + SKIN) / H)
    root = torch.arange(n, device="cuda")
    img = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    sg = s.clone()
    for k in range(3):
        hi = len(sg)
        low = torch.nonzero(sg[:hi, k] <= sh[k]).flatten()
        high = torch.nonzero(1.0 - sh[k] <= sg[:hi, k]).flatten()
        src = torch.cat([low, high])
        add = torch.zeros((len(src), 3), dtype=torch.float64, device="cuda")
        add[:len(low), k], add[len(low):, k] = 1.0, -1.0
        sg, img, root = torch.cat([sg, sg[src] + add]), torch.cat([img, img[src] + add]), torch.cat([root, root[src]])
    x = torch.from_numpy(d["x"]).cuda()
    xg = x[root] + img * H
    I, J = [], []
    step = max(1, min(512, 40_000_000 // len(xg)))
    for a in range(0, n, step):
        xi = x[a:a + step]
        near = torch.nonzero(((xg >= xi.min(0).values - cut) & (xg <= xi.max(0).values + cut)).all(1)).flatten()
        near = near[near > a]
        dx = xi[:, None, :] - xg[None, near, :]
        rsq = (dx * dx).sum(2)
        i, j = torch.nonzero(rsq < cut * cut, as_tuple=True)
        i, j = i + a, near[j]
        keep = j > i
        I.append(i[keep])
        J.append(j[keep])
    i, j = torch.cat(I), torch.cat(J)
    dx = x[i] - xg[j]
    return i, j, root[j], dx, (dx * dx).sum(1), root


def _add(out, idx, v):
    out.index_add_(0, idx, v)


def _virial(dx, wf):
    return [float(-(wf * dx[:, p] * dx[:, q]).sum()) for p, q in ((0, 0), (1, 1), (2, 2), (1, 2), (2, 0), (0, 1))]


def _exact_eam(case, seed):
    d = _inputs(case, seed)
    rho, phi, emb = _tables(case["nt"])
    i, j, jo, dx, rsq, _ = _list(d, _RC)
    ty = torch.from_numpy(d["type"]).cuda().long()
    own = (j < d["n"]).double()
    r = rsq.sqrt()
    m, p = _knot(r, _DR)
    dens = torch.zeros(d["n"], dtype=torch.float64, device="cuda")
    dr, ph, dph = (torch.zeros_like(r) for _ in range(3))
    g = torch.zeros_like(r)
    for a in range(case["nt"]):
        for b in range(case["nt"]):
            k = torch.nonzero((ty[i] == a) & (ty[jo] == b)).flatten()
            g[k], dr[k] = _val(rho[a, b], m[k], p[k]), _der(rho[a, b], m[k], p[k])
            z, dz = _val(phi[a, b], m[k], p[k]), _der(phi[a, b], m[k], p[k])
            ph[k], dph[k] = z / r[k], (dz - z / r[k]) / r[k]
    _add(dens, i, g)
    _add(dens, jo, g * own)
    F, dF = torch.empty_like(dens), torch.empty_like(dens)
    for a in range(case["nt"]):
        k = ty == a
        F[k], dF[k], _ = _F(emb[a], dens[k], False)
    fp = -(dph + dr * (dF[i] + dF[jo])) / r
    f = torch.zeros((d["n"], 3), dtype=torch.float64, device="cuda")
    _add(f, i, fp[:, None] * dx)
    _add(f, jo, -(fp * own)[:, None] * dx)
    w = 0.5 + 0.5 * own
    en = [float(F.sum() + (w * ph).sum())] + _virial(dx, w * fp)
    return dict(f=f, en=np.array(en))


def _smear(tab, odd, r, alpha, xi, w):
    """Value and r, alpha derivatives of one smeared function (odd: r*phi, else rho)."""
    isq = alpha.rsqrt()
    sums = [torch.zeros_like(r) for _ in range(3)]
    for q in range(len(xi)):
        t = r - xi[q] * isq
        m, p = _knot(t.abs(), _DR)
        v = _val(tab, m, p)
        v = v * torch.sign(t) if odd else v * t
        v = torch.where(t.abs() < _RC, v, torch.zeros_like(v))
        for k in range(3):
            sums[k] += w[q] * xi[q]**k * v
    sc = 1.0 / (math.sqrt(math.pi) * r)
    g, gb, gc = (v * sc for v in sums)
    return g, -g / r - 2.0 * alpha.sqrt() * gb, (0.5 * g - gc) / alpha


def _dmd_setup(case, d):
    nt = case["nt"]
    xi, w = (v.tolist() for v in np.polynomial.hermite.hermgauss(case["nq"]))
    rho, phi, emb = _tables(nt)
    i, j, jo, dx, rsq, root = _list(d, _RC + xi[-1] / math.sqrt(A_LO))
    al, c = torch.from_numpy(d["alpha"]).cuda(), torch.from_numpy(d["c"]).cuda()
    r = rsq.sqrt()
    G, P = {}, {}
    for a in range(nt):
        for b in range(nt):
            aa = al[i, a] * al[jo, b] / (al[i, a] + al[jo, b])
            G[a, b] = _smear(rho[a, b], False, r, aa, xi, w)
            if a >= b:
                P[a, b] = P[b, a] = _smear(phi[a, b], True, r, aa, xi, w)
    kb, hbar = 8.617332478e-5, 6.5821192815e-16
    kT = kb * TEMP
    c0 = [1.5 * kT * (math.log(hbar * hbar * 2.0 / (_MASS[a] * 1.0364269184093291236e-28 * kT)) - 1.0) for a in range(nt)]
    return dict(i=i, j=j, jo=jo, dx=dx, rsq=rsq, r=r, own=(j < d["n"]).double(), G=G, P=P, al=al, c=c, emb=emb, kT=kT, c0=c0,
                xi=xi, w=w, rho=rho, phi=phi, root=root)


def _site_energy(S, F):
    c, al = S["c"], S["al"]
    ent = torch.where((c < 1.0e-8) | (c > 0.99999999), torch.zeros_like(c), torch.xlogy(c, c) + torch.xlogy(1.0 - c, 1.0 - c))
    c0 = torch.tensor(S["c0"], dtype=torch.float64, device="cuda")
    return float((c * F + S["kT"] * ent + 1.5 * S["kT"] * c * al.log() + c * c0).sum())


def _exact_dmd(case, seed):
    d, nt = _inputs(case, seed), case["nt"]
    S = _dmd_setup(case, d)
    i, jo, dx, r, own, G, P, al, c = (S[k] for k in ("i", "jo", "dx", "r", "own", "G", "P", "al", "c"))
    E = torch.zeros_like(c)
    e = 0.0
    for a in range(nt):
        for b in range(nt):
            _add(E[:, a], i, G[a, b][0] * c[jo, b])
            _add(E[:, b], jo, G[a, b][0] * c[i, a] * own)
            if a >= b:
                e += float(((0.25 + 0.25 * own) * (c[jo, b] * c[i, a] + c[jo, a] * c[i, b]) * P[a, b][0]).sum())
    F, dE = torch.empty_like(E), torch.empty_like(E)
    for a in range(nt):
        F[:, a], dE[:, a], _ = _F(S["emb"][a], E[:, a].contiguous(), True)
    e += _site_energy(S, F)
    f = torch.zeros((d["n"], 3 + nt), dtype=torch.float64, device="cuda")
    f[:, 3:] = -1.5 * S["kT"] * c / al
    fs = torch.zeros_like(r)
    for a in range(nt):
        for b in range(nt):
            cc = c[i, a] * c[jo, b]
            fs -= (G[b, a][1] * dE[i, a] + G[a, b][1] * dE[jo, b] + P[a, b][1]) * cc / r
            ap = -(G[b, a][2] * dE[i, a] + G[a, b][2] * dE[jo, b] + P[a, b][2]) * cc / (al[i, a] + al[jo, b])**2
            _add(f[:, 3 + a], i, ap * al[jo, b]**2)
            _add(f[:, 3 + b], jo, ap * al[i, a]**2 * own)
    for k in range(3):
        _add(f[:, k], i, fs * dx[:, k])
        _add(f[:, k], jo, -fs * dx[:, k] * own)
    out = dict(f=f, en=np.array([e] + _virial(dx, (0.5 + 0.5 * own) * fs)))
    if case["kind"] == "linesearch":
        # energy_calc: species pairs b >= a for the densities, like pairs for phi
        E = torch.zeros_like(c)
        e = 0.0
        for a in range(nt):
            for b in range(a, nt):
                _add(E[:, a], i, G[a, b][0] * c[jo, b])
                _add(E[:, b], jo, G[a, b][0] * c[i, a] * own)
            e += float(((0.25 + 0.25 * own) * 2.0 * c[jo, a] * c[i, a] * P[a, a][0]).sum())
        for a in range(nt):
            F[:, a], _, _ = _F(S["emb"][a], E[:, a].contiguous(), True)
        out["e"] = e + _site_energy(S, F)
    return out


def _rate(style, beta, ni, nj, ci, cj):
    """Jump rate of one neighbour pair and species, its t terms and its g factors."""
    if style == "DMD_II":
        mt = torch.maximum(ni, nj) + 0.5
        fi, fj = torch.exp(beta * (ni - mt)), torch.exp(beta * (nj - mt))
        ti, tj = ci * (1.0 - cj) * fi, cj * (1.0 - ci) * fj
        up, dn = (ni > nj).double(), (nj > ni).double()
        return tj - ti, ti + up * (tj - ti), tj + dn * (ti - tj), (1.0 - cj) * fi + cj * fj, (1.0 - ci) * fj + ci * fi
    if style == "DMD":
        ei, ej = torch.exp(ni + 5.2 * beta), torch.exp(nj + 5.2 * beta)
        wi, wj = ci * (1.0 - cj) * ei, cj * (1.0 - ci) * ej
        return wj - wi, wi, wj, ei * (1.0 - cj) + ej * cj, ej * (1.0 - ci) + ei * ci
    ei, ej = torch.exp(0.5 * (ni - nj) + 0.4 * beta), torch.exp(0.5 * (nj - ni) + 0.4 * beta)
    wi, wj = ci * (1.0 - cj) * ei, cj * (1.0 - ci) * ej
    return wj - wi, 0.5 * (wi + wj), 0.5 * (wi + wj), ei * (1.0 - cj) + ej * cj, ej * (1.0 - ci) + ei * ci


def _exact_rates(case, seed):
    d, nt = _inputs(case, seed), case["nt"]
    S = _dmd_setup(case, d)
    i, j, jo, own, G, P, al, c = (S[k] for k in ("i", "j", "jo", "own", "G", "P", "al", "c"))
    n, beta, style = d["n"], 1.0 / S["kT"], case["style"]
    a_in = torch.from_numpy(-d["c"] + 1e-3 * np.random.default_rng([seed, 17]).normal(size=d["c"].shape)).cuda()
    E = torch.zeros_like(c)
    for a in range(nt):
        for b in range(nt):
            _add(E[:, a], i, c[jo, b] * G[b, a][0])
            _add(E[:, b], jo, c[i, a] * G[a, b][0] * own)
    N, dE, ddE = torch.empty_like(E), torch.empty_like(E), torch.empty_like(E)
    for a in range(nt):
        N[:, a], dE[:, a], ddE[:, a] = _F(S["emb"][a], E[:, a].contiguous(), True)

    def flat(q):  # dE at the reference's flat index site + species
        return dE[S["root"][torch.div(q, nt, rounding_mode="floor")], q % nt]

    for a in range(nt):
        for b in range(nt):
            _add(N[:, a], i, c[jo, b] * (G[a, b][0] * flat(j + b) + P[a, b][0]))
            _add(N[:, b], jo, c[i, a] * (G[b, a][0] * flat(i + a) + P[a, b][0]) * own)
    N += torch.tensor(S["c0"], dtype=torch.float64, device="cuda") + 1.5 * S["kT"] * al.log()
    if style != "DMD_II":
        N *= beta
    k = torch.nonzero(S["rsq"] < R_CRD * R_CRD).flatten()
    ki, kj, ko = i[k], jo[k], own[k]
    cd, s = torch.zeros_like(c), 2.0 * (c + a_in)
    R = [_rate(style, beta, N[ki, a], N[kj, a], c[ki, a], c[kj, a]) for a in range(nt)]
    for a in range(nt):
        _add(cd[:, a], ki, R[a][0])
        _add(cd[:, a], kj, -R[a][0] * ko)
    alpha = _time_step(cd)
    s -= 2.0 * alpha * cd
    cost = float((s * s).sum()) * 0.25
    g, t, v = -s.clone(), torch.zeros_like(s), torch.zeros_like(s)
    for a in range(nt):
        ds = s[ki, a] - s[kj, a]
        _add(t[:, a], ki, R[a][1] * ds)
        _add(t[:, a], kj, -R[a][2] * ds * ko)
        _add(g[:, a], ki, -alpha * R[a][3] * ds)
        _add(g[:, a], kj, alpha * R[a][4] * ds * ko)
    for a in range(nt):
        for b in range(nt):
            r_ab, r_ba = G[b, a][0], G[a, b][0]  # densities of slots a*nt+b and b*nt+a
            q = beta * alpha * (P[a, b][0] + r_ab * dE[i, a] + r_ba * dE[jo, b])
            _add(v[:, a], i, r_ab * t[jo, b])
            _add(v[:, b], jo, r_ba * t[i, a] * own)
            _add(g[:, a], i, q * t[jo, b])
            _add(g[:, b], jo, q * t[i, a] * own)
    for a in range(nt):
        for b in range(nt):
            _add(g[:, a], i, alpha * beta * G[a, b][0] * (ddE * c * v)[jo, b])
            _add(g[:, b], jo, alpha * beta * G[b, a][0] * (ddE * c * v)[i, a] * own)
    out = dict(cd=cd, g=g)
    if case["form"] != "fp32":
        out["cost"] = cost
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "eam":
        return _exact_eam(case, seed)
    if kind in ("dmd", "linesearch", "relist"):
        return _exact_dmd(case, seed)
    if kind == "rates":
        return _exact_rates(case, seed)
    return None  # runs of many steps, and training
