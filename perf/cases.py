"""The work a Car-Parrinello program has this library do, as cases to time.

Every case goes through the public Python entry points (``StepContext``,
``StepBatch``): whole electronic steps, a batch of systems in one graph, and
the blocks a driver with its own step loop calls (density, V_KS, V.psi, the
EES non-local pass, the overlap / S^(-1/2) / back-multiply chain).  The systems
are the water boxes of ``bench.py`` and the tests (24, 192 and 768 atoms) and
boxes of the same density on the other grids the library is built for.

A case: ``op``; ``grid`` (points per axis); ``ecut`` (Ry); ``box`` (bohr);
``states``; ``precision`` ("fp64", the drop-in path, or "mixed"); ``xc`` for
the ops that have one.  ``batch`` cases hold ``systems``, one
"grid/ecut/box/states" per system.
"""
import ctypes
import functools
import math
import types

import numpy as np
import torch

from openatom_b200 import _lib
from openatom_b200.batch import StepBatch
from openatom_b200.context import StepContext
from openatom_b200.layout import StateLayout
from openatom_b200.system import nonlocal_channels, spline_tables

DEV = "cuda"
DT = 3.0            # a.u.
TAU_FS = 25.0       # CP mass and thermostat time constant
TE_EXT = 1000.0     # K, the isokinetic chains of the coefficients (on in CP dynamics)
TOL_NORB = 0.05     # random starts deviate more than the default 0.003
SEGMENT = 16        # steps of one trajectory before it starts again from psi0
GRIDS = (28, 32, 40, 48, 60, 64, 80, 96, 120, 128)
NL_GRIDS = (16, 20, 24, 28, 32, 40, 42, 48, 60, 64, 80, 96, 120, 128)
SPECIES = ("O", "H")


def listed():
    return [
        # the smallest dynamics users run (24 atoms): launches and latency count
        dict(name="step_water24_mixed", op="step", grid=48, ecut=30.0, box=12.0, states=32,
             precision="mixed", xc="pz_lda"),
        # the benchmark system (192 atoms), production dynamics
        dict(name="step_water192_mixed", op="step", grid=128, ecut=70.0, box=23.5, states=128,
             precision="mixed", xc="pz_lda"),
        # the same system through the plain FP64 path, the drop-in
        dict(name="step_water192_fp64", op="step", grid=128, ecut=70.0, box=23.5, states=128,
             precision="fp64", xc="pz_lda"),
        # the largest system (768 atoms, 200^3), half of its states
        dict(name="step_water768_mixed", op="step", grid=200, ecut=70.0, box=37.2, states=512,
             precision="mixed", xc="pz_lda"),
        # a ragged FP64 system: odd state count, a grid that is no power of two
        dict(name="step_ragged_fp64", op="step", grid=60, ecut=43.0, box=12.3, states=45,
             precision="fp64", xc="pz_lda"),
        # independent uneven systems in one graph (replica and sampling runs)
        dict(name="batch_uneven_mixed", op="batch", precision="mixed", xc="pz_lda",
             systems="32/40/7.2/24 48/55/9.6/58 64/35/16.4/119 96/62/18.9/162"),
        # density of an ordinary system on 96^3, for a driver with its own step loop
        dict(name="density_g96_mixed", op="density", grid=96, ecut=55.0, box=19.6, states=209,
             precision="mixed"),
        # V.psi + kinetic forces in FP64 on a grid with odd radices
        dict(name="vpsi_g120_fp64", op="vpsi", grid=120, ecut=70.0, box=21.4, states=50,
             precision="fp64"),
        # V_KS of a given density with gradient corrections and atom forces
        dict(name="vks_blyp_g128", op="vks", grid=128, ecut=70.0, box=23.5, states=8,
             precision="fp64", xc="blyp"),
        # overlap, S^(-1/2) and back-multiply of many states (512 x 60,000)
        dict(name="ortho_512_mixed", op="ortho", grid=128, ecut=70.0, box=22.8, states=512,
             precision="mixed"),
        # the same chain in FP64 with a ragged state count
        dict(name="ortho_77_fp64", op="ortho", grid=64, ecut=35.0, box=16.4, states=77,
             precision="fp64"),
        # the non-local pass alone, FP64
        dict(name="ees_g80_fp64", op="ees", grid=80, ecut=60.0, box=15.4, states=101,
             precision="fp64"),
    ]


def _kmax(box, ecut):
    """Largest |k| of the states' sphere on an axis and its number of points."""
    v = [ctypes.c_int() for _ in range(4)]
    _lib.lib().cpstep_layout_sizes(float(box), float(ecut), *(ctypes.byref(x) for x in v))
    return v[0].value, v[3].value


def _fits(grid, ecut, box, nonlocal_on=True):
    """The density sphere fits the grid and the library has the non-local grid."""
    k, _ = _kmax(box, ecut)
    nl = _lib.lib().cpstep_nl_grid_size(k, 1.2, 8)
    return grid >= 2 * (2 * k + 1) and (not nonlocal_on or nl in NL_GRIDS)


def _box(rng, grid, nonlocal_on=True):
    """A cutoff and a box for a grid."""
    while True:
        ecut = round(rng.uniform(30.0, 70.0), 1)
        box = round(rng.uniform(0.8, 0.965) * grid * math.pi / (2.0 * math.sqrt(ecut)), 2)
        if _fits(grid, ecut, box, nonlocal_on):
            return ecut, box


def draw(rng):
    op = rng.choice(["step", "step", "batch", "density", "vpsi", "vks", "ortho", "ees"])
    prec = rng.choice(["mixed", "fp64"])
    if op == "batch":
        n = rng.randint(2, 5)
        sys_ = []
        for _ in range(n):
            g = rng.choice((32, 48, 64, 96))
            ec, box = _box(rng, g)
            s = round(math.exp(rng.uniform(math.log(16), math.log(200 if g > 32 else 60))))
            sys_.append("%d/%s/%s/%d" % (g, ec, box, s))
        return dict(op=op, precision=prec, xc="pz_lda", systems=" ".join(sys_))
    grid = rng.choice(GRIDS)
    ecut, box = _box(rng, grid, op in ("step", "ees"))
    most = _kmax(box, ecut)[1] / 6.0
    states = round(math.exp(rng.uniform(math.log(16), math.log(min(256.0, most)))))
    c = dict(op=op, grid=grid, ecut=ecut, box=box, states=states, precision=prec)
    if op == "step":
        c["xc"] = "pz_lda"
    if op == "vks":
        c.update(xc=rng.choice(["pz_lda", "blyp"]), states=8, precision="fp64")
    if op == "ortho":
        c["states"] = round(math.exp(rng.uniform(math.log(16), math.log(min(512.0, most)))))
    return c


# ---------------------------------------------------------------------------
# inputs

@functools.lru_cache(maxsize=8)
def _layout(box, ecut, grid):
    return StateLayout(box, ecut, nfft=grid)


def _atoms(box, seed):
    """Waters at liquid density (one per 200 bohr^3) on jittered lattice sites."""
    nw = max(1, int(round(box ** 3 / 200.0)))
    natm = 3 * nw
    m = int(math.ceil(natm ** (1.0 / 3.0) - 1e-9))
    r = np.random.default_rng(seed)
    cell = r.permutation(m ** 3)[:natm]
    ijk = np.stack([cell // (m * m), (cell // m) % m, cell % m], axis=1)
    pos = (ijk + 0.5 + r.uniform(-0.3, 0.3, (natm, 3))) * (box / m)
    return pos, np.array([0] * nw + [1] * (2 * nw), dtype=np.int32)


def _system(box, ecut, grid, states, seed):
    tpi = 2.0 * math.pi / box
    gmax = math.sqrt(4.0 * ecut) * 4.0 / 3.0 + tpi
    tab = spline_tables(list(SPECIES), 0.75 * tpi, gmax)
    pos, typ = _atoms(box, seed)
    return types.SimpleNamespace(
        layout=_layout(box, ecut, grid), box_len=box, ecut_ry=ecut, nstates=states, tab=tab,
        pos=pos, typ=typ, natm=len(typ), alp_ewd=3.5 / box,
        channels=nonlocal_channels(list(SPECIES), tab["gmin"], tab["dg"], tab["nspl"]))


def _geometry(lay):
    """The packed points on the GPU: k, |G|^2, weight, half-spectrum index."""
    k = [torch.from_numpy(np.asarray(a, dtype=np.int64)).to(DEV) for a in (lay.kx, lay.ky, lay.kz)]
    return _points(k[0], k[1], k[2], lay.box_len, lay.n)


def _points(kx, ky, kz, box, n):
    tpi = 2.0 * math.pi / box
    g2 = (kx * kx + ky * ky + kz * kz).double() * (tpi * tpi)
    return types.SimpleNamespace(
        kx=kx, ky=ky, kz=kz, g2=g2, n=n, npts=len(kx), tpi=tpi, vol=box ** 3,
        w=torch.where(kx == 0, 1.0, 2.0).double(),
        idx=((kz % n) * n + ky % n) * (n // 2 + 1) + kx)


def _mirror(geo):
    """(redundant Gx=0 points, their partners, the index of G=0)."""
    span = 4 * geo.n
    code = torch.where(geo.kx == 0, (geo.ky + geo.n) * span + geo.kz + geo.n, -1)
    red = torch.nonzero((geo.kx == 0) & ((geo.ky < 0) | ((geo.ky == 0) & (geo.kz < 0))))[:, 0]
    order = torch.argsort(code)
    want = (-geo.ky[red] + geo.n) * span - geo.kz[red] + geo.n
    src = order[torch.searchsorted(code[order], want)]
    g0 = torch.nonzero((geo.kx == 0) & (geo.ky == 0) & (geo.kz == 0))[:, 0]
    return red, src, g0


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _coefficients(geo, states, gen):
    """Gaussian-damped random coefficients with the Gamma-point symmetry."""
    c = torch.randn((states, geo.npts, 2), generator=gen, dtype=torch.float64, device=DEV)
    c = torch.view_as_complex(c)
    c *= torch.exp(-geo.g2 / 8.0)
    red, src, g0 = _mirror(geo)
    c[:, red] = c[:, src].conj()
    c[:, g0] = c[:, g0].real.to(c.dtype)
    return c


def _gram(a, b, w):
    """sum_p w Re(conj a_i b_j)."""
    x = torch.view_as_real(a) * w[None, :, None] if w is not None else torch.view_as_real(a)
    return x.reshape(a.shape[0], -1) @ torch.view_as_real(b).reshape(b.shape[0], -1).T


def _inv_sqrt_half(S):
    e, u = torch.linalg.eigh(0.5 * (S + S.T) / 2.0)
    return (u * e.rsqrt()) @ u.T


def _mix(T, x):
    """out_i = sum_j T(j, i) x_j."""
    y = T.T @ torch.view_as_real(x).reshape(x.shape[0], -1)
    return torch.view_as_complex(y.reshape(T.shape[1], -1, 2))


def _orbitals(geo, states, seed):
    """Orthonormal coefficients (S = 2 I)."""
    c = _coefficients(geo, states, _gen(seed))
    return _mix(_inv_sqrt_half(_gram(c, c, geo.w)), c).contiguous()


def _smooth_field(n, box, gen):
    """A smooth random real field on the grid, unit variance."""
    f = torch.randn((n, n, n), generator=gen, dtype=torch.float64, device=DEV)
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=DEV) * (2.0 * math.pi / box)
    kh = k[: n // 2 + 1].abs()
    g2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kh[None, None, :] ** 2
    f = torch.fft.irfftn(torch.fft.rfftn(f) * torch.exp(-g2 / 6.0), s=(n, n, n))
    return f / f.std()


def _context(case, seed, atoms=True):
    sysm = _system(case["box"], case["ecut"], case["grid"], case["states"], seed)
    ctx = StepContext(sysm.layout, sysm.nstates, precision=case["precision"])
    if atoms:
        ctx.set_atoms(sysm)
    return sysm, ctx


def _stepper(case, seed):
    sysm, ctx = _context(case, seed)
    ctx.set_nonlocal(sysm)
    if case["xc"] != "pz_lda":
        ctx.set_xc(case["xc"])
    ctx.set_cp_mass(TAU_FS, case["ecut"])
    ctx.set_cp_thermostat(TE_EXT, TAU_FS)
    ctx.set_constraint("ortho_t", TOL_NORB)
    psi0 = _orbitals(_geometry(sysm.layout), case["states"], seed)
    return dict(sys=sysm, ctx=ctx, psi0=psi0, psi=psi0.clone(), v=torch.zeros_like(psi0),
                occ=torch.ones(case["states"], dtype=torch.float64, device=DEV),
                e=torch.zeros(_lib.NENERGY, dtype=torch.float64, device=DEV),
                f=torch.zeros((sysm.natm, 3), dtype=torch.float64, device=DEV))


def _batch_cases(case):
    for s in case["systems"].split():
        g, ec, box, n = s.split("/")
        yield dict(op="step", grid=int(g), ecut=float(ec), box=float(box), states=int(n),
                   precision=case["precision"], xc=case["xc"])


def prepare(case, seed):
    op = case["op"]
    if op == "step":
        return dict(_stepper(case, seed), op=op, done=0)
    if op == "batch":
        parts = [_stepper(c, seed * 101 + k) for k, c in enumerate(_batch_cases(case))]
        for p in parts:
            p["ctx"].set_graph(False)  # the batch holds the one graph
        return dict(op=op, parts=parts, batch=StepBatch([p["ctx"] for p in parts]), done=0)
    if op == "vks":
        sysm, ctx = _context(case, seed)
        if case["xc"] != "pz_lda":
            ctx.set_xc(case["xc"])
        a = _smooth_field(case["grid"], case["box"], _gen(seed))
        b = _smooth_field(case["grid"], case["box"], _gen(seed + 1000003))
        return dict(op=op, sys=sysm, ctx=ctx, rho=0.03 * (a * a + b * b) + 1e-4)
    sysm, ctx = _context(case, seed, atoms=op == "ees")
    if op == "ees":
        ctx.set_nonlocal(sysm)
    geo = _geometry(sysm.layout)
    st = dict(op=op, sys=sysm, ctx=ctx, psi=_orbitals(geo, case["states"], seed),
              occ=torch.ones(case["states"], dtype=torch.float64, device=DEV))
    if op == "vpsi":
        st["vks"] = 0.8 * _smooth_field(case["grid"], case["box"], _gen(seed + 5)) - 0.5
    if op == "ortho":  # as after an integration step: orthonormal up to a few percent
        d = _coefficients(geo, case["states"], _gen(seed + 9))
        st["psi"] += d * (0.02 / d.abs().square().sum(1).sqrt().mean())
        st["mixed"] = case["precision"] == "mixed"
    return st


def run(st):
    op = st["op"]
    if op == "step":
        it = st["done"] % SEGMENT + 1
        st["done"] += 1
        if it == 1:
            st["psi"].copy_(st["psi0"])
            st["v"].zero_()
        st["ctx"].cp_step(st["psi"], st["v"], st["occ"], DT, it, st["e"], st["f"])
        return st["psi"], st["v"], st["e"], st["f"]
    if op == "batch":
        it, parts = st["done"] % SEGMENT + 1, st["parts"]
        st["done"] += 1
        if it == 1:
            for p in parts:
                p["psi"].copy_(p["psi0"])
                p["v"].zero_()
        st["batch"].step(*([p[k] for p in parts] for k in ("psi", "v", "occ")), DT, it,
                         [p["e"] for p in parts], [p["f"] for p in parts])
        return [(p["psi"], p["v"], p["e"], p["f"]) for p in parts]
    ctx = st["ctx"]
    if op == "density":
        return ctx.density(st["psi"], st["occ"])
    if op == "vpsi":
        return ctx.vks_psi(st["psi"], st["vks"], st["occ"])
    if op == "vks":
        return ctx.vks_from_rho(st["rho"])
    if op == "ees":
        return ctx.ees_nonlocal(st["psi"], st["occ"])
    S = ctx.pc_overlap(st["psi"], st["psi"])
    T, _, _ = ctx.ortho_tmat(S, mixed=st["mixed"], tol=2e-6 if st["mixed"] else 1e-15,
                             max_iter=20 if st["mixed"] else 10)
    return S, T, ctx.pc_backmultiply(T, st["psi"])


# ---------------------------------------------------------------------------
# the least a pass can do

def work(case):
    if case["op"] == "batch":
        parts = [work(c) for c in _batch_cases(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, S, op = case["grid"], case["states"], case["op"]
    kr = math.sqrt(case["ecut"]) * case["box"] / (2.0 * math.pi)   # radius of the sphere in k
    npts = 2.0 / 3.0 * math.pi * kr ** 3
    natm = 3 * max(1, round(case["box"] ** 3 / 200.0))
    n3, coef = float(n) ** 3, 16.0 * S * npts
    fft = 2.5 * n3 * math.log2(n3)                # one real transform of the grid
    gemm = 2.0 * S * S * 2.0 * npts               # one S x S x 2 npts product
    ees = 2.0 * (4 * S) * (5 * natm) * 2.0 * npts  # Z and force sums, psi force; 4 channels
    vks_f = 3.0 * fft + 8.0 * natm * 8.0 * npts   # density transforms, structure factors
    if op == "density":
        return {"bytes": coef + 8.0 * n3, "flops": S * fft}
    if op == "vpsi":
        return {"bytes": 2.0 * coef + 8.0 * n3, "flops": 2.0 * S * fft}
    if op == "vks":
        return {"bytes": 16.0 * n3, "flops": vks_f + (7.0 * fft if case["xc"] == "blyp" else 0.0)}
    if op == "ees":
        return {"bytes": 2.0 * coef, "flops": ees}
    if op == "ortho":
        return {"bytes": 2.0 * coef + 16.0 * S * S, "flops": 2.0 * gemm + 6.0 * S ** 3 * 5}
    return {"bytes": 6.0 * coef, "flops": 3.0 * S * fft + 5.0 * gemm + ees + vks_f + 30.0 * S ** 3}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch

def _to_r(c, geo):
    """psi(r) = sum_G psi e^{-iG.r} (real) of [s, npts] coefficients."""
    n = geo.n
    half = torch.zeros((c.shape[0], n * n * (n // 2 + 1)), dtype=c.dtype, device=DEV)
    half[:, geo.idx] = c.conj()
    return torch.fft.irfftn(half.view(-1, n, n, n // 2 + 1), s=(n, n, n), norm="forward")


def _to_g(f, geo):
    """sum_r f e^{+iG.r} at the packed points of [s, n, n, n] fields."""
    x = torch.fft.rfftn(f, dim=(1, 2, 3)).reshape(f.shape[0], -1)
    return x[:, geo.idx].conj()


def _chunks(S, n):
    step = max(1, int(6e7 // n ** 3))
    return [(a, min(S, a + step)) for a in range(0, S, step)]


def _x_density(psi, geo):
    rho = torch.zeros((geo.n,) * 3, dtype=torch.float64, device=DEV)
    for a, b in _chunks(len(psi), geo.n):
        rho += _to_r(psi[a:b], geo).square().sum(0)
    return rho / geo.vol


def _x_vpsi(psi, vks, geo, ecut):
    force = torch.empty_like(psi)
    for a, b in _chunks(len(psi), geo.n):
        force[a:b] = _to_g(_to_r(psi[a:b], geo) * vks, geo) * (-2.0 / geo.n ** 3)
    wg = torch.where(geo.g2 <= ecut, geo.w * geo.g2, 0.0)
    force = torch.where(geo.g2 <= ecut, force * geo.w - psi * wg, 0.0)
    return force, 0.5 * (psi.abs().square() * wg).sum(1)


def _x_lda(rho, vol):
    """Perdew-Zunger LDA: (v_xc, E_xc, sum v_xc rho)."""
    rs = (3.0 / (4.0 * math.pi * rho)) ** (1.0 / 3.0)
    vx = -((3.0 * rho / math.pi) ** (1.0 / 3.0))
    sq, ln = rs.sqrt(), rs.log()
    b1, b2, au, bu, cu, du = 1.0529, 0.3334, 0.0311, -0.048, 0.002, -0.0116
    den = 1.0 + b1 * sq + b2 * rs
    hi = -0.1423 / den
    ec = torch.where(rs >= 1.0, hi, au * ln + bu + cu * rs * ln + du * rs)
    vc = torch.where(rs >= 1.0, hi * (1.0 + 7.0 / 6.0 * b1 * sq + 4.0 / 3.0 * b2 * rs) / den,
                     au * ln + (bu - au / 3.0) + 2.0 / 3.0 * cu * rs * ln
                     + (2.0 * du - cu) / 3.0 * rs)
    dv = vol / rho.numel()
    return vx + vc, ((0.75 * vx + ec) * rho).sum() * dv, ((vx + vc) * rho).sum() * dv


def _spline(tab, vps, g):
    i = ((g - tab["gmin"]) / tab["dg"] + 1.0).long().clamp(1, tab["nspl"]) - 1
    h = g - (i.double() * tab["dg"] + tab["gmin"])
    v = [torch.from_numpy(np.ascontiguousarray(vps[..., k, :])).to(DEV)[..., i] for k in range(4)]
    return ((v[3] * h + v[2]) * h + v[1]) * h + v[0]


def _x_vks(rho, sysm, ctx):
    """LDA V_KS, energies and local + Ewald atom forces of a density."""
    n, box, vol = rho.shape[0], sysm.box_len, sysm.box_len ** 3
    tab, tpi = sysm.tab, 2.0 * math.pi / sysm.box_len
    k = [torch.from_numpy(a.astype(np.int64)).to(DEV) for a in ctx.rho_layout()]
    geo = _points(k[0], k[1], k[2], box, n)
    vxc, exc, mu = _x_lda(rho, vol)
    rg = torch.fft.rfftn(rho).reshape(-1)[geo.idx] * (vol / n ** 3)
    pos = torch.from_numpy(sysm.pos).to(DEV)
    typ = torch.from_numpy(sysm.typ.astype(np.int64)).to(DEV)
    q = torch.from_numpy(np.asarray(tab["q"])).to(DEV)[typ]
    vg = torch.zeros_like(rg)
    e = torch.zeros(_lib.NENERGY, dtype=torch.float64, device=DEV)
    e[0], e[1] = exc, mu
    force = torch.zeros((len(typ), 3), dtype=torch.float64, device=DEV)
    step = max(1024, int(1.2e8 // max(1, len(typ))))
    for a in range(0, geo.npts, step):
        s = slice(a, a + step)
        kk = torch.stack([geo.kx[s], geo.ky[s], geo.kz[s]]).double() * tpi
        g2, w = geo.g2[s], geo.w[s]
        nz = (g2 > 0) & (g2 <= 4.0 * sysm.ecut_ry)
        ig = torch.where(nz, 4.0 * math.pi / torch.where(nz, g2, 1.0) / vol, 0.0)
        vt = _spline(tab, tab["vps"], g2.sqrt())[typ] / vol
        ph = pos @ kk
        h = torch.polar(torch.ones_like(ph), ph)
        vext, sq = (h * vt).sum(0), (h * q[:, None]).sum(0)
        r = rg[s]
        vg[s] = torch.where(nz, r * ig + vext.conj(), 0.0)
        ew = ig * torch.exp(-g2 / (4.0 * sysm.alp_ewd ** 2)) * w
        e[2] += 0.5 * (ig * w * r.abs().square()).sum()
        e[3] += torch.where(nz, (r * vext).real * w, 0.0).sum()
        e[4] += 0.5 * (ew * sq.abs().square()).sum()
        z = torch.where(nz, r.conj() * w, 0.0)[None] * vt + (sq * ew)[None] * q[:, None]
        force += (z.real * h.imag - z.imag * h.real) @ kk.T
    g0 = torch.nonzero(geo.g2 == 0)[:, 0]
    v0 = torch.from_numpy(np.asarray(tab["gzvps"])).to(DEV)[typ].sum() / vol
    vg[g0] = v0.to(vg.dtype)
    e[3] += (v0 * rg[g0].real).sum()
    return vxc + _to_r(vg.conj()[None], geo)[0], e, force


def _spline_axes(frac, ng, order=8):
    """Cardinal B-spline values and slopes [natm, order] and grid indices."""
    u0 = frac * ng
    it = np.floor(u0).astype(np.int64)
    u = (u0 - it)[:, None] + np.arange(order)[None]

    def m(p, x):
        if p == 2:
            return np.maximum(0.0, 1.0 - np.abs(x - 1.0))
        return (x * m(p - 1, x) + (p - x) * m(p - 1, x - 1.0)) / (p - 1)
    return m(order, u), m(order - 1, u) - m(order - 1, u - 1.0), (it[:, None] - np.arange(order)) % ng


def _x_ees(psi, sysm, geo, nkf):
    """EES non-local pass (s and p channels) by Parseval: (F_psi, E_NL, F_atoms)."""
    order, box, vol = 8, sysm.box_len, sysm.box_len ** 3
    km = int(max(geo.kx.max(), geo.ky.max(), geo.kz.max())) + 1
    kk = np.arange(-km, km + 1)
    knots = _spline_axes(np.zeros(1), nkf)[0][0]                  # M_8(0..7)
    d = (knots[1:] * np.exp(2j * np.pi * np.outer(kk, np.arange(order - 1)) / nkf)).sum(1)
    euler = np.exp(2j * np.pi * (order - 1) * kk / nkf) / d
    eu = torch.from_numpy(euler).to(DEV)
    b = eu[geo.kx + km] * eu[geo.ky + km] * eu[geo.kz + km]
    tabs = []
    for ax in range(3):
        mn, dm, ig = _spline_axes(np.mod(sysm.pos[:, ax] / box, 1.0), nkf)
        e = np.exp(-2j * np.pi * ig[:, :, None] * kk[None, None, :] / nkf)
        tabs.append([torch.from_numpy(np.einsum("aj,ajk->ak", t, e)).to(DEV)
                     for t in (mn, dm * (nkf / box))])
    g = geo.g2.sqrt()
    gs = torch.where(g > 0, g, 1.0)
    ylm = {0: torch.full_like(g, 1.0 / math.sqrt(4.0 * math.pi))}
    fpsi, enl = torch.zeros_like(psi), torch.zeros((), dtype=torch.float64, device=DEV)
    fatm = torch.zeros((sysm.natm, 3), dtype=torch.float64, device=DEV)
    c1 = math.sqrt(3.0 / (4.0 * math.pi)) * geo.tpi
    psi_r = torch.view_as_real(psi)
    for t in range(len(SPECIES)):
        at = torch.from_numpy(np.nonzero(sysm.typ == t)[0]).to(DEV)
        px, py, pz = (geo.kx + km, geo.ky + km, geo.kz + km)
        for a0 in range(0, len(at), 128):
            aa = at[a0:a0 + 128]
            X, Y, Z = ([tb[0][aa], tb[1][aa]] for tb in tabs)
            rows = []
            for dx, dy, dz in ((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)):
                rows.append(X[dx][:, px] * Y[dy][:, py] * Z[dz][:, pz])
            for ch in sysm.channels:
                if ch["type"] != t:
                    continue
                rad = _spline(sysm.tab, ch["vnl"], g)
                if ch["l"] == 0:
                    dyp = b * ylm[0] * torch.where(g > 0, rad, ch["gzvps0"])
                else:
                    k = {0: geo.kz, 1: geo.kx, -1: geo.ky}[ch["m"]].double()
                    dyp = torch.where(g > 0, 1j * b * (c1 * k / gs) * rad, 0.0)
                vn = ch["vnorm"] / vol
                # sum_p w Re(conj(dyp psi) S) = psi . (w conj(S) dyp)^T over the real view
                def dots(S):
                    x = torch.view_as_real((S * (geo.w * dyp.conj())[None])).reshape(len(aa), -1)
                    return psi_r.reshape(len(psi), -1) @ x.T
                z = dots(rows[0])
                enl += vn * z.square().sum()
                zs = 2.0 * vn * z
                for ax in range(3):
                    fatm[aa, ax] -= (zs * dots(rows[1 + ax])).sum(0)
                x = torch.view_as_real(rows[0] * (geo.w * dyp.conj())[None]).reshape(len(aa), -1)
                fpsi -= torch.view_as_complex((zs @ x).reshape(len(psi), -1, 2))
    return fpsi, enl, fatm


def _x_step(p):
    """The first step from psi0 with v = 0 and orthoT = I."""
    sysm, ctx, psi = p["sys"], p["ctx"], p["psi0"]
    geo = _geometry(sysm.layout)
    vks, e, fat = _x_vks(_x_density(psi, geo), sysm, ctx)
    F, eke = _x_vpsi(psi, vks, geo, sysm.ecut_ry)
    fnl, enl, fnl_at = _x_ees(psi, sysm, geo, ctx.nkf)
    F += fnl
    e[6], e[7] = eke.sum(), enl
    e[8] = e[6] + e[7] + e[2] + e[3] + e[0]
    lam = _gram(psi, F, None)
    F -= torch.where(geo.kx == 0, 0.5, 1.0) * _mix(lam, psi)
    red, src, g0 = _mirror(geo)
    F[:, g0] = F[:, g0].real.to(F.dtype)
    m0 = 4.0 * (TAU_FS / 0.0241888) ** 2 * 0.0005
    mass = m0 * torch.clamp(0.5 * geo.g2 / (0.5 * sysm.ecut_ry), min=1.0)
    mass[g0] = 0.5 * m0
    v = F * (0.5 * DT / mass)
    x = psi + v * DT
    x[:, red], v[:, red] = x[:, src].conj(), v[:, src].conj()
    e[12] = len(psi) * TE_EXT / 315777.0   # two chains at kT/2 each, per state
    return _mix(_inv_sqrt_half(_gram(x, x, geo.w)), x), v, e, fat + fnl_at


def exact(case, seed):
    if case.get("xc") == "blyp":
        return None
    st = prepare(case, seed)
    op = case["op"]
    if op == "step":
        return _x_step(st)
    if op == "batch":
        return [_x_step(p) for p in st["parts"]]
    if op == "vks":
        return _x_vks(st["rho"], st["sys"], st["ctx"])
    geo, psi = _geometry(st["sys"].layout), st["psi"]
    if op == "density":
        return _x_density(psi, geo)
    if op == "vpsi":
        return _x_vpsi(psi, st["vks"], geo, case["ecut"])
    if op == "ees":
        f, enl, fat = _x_ees(psi, st["sys"], geo, st["ctx"].nkf)
        e = torch.zeros(_lib.NENERGY, dtype=torch.float64, device=DEV)
        e[7] = enl
        return f, e, fat
    S = _gram(psi, psi, geo.w)
    T = _inv_sqrt_half(S)
    return S, T, _mix(T, psi)
