"""EES non-local on the GPU (cpstep_ees_nonlocal and inside cpstep_cp_step)
against the FP64 oracle (oracle/ees.py, itself pinned to the reference's
cp_ees_nonlocal.C routines by tests/test_ees_oracle.py).

FP64 path: E_NL to 1e-11 relative, psi force and atom forces to 1e-10 of
their largest entry.  Mixed path (FP32 NL FFTs, FP64 sums): E_NL to 1e-5
relative, forces to 1e-5 of their largest entry, both for the NL-grid FFT
form and for the G-space form (the same stencil sums by Parseval, evaluated
as split-BF16 tensor-core products with the separable B-spline transforms);
inside the step, energy per atom <= 1e-6 Ha and atom forces <= 1e-5 Ha/bohr.
"""
import numpy as np
import pytest

from conftest import cuda_ok

pytestmark = pytest.mark.gpu

DT = 5.0


@pytest.fixture(scope="module")
def nlsys():
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from oracle import ees as OE
    from openatom_b200.system import System
    sysm = System(12.0, 30.0, 16, {"O": 4, "H": 8}, nfft=48, seed=21)
    psi = sysm.psi()
    occ_np = np.where(np.arange(sysm.nstates) % 3 == 0, 1.0, 2.0)
    occ = torch.from_numpy(occ_np).cuda()
    nkf = OE.nl_grid_size(sysm.layout.kmax)
    e, fpsi, fatm = OE.nonlocal_ees(psi.cpu().numpy(), sysm.layout, occ_np, sysm.box_len ** 3,
                                    sysm.hmati(), dict(pos=sysm.pos, typ=sysm.typ),
                                    sysm.channels, sysm.tab, nkf)
    return dict(sys=sysm, psi=psi, occ=occ, nkf=nkf, ref=(e, fpsi, fatm))


def _run(nlsys, precision, gspace=None):
    from openatom_b200.context import StepContext
    s = nlsys["sys"]
    ctx = StepContext(s.layout, s.nstates, precision=precision)
    try:
        ctx.set_atoms(s)
        nkf = ctx.set_nonlocal(s)
        if gspace is not None:
            ctx.tune_set({"ees_gspace": int(gspace)})
        assert nkf == nlsys["nkf"]
        fpsi, e, f = ctx.ees_nonlocal(nlsys["psi"], nlsys["occ"])
        return e.cpu().numpy()[7], fpsi.cpu().numpy(), f.cpu().numpy()
    finally:
        ctx.close()


def test_nl_grid_size_entry():
    from openatom_b200 import _lib
    from oracle import ees as OE
    L = _lib.lib()
    for kmax in (6, 10, 31, 49):
        assert L.cpstep_nl_grid_size(kmax, 1.2, 8) == OE.nl_grid_size(kmax)


def test_fp64_ees_matches_oracle(nlsys):
    e, fpsi, f = _run(nlsys, "fp64")
    er, fr, far = nlsys["ref"]
    assert er > 0.0
    assert abs(e - er) <= 1e-11 * abs(er)
    assert np.max(np.abs(fpsi - fr)) <= 1e-10 * np.max(np.abs(fr))
    assert np.max(np.abs(f - far)) <= 1e-10 * np.max(np.abs(far))


@pytest.mark.parametrize("gspace", [True, False])
def test_mixed_ees_within_budget(nlsys, gspace):
    """Mixed contexts: the G-space form on the tensor cores (gspace) and the
    NL-grid FFT form."""
    e, fpsi, f = _run(nlsys, "mixed", gspace)
    er, fr, far = nlsys["ref"]
    assert abs(e - er) <= 1e-5 * abs(er)
    assert np.max(np.abs(fpsi - fr)) <= 1e-5 * np.max(np.abs(fr))
    assert np.max(np.abs(f - far)) <= 1e-5 * np.max(np.abs(far))


def test_ees_accumulates_into_the_force(nlsys):
    import torch
    from openatom_b200.context import StepContext
    s = nlsys["sys"]
    ctx = StepContext(s.layout, s.nstates, precision="fp64")
    try:
        ctx.set_atoms(s)
        ctx.set_nonlocal(s)
        base = torch.full_like(nlsys["psi"], 0.25 - 0.5j)
        fpsi, _, _ = ctx.ees_nonlocal(nlsys["psi"], nlsys["occ"], fpsi=base.clone())
        _, fr, _ = nlsys["ref"]
        got = fpsi.cpu().numpy() - base.cpu().numpy()
        assert np.max(np.abs(got - fr)) <= 1e-10 * np.max(np.abs(fr))
    finally:
        ctx.close()


@pytest.fixture(scope="module")
def nlstep(nlsys):
    from oracle import density as OD
    from oracle import layout as OL
    from oracle import step as OS
    s = nlsys["sys"]
    lay = OL.Layout(12.0, 30.0, grid=48)
    dlay = OD.density_layout(12.0, 30.0, 48)
    cmass = OS.cp_mass(lay, 25.0, 30.0)
    pn = nlsys["psi"].cpu().numpy()
    occ = nlsys["occ"].cpu().numpy()
    p1, v1, en1, f1, _ = OS.cp_step(pn, np.zeros_like(pn), occ, s, lay, dlay, cmass, DT, 1,
                                    nonlocal_on=True, nkf=nlsys["nkf"], tol_norb=1.0)
    return (p1, v1, en1, f1)


def _step(nlsys, precision):
    import torch
    from openatom_b200.context import StepContext
    s = nlsys["sys"]
    ctx = StepContext(s.layout, s.nstates, precision=precision)
    try:
        ctx.set_atoms(s)
        ctx.set_nonlocal(s)
        ctx.set_cp_mass(25.0, 30.0)
        ctx.set_constraint("ortho_t", 1.0)  # cp_norb_tol above this step's deviation
        psi = nlsys["psi"].clone()
        v = torch.zeros_like(psi)
        e, f = ctx.cp_step(psi, v, nlsys["occ"], DT, 1)
        _, ok = ctx.step_status()
        return psi.cpu().numpy(), v.cpu().numpy(), e.cpu().numpy(), f.cpu().numpy(), ok
    finally:
        ctx.close()


def test_fp64_step_with_nonlocal(nlsys, nlstep):
    p, v, e, f, ok = _step(nlsys, "fp64")
    pr, vr, er, fr = nlstep
    assert ok
    for name, slot in (("ENL", 7), ("EKE", 6), ("ETOT", 8)):
        assert abs(e[slot] - er[name]) <= 1e-10 * max(1.0, abs(er[name])), name
    assert np.max(np.abs(p - pr)) < 1e-9
    assert np.max(np.abs(f - fr)) < 1e-9 * max(1.0, np.max(np.abs(fr)))


def test_mixed_step_with_nonlocal(nlsys, nlstep):
    p, v, e, f, ok = _step(nlsys, "mixed")
    pr, vr, er, fr = nlstep
    natm = nlsys["sys"].natm
    assert ok
    assert abs(e[8] - er["ETOT"]) / natm <= 1e-6
    assert np.max(np.abs(f - fr)) <= 1e-5


def _launches(ctx, psi, occ):
    """Kernels of one non-local pass."""
    from openatom_b200 import _lib
    n0 = _lib.lib().cpstep_launch_count()
    ctx.ees_nonlocal(psi, occ)
    return _lib.lib().cpstep_launch_count() - n0


@pytest.mark.parametrize("states,atoms,keep,gspace", [
    (1, {"O": 1, "H": 2}, None, True), (31, {"O": 3, "H": 5}, None, True),
    (33, {"O": 11, "H": 22}, None, True), (65, {"O": 2, "H": 3}, (1, 0), False),
    (65, {"O": 33, "H": 40}, (1, 0), True), (130, {"O": 9, "H": 0}, None, True),
    (64, {"O": 16, "H": 17}, (0, 0), True)])
def test_fp64_gspace_matches_grid_form(states, atoms, keep, gspace):
    """FP64 contexts: the G-space products against the NL-grid transforms at the
    edges of their tiles (32, 64, 128 states; 32 atoms; a ragged last point
    tile), with a type without channels or with one only, and forces added to
    what is there.  Both are FP64 sums of the same terms: 1e-11 of the largest
    entry.  `gspace`: whether choice 1 runs the G-space form (one channel and few
    atoms do not), told by the kernels of a pass."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.system import System
    s = System(12.0, 25.0, states, {k: n for k, n in atoms.items() if n}, nfft=40, seed=5)
    if keep is not None:  # (type, l) of the one channel kept
        s.channels = [c for c in s.channels if (c["type"], c["l"]) == keep]
    g = torch.Generator(device="cuda").manual_seed(states)
    psi = torch.view_as_complex(torch.randn((states, s.layout.npts, 2), generator=g,
                                            dtype=torch.float64, device="cuda"))
    f0 = 0.1 * psi.flip(0).contiguous()
    occ = 1.0 + torch.arange(states, dtype=torch.float64, device="cuda") % 2
    out, n = [], []
    for form in (1, 0):
        ctx = StepContext(s.layout, states, precision="fp64")
        try:
            ctx.set_atoms(s)
            ctx.set_nonlocal(s)
            ctx.tune_set({"ees_gspace": form})
            f, e, fa = ctx.ees_nonlocal(psi, occ, fpsi=f0.clone())
            out.append((e[7:8].cpu().numpy(), f.cpu().numpy(), fa.cpu().numpy()))
            n.append(_launches(ctx, psi, occ))
            f2, e2, _ = ctx.ees_nonlocal(psi, occ, fpsi=f0.clone(), forces=False)
            assert bool((f2 == f).all()) and bool((e2[7] == e[7]).all())
        finally:
            ctx.close()
    assert (n[0] < n[1]) == gspace and (gspace or n[0] == n[1])
    for a, b in zip(*out):
        assert np.max(np.abs(b)) > 0.0
        assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(b))


@pytest.mark.parametrize("states,atoms,keep", [
    (1, {"H": 1}, None), (16, {"O": 31, "H": 1}, None), (17, {"O": 32, "H": 33}, None),
    (33, {"O": 3, "H": 6}, (0, 1)), (33, {"O": 3, "H": 6}, (1, 0))])
def test_mixed_atom_forces_tile_edges(states, atoms, keep):
    """Mixed contexts: energy, psi force and atom forces of the G-space form
    against an FP64 context at the edges of the tiles (32 atoms; 16 states) and
    with a type without channels.  FP16 pairs hold 22 bits and the sums FP32's 24
    in chunks, added to the forces' largest entry: the module's 1e-5."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.system import System
    s = System(12.0, 25.0, states, atoms, nfft=40, seed=5)
    if keep is not None:
        s.channels = [c for c in s.channels if (c["type"], c["l"]) == keep]
    g = torch.Generator(device="cuda").manual_seed(states)
    psi = torch.view_as_complex(torch.randn((states, s.layout.npts, 2), generator=g,
                                            dtype=torch.float64, device="cuda"))
    f0 = 0.1 * psi.flip(0).contiguous()
    occ = 1.0 + torch.arange(states, dtype=torch.float64, device="cuda") % 2
    out = []
    for precision in ("mixed", "fp64"):
        ctx = StepContext(s.layout, states, precision=precision)
        try:
            ctx.set_atoms(s)
            ctx.set_nonlocal(s)
            ctx.tune_set({"ees_gspace": 1})
            f, e, fa = ctx.ees_nonlocal(psi, occ, fpsi=f0.clone())
            out.append((e[7:8].cpu().numpy(), f.cpu().numpy(), fa.cpu().numpy()))
            assert ctx.device_errors() == 0
        finally:
            ctx.close()
    for a, b in zip(*out):
        assert np.max(np.abs(b)) > 0.0
        assert np.max(np.abs(a - b)) <= 1e-5 * np.max(np.abs(b))


def _retyped(s, typ):
    """`s` with the same positions and other atom types."""
    import copy
    t = copy.copy(s)
    t.typ = np.ascontiguousarray(typ, dtype=np.asarray(s.typ).dtype)
    return t


@pytest.mark.parametrize("precision,form,keep", [
    ("fp64", 1, None), ("fp64", 1, (0, 0)), ("fp64", 0, None), ("mixed", 1, None),
    ("mixed", 1, (0, 0)), ("mixed", 0, None)])
def test_atoms_of_other_types_after_set_nonlocal(precision, form, keep):
    """set_atoms with the same number of atoms and other types after
    set_nonlocal (the types permuted, and other counts of each): the pass is the
    one of a context that saw these atoms only, bit for bit.  `keep`: one channel
    on type 0 only, so that atoms gain and lose their projectors."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.system import System
    s = System(12.0, 25.0, 33, {"O": 9, "H": 27}, nfft=40, seed=5)
    if keep is not None:
        s.channels = [c for c in s.channels if (c["type"], c["l"]) == keep]
    typ = np.asarray(s.typ)
    sets = [_retyped(s, typ[::-1]), _retyped(s, 1 - typ), s]
    psi, occ = s.psi(), torch.ones(s.nstates, dtype=torch.float64, device="cuda")

    def results(ctx):
        f, e, fa = ctx.ees_nonlocal(psi, occ)
        return float(e[7]), f.cpu().numpy(), fa.cpu().numpy()

    def context(t):
        ctx = StepContext(s.layout, s.nstates, precision=precision)
        ctx.set_atoms(t)
        ctx.set_nonlocal(t)
        ctx.tune_set({"ees_gspace": form})
        return ctx

    ctx = context(s)
    try:
        results(ctx)
        for t in sets:
            ctx.set_atoms(t)
            got = results(ctx)
            ref = context(t)
            try:
                want = results(ref)
            finally:
                ref.close()
            assert want[0] != 0.0 and np.max(np.abs(want[2])) > 0.0
            for a, b in zip(got, want):
                assert np.array_equal(a, b)
    finally:
        ctx.close()


def test_other_atom_count_after_set_nonlocal_is_refused():
    """Another number of atoms, or fewer types than the channels name, leaves the
    non-local data stale: an error, and the first atoms again make it good."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import copy
    import torch
    from openatom_b200 import _lib
    from openatom_b200.context import StepContext
    from openatom_b200.system import System
    s = System(12.0, 25.0, 8, {"O": 3, "H": 6}, nfft=40, seed=5)
    fewer = copy.copy(s)
    fewer.pos, fewer.typ = s.pos[:-1], s.typ[:-1]
    one = copy.copy(s)  # all atoms of one type: type 1 and its channels are gone
    one.typ = np.zeros_like(s.typ)
    one.tab = dict(s.tab, q=s.tab["q"][:1], vps=s.tab["vps"][:1], gzvps=s.tab["gzvps"][:1])
    psi, occ = s.psi(), torch.ones(s.nstates, dtype=torch.float64, device="cuda")
    ctx = StepContext(s.layout, s.nstates, precision="fp64")
    try:
        ctx.set_atoms(s)
        ctx.set_nonlocal(s)
        e0 = float(ctx.ees_nonlocal(psi, occ)[1][7])
        for t in (fewer, one):
            ctx.set_atoms(t)
            with pytest.raises(_lib.CpstepError) as err:
                ctx.ees_nonlocal(psi, occ)
            assert err.value.code == 5 and "atoms changed" in str(err.value)
            ctx.set_atoms(s)
            assert float(ctx.ees_nonlocal(psi, occ)[1][7]) == e0
    finally:
        ctx.close()


def test_mixed_atom_forces_do_not_lose_with_states():
    """Mixed atom forces at 256 states, where one accumulator takes the whole sum over
    the states, and at 257, 512, 513 and 1030, where two, a full pair and further
    pairs do: an accumulator never takes more than 256, so the relative error
    against FP64 stays that of 256 states.  144 force components scatter an error's
    norm by 1 / sqrt(288) = 6 %, a ratio of two by 8 %: at most 1.3."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.system import System
    s = System(12.0, 25.0, 8, {"O": 16, "H": 32}, nfft=40, seed=5)
    g = torch.Generator(device="cuda").manual_seed(4)
    psi = torch.view_as_complex(torch.randn((1030, s.layout.npts, 2), generator=g,
                                            dtype=torch.float64, device="cuda"))
    psi /= 8.0  # the mixed operands' FP16 levels hold |psi| < 4 (else a device error)
    err = {}
    for states in (256, 257, 512, 513, 1030):
        occ = torch.ones(states, dtype=torch.float64, device="cuda")
        f = []
        for precision in ("mixed", "fp64"):
            ctx = StepContext(s.layout, states, precision=precision)
            try:
                ctx.set_atoms(s)
                ctx.set_nonlocal(s)
                f.append(ctx.ees_nonlocal(psi[:states], occ)[2].cpu().numpy())
                assert ctx.device_errors() == 0
            finally:
                ctx.close()
        err[states] = np.linalg.norm(f[0] - f[1]) / np.linalg.norm(f[1])
    assert max(err.values()) <= 1.3 * err[256], err


@pytest.mark.parametrize("states,gspace", [(1, False), (8, False), (64, True), (128, True)])
def test_fp64_form_follows_the_states(states, gspace):
    """195 atoms: the G-space products pay for whole tiles of states, so few states
    take the NL-grid form (8 states: 0.9 ms against 1.6) and many the G-space one
    (128: 3.4 ms against 8.9).  The form is told by the kernels of a pass."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.system import System
    s = System(23.5, 70.0, states, {"O": 65, "H": 130}, nfft=128, seed=5)
    g = torch.Generator(device="cuda").manual_seed(states)
    psi = torch.view_as_complex(torch.randn((states, s.layout.npts, 2), generator=g,
                                            dtype=torch.float64, device="cuda"))
    occ = torch.ones(states, dtype=torch.float64, device="cuda")
    ctx = StepContext(s.layout, states, precision="fp64")
    try:
        ctx.set_atoms(s)
        ctx.set_nonlocal(s)
        n = _launches(ctx, psi, occ)
        ctx.tune_set({"ees_gspace": 0})
        ngrid = _launches(ctx, psi, occ)
        assert ngrid > 3 * len(s.channels)  # projection, sums and force of each channel
        assert (n < ngrid) == gspace and (gspace or n == ngrid)
    finally:
        ctx.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_three_types_with_projectors(precision):
    """Three types with projectors, two of them the same element: the mixed pass takes
    the types two at a time, with psi's transposed levels kept from the first pair.
    The sums are those of the two-type system in another order: FP64 to 1e-11 of the
    largest entry, mixed to the module's 1e-5, and the mixed pass to FP64 as well."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import copy
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.system import System
    s = System(12.0, 25.0, 37, {"O": 9, "H": 20}, nfft=40, seed=5)
    t = copy.copy(s)
    t.typ = np.array(s.typ)
    t.typ[np.nonzero(t.typ == 0)[0][::2]] = 2
    t.tab = dict(s.tab)
    for k in ("q", "vps", "gzvps"):
        t.tab[k] = np.concatenate([s.tab[k], s.tab[k][:1]])
    t.channels = s.channels + [dict(c, type=2) for c in s.channels if c["type"] == 0]
    psi = s.psi()
    occ = 1.0 + torch.arange(37, dtype=torch.float64, device="cuda") % 2
    out = []
    for system, prec in ((s, "fp64"), (s, precision), (t, precision)):
        ctx = StepContext(s.layout, 37, precision=prec)
        try:
            ctx.set_atoms(system)
            ctx.set_nonlocal(system)
            f, e, fa = ctx.ees_nonlocal(psi, occ, fpsi=0.1 * psi)
            out.append((e[7:8].cpu().numpy(), f.cpu().numpy(), fa.cpu().numpy()))
            f2, e2, _ = ctx.ees_nonlocal(psi, occ, fpsi=0.1 * psi, forces=False)
            assert bool((f2 == f).all()) and bool((e2[7] == e[7]).all())
            assert ctx.device_errors() == 0
        finally:
            ctx.close()
    tol = 1e-11 if precision == "fp64" else 1e-5
    for a, b, c in zip(*out):
        assert np.max(np.abs(c - b)) <= tol * np.max(np.abs(b)) and np.max(np.abs(b)) > 0.0
        assert np.max(np.abs(c - a)) <= tol * np.max(np.abs(a))
