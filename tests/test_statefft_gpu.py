"""State FFT path on the GPU (through the C ABI) against the FP64 oracle.

Tolerances (relative to the largest magnitude of the oracle result):
FP64 path 1e-11; mixed path (FP32 FFTs, FP64 accumulation) 2e-5.
"""
import numpy as np
import pytest

from conftest import cuda_ok

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-11, "mixed": 2e-5}
# (box bohr, ecut Ry, grid) -> grids 28, 42 (reference radixme), 48 (grid override);
# 32, 64, 80, 96 and 128 run the register (shuffle) plane FFTs
CASES = [(9.0, 20.0, None), (12.0, 30.0, None), (12.0, 30.0, 48), (9.0, 20.0, 32),
         (12.0, 30.0, 64), (12.0, 30.0, 80), (12.0, 30.0, 96), (12.0, 30.0, 128)]


def relerr(a, b):
    a = np.asarray(a)
    b = np.asarray(b)
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


@pytest.fixture(scope="module", params=CASES, ids=lambda c: "L%g_E%g_n%s" % c)
def system(request):
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from oracle import layout as OL
    from openatom_b200.layout import StateLayout
    from openatom_b200.system import make_psi
    box, ecut, grid = request.param
    lay = StateLayout(box, ecut, nfft=grid)
    olay = OL.Layout(box, ecut, grid=grid)
    assert np.array_equal(lay.kx, olay.kx)
    S = 6
    psi = make_psi(lay, S, seed=5, device="cuda")
    occ = torch.tensor([1.0, 1.0, 0.5, 1.0, 0.25, 1.0], dtype=torch.float64, device="cuda")
    return dict(lay=lay, olay=olay, psi=psi, occ=occ, S=S)


@pytest.fixture(params=["fp64", "mixed"])
def ctx(request, system):
    from openatom_b200.context import StepContext
    c = StepContext(system["lay"], system["S"], precision=request.param)
    yield c
    c.close()


def test_expand_pack_roundtrip(system, ctx):
    from oracle import fftpath as OF
    psi = system["psi"]
    lines = ctx.expand_gspace(psi)
    ref = OF.expand(psi.cpu().numpy(), system["olay"])
    assert np.array_equal(lines.cpu().numpy(), ref)
    back = ctx.pack_gspace(lines)
    assert np.array_equal(back.cpu().numpy(), psi.cpu().numpy())


def test_g_to_r_matches_oracle(system, ctx):
    from oracle import fftpath as OF
    pr = ctx.fft_g_to_r(system["psi"]).cpu().numpy()
    ref = OF.state_g_to_r(system["psi"].cpu().numpy(), system["olay"])
    assert relerr(pr, ref) < TOL[ctx.precision]


def test_r_to_g_matches_oracle(system, ctx):
    import torch
    from oracle import fftpath as OF
    n = system["lay"].n
    g = torch.Generator(device="cpu").manual_seed(3)
    f = torch.randn((system["S"], n, n, n), generator=g, dtype=torch.float64)
    out = ctx.fft_r_to_g(f.cuda()).cpu().numpy()
    ref = OF.state_r_to_g(f.numpy(), system["olay"])
    assert relerr(out, ref) < TOL[ctx.precision]


def test_density_matches_oracle(system, ctx):
    from oracle import fftpath as OF
    rho = ctx.density(system["psi"], system["occ"]).cpu().numpy()
    lay = system["lay"]
    ref = OF.density(system["psi"].cpu().numpy(), system["olay"], system["occ"].cpu().numpy(),
                     lay.vol)
    assert relerr(rho, ref) < TOL[ctx.precision]
    # electron count: states normalised to 2 (S = 2 I)
    nel = rho.sum() * lay.vol / lay.n ** 3
    assert abs(nel - 2.0 * float(system["occ"].sum())) < 1e-9 * nel + (1e-5 if ctx.precision == "mixed" else 0)


def test_vks_psi_and_kinetic_match_oracle(system, ctx):
    import torch
    from oracle import fftpath as OF
    lay = system["lay"]
    n = lay.n
    g = torch.Generator(device="cpu").manual_seed(9)
    vks = torch.randn((n, n, n), generator=g, dtype=torch.float64)
    psi = system["psi"]
    occ = system["occ"]
    force, eke = ctx.vks_psi(psi, vks.cuda(), occ, kinetic=True)
    pn, on = psi.cpu().numpy(), occ.cpu().numpy()
    fv = OF.vpsi_force(pn, vks.numpy(), system["olay"], on)
    f_ref = OF.add_forces(fv, None, system["olay"])
    f_ref, e_ref = OF.eke(f_ref, pn, system["olay"], on, lay.ecut_ry)
    assert relerr(force.cpu().numpy(), f_ref) < TOL[ctx.precision]
    assert relerr(eke.cpu().numpy(), e_ref) < 1e-12


def test_eke_entry_matches_oracle(system, ctx):
    import torch
    from oracle import fftpath as OF
    psi = system["psi"]
    occ = system["occ"]
    f0 = torch.zeros_like(psi)
    e = ctx.eke(f0, psi, occ)
    f_ref, e_ref = OF.eke(np.zeros(psi.shape, complex), psi.cpu().numpy(), system["olay"],
                          occ.cpu().numpy(), system["lay"].ecut_ry)
    assert relerr(f0.cpu().numpy(), f_ref) < 1e-13
    assert relerr(e.cpu().numpy(), e_ref) < 1e-13


def test_adjointness_of_the_two_transforms(system, ctx):
    """<F(psi), f> = sum_r psi(r) f(r) with the double-pack weights (size independent)."""
    import torch
    lay = system["lay"]
    n = lay.n
    psi = system["psi"]
    g = torch.Generator(device="cpu").manual_seed(4)
    f = torch.randn((system["S"], n, n, n), generator=g, dtype=torch.float64).cuda()
    pr = ctx.fft_g_to_r(psi)
    lhs = (pr * f).sum(dim=(1, 2, 3))
    Fg = ctx.fft_r_to_g(f)
    w = torch.from_numpy(np.where(lay.kx == 0, 1.0, 2.0)).cuda()
    rhs = (w[None] * (psi.conj() * Fg).real).sum(dim=1)
    tol = 1e-10 if ctx.precision == "fp64" else 1e-4
    assert float((lhs - rhs).abs().max() / lhs.abs().max()) < tol


@pytest.mark.parametrize("form", [0, 1, 2])
def test_plane_pass_forms_match_oracle(system, form):
    """Density and V.psi in a mixed context with each plane-pass form: 0
    shared-memory Stockham, 1 register shuffles, 2 the two-stage form."""
    import torch
    from oracle import fftpath as OF
    from openatom_b200.context import StepContext
    lay, olay = system["lay"], system["olay"]
    psi, occ = system["psi"], system["occ"]
    ctx = StepContext(lay, system["S"], precision="mixed")
    try:
        ctx.tune_set({"plane_shfl": form})
        pn, on = psi.cpu().numpy(), occ.cpu().numpy()
        rho = ctx.density(psi, occ).cpu().numpy()
        ref = OF.density(pn, olay, on, lay.vol)
        assert relerr(rho, ref) < TOL["mixed"]
        n = lay.n
        g = torch.Generator(device="cpu").manual_seed(9)
        vks = torch.randn((n, n, n), generator=g, dtype=torch.float64)
        force, eke = ctx.vks_psi(psi, vks.cuda(), occ, kinetic=True)
        fv = OF.vpsi_force(pn, vks.numpy(), olay, on)
        f_ref = OF.add_forces(fv, None, olay)
        f_ref, e_ref = OF.eke(f_ref, pn, olay, on, lay.ecut_ry)
        assert relerr(force.cpu().numpy(), f_ref) < TOL["mixed"]
        assert ctx.device_errors() == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("form", [0, 2])
def test_plane_pass_forms_n200(form):
    """The 200^3 grid (the largest benchmark system's): density and V.psi in a mixed
    context with the shared-memory Stockham form (0) and the two-stage 20 x 10 form
    (2), against the oracle."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from oracle import fftpath as OF
    from oracle import layout as OL
    from openatom_b200.context import StepContext
    from openatom_b200.layout import StateLayout
    from openatom_b200.system import make_psi
    lay = StateLayout(12.0, 30.0, nfft=200)
    olay = OL.Layout(12.0, 30.0, grid=200)
    S = 6
    psi = make_psi(lay, S, seed=5, device="cuda")
    occ = torch.tensor([1.0, 1.0, 0.5, 1.0, 0.25, 1.0], dtype=torch.float64, device="cuda")
    ctx = StepContext(lay, S, precision="mixed")
    try:
        ctx.tune_set({"plane_shfl": form})
        pn, on = psi.cpu().numpy(), occ.cpu().numpy()
        rho = ctx.density(psi, occ).cpu().numpy()
        assert relerr(rho, OF.density(pn, olay, on, lay.vol)) < TOL["mixed"]
        g = torch.Generator(device="cpu").manual_seed(9)
        vks = torch.randn((200, 200, 200), generator=g, dtype=torch.float64)
        force, eke = ctx.vks_psi(psi, vks.cuda(), occ, kinetic=True)
        fv = OF.vpsi_force(pn, vks.numpy(), olay, on)
        f_ref = OF.add_forces(fv, None, olay)
        f_ref, e_ref = OF.eke(f_ref, pn, olay, on, lay.ecut_ry)
        assert relerr(force.cpu().numpy(), f_ref) < TOL["mixed"]
        assert ctx.device_errors() == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("grid,box,states", [
    (28, 9.0, 1), (32, 9.0, 7), (40, 9.0, 33), (42, 9.0, 5), (48, 9.0, 150), (60, 9.0, 3),
    (64, 12.0, 9), (80, 12.0, 4), (96, 12.0, 2), (120, 12.0, 5), (128, 12.0, 3), (200, 12.0, 2)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_two_stage_planes_match_stockham(grid, box, states, precision):
    """Every grid of the two-stage P x Q passes (form 2) against the shared-memory
    Stockham passes (form 0): one state and many (blocks over several planes and
    several blocks per plane), empty and ragged rounds of line tasks.  Both are
    transforms of the same rounding order: the oracle tests' tolerances.  That form 2
    ran is told by its other rounding; 200^3 in FP64 has no two-stage form and runs
    form 0 both times."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.layout import StateLayout
    lay = StateLayout(box, 20.0, nfft=grid)
    g = torch.Generator(device="cuda").manual_seed(grid)
    psi = torch.view_as_complex(torch.randn((states, lay.npts, 2), generator=g,
                                            dtype=torch.float64, device="cuda"))
    occ = 0.5 + torch.arange(states, dtype=torch.float64, device="cuda") % 3
    vks = torch.randn((grid, grid, grid), generator=g, dtype=torch.float64, device="cuda")
    ctx = StepContext(lay, states, precision=precision)
    out = []
    try:
        for form in (2, 0):
            ctx.tune_set({"plane_shfl": form})
            rho = ctx.density(psi, occ).clone()
            force, eke = ctx.vks_psi(psi, vks, occ)
            out.append((rho, torch.view_as_real(force), eke))
        for a, b in zip(*out):
            assert bool(torch.isfinite(a).all())
            assert relerr(a.cpu().numpy(), b.cpu().numpy()) < TOL[precision]
        two = not (precision == "fp64" and grid == 200)
        assert torch.equal(out[0][0], out[1][0]) != two
        assert torch.equal(out[0][1], out[1][1]) != two
    finally:
        ctx.close()


@pytest.mark.parametrize("grid,box,states", [
    (28, 9.0, 3), (32, 9.0, 1), (40, 12.0, 2), (42, 9.0, 7), (48, 12.0, 2), (60, 12.0, 3),
    (64, 12.0, 1), (80, 12.0, 2), (96, 12.0, 1), (120, 12.0, 2), (128, 12.0, 1), (200, 12.0, 1)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_line_and_real_passes_match_oracle(grid, box, states, precision):
    """The z passes and the passes to and from a real array on every grid of the
    two-stage form, with a ragged last block of lines.  The oracle tests'
    tolerances."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from oracle import fftpath as OF
    from oracle import layout as OL
    from openatom_b200.context import StepContext
    from openatom_b200.layout import StateLayout
    lay = StateLayout(box, 20.0, nfft=grid)
    olay = OL.Layout(box, 20.0, grid=grid)
    g = torch.Generator(device="cuda").manual_seed(grid)
    psi = torch.view_as_complex(torch.randn((states, lay.npts, 2), generator=g,
                                            dtype=torch.float64, device="cuda"))
    f = torch.randn((states, grid, grid, grid), generator=g, dtype=torch.float64, device="cuda")
    ctx = StepContext(lay, states, precision=precision)
    try:
        pr = ctx.fft_g_to_r(psi).cpu().numpy()
        assert relerr(pr, OF.state_g_to_r(psi.cpu().numpy(), olay)) < TOL[precision]
        out = ctx.fft_r_to_g(f).cpu().numpy()
        assert relerr(out, OF.state_r_to_g(f.cpu().numpy(), olay)) < TOL[precision]
    finally:
        ctx.close()


@pytest.mark.parametrize("grid,box,ecut,vpsi,density", [
    (28, 8.0, 18.0, 1.937e-08, 8.421e-08), (32, 8.0, 24.0, 2.624e-08, 1.545e-07),
    (40, 8.7, 45.0, 1.938e-08, 1.020e-07), (42, 9.0, 45.0, 2.518e-08, 1.186e-07),
    (48, 10.4, 45.0, 2.996e-08, 1.582e-07), (60, 13.0, 45.0, 1.868e-08, 8.599e-08),
    (64, 13.9, 45.0, 2.937e-08, 1.833e-07), (80, 17.4, 45.0, 2.197e-08, 1.001e-07),
    (96, 20.0, 45.0, 3.896e-08, 2.087e-07), (120, 22.0, 45.0, 1.943e-08, 9.152e-08),
    (128, 23.5, 45.0, 2.925e-08, 1.883e-07)])
def test_fp32_error_by_grid(grid, box, ecut, vpsi, density):
    """Relative error of FP32 V.psi and density against an FP64 context on every
    grid, no larger than the shuffle and Stockham line FFTs had on the same inputs
    (the numbers given).  Some 1e5 rounding errors make up a norm, four draws: it
    scatters by a few tenths of a percent, 1 % is allowed."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.layout import StateLayout
    from openatom_b200.system import make_psi
    lay = StateLayout(box, ecut, nfft=grid)
    ctx = {p: StepContext(lay, 16, precision=p) for p in ("mixed", "fp64")}
    try:
        occ = torch.ones(16, dtype=torch.float64, device="cuda")
        x = torch.arange(grid, dtype=torch.float64, device="cuda") * (2 * np.pi / grid)
        c = torch.cos(x)
        vks = -0.5 + 0.4 * (c[:, None, None] + torch.cos(2 * x)[None, :, None] * c[None, None, :])
        e2 = np.zeros(2)
        for seed in range(4):
            psi = make_psi(lay, 16, seed=seed, device="cuda")
            got, ref = ((torch.view_as_real(k.vks_psi(psi, vks, occ)[0]), k.density(psi, occ))
                        for k in (ctx["mixed"], ctx["fp64"]))
            e2 += [float((a - b).norm() / b.norm()) ** 2 for a, b in zip(got, ref)]
        err = np.sqrt(e2 / 4)
        assert (err > 0.0).all() and (err <= 1.01 * np.array([vpsi, density])).all(), err
    finally:
        for k in ctx.values():
            k.close()
