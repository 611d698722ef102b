"""PairCalculator products and the Ortho S -> T iteration on the GPU vs the oracle."""
import numpy as np
import pytest

from conftest import cuda_ok

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pc():
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.layout import StateLayout
    from openatom_b200.system import make_psi
    lay = StateLayout(12.0, 30.0)
    S = 37  # not a tile multiple
    psi = make_psi(lay, S, seed=21, device="cuda")
    g = torch.Generator(device="cpu").manual_seed(2)
    f = (torch.randn((S, lay.npts), generator=g, dtype=torch.float64)
         + 1j * torch.randn((S, lay.npts), generator=g, dtype=torch.float64)).to(torch.complex128).cuda()
    ctx = StepContext(lay, S, precision="fp64")
    yield dict(lay=lay, psi=psi, f=f, ctx=ctx, S=S)
    ctx.close()


def colmajor(t):
    return t.cpu().numpy().T  # tensors hold column-major matrices as [ncol][ld]


def test_overlap_symmetric_matches_oracle(pc):
    from oracle import ortho as OO
    out = pc["ctx"].pc_overlap(pc["psi"], pc["psi"])
    ref = OO.pc_overlap(pc["psi"].cpu().numpy(), pc["psi"].cpu().numpy(), pc["lay"].kx)
    assert np.max(np.abs(colmajor(out) - ref)) < 1e-12
    # orthonormalised input: S = 2 I
    assert np.max(np.abs(ref - 2.0 * np.eye(pc["S"]))) < 1e-10


def test_overlap_asymmetric_lambda_matches_oracle(pc):
    from oracle import ortho as OO
    out = pc["ctx"].pc_overlap(pc["psi"], pc["f"])
    ref = OO.pc_overlap(pc["psi"].cpu().numpy(), pc["f"].cpu().numpy(), pc["lay"].kx)
    assert np.max(np.abs(colmajor(out) - ref)) / np.max(np.abs(ref)) < 1e-13


def test_overlap_alpha_beta(pc):
    from oracle import ortho as OO
    import torch
    c0 = torch.ones((pc["S"], pc["S"]), dtype=torch.float64, device="cuda")
    out = pc["ctx"].pc_overlap(pc["psi"], pc["f"], alpha=-0.5, beta=2.0, out=c0)
    ref = -0.5 * OO.pc_overlap(pc["psi"].cpu().numpy(), pc["f"].cpu().numpy(), pc["lay"].kx) + 2.0
    assert np.max(np.abs(colmajor(out) - ref)) < 1e-11


def test_backmultiply_matches_oracle(pc):
    import torch
    S = pc["S"]
    rng = np.random.default_rng(4)
    M = rng.standard_normal((S, S))  # column-major matrix M(j,i) = M[j, i]
    Mt = torch.from_numpy(np.ascontiguousarray(M.T)).cuda()  # [col][row] storage
    out = pc["ctx"].pc_backmultiply(Mt, pc["psi"], alpha=1.0, beta=0.0)
    ref = M.T @ pc["psi"].cpu().numpy()
    assert np.max(np.abs(out.cpu().numpy() - ref)) / np.max(np.abs(ref)) < 1e-13
    out2 = pc["ctx"].pc_backmultiply(Mt, pc["psi"], alpha=-1.0, beta=1.0, out=pc["f"].clone())
    ref2 = pc["f"].cpu().numpy() - ref
    assert np.max(np.abs(out2.cpu().numpy() - ref2)) / np.max(np.abs(ref2)) < 1e-13


def test_dgemm_all_transposes(pc):
    import torch
    rng = np.random.default_rng(8)
    m, n, k = 45, 70, 33
    for ta in "NT":
        for tb in "NT":
            A = rng.standard_normal((m, k) if ta == "N" else (k, m))
            B = rng.standard_normal((k, n) if tb == "N" else (n, k))
            C = rng.standard_normal((m, n))
            opA = A if ta == "N" else A.T
            opB = B if tb == "N" else B.T
            ref = 1.5 * opA @ opB - 0.5 * C
            dA = torch.from_numpy(np.asfortranarray(A).T.copy()).cuda()
            dB = torch.from_numpy(np.asfortranarray(B).T.copy()).cuda()
            dC = torch.from_numpy(np.asfortranarray(C).T.copy()).cuda()
            pc["ctx"].dgemm(ta, tb, m, n, k, 1.5, dA, A.shape[0], dB, B.shape[0], -0.5, dC, m)
            assert np.max(np.abs(dC.cpu().numpy().T - ref)) < 1e-12


@pytest.mark.parametrize("n,lo,hi", [(37, 1.7, 2.3), (128, 0.5, 2.0)])
def test_ortho_fp64_matches_oracle(pc, n, lo, hi):
    import torch
    from oracle import ortho as OO
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    S = (Q * np.exp(rng.uniform(np.log(lo), np.log(hi), n))) @ Q.T
    S = 0.5 * (S + S.T)
    T, it, rms = pc["ctx"].ortho_tmat(torch.from_numpy(S).cuda(), tol=1e-14, max_iter=12)
    To, ito, _ = OO.schulz_tmat(S, tol=1e-14, max_iter=12)
    T = T.cpu().numpy()
    assert np.max(np.abs(T - To)) < 1e-12
    assert np.max(np.abs(T @ (S / 2) @ T - np.eye(n))) < 1e-12


@pytest.mark.parametrize("lo,hi,scale", [(1.6, 2.4, False), (0.5, 2.0, False), (0.05, 5.0, True)])
def test_ortho_mixed_is_orthonormal_to_fp64(pc, lo, hi, scale):
    import torch
    n = 96
    rng = np.random.default_rng(7)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    S = (Q * np.exp(rng.uniform(np.log(lo), np.log(hi), n))) @ Q.T
    S = 0.5 * (S + S.T)
    T, it, rms = pc["ctx"].ortho_tmat(torch.from_numpy(S).cuda(), mixed=True, scale=scale,
                                      tol=2e-6, max_iter=40)
    T = T.cpu().numpy()
    # |T^T (S/2) T - I| at FP64 rounding after the FP64 correction
    assert np.max(np.abs(T.T @ (S / 2) @ T - np.eye(n))) < 1e-12
    w, V = np.linalg.eigh(S / 2)
    Z = (V * w ** -0.5) @ V.T
    assert np.max(np.abs(T - Z)) < 1e-4


def test_ortho_reports_non_convergence(pc):
    import torch
    from openatom_b200 import _lib
    S = torch.diag(torch.tensor([0.05, 2.0, 5.0], dtype=torch.float64)).cuda()
    with pytest.raises(_lib.CpstepError) as e:
        pc["ctx"].ortho_tmat(S)
    assert e.value.code == _lib.CPSTEP_ERR_NOCONV


@pytest.mark.parametrize("na,nb", [(1, 1), (32, 33), (64, 64), (65, 64), (64, 65), (128, 129), (200, 3)])
def test_fp64_product_tile_edges(na, nb):
    """The FP64 products at the edges of their tiles (32 rows per warp, 64 and 128
    per block; ragged K), a operand equal to or other than b, an odd leading
    dimension, an output that is only 8-byte aligned.  K = 2 npts terms of
    order 1, so rounding stays below eps K = 2.6e-13 of the largest entry: 1e-12."""
    if not cuda_ok():
        pytest.skip("no CUDA device")
    import torch
    from openatom_b200.context import StepContext
    from openatom_b200.layout import StateLayout
    from oracle import ortho as OO
    lay = StateLayout(9.0, 20.0, nfft=28)
    g = torch.Generator(device="cuda").manual_seed(na * 1000 + nb)
    mk = lambda n: torch.view_as_complex(torch.randn((n, lay.npts, 2), generator=g,
                                                     dtype=torch.float64, device="cuda"))
    a, b = mk(na), mk(nb)
    ctx = StepContext(lay, max(na, nb), precision="fp64")
    try:
        out = ctx.pc_overlap(a, b)
        ref = OO.pc_overlap(a.cpu().numpy(), b.cpu().numpy(), lay.kx)
        assert np.max(np.abs(colmajor(out) - ref)) <= 1e-12 * np.max(np.abs(ref))
        s = ctx.pc_overlap(a, a)
        assert bool((s == s.t()).all())
        refs = OO.pc_overlap(a.cpu().numpy(), a.cpu().numpy(), lay.kx)
        assert np.max(np.abs(s.cpu().numpy() - refs)) <= 1e-12 * np.max(np.abs(refs))
        M = torch.randn((nb, na + 1), generator=g, dtype=torch.float64, device="cuda")
        want = (M[:, :na].cpu().numpy() @ a.cpu().numpy())
        got = ctx.pc_backmultiply(M, a, nout=nb)
        assert np.max(np.abs(got.cpu().numpy() - want)) <= 1e-12 * np.max(np.abs(want))
        buf = torch.ones(2 * nb * lay.npts + 1, dtype=torch.float64, device="cuda")
        odd = buf[1:]  # 8 bytes past a 16-byte boundary
        ctx.pc_backmultiply(M, a, nout=nb, alpha=-2.0, beta=3.0, out=odd)
        want2 = 3.0 * (1 + 1j) - 2.0 * want
        got2 = odd.cpu().numpy().view(np.complex128).reshape(nb, -1)
        assert np.max(np.abs(got2 - want2)) <= 1e-12 * np.max(np.abs(want2))
    finally:
        ctx.close()


@pytest.mark.parametrize("n", [1, 16, 17, 63, 64, 65, 96, 127, 128, 129, 200])
@pytest.mark.parametrize("mixed", [False, True])
def test_ortho_tile_edges(pc, n, mixed):
    """One block (64 states at most), one K chunk (128) and more, odd and even row
    strides: T (S/2) T = I.  The products have n terms of order 1, rounding
    below n eps = 5e-14 each over four of them: 1e-12."""
    import torch
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    S = (Q * rng.uniform(1.7, 2.3, n)) @ Q.T
    S = 0.5 * (S + S.T)
    T, it, rms = pc["ctx"].ortho_tmat(torch.from_numpy(S).cuda(), mixed=mixed,
                                      tol=2e-6 if mixed else 1e-13, max_iter=12)
    T = T.cpu().numpy()
    assert np.max(np.abs(T.T @ (S / 2) @ T - np.eye(n))) < 1e-12


@pytest.mark.parametrize("n", [1, 33, 64, 65, 130])
@pytest.mark.parametrize("mixed,scale", [(False, False), (False, True), (True, False), (True, True)])
def test_ortho_without_an_iteration(pc, n, mixed, scale):
    """tol >= 1 runs no iteration: T is the starting iterate I times (sigma/2)^(-1/2),
    in the mixed mode with the correction X (I - R/2 + 3 R^2/8), R = X (S/2) X - I,
    whatever an earlier call left in the workspace.  At most 130 terms of order 1
    in three products: 1e-12."""
    import torch
    rng = np.random.default_rng(n)
    R = rng.standard_normal((n, n)) / (20.0 * np.sqrt(n))
    S = 2.0 * np.eye(n) + R + R.T
    d = torch.from_numpy(S).cuda()
    pc["ctx"].ortho_tmat(d, mixed=mixed, scale=True, tol=2e-6, max_iter=40)
    T, it, rms = pc["ctx"].ortho_tmat(d, mixed=mixed, scale=scale, tol=1.0, max_iter=10)
    sigma = max(2.0, 1.0001 * np.abs(S).sum(1).max()) if scale else 2.0
    want = np.eye(n) * np.sqrt(2.0 / sigma)
    if mixed:
        E = want @ (S / 2) @ want - np.eye(n)
        want = want @ (np.eye(n) - 0.5 * E + 0.375 * E @ E)
    assert it == 0 and rms == 1.0
    assert np.max(np.abs(T.cpu().numpy() - want)) < 1e-12


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (32, 33, 15), (31, 32, 128), (64, 1, 129), (97, 65, 16),
                                   (128, 128, 300)])
def test_dgemm_tile_edges(pc, m, n, k):
    """Edges of the 32 x 32 tiles, of a warp's 16 and a chunk's 128 of K, leading
    dimensions beyond the matrices, beta = 0 over NaN.  At most 300 terms of
    order 1: rounding below 300 eps times a few: 1e-12."""
    import torch
    rng = np.random.default_rng(m * 1000 + n)
    for ta in "NT":
        for tb in "NT":
            A = rng.standard_normal((m + 3, k) if ta == "N" else (k + 3, m))
            B = rng.standard_normal((k + 5, n) if tb == "N" else (n + 5, k))
            opA = A[:m] if ta == "N" else A[:k].T
            opB = B[:k] if tb == "N" else B[:n].T
            dA, dB = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (A, B))
            dC = torch.full((n, m + 1), float("nan"), dtype=torch.float64, device="cuda")
            pc["ctx"].dgemm(ta, tb, m, n, k, -0.5, dA, A.shape[0], dB, B.shape[0], 0.0, dC, m + 1)
            got = dC.cpu().numpy()
            assert np.max(np.abs(got[:, :m].T + 0.5 * opA @ opB)) < 1e-12
            assert np.isnan(got[:, m]).all()
