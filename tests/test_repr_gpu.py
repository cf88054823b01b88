"""FCHL19 descriptors and Jacobians on the GPU (kfb_fchl19_repr) against the
reference's own outputs (tests/golden/golden_repr.npz) and the torch restatement.
FP64: X at rtol 1e-10, Jacobians at 1e-9 of their largest entry (both sides are
analytic); float32 storage (cuda_fchl19_repr): 1e-5."""
import ast
import math

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def golden():
    g = load_golden("golden_repr.npz")
    return g, ast.literal_eval(str(g["nondefault"]))


def close_x(got, ref, rtol=1e-10):
    np.testing.assert_allclose(got, ref, rtol=rtol, atol=rtol * max(1e-3, np.abs(ref).max()))


def close_g(got, ref, tol=1e-9):
    np.testing.assert_allclose(got, ref, rtol=tol, atol=tol * max(1e-3, np.abs(ref).max()))


@pytest.mark.parametrize("c", range(6))
def test_golden_default(c):
    from kernelforge_b200 import fchl19_repr as fr
    g, _ = golden()
    R, Z = g[f"d{c}_R"], g[f"d{c}_Z"]
    X = fr.generate_fchl_acsf(R, Z)
    assert X.shape == g[f"d{c}_X"].shape and X.dtype == np.float64
    close_x(X, g[f"d{c}_X"])
    X2, J = fr.generate_fchl_acsf_and_gradients(R, Z)
    close_x(X2, g[f"d{c}_X"])
    assert J.shape == g[f"d{c}_G"].shape
    close_g(J, g[f"d{c}_G"])


@pytest.mark.parametrize("c", range(3))
def test_golden_nondefault(c):
    from kernelforge_b200 import fchl19_repr as fr
    g, nd = golden()
    X, J = fr.generate_fchl_acsf_and_gradients(g[f"n{c}_R"], g[f"n{c}_Z"], **nd)
    close_x(X, g[f"n{c}_X"])
    close_g(J, g[f"n{c}_G"])


def test_golden_nfourier2():
    from kernelforge_b200 import fchl19_repr as fr
    g, _ = golden()
    X = fr.generate_fchl_acsf(g["f_R"].reshape(-1), g["f_Z"], elements=[1, 6, 7, 8],
                              nFourier=2)
    close_x(X, g["f_X"])


def test_batched_padding_and_float32():
    """Several molecules in one launch, padded; float32 storage through the
    torch-facing module with element indices."""
    import torch
    from kernelforge_b200 import cuda_fchl19_repr as cr
    from kernelforge_b200 import fchl19_repr as fr
    g, _ = golden()
    mols = [(g[f"d{c}_R"], g[f"d{c}_Z"]) for c in (2, 3, 4, 5)]
    nm, ma = len(mols), max(len(z) for _, z in mols)
    C = np.zeros((nm, ma, 3))
    Zp = np.zeros((nm, ma), np.int32)
    N = np.array([len(z) for _, z in mols], np.int32)
    for m, (R, Z) in enumerate(mols):
        C[m, :len(Z)] = R
        Zp[m, :len(Z)] = Z
    X, dX = fr.generate_batched(C, Zp, N, gradients=True, dtype="float64")
    X, dX = X.cpu().numpy(), dX.cpu().numpy()
    for m, (R, Z) in enumerate(mols):
        n = len(Z)
        close_x(X[m, :n], g[f"d{[2, 3, 4, 5][m]}_X"])
        close_g(dX[m, :n, :, :3 * n], g[f"d{[2, 3, 4, 5][m]}_G"])
        assert not X[m, n:].any() and not dX[m, n:].any() and not dX[m, :, :, 3 * n:].any()
    lut = {e: k for k, e in enumerate((1, 6, 7, 8, 16))}
    Q = np.vectorize(lambda z: lut.get(int(z), 0))(Zp).astype(np.int32)
    ct = torch.tensor(C, dtype=torch.float32, device="cuda")
    rep, grad = cr.generate_fchl_acsf_and_gradients(
        ct, torch.tensor(Q, device="cuda"), torch.tensor(N, device="cuda"), 5)
    assert rep.dtype == torch.float32 and tuple(grad.shape) == (nm, ma, 720, ma, 3)
    # float32 coordinates: compare with the FP64 result on the same rounded coordinates
    X32, dX32 = fr.generate_batched(C.astype(np.float32).astype(np.float64), Zp, N,
                                    gradients=True, dtype="float64")
    close_x(rep.double().cpu().numpy(), X32.cpu().numpy(), 1e-5)
    close_g(grad.double().cpu().numpy().reshape(dX32.shape), dX32.cpu().numpy(), 1e-5)
    rep2 = cr.generate_fchl_acsf(ct, torch.tensor(Q, device="cuda"),
                                 torch.tensor(N, device="cuda"), 5)
    assert torch.equal(rep2, rep)


def test_against_restatement_and_finite_differences():
    """A 16-atom molecule: the torch restatement (autograd) and central finite
    differences of the GPU descriptor itself."""
    import torch
    from kernelforge_b200 import fchl19_repr as fr
    from kernelforge_b200 import synthetic
    mols = synthetic.make_molecules(1, 16, 16, seed=5)
    R, Z = mols.R[0], mols.Z[0]
    X, J = fr.generate_fchl_acsf_and_gradients(R, Z)
    zi = synthetic._zidx(Z)
    f = lambda r: synthetic._fchl19_one(r, zi)
    Rt = torch.tensor(R, dtype=torch.float64)
    close_x(X, f(Rt).numpy())
    close_g(J, torch.func.jacfwd(f)(Rt).numpy().reshape(J.shape))
    h = 1e-5
    for a, t in [(0, 0), (7, 1), (15, 2)]:
        Rp, Rm = R.copy(), R.copy()
        Rp[a, t] += h
        Rm[a, t] -= h
        fd = (fr.generate_fchl_acsf(Rp, Z) - fr.generate_fchl_acsf(Rm, Z)) / (2 * h)
        np.testing.assert_allclose(J[:, :, 3 * a + t], fd, rtol=1e-5,
                                   atol=1e-6 * np.abs(J).max())


@pytest.mark.parametrize("n", [1, 2, 9, 20, 33, 41])
@pytest.mark.parametrize("hyper", [{}, dict(nRs2=7, nRs3=5, rcut=3.0, acut=2.5)])
def test_row_wise_gradients_match_large_molecule_kernel(n, hyper):
    """Up to 41 padded atoms the Jacobian rows come from shared-memory pair terms, above from the
    kernel that forms them as it goes: the same molecules padded to 41 and to 42 atoms.  Both sum
    the same FP64 terms in another order (1e-13 of the largest entry); atoms beyond the cutoffs,
    elements that one or no atom has, partial row groups."""
    import torch
    from kernelforge_b200 import fchl19_repr as fr
    rng = np.random.default_rng(n)
    nm = 3
    C = np.zeros((nm, 42, 3))
    Z = np.zeros((nm, 42), np.int32)
    grid = np.stack(np.meshgrid(*[np.arange(4)] * 3), -1).reshape(-1, 3) * 1.3
    for m in range(nm):
        C[m, :n] = grid[rng.permutation(64)[:n]] + rng.uniform(-0.2, 0.2, (n, 3))
        Z[m, :n] = rng.choice([[1], [1, 6], [1, 6, 8, 16]][m], n)
    N = np.array([n, n, max(n - 1, 0)], np.int32)
    out = []
    for ma in (41, 42):
        X, dX = fr.generate_batched(C[:, :ma], Z[:, :ma], N, gradients=True, dtype="float64",
                                    **hyper)
        assert not dX[:, :, :, 3 * n:].any() and not X[2, N[2]:].any()
        out.append((X[:, :41].cpu().numpy(), dX[:, :41, :, :123].cpu().numpy()))
    for a, b in zip(*out):
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-13 * max(1e-3, np.abs(b).max()))


def test_edge_cases_and_errors():
    from kernelforge_b200 import fchl19_repr as fr
    X, J = fr.generate_fchl_acsf_and_gradients(np.zeros((1, 3)), [6])
    assert X.shape == (1, 720) and not X.any() and J.shape == (1, 720, 3) and not J.any()
    with pytest.raises(RuntimeError):
        fr.generate_fchl_acsf(np.zeros((2, 3)) + [[0, 0, 0], [1, 0, 0]], [6, 9])
    with pytest.raises(ValueError):
        fr.generate_fchl_acsf(np.zeros((3, 2)), [1, 1, 1])
    with pytest.raises(ValueError):
        fr.generate_fchl_acsf(np.zeros((0, 3)), [])
    with pytest.raises(ValueError):
        fr.generate_fchl_acsf_and_gradients(np.eye(3), [1, 1, 1], nFourier=2)
    assert fr.compute_rep_size(5, 24, 20, 2) == 720


@pytest.mark.parametrize("far", [50.0, 1e30, 1e200, np.inf, np.nan])
def test_atoms_beyond_every_cutoff(far):
    """An atom beyond the cutoffs, also at a distance whose square is no FP64 number: the others'
    descriptors and Jacobians are those of the molecule without it.  One at no finite place
    leaves their descriptors (not their Jacobians) as they are."""
    from kernelforge_b200 import fchl19_repr as fr
    rng = np.random.default_rng(3)
    n = 9
    grid = np.stack(np.meshgrid(*[np.arange(3)] * 3), -1).reshape(-1, 3) * 1.3
    C = np.zeros((1, n + 1, 3))
    C[0, :n] = grid[:n] + rng.uniform(-0.2, 0.2, (n, 3))
    C[0, n, 1] = far
    Z = rng.choice([1, 6, 8], (1, n + 1)).astype(np.int32)
    Z[0, n] = 6
    kw = dict(gradients=True, dtype="float64")
    X, dX = (t.cpu().numpy() for t in fr.generate_batched(C, Z, np.array([n + 1], np.int32), **kw))
    X0, dX0 = (t.cpu().numpy() for t in fr.generate_batched(C, Z, np.array([n], np.int32), **kw))
    # (the atoms of an element are added up in an order that does not depend on the far one)
    np.testing.assert_allclose(X[0, :n], X0[0, :n], rtol=0, atol=1e-15 * np.abs(X0).max())
    if np.isfinite(far):
        np.testing.assert_allclose(dX[0, :n], dX0[0, :n], rtol=0, atol=1e-15 * np.abs(dX0).max())
    V = fr.generate_batched(C, Z, np.array([n + 1], np.int32), dtype="float64").cpu().numpy()
    np.testing.assert_allclose(X[0, :n], V[0, :n], rtol=0, atol=1e-13 * np.abs(X0).max())
    if np.isfinite(far):
        assert not X[0, n].any() and not dX[0, n].any()


@pytest.mark.parametrize("n", [42, 57])
def test_large_molecules(n):
    """More atoms than the row-wise kernel takes: descriptors as the kernel without gradients
    gives them, Jacobians against central finite differences of those (h = 1e-5: 1e-10 of the
    values' rounding over h, and h^2 times third derivatives), rows that sum to zero."""
    from kernelforge_b200 import fchl19_repr as fr
    rng = np.random.default_rng(n)
    grid = np.stack(np.meshgrid(*[np.arange(4)] * 3), -1).reshape(-1, 3) * 1.4
    R = grid[rng.permutation(64)[:n]] + rng.uniform(-0.2, 0.2, (n, 3))
    Z = rng.choice([1, 6, 7, 8, 16], n).astype(np.int32)
    X, J = fr.generate_fchl_acsf_and_gradients(R, Z)
    X0 = fr.generate_fchl_acsf(R, Z)
    np.testing.assert_allclose(X, X0, rtol=0, atol=1e-13 * np.abs(X0).max())
    J = J.reshape(n, -1, n, 3)
    assert np.abs(J.sum(2)).max() <= 1e-12 * np.abs(J).max()
    h = 1e-5
    for a, t in [(0, 0), (n // 2, 1), (n - 1, 2)]:
        Rp, Rm = R.copy(), R.copy()
        Rp[a, t] += h
        Rm[a, t] -= h
        fd = (fr.generate_fchl_acsf(Rp, Z) - fr.generate_fchl_acsf(Rm, Z)) / (2 * h)
        np.testing.assert_allclose(J[:, :, a, t], fd, rtol=1e-5, atol=1e-6 * np.abs(J).max())


def test_coincident_atoms_without_a_triple():
    """Two atoms at one place, the others beyond the cutoff of both: their pair terms are
    undefined, the three-body rows, which hold no triple, are zero."""
    from kernelforge_b200 import fchl19_repr as fr
    R = np.array([[[0, 0, 0], [2, 0, 0], [2, 0, 0], [0, 1, 0]]], float)
    Z = np.array([[1, 6, 6, 8]], np.int32)
    X, dX = fr.generate_batched(R, Z, np.array([4], np.int32), gradients=True, dtype="float64",
                                rcut=1.0, acut=1.0)
    assert not X[..., 120:].any() and not dX[:, :, 120:].any()
    assert not np.isfinite(X[0, 1, 24:48].cpu().numpy()).any()
