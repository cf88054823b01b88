"""Contracted energy/force prediction on the GPU (kfb_local_alpha_desc,
kfb_local_matvec) against the reference's golden outputs and the oracle.
FP64 inputs: rtol 1e-10 (the reference's own matvec tests use 1e-8 to 1e-12);
float32 inputs (the torch-facing module): FP64 arithmetic on the rounded
inputs, compared with the oracle on the same rounded inputs at rtol 1e-9 and
the float32 outputs at rtol 1e-6."""
import os

import numpy as np
import pytest

from conftest import load_golden, make_set
from oracle import matvec as om

pytestmark = pytest.mark.gpu


def _case(tag):
    g = load_golden("golden_matvec.npz")
    return {k[len(tag) + 1:]: v for k, v in g.items() if k.startswith(tag + "_")}


def close(got, ref, rtol=1e-10):
    ref = np.asarray(ref)
    np.testing.assert_allclose(got, ref, rtol=rtol, atol=rtol * max(1.0, np.abs(ref).max()))


@pytest.mark.parametrize("tag", ["r", "f"])
def test_golden_alpha_desc(tag):
    from kernelforge_b200 import local_kernels as lk
    c = _case(tag)
    ad = lk.kernel_gaussian_local_compute_alpha_desc(c["dX2"], c["Q2"], c["N2"], c["alpha_F"])
    assert ad.shape == c["alpha_desc"].shape and ad.dtype == np.float64
    close(ad, c["alpha_desc"], 1e-12)


@pytest.mark.parametrize("tag", ["r", "f"])
def test_golden_matvecs(tag):
    from kernelforge_b200 import local_kernels as lk
    c = _case(tag)
    tail = (c["Q1"], c["Q2"], c["N1"], c["N2"], float(c["sigma"]))
    E = lk.kernel_gaussian_local_jacobian_t_matvec(c["X1"], c["X2"], c["alpha_desc"], *tail)
    assert E.shape == c["jacobian_t_matvec"].shape
    close(E, c["jacobian_t_matvec"])
    F = lk.kernel_gaussian_local_hessian_matvec(c["X1"], c["dX1"], c["X2"], c["alpha_desc"],
                                                *tail)
    assert F.shape == c["hessian_matvec"].shape
    close(F, c["hessian_matvec"])
    E, F = lk.kernel_gaussian_local_full_matvec(c["X1"], c["dX1"], c["X2"], c["alpha_desc"],
                                                c["alpha_E"], *tail)
    close(E, c["full_matvec_E"])
    close(F, c["full_matvec_F"])


def _problem(seed, nm1=7, nm2=9, ma1=6, ma2=8, rep=24, species=3, scale=0.35):
    X1, dX1, Q1, N1 = make_set(nm1, ma1, rep, species, seed)
    X2, dX2, Q2, N2 = make_set(nm2, ma2, rep, species, seed + 1)
    rng = np.random.default_rng(seed + 2)
    aE = rng.standard_normal(nm2)
    aF = rng.standard_normal(int(3 * N2.sum()))
    return (X1 * scale, dX1 * 0.3, Q1, N1, X2 * scale, dX2 * 0.3, Q2, N2, aE, aF)


@pytest.mark.parametrize("sigma", [0.2, 0.5, 1.0, 2.0, 5.0])
def test_sigmas_against_oracle(sigma):
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(11)
    ad = om.alpha_desc(dX2, Q2, N2, aF)
    close(lk.kernel_gaussian_local_compute_alpha_desc(dX2, Q2, N2, aF), ad, 1e-12)
    Er, Fr = om.matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1, N2, sigma)
    E, F = lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1, N2, sigma)
    close(E, Er)
    close(F, Fr)


def test_equals_full_kernel_times_coefficients():
    """E, F equal the GPU's own kernel_gaussian_full(query, training) @ [aE; aF]."""
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(21, nm1=12, nm2=15, rep=40)
    sigma = 1.3
    K = lk.kernel_gaussian_full(X1, dX1, X2, dX2, Q1, Q2, N1, N2, sigma)
    v = np.concatenate([aE, aF])
    ad = lk.kernel_gaussian_local_compute_alpha_desc(dX2, Q2, N2, aF)
    E, F = lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1, N2, sigma)
    close(E, K[:len(N1)] @ v)
    close(F, K[len(N1):] @ v)


def test_chunked_query_rows(monkeypatch):
    """A workspace budget far below one label's rows forces many query chunks."""
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(31, nm1=40, nm2=30, rep=32)
    ad = om.alpha_desc(dX2, Q2, N2, aF)
    Er, Fr = om.matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1, N2, 1.1)
    monkeypatch.setenv("KFB_WORKSPACE_GB", "0.00002")  # ~21 kB: a handful of rows
    E, F = lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1, N2, 1.1)
    close(E, Er)
    close(F, Fr)


@pytest.mark.parametrize("nm1,nm2,ma,rep", [(1, 1, 1, 7), (1, 5, 7, 8), (2, 9, 8, 31),
                                            (3, 11, 11, 32), (4, 13, 16, 33), (5, 17, 16, 64),
                                            (7, 19, 13, 65), (9, 33, 12, 72)])
def test_direct_products_tile_edges(nm1, nm2, ma, rep, monkeypatch):
    """Few atom pairs take the FP64 mma kernels, more than the workspace holds the digit planes:
    both against the oracle with one label (rows at and around the 16-, 32- and 64-row tiles and
    the 32- and 64-column slices) and three, with and without alpha_E, energies or forces alone.
    The error of either is a few hundred roundings of sums of a few thousand terms."""
    from kernelforge_b200 import local_kernels as lk
    for species in (1, 3):
        X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(81 + rep, nm1=nm1, nm2=nm2, ma1=ma,
                                                            ma2=ma, rep=rep, species=species)
        N1[0] = ma
        ad = om.alpha_desc(dX2, Q2, N2, np.resize(aF, int(3 * N2.sum())))
        tail = (Q1, Q2, N1, N2, 0.9)
        Er, Fr = om.matvec(X1, dX1, X2, ad, aE, *tail)
        Er0, Fr0 = om.matvec(X1, dX1, X2, ad, 0 * aE, *tail)
        for budget, tol in (("4", 1e-11), ("0.0000001", 1e-10)):
            monkeypatch.setenv("KFB_WORKSPACE_GB", budget)
            E, F = lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad, aE, *tail)
            close(E, Er, tol)
            close(F, Fr, tol)
            close(lk.kernel_gaussian_local_jacobian_t_matvec(X1, X2, ad, *tail), Er0, tol)
            close(lk.kernel_gaussian_local_hessian_matvec(X1, dX1, X2, ad, *tail), Fr0, tol)


@pytest.mark.parametrize("rep", [24, 40, 720, 43])
def test_direct_products_unused_groups(rep):
    """Groups of 8 columns that are zero in the training rows and their coefficients are skipped:
    the query rows are not zero there (their norms count), one group holds a single coefficient
    and one a single descriptor value; no group at all is used with zero training data."""
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(91 + rep, nm1=5, nm2=9, ma1=7, ma2=7,
                                                        rep=rep, scale=0.35 * (24 / rep) ** 0.5)
    ad = om.alpha_desc(dX2, Q2, N2, np.resize(aF, int(3 * N2.sum())))
    groups = np.arange(rep) // 8
    off = np.isin(groups, np.unique(groups)[::2])
    X2[:, :, off] = 0.0
    ad[:, :, off] = 0.0
    ad[1, 0, 3] = 0.7
    X2[2, 0, min(19, rep - 1)] = 0.4
    tail = (Q1, Q2, N1, N2, 0.9)
    for scale in (1.0, 0.0):
        X2s, ads = X2 * scale, ad * scale
        Er, Fr = om.matvec(X1, dX1, X2s, ads, aE, *tail)
        E, F = lk.kernel_gaussian_local_full_matvec(X1, dX1, X2s, ads, aE, *tail)
        close(E, Er, 1e-11)
        close(F, Fr, 1e-11)


def test_edge_cases():
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(41)
    ad = om.alpha_desc(dX2, Q2, N2, aF)
    # query labels absent from the training set: all zero
    Q1x = np.where(Q1 > 0, Q1 + 50, 0).astype(np.int32)
    E, F = lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad, aE, Q1x, Q2, N1, N2, 1.0)
    assert not E.any() and not F.any() and F.shape == (3 * N1.sum(),)
    # empty query molecules and a single query molecule
    N1e = N1.copy()
    N1e[[0, 3]] = 0
    Er, Fr = om.matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1e, N2, 0.9)
    E, F = lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1e, N2, 0.9)
    close(E, Er)
    close(F, Fr)
    assert E[0] == 0.0 and E[3] == 0.0
    E1, F1 = lk.kernel_gaussian_local_full_matvec(X1[:1], dX1[:1], X2, ad, aE, Q1[:1], Q2,
                                                  N1[:1], N2, 0.9)
    Er1, Fr1 = om.matvec(X1[:1], dX1[:1], X2, ad, aE, Q1[:1], Q2, N1[:1], N2, 0.9)
    close(E1, Er1)
    close(F1, Fr1)
    # all query molecules empty
    Z = np.zeros_like(N1)
    F = lk.kernel_gaussian_local_hessian_matvec(X1, dX1, X2, ad, Q1, Q2, Z, N2, 1.0)
    assert F.shape == (0,)
    E = lk.kernel_gaussian_local_jacobian_t_matvec(X1, X2, ad, Q1, Q2, Z, N2, 1.0)
    assert E.shape == (len(N1),) and not E.any()


def test_bad_arguments():
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(51)
    ad = om.alpha_desc(dX2, Q2, N2, aF)
    with pytest.raises(ValueError):
        lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad[:-1], aE, Q1, Q2, N1, N2, 1.0)
    with pytest.raises(ValueError):
        lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad, aE[:-1], Q1, Q2, N1, N2, 1.0)
    with pytest.raises(ValueError):
        lk.kernel_gaussian_local_hessian_matvec(X1, dX1[:, :, :-1], X2, ad, Q1, Q2, N1, N2, 1.0)
    with pytest.raises(ValueError):
        lk.kernel_gaussian_local_jacobian_t_matvec(X1, X2, ad, Q1, Q2, N1, N2, 0.0)
    with pytest.raises(ValueError):
        lk.kernel_gaussian_local_compute_alpha_desc(dX2[..., :-1], Q2, N2, aF)


def test_torch_module_float32():
    import torch
    from kernelforge_b200 import cuda_local_kernels as clk
    X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(61, nm1=10, nm2=12, rep=48)
    f32 = lambda a: torch.tensor(np.asarray(a, np.float32), device="cuda")
    i32 = lambda a: torch.tensor(np.asarray(a, np.int32), device="cuda")
    r = lambda a: np.asarray(a, np.float32).astype(np.float64)
    ad = clk.compute_alpha_desc(f32(dX2), i32(N2), f32(aF))
    assert ad.dtype == torch.float32 and tuple(ad.shape) == X2.shape
    ad_ref = om.alpha_desc(r(dX2), Q2, N2, r(aF))
    close(ad.double().cpu().numpy(), ad_ref, 1e-6)
    sigma = 1.2
    E, F = clk.kernel_gaussian_full_matvec(f32(X1), f32(dX1), i32(Q1), i32(N1), f32(X2),
                                           i32(Q2), i32(N2), f32(aE), ad, sigma)
    assert E.dtype == torch.float32 and F.dtype == torch.float32
    Er, Fr = om.matvec(r(X1), r(dX1), r(X2), r(ad.cpu().numpy()), r(aE), Q1, Q2, N1, N2, sigma)
    close(E.double().cpu().numpy(), Er, 1e-6)
    close(F.double().cpu().numpy(), Fr, 1e-6)


def test_fp32_inputs_fp64_arithmetic():
    """x_dt = KFB_F32 through the C-ABI: FP64 arithmetic on the float32 values."""
    import ctypes
    import torch
    from kernelforge_b200 import _lib
    X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(71)
    r = lambda a: np.asarray(a, np.float32).astype(np.float64)
    ad = om.alpha_desc(r(dX2), Q2, N2, aF)
    Er, Fr = om.matvec(r(X1), r(dX1), r(X2), ad, aE, Q1, Q2, N1, N2, 0.8)
    d = lambda a, dt: torch.tensor(np.asarray(a), dtype=dt, device="cuda")
    x1, dx1, x2 = d(X1, torch.float32), d(dX1, torch.float32), d(X2, torch.float32)
    adt, aet = d(ad, torch.float64), d(aE, torch.float64)
    e = torch.empty(len(N1), dtype=torch.float64, device="cuda")
    f = torch.empty(int(3 * N1.sum()), dtype=torch.float64, device="cuda")
    Q1c, Q2c, N1c, N2c = (np.ascontiguousarray(a, np.int32) for a in (Q1, Q2, N1, N2))
    nm1, ma1, rep = X1.shape
    nm2, ma2, _ = X2.shape
    _lib.check(_lib.lib().kfb_local_matvec(
        x1.data_ptr(), dx1.data_ptr(), x2.data_ptr(), adt.data_ptr(), aet.data_ptr(),
        Q1c.ctypes.data, Q2c.ctypes.data, N1c.ctypes.data, N2c.ctypes.data, nm1, nm2, ma1, ma2,
        rep, ctypes.c_double(0.8), _lib.KFB_F32, e.data_ptr(), f.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    close(e.cpu().numpy(), Er, 1e-9)
    close(f.cpu().numpy(), Fr, 1e-9)


def test_squared_norm_beyond_fp64():
    """A query atom of finite values whose squared norm is not: its pairs' kernels are zero, and
    so is all that it adds; one that holds an infinity leaves its molecule's energy undefined and
    no other."""
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(81)
    ad = om.alpha_desc(dX2, Q2, N2, aF)
    a = [m for m in range(len(N1)) if N1[m] and Q1[m, 0] in Q2[:, 0]][:2]
    X1[a[0], 0, 1] = 1e160
    with np.errstate(over="ignore"):
        Er, Fr = om.matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1, N2, 0.9)
    E, F = lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1, N2, 0.9)
    close(E, Er)
    close(F, Fr)
    X1[a[1], 0, 1] = np.inf
    E, F = lk.kernel_gaussian_local_full_matvec(X1, dX1, X2, ad, aE, Q1, Q2, N1, N2, 0.9)
    assert np.isnan(E[a[1]])
    keep = np.arange(len(N1)) != a[1]
    close(E[keep], Er[keep])
    # energies alone (no Ad) of an energy-trained model: an infinite distance is a zero
    import ctypes
    import torch
    from kernelforge_b200 import _lib
    with np.errstate(invalid="ignore"):
        Er, _ = om.matvec(X1, None, X2, None, aE, Q1, Q2, N1, N2, 0.9)
    x1, x2, ae = (torch.tensor(v, device="cuda") for v in (X1, X2, aE))
    e = torch.empty(len(N1), dtype=torch.float64, device="cuda")
    i = [np.ascontiguousarray(v, np.int32) for v in (Q1, Q2, N1, N2)]
    _lib.check(_lib.lib().kfb_local_matvec(
        x1.data_ptr(), None, x2.data_ptr(), None, ae.data_ptr(), *(v.ctypes.data for v in i),
        len(N1), len(N2), X1.shape[1], X2.shape[1], X1.shape[2], ctypes.c_double(0.9),
        _lib.KFB_F64, e.data_ptr(), None, torch.cuda.current_stream().cuda_stream))
    assert np.isfinite(Er).all()
    close(e.cpu().numpy(), Er)


@pytest.mark.parametrize("kind", ["matvec", "descriptors"])
def test_calls_of_different_sizes_in_threads(kind):
    """Calls that take more and less shared memory (long and short descriptors, large and small
    molecules), each from its own thread and stream: all run, with one thread's results."""
    import threading
    import torch
    from kernelforge_b200 import cuda_local_kernels as clk
    from kernelforge_b200 import fchl19_repr as fr
    f32 = lambda a: torch.tensor(np.asarray(a, np.float32), device="cuda")
    i32 = lambda a: torch.tensor(np.asarray(a, np.int32), device="cuda")
    calls = []
    for size in (0, 1):
        if kind == "matvec":
            X1, dX1, Q1, N1, X2, dX2, Q2, N2, aE, aF = _problem(91, nm1=2, nm2=3,
                                                                rep=(16, 24576)[size])
            ad = om.alpha_desc(dX2, Q2, N2, aF)
            args = (f32(X1), f32(dX1), i32(Q1), i32(N1), f32(X2), i32(Q2), i32(N2), f32(aE),
                    f32(ad), 50.0)
            calls.append(lambda args=args: clk.kernel_gaussian_full_matvec(*args)[1])
        else:
            ma = (3, 40)[size]
            grid = np.stack(np.meshgrid(*[np.arange(4.0)] * 3), -1).reshape(-1, 3)[:ma]
            args = (f32(grid[None]), np.full((1, ma), 6, np.int32), np.array([ma], np.int32))
            calls.append(lambda args=args: fr.generate_batched(*args, gradients=True)[1])
    refs = [c().double().cpu().numpy() for c in calls]
    failed = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(300):
                try:
                    close(calls[k]().double().cpu().numpy(), refs[k], 1e-6)
                except Exception as e:
                    failed.append(repr(e)[:300])
                    return
    threads = [threading.Thread(target=work, args=(k % 2,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
