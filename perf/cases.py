"""The timed cases: what a user of the FCHL19 kernel-ridge path calls, at the sizes of this
repository's own workloads and below them.

Molecules are the repository's synthetic ones: H/C/N/O at 0.5/0.3/0.1/0.1 in a 6 A box with a
0.9 A minimum distance, FCHL19 descriptors with the default hyper-parameters (720 dimensions),
sigma = 2.  Descriptors and Jacobians come from the package's own generator, which is what a
program calls before the kernels; labels and atom counts are host arrays, as the calls take them.

Kinds of a case:

symm       symmetric energy kernel, packed (RFP) or dense: the training matrix of an energy model
rect       rectangular energy kernel: energies of query molecules from a trained model
solve      the mixed-precision ridge solve of a packed training matrix
jacobian   kernel gradients (C ABI): force predictions and force rows of a training matrix
ef_symm    symmetric energy + force kernel, packed or dense: the training matrix of a force field
ef_predict contracted energy + force prediction of a batch
md         one molecular-dynamics step: descriptors, then energy and forces of one molecule
repr       descriptors and their Jacobians of a batch
rff        random Fourier features of energies and forces
mlp        one training step of the learned cos-MLP feature map
"""
import math

import numpy as np
import torch

SIGMA = 2.0
ELEMENTS = (1, 6, 7, 8, 16)        # descriptor channels (the generator's default)
CHARGES = (1, 6, 7, 8)             # elements of the molecules
FRACTIONS = (0.5, 0.3, 0.1, 0.1)
REP = 720


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a first small training set: launches and host planning count
        dict(name="symm_60", kind="symm", nm=60, nmin=9, nmax=21, precision="split_f16", rfp=True),
        # the headline fit's kernel: 10,000 molecules of 9 to 21 atoms
        dict(name="symm_10000", kind="symm", nm=10000, nmin=9, nmax=21, precision="split_f16",
             rfp=True),
        # plain FP64 energy model of 1,000 molecules, dense float64 result
        dict(name="symm_1000_fp64", kind="symm", nm=1000, nmin=9, nmax=21, precision="fp64",
             rfp=False),
        # energies of a few hundred new molecules against a training set (odd sizes)
        dict(name="rect_501x4003", kind="rect", nq=501, nt=4003, nmin=9, nmax=30),
        # the headline fit's solve
        dict(name="solve_10000", kind="solve", n=10000, l2=1e-2),
        # kernel gradients of molecules of 9 to 30 atoms
        dict(name="jacobian_403x333", kind="jacobian", nq=403, nt=333, nmin=9, nmax=30),
        # force-field training matrix: 300 molecules of 21 atoms, 19,200 rows
        dict(name="ef_symm_300x21", kind="ef_symm", nm=300, nmin=21, nmax=21, rfp=True),
        # force-field prediction of a test set
        dict(name="ef_predict_100x300", kind="ef_predict", nq=100, nt=300, nmin=21, nmax=21),
        # one step of molecular dynamics with that model
        dict(name="md_1x300", kind="md", nt=300, nmin=21, nmax=21),
        # descriptors and Jacobians of the training set
        dict(name="repr_300x21", kind="repr", nm=300, nmin=21, nmax=21),
        # random Fourier features of energies and forces, 4,096 features
        dict(name="rff_150x21", kind="rff", nm=150, nmin=21, nmax=21, d=4096),
        # a training step of the learned map: 4,096 atom pairs
        dict(name="mlp_4096", kind="mlp", pairs=4096, d=4096),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["symm", "symm", "rect", "solve", "jacobian", "ef_symm", "ef_symm",
                       "ef_predict", "md", "repr", "rff", "mlp"])
    nmin = rng.randint(5, 21)
    nmax = rng.randint(nmin, 21)
    if kind == "symm":
        precision = rng.choice(["split_f16", "split_f16", "fp64"])
        return dict(kind=kind, nm=_log_int(rng, 20, 10000 if precision == "split_f16" else 1500),
                    nmin=nmin, nmax=nmax, precision=precision, rfp=rng.random() < 0.5)
    if kind == "rect":
        return dict(kind=kind, nq=_log_int(rng, 1, 2000), nt=_log_int(rng, 50, 5000), nmin=nmin,
                    nmax=nmax)
    if kind == "solve":
        return dict(kind=kind, n=_log_int(rng, 200, 10000), l2=rng.choice([1e-2, 1e-1]))
    if kind == "jacobian":
        return dict(kind=kind, nq=_log_int(rng, 4, 400), nt=_log_int(rng, 8, 333), nmin=nmin,
                    nmax=nmax)
    if kind == "ef_symm":
        return dict(kind=kind, nm=_log_int(rng, 4, 300), nmin=nmin, nmax=nmax,
                    rfp=rng.random() < 0.5)
    if kind == "ef_predict":
        return dict(kind=kind, nq=_log_int(rng, 1, 200), nt=_log_int(rng, 20, 300), nmin=nmin,
                    nmax=nmax)
    if kind == "md":
        return dict(kind=kind, nt=_log_int(rng, 20, 300), nmin=nmin, nmax=nmax)
    if kind == "repr":
        return dict(kind=kind, nm=_log_int(rng, 1, 300), nmin=nmin, nmax=nmax)
    if kind == "rff":
        return dict(kind=kind, nm=_log_int(rng, 8, 150), nmin=nmin, nmax=nmax,
                    d=rng.choice([1000, 2048, 4096]))
    return dict(kind=kind, pairs=_log_int(rng, 200, 4096), d=rng.choice([1024, 2048, 4096]))


# ----------------------------------------------------------------- inputs
def _molecules(nm, nmin, nmax, g, box=6.0, dmin=0.9):
    """Random molecules on the GPU: coordinates (nm, ma, 3) float32 (rejection sampling, atom by
    atom, a few candidates at a time), charges (nm, ma) and atom counts (nm,) on the host.  Every
    size from nmax down to nmin comes equally often, in an order that the seed gives, so that the
    outputs have one shape for all seeds."""
    dev = "cuda"
    N = nmax - torch.arange(nm, device=dev) % (nmax - nmin + 1)
    N = N[torch.randperm(nm, generator=g, device=dev)]
    ma = nmax
    R = torch.zeros((nm, ma, 3), device=dev)
    for k in range(ma):
        todo = torch.ones(nm, dtype=torch.bool, device=dev)
        pos = torch.zeros((nm, 3), device=dev)
        while True:
            c = torch.rand((nm, 16, 3), generator=g, device=dev) * box
            if k:
                ok = torch.cdist(c, R[:, :k], compute_mode="donot_use_mm_for_euclid_dist")
                ok = ok.amin(dim=2) >= dmin
            else:
                ok = torch.ones((nm, 16), dtype=torch.bool, device=dev)
            first = ok.to(torch.int32).argmax(dim=1)
            pick = c.gather(1, first[:, None, None].expand(nm, 1, 3))[:, 0]
            take = todo & ok.any(dim=1)
            pos = torch.where(take[:, None], pick, pos)
            todo &= ~take
            if not bool(todo.any()):
                break
        R[:, k] = pos
    p = torch.tensor(FRACTIONS, device=dev)
    z = torch.multinomial(p, nm * ma, replacement=True, generator=g).reshape(nm, ma)
    Z = torch.tensor(CHARGES, device=dev)[z]
    real = torch.arange(ma, device=dev)[None, :] < N[:, None]
    R = torch.where(real[:, :, None], R, torch.zeros_like(R))
    Z = torch.where(real, Z, torch.zeros_like(Z))
    return R.contiguous(), Z.to(torch.int32).cpu().numpy(), N.to(torch.int32).cpu().numpy()


def _described(nm, nmin, nmax, g, gradients):
    from kernelforge_b200 import fchl19_repr
    R, Z, N = _molecules(nm, nmin, nmax, g)
    out = fchl19_repr.generate_batched(R, Z, N, gradients=gradients)
    X, dX = out if gradients else (out, None)
    return X, dX, Z, N


def _energies(R, N):
    """Morse energies sum_{i<j} (1 - exp(-1.5 (r - 1.2)))^2, the labels of the synthetic sets."""
    ma = R.shape[1]
    real = torch.arange(ma, device=R.device) < torch.as_tensor(N, device=R.device)[:, None]
    pair = torch.triu(real[:, :, None] & real[:, None, :], 1)
    r = (R[:, :, None].double() - R[:, None, :].double()).norm(dim=-1)
    e = (1.0 - torch.exp(-1.5 * (r - 1.2))).square()
    return (e * pair).sum((1, 2))


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _element_index(Z):
    q = np.full(Z.shape, -1, np.int32)
    for k, z in enumerate(CHARGES):
        q[Z == z] = k
    return q


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    s = dict(case)
    span = (case.get("nmin"), case.get("nmax"))
    if kind == "symm":
        s["X"], _, s["Q"], s["N"] = _described(case["nm"], *span, g, False)
    elif kind == "rect":
        s["Xq"], _, s["Qq"], s["Nq"] = _described(case["nq"], *span, g, False)
        s["Xt"], _, s["Qt"], s["Nt"] = _described(case["nt"], *span, g, False)
    elif kind == "solve":
        # the training matrix of n molecules, held in FP32 as the kernel call returns it
        from kernelforge_b200 import fchl19_repr
        R, Z, N = _molecules(case["n"], 9, 21, g)
        X = fchl19_repr.generate_batched(R, Z, N)
        s["K"] = _rfp_lower(_scalar(X, Z, N, X, Z, N, torch.float32))
        s["y"] = _energies(R, N)
        s["y"] -= s["y"].mean()
    elif kind == "jacobian":
        s["Xq"], _, s["Qq"], s["Nq"] = _described(case["nq"], *span, g, False)
        s["Xt"], s["dXt"], s["Qt"], s["Nt"] = _described(case["nt"], *span, g, True)
    elif kind == "ef_symm":
        s["X"], s["dX"], s["Q"], s["N"] = _described(case["nm"], *span, g, True)
    elif kind in ("ef_predict", "md"):
        # a trained model: descriptors, energy coefficients and J^T alpha of the training set
        s["Xt"], _, s["Qt"], s["Nt"] = _described(case["nt"], *span, g, False)
        s["aE"] = torch.randn(case["nt"], dtype=torch.float64, generator=g, device="cuda")
        ad = torch.randn(s["Xt"].shape, dtype=torch.float64, generator=g, device="cuda")
        # J^T alpha of a padded atom is zero, and so is that of a feature no atom has
        real = torch.arange(ad.shape[1])[None, :] < torch.as_tensor(s["Nt"])[:, None]
        used = (s["Xt"] != 0).any(dim=0).any(dim=0)
        s["ad"] = ad * real.to("cuda")[:, :, None] * used
        if kind == "md":
            s["R"], Z, s["Nq"] = _molecules(1, *span, g)
            s["Qq"] = Z
            s["elem"] = np.searchsorted(ELEMENTS, np.where(Z == 0, 1, Z)).astype(np.int32)
        else:
            s["Xq"], s["dXq"], s["Qq"], s["Nq"] = _described(case["nq"], *span, g, True)
    elif kind == "repr":
        s["R"], s["Z"], s["N"] = _molecules(case["nm"], *span, g)
    elif kind == "rff":
        s["X"], s["dX"], Z, s["N"] = _described(case["nm"], *span, g, True)
        s["Q"] = _element_index(Z)
        d = case["d"]
        s["W"] = torch.randn((4, REP, d), generator=g, device="cuda") / SIGMA
        s["b"] = torch.rand((4, d), generator=g, device="cuda") * (2 * math.pi)
    elif kind == "mlp":
        from kernelforge_b200 import feature_maps
        X, _, Q, N = _described(400, 9, 30, g, False)
        s["X"] = X.reshape(-1, REP)
        rows = torch.as_tensor(np.flatnonzero(Q.reshape(-1) == 1), device="cuda")
        n = case["pairs"]
        for k in ("pi", "pj"):
            at = torch.randint(0, rows.numel(), (n,), generator=g, device="cuda")
            s[k] = rows[at].to(torch.int32)
        d2 = (s["X"][s["pi"].long()].double() - s["X"][s["pj"].long()].double()).square().sum(1)
        s["t"] = torch.exp(-d2 / (2 * SIGMA * SIGMA)).float()
        s["map"] = feature_maps.CosMLPFeatureMap(1, REP, 512, case["d"], sigma=SIGMA,
                                                 seed=int(seed) & 0xFFFF, max_pairs=n)
    return s


# -------------------------------------------------------------- the calls
def run(s):
    kind = s["kind"]
    if kind == "symm":
        from kernelforge_b200 import cuda_local_kernels as clk
        call = clk.kernel_gaussian_symm_rfp if s["rfp"] else clk.kernel_gaussian_symm
        return call(s["X"], s["Q"], s["N"], SIGMA, precision=s["precision"])
    if kind == "rect":
        from kernelforge_b200 import cuda_local_kernels as clk
        return clk.kernel_gaussian_rect(s["Xq"], s["Qq"], s["Nq"], s["Xt"], s["Qt"], s["Nt"],
                                        SIGMA)
    if kind == "solve":
        from kernelforge_b200 import cuda_global_kernels as cgk
        return cgk.krr_solve_mixed(s["K"], s["y"], l2=s["l2"], uplo="L", tol=1e-10)[0]
    if kind == "jacobian":
        from kernelforge_b200 import _lib
        (nq, ma1, rep), (nt, ma2) = s["Xq"].shape, s["Xt"].shape[:2]
        naq = 3 * int(s["Nt"].sum())
        out = torch.empty((nq, naq), dtype=torch.float32, device="cuda")
        _lib.check(_lib.lib().kfb_kernel_gaussian_jacobian(
            s["Xq"].data_ptr(), s["Xt"].data_ptr(), s["dXt"].data_ptr(), s["Qq"].ctypes.data,
            s["Qt"].ctypes.data, s["Nq"].ctypes.data, s["Nt"].ctypes.data, nq, nt, ma1, ma2, rep,
            naq, SIGMA, _lib.KFB_F32, _lib.PREC["split_f16"], out.data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        return out
    if kind == "ef_symm":
        from kernelforge_b200 import cuda_local_kernels as clk
        call = clk.kernel_gaussian_full_symm_rfp if s["rfp"] else clk.kernel_gaussian_full_symm
        return call(s["X"], s["dX"], s["Q"], s["N"], SIGMA)
    if kind in ("ef_predict", "md"):
        from kernelforge_b200 import cuda_fchl19_repr, cuda_local_kernels as clk
        if kind == "md":
            X, dX = cuda_fchl19_repr.generate_fchl_acsf_and_gradients_md_single(
                s["R"], s["elem"], s["Nq"], len(ELEMENTS))
            dX = dX.reshape(dX.shape[:3] + (-1,))
        else:
            X, dX = s["Xq"], s["dXq"]
        return clk.kernel_gaussian_full_matvec(X, dX, s["Qq"], s["Nq"], s["Xt"], s["Qt"], s["Nt"],
                                               s["aE"], s["ad"], SIGMA)
    if kind == "repr":
        from kernelforge_b200 import fchl19_repr
        return fchl19_repr.generate_batched(s["R"], s["Z"], s["N"], gradients=True)
    if kind == "rff":
        from kernelforge_b200 import cuda_rff_features as crf
        return (crf.rff_features_elemental(s["X"], s["Q"], s["N"], s["W"], s["b"]),
                crf.rff_gradient_elemental(s["X"], s["dX"], s["Q"], s["N"], s["W"], s["b"]))
    fm = s["map"]
    loss = fm.step(0, s["X"], s["pi"], s["pj"], s["t"])
    grads, weights = fm.grads(), fm.parameters()
    for view in grads + weights:
        view.owner = fm                    # the views are valid while the map lives
    return {"loss": loss, "grads": grads, "weights": weights}


# ------------------------------------------------------------------- work
def _pairs_per_pair(case):
    """Same-label atom pairs of a molecule pair, and atoms of a molecule, on average."""
    n = 0.5 * (case["nmin"] + case["nmax"])
    return n * n * sum(f * f for f in FRACTIONS), n


def work(case):
    """Inputs read once, outputs written once; a multiply and an add for each term of the dot
    products x_i . x_j, J^T (x_i - x_j), J^T Y, x W and so on that define the results."""
    kind = case["kind"]
    if kind in ("solve",):
        n = case["n"]
        return {"bytes": 2.0 * n * (n + 1) + 16 * n, "flops": n ** 3 / 3}
    if kind == "mlp":
        p, d = case["pairs"], case["d"]
        weights = 512 * REP + 512 + d * 512 + d
        return {"bytes": 4.0 * (2 * p * REP + 6 * weights + 3 * p),
                "flops": 6.0 * 2 * p * (REP * 512 + 512 * d) - 2.0 * 2 * p * REP * 512}
    pp, n = _pairs_per_pair(case)
    if kind == "symm":
        nm = case["nm"]
        out = (nm * (nm + 1) // 2) * 4 if case["rfp"] else nm * nm * 8
        return {"bytes": 4.0 * nm * n * REP + out, "flops": 2 * REP * pp * nm * (nm + 1) / 2}
    if kind == "rect":
        nq, nt = case["nq"], case["nt"]
        return {"bytes": 4.0 * (nq + nt) * n * REP + 8.0 * nq * nt,
                "flops": 2 * REP * pp * nq * nt}
    jac = 3 * n * n * REP * 4.0            # bytes of a molecule's Jacobian
    if kind == "jacobian":
        nq, nt = case["nq"], case["nt"]
        return {"bytes": nt * jac + 4.0 * (nq + nt) * n * REP + 4.0 * nq * nt * 3 * n,
                "flops": nq * nt * (4 * REP * pp + 2 * n * REP * 3 * n)}
    if kind == "ef_symm":
        nm = case["nm"]
        big = nm * (1 + 3 * n)
        out = big * (big + 1) / 2 if case["rfp"] else big * big
        # per molecule pair: w J (same-label pairs), J^T Y, and the rank-one terms
        pair = 2 * REP * 3 * n * pp + 2 * REP * 9 * n * n * n + 2 * 9 * n * n * pp
        return {"bytes": nm * (jac + 4.0 * n * REP) + 4.0 * out,
                "flops": pair * nm * (nm + 1) / 2}
    if kind in ("ef_predict", "md"):
        nq, nt = case.get("nq", 1), case["nt"]
        return {"bytes": nq * jac * (2 if kind == "md" else 1) + nt * n * REP * 12.0 +
                4.0 * nq * n * REP + 8.0 * (nq * (1 + 3 * n)),
                "flops": 8 * REP * pp * nq * nt + 6 * REP * n * n * nq}
    if kind == "repr":
        nm = case["nm"]
        # two Gaussian terms and three derivative columns for each triple and radial channel
        return {"bytes": nm * (jac + 4.0 * n * REP + 12.0 * n),
                "flops": nm * n * (n - 1) * (n - 2) / 2 * 20 * 2 * 22.0}
    nm, d = case["nm"], case["d"]
    return {"bytes": nm * (jac + 4.0 * n * REP) + 4.0 * 4 * (REP + 1) * d +
            4.0 * nm * (1 + 3 * n) * d, "flops": nm * 2 * REP * d * (n + 3 * n * n)}


def tolerance(case):
    """About four times the largest error against the 64-bit results over the ranges above."""
    kind = case["kind"]
    if kind == "symm" and case["precision"] == "fp64":
        return {"rel": 1e-14}
    return {"symm": {"rel": 8e-7}, "rect": {"rel": 8e-7}, "solve": {"rel": 1e-8},
            "jacobian": {"rel": 5e-5}, "ef_symm": {"rel": 2e-5}, "ef_predict": {"rel": 1e-12},
            "md": {"rel": 2e-7}, "repr": {"rel": 1e-7}, "rff": {"rel": 2e-5},
            "mlp": {"rel": 2e-2}}[kind]


# ----------------------------------------------------- results in 64 bits
def _by_label(X, Q, N):
    """{label: (padded rows (nm, m, rep), mask (nm, m), atoms (nm, m))} of the real atoms."""
    dev = X.device
    q = torch.as_tensor(Q, device=dev)
    real = torch.arange(q.shape[1], device=dev)[None, :] < torch.as_tensor(N, device=dev)[:, None]
    out = {}
    for l in CHARGES:
        has = (q == l) & real
        m = int(has.sum(1).max()) if has.numel() else 0
        if m:
            at = torch.sort((~has).to(torch.int8), dim=1, stable=True).indices[:, :m]
            out[l] = (X.gather(1, at[:, :, None].expand(-1, -1, X.shape[2])), has.gather(1, at), at)
    return out


def _scalar(X1, Q1, N1, X2, Q2, N2, dt):
    """K[a, b] = sum over same-label atom pairs of exp(-|x - y|^2 / (2 sigma^2)) in type dt."""
    K = torch.zeros((X1.shape[0], X2.shape[0]), dtype=dt, device=X1.device)
    A, B = _by_label(X1, Q1, N1), _by_label(X2, Q2, N2)
    for l in A:
        if l not in B:
            continue
        (a, ha, _), (b, hb, _) = A[l], B[l]
        mu = (b.double() * hb[:, :, None]).sum((0, 1)) / hb.sum()
        b = (b.double() - mu).to(dt).reshape(-1, b.shape[2])
        nb = b.square().sum(1)
        step = max(1, int(3e8 // max(1, b.shape[0] * a.shape[1])))
        for i in range(0, a.shape[0], step):
            x = (a[i:i + step].double() - mu).to(dt)
            x, w = x.reshape(-1, x.shape[2]), ha[i:i + step]
            e = torch.addmm(x.square().sum(1)[:, None] + nb[None, :], x, b.T, alpha=-2.0)
            e = e.clamp_(min=0).mul_(-1.0 / (2 * SIGMA * SIGMA)).exp_()
            e = e.reshape(w.shape[0], w.shape[1], K.shape[1], -1)
            e = (e * hb[None, None].to(dt)).sum(3)
            K[i:i + step] += (e * w[:, :, None].to(dt)).sum(1)
    return K


def _rfp_lower(A):
    """RFP (TRANSR='N', UPLO='L') of a symmetric matrix: an (n + 1 or n) x ceil(n / 2) array in
    column order with the trailing triangle turned over the leading one."""
    n = A.shape[0]
    k = (n + 1) // 2                       # columns of the leading trapezoid
    odd = n & 1
    c = torch.arange(k, device=A.device)
    M = torch.zeros((k, n + 1 - odd), dtype=A.dtype, device=A.device)
    if odd:
        M[:] = A[:k]
        tail = torch.zeros((k, k), dtype=A.dtype, device=A.device)
        tail[1:, :k - 1] = A[k:, k:]
        below = c[None, :] < c[:, None]
    else:
        M[:, 1:] = A[:k]
        tail = A[k:, k:]
        below = c[None, :] <= c[:, None]
    M[:, :k] = torch.where(below, tail, M[:, :k])
    return M.reshape(-1)


def _weights(x, y, Qx, Qy):
    """e (..., i, j) of same-label pairs for x (..., i, rep) against y (j, rep); zero elsewhere."""
    d2 = x.square().sum(-1)[..., :, None] + y.square().sum(-1) - 2 * x @ y.T
    same = (Qx[..., :, None] == Qy) & (Qx[..., :, None] > 0)
    return torch.exp(-d2.clamp(min=0) / (2 * SIGMA * SIGMA)) * same


def _jacobian(X1, Q1, X2, dX2, Q2, N2):
    """+dK/dR of set 2: (nm1, 3 sum(N2)); labels 0 are padding."""
    q1, q2 = (torch.as_tensor(q, device=X1.device) for q in (Q1, Q2))
    cols = []
    for m in range(X2.shape[0]):
        n = int(N2[m])
        y, J = X2[m, :n].double(), dX2[m, :n, :, :3 * n].double()
        parts = []
        for o in range(0, X1.shape[0], 256):
            x = X1[o:o + 256].double()
            w = _weights(x, y, q1[o:o + 256], q2[m, :n]) / SIGMA ** 2
            v = w.transpose(1, 2) @ x - w.sum(1)[:, :, None] * y
            parts.append(v.reshape(v.shape[0], -1) @ J.reshape(-1, 3 * n))
        cols.append(torch.cat(parts))
    return torch.cat(cols, 1)


def _hessian(X, dX, Q, N):
    """The symmetric Hessian block, square of 3 sum(N)."""
    nm, ma, rep = X.shape
    q = torch.as_tensor(Q, device=X.device)
    keep = torch.cat([m * 3 * ma + torch.arange(3 * int(N[m])) for m in range(nm)]).to(X.device)
    H = torch.zeros((len(keep), nm * 3 * ma), dtype=torch.float64, device=X.device)
    x, row = X.double(), 0
    step = max(1, int(1.5e8 // (ma * rep * 3 * ma)))
    for a in range(nm):
        n = int(N[a])
        J = dX[a, :n, :, :3 * n].double()
        for b0 in range(0, nm, step):
            b = slice(b0, min(nm, b0 + step))
            k = b.stop - b0
            Jb = dX[b].double()
            e = _weights(x[a, :n], x[b].reshape(-1, rep), q[a, :n], q[b].reshape(-1))
            e = e.reshape(n, k, ma).transpose(0, 1)                     # (b, i, j)
            y = torch.bmm(e, Jb.reshape(k, ma, -1)) / SIGMA ** 2         # (b, i, rep 3 ma)
            h = J.reshape(n * rep, -1).T @ y.reshape(k, n * rep, -1)
            # rank-one terms: J_i^T d and J_j^T d with d = x_i - x_j
            d = x[a, :n][None, :, None] - x[b][:, None]                 # (b, i, j, rep)
            ti = torch.einsum("bijk,ikc->bijc", d, J)
            tj = torch.einsum("bijk,bjkc->bijc", d, Jb)
            ti = ti * e[..., None] / SIGMA ** 4
            h -= ti.reshape(k, -1, ti.shape[3]).transpose(1, 2) @ tj.reshape(k, -1, tj.shape[3])
            H[row:row + 3 * n, b0 * 3 * ma:b.stop * 3 * ma] = h.permute(1, 0, 2).reshape(3 * n, -1)
        row += 3 * n
    return H[:, keep]


def _predict(Xq, dXq, Qq, Nq, Xt, Qt, aE, ad):
    qq, qt = (torch.as_tensor(q, device=Xt.device) for q in (Qq, Qt))
    y, a = Xt.double().reshape(-1, Xt.shape[2]), ad.reshape(-1, Xt.shape[2])
    ae, qt = aE[:, None].expand(Xt.shape[:2]).reshape(-1), qt.reshape(-1)
    ya = (y * a).sum(1)
    E, F = [], []
    for m in range(Xq.shape[0]):
        n = int(Nq[m])
        x = Xq[m, :n].double()
        e = _weights(x, y, qq[m, :n], qt)
        p = x @ a.T - ya                                                # d . (J alpha)
        E.append((e * ae + e * p / SIGMA ** 2).sum())
        v = -e * ae / SIGMA ** 2 - e * p / SIGMA ** 4
        g = e @ a / SIGMA ** 2 + v.sum(1)[:, None] * x - v @ y
        F.append(torch.einsum("ik,ikc->c", g, dXq[m, :n, :, :3 * n].double()))
    return torch.stack(E), torch.cat(F)


def _fchl19(R, z):
    """FCHL19 descriptors (n, 720) of one molecule from coordinates (n, 3) and element channels
    z (n,), default hyper-parameters: log-normal two-body terms on each neighbour's element, and
    Axilrod-Teller-weighted radial x first-order Fourier terms on each pair of elements."""
    n, ne, n2, n3 = R.shape[0], len(ELEMENTS), 24, 20
    eta2, eta3, cut, w3 = 0.32, 2.7, 8.0, 13.4
    eye = torch.eye(n, dtype=torch.bool, device=R.device)
    v = R[None] - R[:, None]
    r = torch.sqrt(torch.where(eye, torch.ones_like(v[..., 0]), v.square().sum(-1)))
    near = (~eye) & (r <= cut)
    fc = 0.5 * (torch.cos(math.pi * r / cut) + 1) * near
    grid = torch.arange(1, n2 + 1, dtype=R.dtype, device=R.device) * (cut / n2)
    s2 = torch.log1p(eta2 / r ** 2)
    mu = torch.log(r) - 0.5 * s2
    two = torch.exp(-0.5 * (torch.log(grid) - mu[..., None]) ** 2 / s2[..., None]) / grid
    two = two * (fc / (torch.sqrt(2 * math.pi * s2) * r ** 1.8))[..., None]
    one = (z[:, None] == torch.arange(ne, device=R.device)).to(R.dtype)
    out2 = torch.einsum("ijk,je->iek", two, one).reshape(n, -1)
    u = v / r[..., None]
    ci = torch.einsum("ijx,ikx->ijk", u, u)
    cj = -torch.einsum("ijx,jkx->ijk", u, u)
    ck = torch.einsum("ikx,jkx->ijk", u, u)
    ok = torch.triu(torch.ones((n, n), dtype=torch.bool, device=R.device), 1)[None]
    ok = ok & ~eye[:, :, None] & ~eye[:, None, :]
    lift = math.sqrt(eta3 / math.pi) * w3
    atm = (1 + 3 * ci * cj * ck) * lift / (r[:, :, None] * r[:, None, :] * r[None]) ** 0.57
    atm = atm * ok * fc[:, :, None] * fc[:, None, :]
    ang = 2 * math.exp(-0.5 * math.pi ** 2)
    si = torch.sqrt(torch.where(ok, 1 - ci * ci, torch.ones_like(ci)).clamp(min=1e-30))
    grid = torch.arange(1, n3 + 1, dtype=R.dtype, device=R.device) * (cut / n3)
    rad = torch.exp(-eta3 * (0.5 * (r[:, :, None] + r[:, None, :])[..., None] - grid) ** 2)
    both = torch.stack([ang * ci * atm, ang * si * atm], -1)            # (i, j, k, 2)
    lo, hi = torch.minimum(z[:, None], z[None]), torch.maximum(z[:, None], z[None])
    ch = hi + ne * lo - lo * (lo + 1) // 2
    np_ = ne * (ne + 1) // 2
    chan = (ch[..., None] == torch.arange(np_, device=R.device)).to(R.dtype).reshape(n * n, np_)
    t3 = (rad[..., :, None] * both[..., None, :]).reshape(n, n * n, n3 * 2)
    out3 = torch.matmul(chan.T, t3).reshape(n, -1)
    return torch.cat([out2, out3], 1)


def _described64(R, Z, N):
    nm, ma = Z.shape
    X = torch.zeros((nm, ma, REP), dtype=torch.float64, device=R.device)
    dX = torch.zeros((nm, ma, REP, 3 * ma), dtype=torch.float64, device=R.device)
    chan = torch.as_tensor(np.searchsorted(ELEMENTS, np.where(Z == 0, 1, Z)), device=R.device)
    both = torch.func.vmap(lambda r, z: (_fchl19(r, z), torch.func.jacfwd(_fchl19)(r, z)))
    for n in sorted(set(int(v) for v in N)):
        ids = np.flatnonzero(N == n)
        for k in range(0, len(ids), 8):
            at = torch.as_tensor(ids[k:k + 8], device=R.device)
            x, j = both(R[at, :n].double(), chan[at, :n])
            X[at, :n] = x
            dX[at, :n, :, :3 * n] = j.reshape(len(at), n, REP, 3 * n)
    return X, dX


def _rff64(s):
    d = s["d"]
    q, c = torch.as_tensor(s["Q"], device="cuda"), math.sqrt(2.0 / d)
    W, b = s["W"].double(), s["b"].double()
    Z = torch.zeros((s["nm"], d), dtype=torch.float64, device="cuda")
    G = []
    for m in range(s["nm"]):
        n = int(s["N"][m])
        J = s["dX"][m, :n, :, :3 * n].double()
        g = torch.zeros((3 * n, d), dtype=torch.float64, device="cuda")
        for e in range(len(CHARGES)):
            at = torch.nonzero(q[m, :n] == e)[:, 0]
            if len(at):
                z = s["X"][m, at].double() @ W[e] + b[e]
                Z[m] += c * torch.cos(z).sum(0)
                p = J[at].transpose(1, 2) @ W[e]                        # (atoms, 3 n, d)
                g += c * torch.einsum("ad,acd->cd", torch.sin(z), p)
        G.append(g)
    return Z, torch.cat(G)


def _mlp64(s, lr=1e-3, eps=1e-8):
    p = [t[0].double().clone().requires_grad_(True) for t in s["map"].parameters()]
    W1, b1, W2, b2 = p
    d = s["d"]
    k = 0.0
    feats = []
    for rows in (s["pi"], s["pj"]):
        h = torch.cos(s["X"][rows.long()].double() @ W1.T + b1)
        feats.append(math.sqrt(2.0 / d) * torch.cos(h @ W2.T + b2))
    k = (feats[0] * feats[1]).sum(1)
    loss = (k - s["t"].double()).square().mean()
    grads = torch.autograd.grad(loss, p)
    # Adam's first step
    new = [(w - lr * g / (g.abs() + eps)).detach()[None] for w, g in zip(p, grads)]
    return {"loss": float(loss), "grads": list(grads), "weights": new}


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "symm":
        K = _scalar(s["X"], s["Q"], s["N"], s["X"], s["Q"], s["N"], torch.float64)
        return _rfp_lower(K) if s["rfp"] else K
    if kind == "rect":
        return _scalar(s["Xq"], s["Qq"], s["Nq"], s["Xt"], s["Qt"], s["Nt"], torch.float64)
    if kind == "solve":
        # unpack: the leading trapezoid, then the trailing triangle
        n = case["n"]
        k, odd = (n + 1) // 2, n & 1
        M = s["K"].double().reshape(k, -1)
        A = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        A[:, :k] = torch.tril(M.T[1 - odd:])
        A[k:, k:] = torch.tril(M[odd:, :n - k])
        A = A + torch.tril(A, -1).T
        A.diagonal().add_(case["l2"])
        L = torch.linalg.cholesky(A)
        x = torch.cholesky_solve(s["y"][:, None], L)
        x = x + torch.cholesky_solve(s["y"][:, None] - A @ x, L)
        return x[:, 0]
    if kind == "jacobian":
        return _jacobian(s["Xq"], s["Qq"], s["Xt"], s["dXt"], s["Qt"], s["Nt"])
    if kind == "ef_symm":
        X, dX, Q, N = s["X"], s["dX"], s["Q"], s["N"]
        S = _scalar(X, Q, N, X, Q, N, torch.float64)
        J = _jacobian(X, Q, X, dX, Q, N)
        K = torch.cat([torch.cat([S, J], 1), torch.cat([J.T, _hessian(X, dX, Q, N)], 1)])
        return _rfp_lower(K) if s["rfp"] else K
    if kind == "ef_predict":
        return _predict(s["Xq"], s["dXq"], s["Qq"], s["Nq"], s["Xt"], s["Qt"], s["aE"], s["ad"])
    if kind == "md":
        X, dX = _described64(s["R"], s["Qq"], s["Nq"])
        return _predict(X, dX, s["Qq"], s["Nq"], s["Xt"], s["Qt"], s["aE"], s["ad"])
    if kind == "repr":
        return _described64(s["R"], s["Z"], s["N"])
    if kind == "rff":
        return _rff64(s)
    return _mlp64(s)
