"""Jacobian / Hessian / full kernels on the GPU against the oracle and the
reference's golden outputs.  FP64: rtol 1e-10 (the reference's own tolerance
for these kernels); FP32: rtol 1e-4 relative to max|K|."""
import numpy as np
import pytest

from conftest import load_golden, make_set
from oracle import oracle as o

pytestmark = pytest.mark.gpu


def close(got, ref, precision):
    if precision == "fp64":
        np.testing.assert_allclose(got, ref, rtol=1e-10, atol=1e-10 * max(1.0, np.abs(ref).max()))
    else:
        np.testing.assert_allclose(got, ref, rtol=1e-3, atol=1e-4 * max(1.0, np.abs(ref).max()))


GOLDEN_CASES = [
    ("kernel_gaussian_jacobian", ("X1", "X2", "dX2", "Q1", "Q2", "N1", "N2")),
    ("kernel_gaussian_jacobian_t", ("X1", "dX1", "X2", "Q1", "Q2", "N1", "N2")),
    ("kernel_gaussian_hessian", ("X1", "dX1", "X2", "dX2", "Q1", "Q2", "N1", "N2")),
    ("kernel_gaussian_hessian_symm", ("X1", "dX1", "Q1", "N1")),
    ("kernel_gaussian_hessian_symm_rfp", ("X1", "dX1", "Q1", "N1")),
    ("kernel_gaussian_full", ("X1", "dX1", "X2", "dX2", "Q1", "Q2", "N1", "N2")),
    ("kernel_gaussian_full_symm", ("X1", "dX1", "Q1", "N1")),
    ("kernel_gaussian_full_symm_rfp", ("X1", "dX1", "Q1", "N1")),
]


@pytest.mark.parametrize("name,args", GOLDEN_CASES)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_golden_random(name, args, precision):
    from kernelforge_b200 import local_kernels as lk
    g = load_golden("golden_random.npz")
    got = getattr(lk, name)(*[g[a] for a in args], float(g["sigma"]), precision=precision)
    assert got.shape == g[name].shape
    close(got, g[name], precision)


def test_golden_fchl19():
    from kernelforge_b200 import local_kernels as lk
    g = load_golden("golden_fchl19.npz")
    X, dX, Q, N, s = g["X"], g["dX"], g["Q"], g["N"], float(g["sigma"])
    close(lk.kernel_gaussian_jacobian(X[:4], X[2:], dX[2:], Q[:4], Q[2:], N[:4], N[2:], s),
          g["kernel_gaussian_jacobian"], "fp64")
    close(lk.kernel_gaussian_hessian_symm_rfp(X, dX, Q, N, s), g["kernel_gaussian_hessian_symm_rfp"],
          "fp64")
    close(lk.kernel_gaussian_full_symm_rfp(X, dX, Q, N, s), g["kernel_gaussian_full_symm_rfp"],
          "fp64")


@pytest.mark.parametrize("seed", [1, 2])
def test_larger_ragged_sets(seed):
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1 = make_set(9, 7, 33, 3, seed)
    X2, dX2, Q2, N2 = make_set(6, 5, 33, 3, seed + 10)
    X1 *= 0.4
    X2 *= 0.4
    s = 2.0
    close(lk.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s),
          o.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s), "fp64")
    close(lk.kernel_gaussian_jacobian_t(X1, dX1, X2, Q1, Q2, N1, N2, s),
          o.kernel_gaussian_jacobian_t(X1, dX1, X2, Q1, Q2, N1, N2, s), "fp64")
    close(lk.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s),
          o.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s), "fp64")
    close(lk.kernel_gaussian_full(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s),
          o.kernel_gaussian_full(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s), "fp64")


def test_jacobian_t_is_minus_jacobian_transposed():
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1 = make_set(5, 6, 10, 2, 3)
    X2, dX2, Q2, N2 = make_set(4, 6, 10, 2, 4)
    jt = lk.kernel_gaussian_jacobian_t(X1, dX1, X2, Q1, Q2, N1, N2, 2.0)
    j = lk.kernel_gaussian_jacobian(X2, X1, dX1, Q2, Q1, N2, N1, 2.0)
    np.testing.assert_allclose(jt, -j.T, rtol=1e-12, atol=1e-12)


def test_full_symm_is_symmetric_and_matches_asym():
    from kernelforge_b200 import local_kernels as lk
    X, dX, Q, N = make_set(5, 5, 12, 2, 8)
    F = lk.kernel_gaussian_full_symm(X, dX, Q, N, 2.0)
    np.testing.assert_allclose(F, F.T, rtol=1e-12, atol=1e-12)
    Fa = lk.kernel_gaussian_full(X, dX, X, dX, Q, Q, N, N, 2.0)
    np.testing.assert_allclose(F, Fa, rtol=1e-10, atol=1e-10)


@pytest.mark.parametrize("rep", [48, 720])
def test_tensor_core_contractions_match_oracle(rep):
    """precision='split_f16' runs the Jacobian and Hessian contraction GEMMs on
    the tcgen05 tensor cores (rep a multiple of 16): FP32-level agreement."""
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1 = make_set(7, 6, rep, 3, 21)
    X2, dX2, Q2, N2 = make_set(5, 6, rep, 3, 22)
    sc = 1.0 / np.sqrt(rep)
    X1 *= 2 * sc
    X2 *= 2 * sc
    dX1 *= sc
    dX2 *= sc
    s = 2.0
    p = "split_f16"
    close(lk.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s), p)
    close(lk.kernel_gaussian_jacobian_t(X1, dX1, X2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_jacobian_t(X1, dX1, X2, Q1, Q2, N1, N2, s), p)
    close(lk.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s), p)
    close(lk.kernel_gaussian_hessian_symm_rfp(X1, dX1, Q1, N1, s, precision=p),
          o.kernel_gaussian_hessian_symm_rfp(X1, dX1, Q1, N1, s), p)
    close(lk.kernel_gaussian_full_symm_rfp(X1, dX1, Q1, N1, s, precision=p),
          o.kernel_gaussian_full_symm_rfp(X1, dX1, Q1, N1, s), p)
    close(lk.kernel_gaussian_full(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_full(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s), p)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "split_f16"])
@pytest.mark.parametrize("rep,used", [(48, 0), (48, 5), (48, 30), (48, 31), (96, 17), (50, 20)])
def test_unused_columns(rep, used, precision):
    """Columns that no real atom of either set uses are left out (when they are an eighth of the
    columns or more after rounding up to 16, 32 and 33 of 48): padding holds values there, one column is used by a single
    Jacobian entry of set 2 alone, another by a descriptor of set 1 alone."""
    from kernelforge_b200 import local_kernels as lk
    X1, dX1, Q1, N1 = make_set(7, 6, rep, 3, 31 + used)
    X2, dX2, Q2, N2 = make_set(5, 5, rep, 3, 32 + used)
    sc = 1.0 / np.sqrt(max(used, 1))
    rng = np.random.default_rng(used)
    off = rng.permutation(rep)[used:]
    for X, dX in ((X1, dX1), (X2, dX2)):
        X *= 2 * sc
        dX *= sc
        X[:, :, off] = 0.0
        dX[:, :, off] = 0.0
    for m in range(len(N1)):     # padding is not read
        X1[m, N1[m]:] = 7.0
        dX1[m, N1[m]:] = 7.0
        dX1[m, :, :, 3 * N1[m]:] = 7.0
    dX2[1, 0, off[0], 1] = 0.5
    X1[2, 0, off[-1]] = 0.5
    s, p = 2.0, precision
    close(lk.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s), p)
    close(lk.kernel_gaussian_jacobian_t(X1, dX1, X2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_jacobian_t(X1, dX1, X2, Q1, Q2, N1, N2, s), p)
    close(lk.kernel_gaussian_full(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_full(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s), p)
    close(lk.kernel_gaussian_full_symm_rfp(X1, dX1, Q1, N1, s, precision=p),
          o.kernel_gaussian_full_symm_rfp(X1, dX1, Q1, N1, s), p)
    # one array, two sets of atom counts
    N3 = np.maximum(N1 - 1, 0).astype(np.int32)
    close(lk.kernel_gaussian_hessian(X1, dX1, X1, dX1, Q1, Q1, N3, N1, s, precision=p),
          o.kernel_gaussian_hessian(X1, dX1, X1, dX1, Q1, Q1, N3, N1, s), p)


@pytest.mark.parametrize("precision,rep", [("fp64", 33), ("fp32", 33), ("split_f16", 48)])
def test_jacobian_chunked_outer_molecules(precision, rep, monkeypatch):
    """A workspace of a few kB splits the outer molecules into chunks (each with
    its own dot-product block and label tiles).  Outer molecules lacking a label
    (zero rows of V), an outer label the inner set lacks, empty molecules and
    rep not a multiple of 4 (scalar row edges) on the CUDA-core paths."""
    from kernelforge_b200 import local_kernels as lk
    monkeypatch.setenv("KFB_WORKSPACE_GB", "0.00002")
    X1, dX1, Q1, N1 = make_set(9, 7, rep, 3, 31)
    X2, dX2, Q2, N2 = make_set(6, 5, rep, 3, 32)
    sc = 1.0 / np.sqrt(rep)
    X1 *= 2 * sc
    X2 *= 2 * sc
    dX1 *= sc
    dX2 *= sc
    Q1[2, :] = 1          # outer molecule with one label only
    Q1[4, :2] = 9         # an outer label the inner set lacks
    N1[6] = 0             # empty outer molecule
    s = 2.0
    if precision == "fp64":
        close(lk.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s),
              o.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s), "fp64")
        close(lk.kernel_gaussian_jacobian_t(X2, dX2, X1, Q2, Q1, N2, N1, s),
              o.kernel_gaussian_jacobian_t(X2, dX2, X1, Q2, Q1, N2, N1, s), "fp64")
    else:
        close(lk.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s, precision=precision),
              o.kernel_gaussian_jacobian(X1, X2, dX2, Q1, Q2, N1, N2, s), precision)


@pytest.mark.parametrize("ma1,ma2", [(23, 5), (4, 23)])
def test_tensor_core_hessian_large_molecules(ma1, ma2):
    """Set-1 molecules of more than 21 atoms (more than 64 Jacobian rows) take
    the contraction with their Jacobian rows as M; smaller ones take the pairs'
    Y rows as M and 64-column tiles; 23-atom molecules b (69 columns of Y) are
    never merged into one problem.  Both sides, asymmetric and symmetric,
    against the oracle at the split-fp16 tolerance."""
    from kernelforge_b200 import local_kernels as lk
    rep = 48
    X1, dX1, Q1, N1 = make_set(4, ma1, rep, 3, 51, n_min=ma1 - 2)
    X2, dX2, Q2, N2 = make_set(3, ma2, rep, 3, 52, n_min=ma2 - 2)
    sc = 1.0 / np.sqrt(rep)
    X1 *= 2 * sc
    X2 *= 2 * sc
    dX1 *= sc
    dX2 *= sc
    s = 2.0
    p = "split_f16"
    close(lk.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s), p)
    Xs, dXs, Qs, Ns = (X1, dX1, Q1, N1) if ma1 > ma2 else (X2, dX2, Q2, N2)
    close(lk.kernel_gaussian_hessian_symm_rfp(Xs, dXs, Qs, Ns, s, precision=p),
          o.kernel_gaussian_hessian_symm_rfp(Xs, dXs, Qs, Ns, s), p)


def test_tensor_core_hessian_disjoint_labels():
    """No atom of set 2 shares a label with set 1: every projection problem
    list is empty and the tensor-core Hessian is exactly zero."""
    from kernelforge_b200 import local_kernels as lk
    rep = 48
    X1, dX1, Q1, N1 = make_set(3, 6, rep, 1, 53, species=[1])
    X2, dX2, Q2, N2 = make_set(4, 6, rep, 1, 54, species=[2])
    H = lk.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, 2.0, precision="split_f16")
    assert H.shape == (int(3 * N1.sum()), int(3 * N2.sum()))
    assert not np.any(H)


@pytest.mark.parametrize("gb,ycore,path", [
    ("0.00005", None, ["hessian:rank-in-y", "hessian:y-cuda-core"]),
    ("0.0001", None, ["hessian:rank-kernel", "hessian:y-gemm"]),
    ("4", None, ["hessian:rank-kernel", "hessian:y-gemm"]),
    ("4", "cuda-core", ["hessian:rank-kernel", "hessian:y-cuda-core"])])
def test_hessian_tensor_core_batches(gb, ycore, path, monkeypatch):
    """Tensor-core Hessians with kernel 1 in GEMM form: a workspace of ~100 kB
    gives batches of a few molecule pairs spanning at most two molecules b (the
    projection buffer's capacity), the default one batch; symmetric RFP,
    asymmetric and full energy+force kernels against the oracle.  At ~54 kB the
    projection and rank buffers (18 kB each here) no longer fit half the
    workspace together, so the rank term stays inside Y (CUDA-core Y kernel);
    with the rank term outside, Y is a tensor-core GEMM per molecule b unless
    KFB_HESSIAN_Y=cuda-core keeps the CUDA-core kernel.  The path log shows
    which forms each call took."""
    from kernelforge_b200 import _lib
    from kernelforge_b200 import local_kernels as lk
    monkeypatch.setenv("KFB_WORKSPACE_GB", gb)
    if ycore:
        monkeypatch.setenv("KFB_HESSIAN_Y", ycore)
    rep = 48
    X1, dX1, Q1, N1 = make_set(7, 6, rep, 3, 41)
    X2, dX2, Q2, N2 = make_set(5, 6, rep, 3, 42)
    sc = 1.0 / np.sqrt(rep)
    X1 *= 2 * sc
    X2 *= 2 * sc
    dX1 *= sc
    dX2 *= sc
    Q2[1, :2] = 9   # a set-2 label set 1 lacks
    s = 2.0
    p = "split_f16"
    _lib.path_log_clear()
    close(lk.kernel_gaussian_hessian_symm_rfp(X1, dX1, Q1, N1, s, precision=p),
          o.kernel_gaussian_hessian_symm_rfp(X1, dX1, Q1, N1, s), p)
    assert _lib.path_log() == path
    _lib.path_log_clear()
    close(lk.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s), p)
    assert _lib.path_log() == path
    close(lk.kernel_gaussian_full(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s, precision=p),
          o.kernel_gaussian_full(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s), p)


@pytest.mark.parametrize("ycore", [None, "cuda-core"])
def test_hessian_of_far_apart_sets(ycore, monkeypatch):
    """Set-2 molecules whose weights are all about 2^-4, 2^-13 and 2^-22, 30 atoms of one element
    each, a batch per molecule b (workspace of 5.7 MB): every block against its own norm.  The
    distance lies along a column that no Jacobian uses, so that the block is J^T Y alone.  Y's
    fp16 pair is scaled by the batch's bound; with one scale for weights of up to 1 its absolute
    floor of 2^-25 leaves 14 bits of the last block (5e-5).  What remains: the weights' pair,
    2^-25 below 2^-8 (4e-6 on average), and the FP32 exponents of 15 (5e-6): 2e-5."""
    from kernelforge_b200 import _lib
    from kernelforge_b200 import local_kernels as lk
    monkeypatch.setenv("KFB_WORKSPACE_GB", "0.0053")
    if ycore:
        monkeypatch.setenv("KFB_HESSIAN_Y", ycore)
    rng = np.random.default_rng(61)
    rep, ma, s = 48, 30, 2.0
    bits = (4, 13, 22)

    def one(nm):
        X = rng.standard_normal((nm, ma, rep)) * 0.02
        dX = rng.standard_normal((nm, ma, rep, 3 * ma)) / np.sqrt(rep)
        dX[:, :, 0] = 0.0
        return X, dX, np.full((nm, ma), 6, np.int32), np.full(nm, ma, np.int32)
    X1, dX1, Q1, N1 = one(4)
    X2, dX2, Q2, N2 = one(len(bits))
    for b, e in enumerate(bits):
        X2[b, :, 0] += np.sqrt(2 * s * s * e * np.log(2.0))
    _lib.path_log_clear()
    H = lk.kernel_gaussian_hessian(X1, dX1, X2, dX2, Q1, Q2, N1, N2, s, precision="split_f16")
    assert _lib.path_log() == ["hessian:rank-kernel",
                               "hessian:y-cuda-core" if ycore else "hessian:y-gemm"]
    f = lambda a: a.astype(np.float32).astype(np.float64)
    R = o.kernel_gaussian_hessian(f(X1), f(dX1), f(X2), f(dX2), Q1, Q2, N1, N2, s)
    for b in range(len(bits)):
        c = slice(3 * ma * b, 3 * ma * (b + 1))
        assert np.linalg.norm(H[:, c] - R[:, c]) <= 2e-5 * np.linalg.norm(R[:, c])


_FULL_GPU = r"""
import sys
import numpy as np
import torch
from kernelforge_b200 import cuda_local_kernels as clk, _lib
kind = sys.argv[1]
nm, ma, rep, used = 150, 24, 720, 480
g = torch.Generator(device="cuda")
g.manual_seed(5)
X = torch.randn((nm, ma, rep), generator=g, device="cuda") * 0.1
dX = torch.randn((nm, ma, rep, 3 * ma), generator=g, device="cuda") * 0.1
off = torch.arange(rep, device="cuda") % 3 == 2
Q = np.random.default_rng(5).choice([1, 6, 8], (nm, ma)).astype(np.int32)
N = np.full(nm, ma, np.int32)
N[::3] -= 3
naq = 3 * int(N.sum())
J = torch.empty((nm, naq), device="cuda")

def call():
    if kind == "ef":
        return clk.kernel_gaussian_full_symm_rfp(X, dX, Q, N, 2.0)
    J.fill_(float("nan"))
    _lib.check(_lib.lib().kfb_kernel_gaussian_jacobian(
        X.data_ptr(), X.data_ptr(), dX.data_ptr(), Q.ctypes.data, Q.ctypes.data, N.ctypes.data,
        N.ctypes.data, nm, nm, ma, ma, rep, naq, 2.0, _lib.KFB_F32, _lib.PREC["split_f16"],
        J.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return J

def needs(limit_mb, step_mb):
    # the smallest free memory, in steps, at which the call still runs; the results agree
    K, good = None, None
    for mb in range(limit_mb, 0, -step_mb):
        torch.cuda.synchronize()      # (the pool keeps nothing: KFB_POOL_KEEP_GB=0)
        free = torch.cuda.mem_get_info()[0]
        fill = torch.empty(free - (mb << 20), dtype=torch.uint8, device="cuda")
        try:
            out = call()
            torch.cuda.synchronize()
        except _lib.KfbError as e:
            assert "cudaMallocAsync" in str(e), e
            out = None
        del fill
        torch.cuda.empty_cache()
        if out is None:
            return good
        good = mb
        if K is None:
            K = out.clone()
        # (two widths: FP32 sums of 17,280 terms in two orders, each 1e-5 from 64 bits)
        assert torch.linalg.norm(out - K) <= 5e-5 * torch.linalg.norm(K)
        del out
    return good

call(), torch.cuda.synchronize()
limit = 3072 if kind == "jacobian" else 6144
dense = needs(limit, 128)
X[:, :, off] = 0
dX[:, :, off] = 0
sparse = needs(limit, 128)
print("full width", dense, "MB, unused columns", sparse, "MB")
assert dense < limit and sparse <= dense
"""


@pytest.mark.parametrize("kind", ["jacobian", "ef"])
def test_derivative_kernels_on_a_nearly_full_gpu(kind):
    """A third of the columns unused: the copies without them, and the Y GEMM's operand, are
    taken where they can be allocated.  The call runs wherever one of the same size that uses
    every column does, with the same result at every amount of free memory (an ordinary
    allocation holds the rest).  In a process of its own: the memory pool's settings are read
    once."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, KFB_POOL_KEEP_GB="0", KFB_WORKSPACE_GB="1", PYTHONPATH=root)
    r = subprocess.run([sys.executable, "-c", _FULL_GPU, kind], env=env, cwd=root,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
