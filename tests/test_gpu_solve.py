"""GPU solver parity: x = A \\ b against the oracle (sparse direct solve in
complex128), in both precisions and both Krylov methods.

Tolerances: the true relative residual ‖b − A x‖/‖b‖, recomputed here with
the oracle's sparse A, must meet the requested tol; the field error against
the direct solve must be ≤ 1e-5 (relative 2-norm) at tol = 1e-7.
"""
import numpy as np
import pytest
import scipy.sparse.linalg as spla

pytestmark = pytest.mark.gpu


def _system(O, N=(16, 14, 12), spheres=True):
    g = O.uniform_grid(N)
    objs = [O.Sphere((8.2, 7.1, 6.3), 3.1, 6.0)] if spheres else []
    S = O.System(g, 2 * np.pi / 7.0, ((3, 3, 3), (3, 3, 3)), objs)
    S.add_pointsrc((7.6, 6.5, 6.0), (0.3, 0.2, 1.0))
    return S


def _op(pkg, S):
    A = pkg.FDFDOperator(S.grid.N, S.omega, S.sdl_e, S.sdl_m)
    A.set_eps(S.eps_diag, S.eps_off)
    return A


@pytest.fixture(scope="module")
def sysx(oracle):
    S = _system(oracle)
    b = S.b()
    xd = spla.spsolve(S.A.tocsc(), b)
    return S, b, xd


@pytest.mark.parametrize("precision,method", [("fp64", "bicgstab"), ("mixed", "bicgstab"), ("fp64", "cocg"),
                                              ("fp64", "bicgstabl"), ("mixed", "bicgstabl")])
def test_solve_matches_direct(pkg, sysx, precision, method):
    S, b, xd = sysx
    A = _op(pkg, S)
    tol = 1e-7
    x, st = A.solve(b, tol=tol, precision=precision, method=method)
    rel = np.linalg.norm(b - S.A @ x) / np.linalg.norm(b)
    assert rel <= tol * 1.01, (rel, st)
    assert abs(st[0]["relres"] - rel) < 1e-9 + 0.05 * rel
    ferr = np.linalg.norm(x - xd) / np.linalg.norm(xd)
    assert ferr < 1e-5, (ferr, st)
    if precision == "mixed":
        assert st[0]["refinements"] >= 1
    A.close()


def test_transpose_solve(pkg, sysx):
    S, b, _ = sysx
    A = _op(pkg, S)
    x, st = A.solve(b, tol=1e-8, precision="mixed", transpose=True)
    rel = np.linalg.norm(b - S.A.T @ x) / np.linalg.norm(b)
    assert rel <= 1e-8 * 1.01, (rel, st)
    A.close()


def test_multiple_rhs_and_x0(pkg, oracle, sysx):
    S, b, xd = sysx
    A = _op(pkg, S)
    b2 = np.stack([b, 2j * b, np.roll(b, 7)])
    x, st = A.solve(b2, tol=1e-7, precision="mixed")
    for q in range(3):
        rel = np.linalg.norm(b2[q] - S.A @ x[q]) / np.linalg.norm(b2[q])
        assert rel <= 1.01e-7, (q, rel)
    assert np.allclose(x[1], 2j * x[0], rtol=0, atol=1e-5 * np.abs(x[0]).max())
    # warm start from the converged answer: no iteration needed
    x3, st3 = A.solve(b, tol=1e-6, precision="mixed", x0=xd)
    assert st3[0]["iterations"] == 0
    A.close()


def test_zero_rhs_and_maxit(pkg, sysx):
    S, b, _ = sysx
    A = _op(pkg, S)
    x, st = A.solve(np.zeros_like(b), precision="mixed")
    assert np.all(x == 0) and st[0]["status"] == 0
    with pytest.raises(pkg.FDFDError) as ei:
        A.solve(b, tol=1e-12, precision="mixed", maxit=3, check_every=1)
    assert ei.value.code == 5
    assert ei.value.stats[0]["iterations"] >= 3
    A.close()


def test_graph_and_plain_agree(pkg, sysx):
    """The CUDA-graph replay and direct launches run the same recurrence."""
    S, b, _ = sysx
    A = _op(pkg, S)
    x1, s1 = A.solve(b, tol=1e-6, precision="fp64", use_graph=True, check_every=10)
    x2, s2 = A.solve(b, tol=1e-6, precision="fp64", use_graph=False, check_every=10)
    assert s1[0]["iterations"] == s2[0]["iterations"]
    assert np.array_equal(x1, x2)
    A.close()


def test_unsupported_cocg_forms_rejected(pkg, sysx):
    S, b, _ = sysx
    A = _op(pkg, S)
    for kw in ({"precision": "fp64", "transpose": True}, {"precision": "mixed"}):
        with pytest.raises(pkg.FDFDError) as ei:
            A.solve(b, method="cocg", **kw)
        assert ei.value.code == 2
    A.close()


@pytest.mark.parametrize("ell", [1, 2, 3, 4])
def test_bicgstabl_degrees(pkg, sysx, ell):
    """BiCGStab(ℓ) for every supported ℓ, mixed precision with reliable
    updates, transposed as well (the adjoint path)."""
    S, b, xd = sysx
    A = _op(pkg, S)
    for tr in (False, True):
        x, st = A.solve(b, tol=1e-8, precision="mixed", method="bicgstabl", ell=ell, transpose=tr)
        M = S.A.T if tr else S.A
        rel = np.linalg.norm(b - M @ x) / np.linalg.norm(b)
        assert rel <= 1e-8 * 1.01, (ell, tr, rel, st)
        assert st[0]["matvecs"] >= 2 * ell
    A.close()


@pytest.mark.parametrize("ell", [1, 2, 3, 4])
@pytest.mark.parametrize("N", [(4, 3, 2), (33, 9, 7), (40, 24, 26)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_reductions_of_every_ell(pkg, oracle, N, ell, precision):
    """The Gram matrix, the closing update and the dot products of
    BiCGStab(1 … 4) on systems of 72 to 75 k unknowns — fewer element pairs
    than one block's threads, an odd count, and several blocks: the true
    residual, recomputed with the oracle's matrix, meets the tolerance."""
    S = _system(oracle, N, spheres=False) if min(N) > 6 else None
    if S is None:
        g = oracle.uniform_grid(N)
        S = oracle.System(g, 2 * np.pi / 7.0, ((0, 0, 0), (0, 0, 0)), [])
    A = _op(pkg, S)
    rng = np.random.default_rng(5)
    b = rng.standard_normal(A.n) + 1j * rng.standard_normal(A.n)
    x, st = A.solve(b, tol=1e-8, precision=precision, ell=ell)
    rel = np.linalg.norm(b - S.A @ x) / np.linalg.norm(b)
    assert rel <= 1e-8 * 1.01, (rel, st)
    A.close()


@pytest.mark.parametrize("N", [(2, 2, 2), (31, 9, 2), (64, 40, 70)])
def test_residual_norm(pkg, oracle, N):
    """‖b − A x‖² of fdfd_residual_dev (the FP64 block and grid sums) against
    numpy: one block, a partial block, many blocks."""
    torch = pytest.importorskip("torch")
    g = oracle.uniform_grid(N)
    S = oracle.System(g, 2 * np.pi / 7.0, ((0, 0, 0), (0, 0, 0)), [])
    A = _op(pkg, S)
    rng = np.random.default_rng(6)
    v = [torch.from_numpy(rng.standard_normal((A.n, 2))).cuda() for _ in range(2)]
    r = torch.empty_like(v[0])
    rr = A.residual_dev(v[0].data_ptr(), v[1].data_ptr(), r.data_ptr())
    ref = np.linalg.norm(r.cpu().numpy()) ** 2
    assert abs(rr - ref) <= 1e-13 * ref
    A.close()


@pytest.mark.parametrize("ell", [1, 2, 4])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_exact_after_one_step(pkg, oracle, precision, ell):
    """A right-hand side on a pinned wall DOF only (its row of A is
    −ω²ε alone): the first BiCG step solves it exactly and the second breaks
    down (A u = 0); the completed step's update of x must survive that."""
    g = oracle.uniform_grid((6, 5, 4))
    om = 0.5  # −ω² = −1/4: every product of the step is exact
    S = oracle.System(g, om, ((0, 0, 0), (0, 0, 0)), [])
    A = _op(pkg, S)
    b = np.zeros(A.n, complex)
    b[1 + 3 * (0 + 6 * (2 + 5 * 1))] = 1.0  # E_y at i = 0
    x, st = A.solve(b, tol=1e-10, precision=precision, ell=ell)
    assert np.linalg.norm(b - S.A @ x) <= 1e-10, st
    A.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_methods_in_turn_on_one_handle(pkg, sysx, precision):
    """BiCGSTAB, BiCGStab(4) and BiCGSTAB again on one handle, each from its
    captured graph: the second BiCGSTAB solve replays the first one's, whose
    reduction buffer the solve between them must not have replaced, and takes
    the same steps to the same result."""
    S, b, xd = sysx
    A = _op(pkg, S)
    got = [A.solve(b, tol=1e-8, precision=precision, method=m) for m in ("bicgstab", "bicgstabl", "bicgstab")]
    for x, st in got:
        assert np.linalg.norm(b - S.A @ x) <= 1.01e-8 * np.linalg.norm(b), st
    assert np.array_equal(got[0][0], got[2][0])
    assert got[0][1][0]["iterations"] == got[2][1][0]["iterations"]
    A.close()


def _shadow(dof):
    """The library's BiCGStab(l) shadow vector, in units of 1/32768: both halves of the 32-bit hash, as signed integers."""
    x = dof.astype(np.uint64)
    for mul, shift in ((0x7feb352d, 16), (0x846ca68b, 15)):
        x = ((x ^ (x >> np.uint64(shift))) * np.uint64(mul)) & np.uint64(0xffffffff)
    x ^= x >> np.uint64(16)
    return (x & np.uint64(0xffff)).astype(np.uint16).view(np.int16).astype(np.int64), \
        (x >> np.uint64(16)).astype(np.uint16).view(np.int16).astype(np.int64)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_breakdown_at_the_end_of_a_cycle(pkg, precision):
    """A cycle of BiCGStab(1) whose minimal-residual coefficient is exactly 0
    ends in a breakdown with its step already in x, once.  On pinned wall
    DOFs A is diagonal; with d = 2 on the set P, d = −1 on Q and b the shadow
    vector r̂ there, α = (r̂, b)/(r̂, D b) = 1 and (D r, r) = 0 when
    Σ_P |r̂|² = 2 Σ_Q |r̂|² — on entries of r̂ with so few bits that every
    product and sum is exact.  One step: x = b, ‖b − A x‖ = √2 ‖b‖."""
    N = (128, 128, 4)
    cell = np.arange(N[0] * N[1])
    dof = np.sort(np.concatenate([3 * cell, 3 * cell + 1]))  # E_x, E_y on the plane k = 0
    re, im = _shadow(dof)
    few = (re % 16 == 0) & (im % 16 == 0) & (re != 0)
    dof, re, im = dof[few][:60], re[few][:60] // 16, im[few][:60] // 16
    K = re * re + im * im
    i, j = np.triu_indices(len(dof), 1)
    pair = {int(s): q for q, s in enumerate(K[i] + K[j])}
    found = None
    for q in range(len(i)):  # Σ over two pairs = 2 Σ over a third one
        for p in range(len(i)):
            r = pair.get(int(2 * (K[i[q]] + K[j[q]]) - K[i[p]] - K[j[p]]))
            if r is not None and len({i[q], j[q], i[p], j[p], i[r], j[r]}) == 6:
                found = ([i[p], j[p], i[r], j[r]], [i[q], j[q]])
                break
        if found:
            break
    P, Q = (dof[f] for f in found)
    sdl = [np.ones(n, complex) for n in N]
    A = pkg.FDFDOperator(N, 1.0, sdl, sdl)  # pinned rows: −ω² ε = −ε
    eps = np.ones(N + (3,))
    for d in P:
        eps[(d // 3) % N[0], (d // 3) // N[0], 0, d % 3] = -2.0
    A.set_eps(eps)
    b = np.zeros(A.n, complex)
    for f in found:
        b[dof[f]] = (re[f] + 1j * im[f]) / 2048.0
    with pytest.raises(pkg.FDFDError) as ei:
        A.solve(b, tol=1e-6, precision=precision, ell=1, maxit=1, check_every=1)
    st = ei.value.stats[0]
    assert st["iterations"] == 1
    assert abs(st["relres"] - np.sqrt(2.0)) <= 1e-12
    assert np.array_equal(ei.value.x, b)
    A.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_graphs_follow_the_off_diagonal_tensor(pkg, oracle, sysx, monkeypatch, precision):
    """Vacuum, a smoothed sphere and vacuum again on one handle with a forced
    z-chunk (no tuning in between): each solve's captured batch has the
    operator of its own ε, so it takes the steps of a fresh handle's solve."""
    monkeypatch.setenv("FDFD_KCHUNK", "4")
    S, b, xd = sysx
    ones = np.ones(S.grid.N + (3,))
    A = pkg.FDFDOperator(S.grid.N, S.omega, S.sdl_e, S.sdl_m)
    for eps in ((ones, None), (S.eps_diag, S.eps_off), (ones, None)):
        A.set_eps(*eps)
        x, st = A.solve(b, tol=1e-8, precision=precision, maxit=5000)
        B = pkg.FDFDOperator(S.grid.N, S.omega, S.sdl_e, S.sdl_m)
        B.set_eps(*eps)
        y, sb = B.solve(b, tol=1e-8, precision=precision, maxit=5000)
        assert st[0]["iterations"] == sb[0]["iterations"]
        assert np.array_equal(x, y)
        B.close()
    A.close()
