"""Field post-processing on the GPU against the oracle: h_from_e
(src/model/model.jl:276-279) and the create_Mcs corner means (:287-306),
on PEC and Bloch grids with SC-PML, ≤ 1e-12 relative (FP64 both sides).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(O, bloch):
    rng = np.random.default_rng(31)
    lp = tuple(np.concatenate([[0.0], np.cumsum(rng.uniform(0.6, 1.4, n))]) for n in (13, 11, 9))
    return O.Grid(lp, bloch)


CASES = [((False, False, False), (0.0, 0.0, 0.0)), ((True, False, True), (0.13, 0.0, -0.21))]


@pytest.mark.parametrize("bloch,kb", CASES)
def test_h_from_e(pkg, oracle, bloch, kb):
    O = oracle
    g = _grid(O, bloch)
    om = 2 * np.pi / 6.5
    npml = ((0 if bloch[0] else 2, 2, 0 if bloch[2] else 2), (0 if bloch[0] else 2, 2, 0 if bloch[2] else 2))
    sdl_e, sdl_m = O.stretched_dl(g, om, npml)
    Ce, _ = O.create_curls(g, sdl_e, sdl_m, kb)
    ph = [np.exp(-1j * kb[w] * g.L[w]) for w in range(3)]
    A = pkg.FDFDOperator(g.N, om, sdl_e, sdl_m, bloch, ph)
    rng = np.random.default_rng(32)
    n = 3 * g.ncell
    e = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    jm = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    for j in (None, jm):
        ref = O.h_from_e(e, om, Ce, j)
        got = A.h_from_e(e, j)
        assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
    A.close()


@pytest.mark.parametrize("bloch,kb", CASES)
def test_corner_means(pkg, oracle, bloch, kb):
    O = oracle
    g = _grid(O, bloch)
    om = 2 * np.pi / 6.5
    npml = ((0 if bloch[0] else 2, 2, 0 if bloch[2] else 2), (0 if bloch[0] else 2, 2, 0 if bloch[2] else 2))
    sdl_e, sdl_m = O.stretched_dl(g, om, npml)
    Mce, Mcm = O.create_Mcs(g, sdl_e, sdl_m, kb)
    ph = [np.exp(-1j * kb[w] * g.L[w]) for w in range(3)]
    A = pkg.FDFDOperator(g.N, om, sdl_e, sdl_m, bloch, ph)
    rng = np.random.default_rng(33)
    n = 3 * g.ncell
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    for field, M in (("E", Mce), ("H", Mcm)):
        ref = M @ v
        got = A.corner_mean(v, field)
        assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref)), field
    A.close()


@pytest.mark.parametrize("bloch,kb", CASES)
def test_e_from_h(pkg, oracle, bloch, kb):
    """e_from_h (model.jl:281-284) with a diagonal ε against the oracle, and
    its rejection of an off-diagonal ε (the reference's Pε \\ needs a
    diagonal one)."""
    O = oracle
    g = _grid(O, bloch)
    om = 2 * np.pi / 6.5
    npml = ((0 if bloch[0] else 2, 2, 0 if bloch[2] else 2), (0 if bloch[0] else 2, 2, 0 if bloch[2] else 2))
    sdl_e, sdl_m = O.stretched_dl(g, om, npml)
    _, Cm = O.create_curls(g, sdl_e, sdl_m, kb)
    ph = [np.exp(-1j * kb[w] * g.L[w]) for w in range(3)]
    A = pkg.FDFDOperator(g.N, om, sdl_e, sdl_m, bloch, ph)
    rng = np.random.default_rng(34)
    ed = rng.uniform(1.0, 12.25, g.N + (3,))
    A.set_eps(ed)
    n = 3 * g.ncell
    h = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    je = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    for j in (None, je):
        ref = O.e_from_h(h, om, O.field_to_vec(ed), Cm, j)
        got = A.e_from_h(h, j)
        assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
    eo = np.zeros(g.N + (3,))
    eo[2, 2, 2, 0] = 0.5
    A.set_eps(ed, eo)
    with pytest.raises(pkg.FDFDError):
        A.e_from_h(h)
    A.close()


@pytest.mark.parametrize("bloch", [(False, False, False), (True, False, False), (False, True, False),
                                   (False, False, True), (True, True, True)])
@pytest.mark.parametrize("N", [(2, 2, 2), (3, 43, 2), (64, 4, 5), (129, 2, 35)])
def test_field_kernels_plane_edges(pkg, oracle, bloch, N):
    """h_from_e and the corner means where their kernels can go wrong: planes
    of one cell more or less than the 256-thread block, of several blocks,
    one-plane and several-plane z-chunks, each axis periodic in turn, and
    real and complex ω (the factor i/ω folded into the curl or not).  The
    bound is that of the other tests here (FP64 on both sides)."""
    O = oracle
    rng = np.random.default_rng(41)
    lp = tuple(np.concatenate([[0.0], np.cumsum(rng.uniform(0.6, 1.4, n))]) for n in N)
    g = O.Grid(lp, bloch)
    kb = tuple(0.17 if b else 0.0 for b in bloch)
    npml = tuple(0 if bloch[w] or N[w] < 8 else 3 for w in range(3))
    for om in (2 * np.pi / 6.5, 0.9 + 0.2j):
        sdl_e, sdl_m = O.stretched_dl(g, 2 * np.pi / 6.5, (npml, npml))
        Ce, _ = O.create_curls(g, sdl_e, sdl_m, kb)
        Mce, Mcm = O.create_Mcs(g, sdl_e, sdl_m, kb)
        A = pkg.FDFDOperator(g.N, om, sdl_e, sdl_m, bloch, [np.exp(-1j * kb[w] * g.L[w]) for w in range(3)])
        n = 3 * g.ncell
        v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        jm = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        for got, ref in ((A.h_from_e(v, jm), O.h_from_e(v, om, Ce, jm)), (A.h_from_e(v), O.h_from_e(v, om, Ce, None)),
                         (A.corner_mean(v, "E"), Mce @ v), (A.corner_mean(v, "H"), Mcm @ v)):
            assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
        A.close()


@pytest.mark.parametrize("N,bloch", [((1, 1, 37), (True, True, False)), ((2, 2, 19), (False, False, True)),
                                     ((3, 5, 7), (False, True, False)), ((16, 1, 5), (False, True, True)),
                                     ((4, 4, 40), (False, False, False)), ((17, 1, 6), (True, True, False))])
def test_field_kernels_thin_planes(pkg, oracle, N, bloch):
    """h_from_e and the corner means on planes of 1, 4, 15, 16 and 17 cells,
    where several z-chunks share a warp (and where they just do not), with
    the last warp part full; the bound is that of the other tests here."""
    O = oracle
    rng = np.random.default_rng(43)
    lp = tuple(np.concatenate([[0.0], np.cumsum(rng.uniform(0.6, 1.4, n))]) for n in N)
    g = O.Grid(lp, bloch)
    kb = tuple(0.17 if b else 0.0 for b in bloch)
    npml = tuple(0 if bloch[w] or N[w] < 8 else 3 for w in range(3))
    om = 2 * np.pi / 6.5
    sdl_e, sdl_m = O.stretched_dl(g, om, (npml, npml))
    Ce, _ = O.create_curls(g, sdl_e, sdl_m, kb)
    Mce, Mcm = O.create_Mcs(g, sdl_e, sdl_m, kb)
    A = pkg.FDFDOperator(g.N, om, sdl_e, sdl_m, bloch, [np.exp(-1j * kb[w] * g.L[w]) for w in range(3)])
    v = rng.standard_normal(A.n) + 1j * rng.standard_normal(A.n)
    jm = rng.standard_normal(A.n) + 1j * rng.standard_normal(A.n)
    for got, ref in ((A.h_from_e(v, jm), O.h_from_e(v, om, Ce, jm)), (A.corner_mean(v, "E"), Mce @ v),
                     (A.corner_mean(v, "H"), Mcm @ v)):
        assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
    A.close()
