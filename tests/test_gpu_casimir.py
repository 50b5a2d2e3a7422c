"""The scuff-cas3D integrand on the GPU: two PEC icospheres (subdivision 3,
1280 panels and 1920 RWG edges each, N = 3840 real), centres 3 apart, at the
20-point Gauss-Laguerre frequencies xi = x_j / g for g = 1 (surface gap) and
g = 3 (centre gap).

* The energy and z-force integrands against the reference's own (its
  unchanged scuff-cas3D, GetCasimirIntegrand, CasimirIntegrand.cc:243-480,
  run by tests/golden/make_golden.py on the same mesh).
* The U block and its derivative dU/dz against the oracle (assembly, and
  central differences of the assembly) at one frequency."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bodies():
    from gbem import mesh
    V, P = mesh.icosphere(3)
    return V, P, [{"V": V, "P": P, "material": None}, {"V": V + [0.0, 0.0, 3.0], "P": P, "material": None}]


@pytest.fixture(scope="module")
def cas():
    from gbem.casimir import CasimirIntegrand
    return CasimirIntegrand(_bodies()[2])


def test_casimir_integrand_matches_reference(cas, golden):
    d = golden("ref_pec2_s3_casimir.npz")
    E = np.zeros(len(d["xi"]))
    F = np.zeros(len(d["xi"]))
    for i, xi in enumerate(d["xi"]):
        E[i], F[i] = cas(float(xi))
    for g in (1.0, 3.0):
        sel = d["gap"] == g
        # scale: the largest integrand over the rule (the integrands fall off
        # by e^{-2 xi gap}); the reference's adaptive near-field cubature
        # carries ~1e-6 relative of each T block's entries
        eE = np.abs(E[sel] - d["energy"][sel]).max() / np.abs(d["energy"][sel]).max()
        eF = np.abs(F[sel] - d["zforce"][sel]).max() / np.abs(d["zforce"][sel]).max()
        print("gap %g: energy %.2e force %.2e" % (g, eE, eF))
        assert eE < 1e-5, (g, eE)
        assert eF < 1e-5, (g, eF)


def test_u_block_and_gradient_match_oracle(cas, golden):
    from oracle import oracle
    V, P, bodies = _bodies()
    G = cas.G
    xi = float(golden("ref_pec2_s3_casimir.npz")["xi"][9])
    n1 = G.NumBFs(0)
    U = G.AssembleBEMMatrixBlock(0, 1, 1j * xi, real=True)
    dUz = G.AssembleBEMMatrixBlockGradient(0, 1, 1j * xi, real=True, components=(2,))[2]
    rng = np.random.default_rng(4)
    cols = np.sort(rng.choice(n1, 12, replace=False))

    def ora_u(dz):
        Sa = oracle.Surface(V + [0.0, 0.0, dz], P)
        Sb = oracle.Surface(V + [0.0, 0.0, 3.0], P)
        M = oracle.assemble_cols([Sa, Sb], [(0, -1), (0, -1)], [True, True], 1j * xi, [1.0], [1.0], n1 + cols)
        return M[:n1]

    Uo = ora_u(0.0)
    assert np.abs(Uo.imag).max() <= 1e-14 * np.abs(Uo).max()
    assert np.abs(U[:, cols] - Uo.real).max() / np.abs(Uo).max() < 1e-11
    h = 1e-4
    dUo = (ora_u(h) - ora_u(-h)).real / (2 * h)
    # central differences: truncation ~h^2 of the entries' third derivative
    assert np.abs(dUz[:, cols] - dUo).max() / np.abs(dUo).max() < 1e-6


def _three_bodies(pec, gap):
    from gbem import RWGGeometry, mesh
    from gbem.api import Material
    m = None if pec else Material(2.5)
    V0, P0 = mesh.icosphere(1)
    V1, P1 = mesh.rounded_cube(108, seed=4)
    V2, P2 = mesh.icosphere(0)
    return RWGGeometry([{"V": V0, "P": P0, "material": m},
                        {"V": V1 + [0.2, 0.1, 1.5 + gap], "P": P1, "material": m},
                        {"V": 0.7 * V2 - [1.8 + gap, 0.3, 0.0], "P": P2, "material": None}])


@pytest.mark.parametrize("gap", [0.1, 4.0])
@pytest.mark.parametrize("pec", [True, False])
@pytest.mark.parametrize("omega", [0.5j, 1.1, 0.8 + 0.2j])
def test_trace_of_a_displacement_equals_the_trace_of_its_blocks(omega, pec, gap):
    """Bodies of unequal size, with (gap 0.1) and without near pairs, every axis,
    real and complex storage: the trace with dM assembled on the device equals the
    trace with the same gradient blocks put in place on the host.  The blocks
    are the same numbers, and so is the solve: equal to the last bit."""
    from gbem._lib import C128, F64
    from gbem.api import HMatrix
    G = _three_bodies(pec, gap)
    off = np.concatenate([[0], np.cumsum([G.NumBFs(s) for s in range(3)])])
    for dt in (F64, C128) if omega == 0.5j else (C128,):
        M = G.AssembleBEMMatrix(omega, HMatrix(G, dt))
        assert M.LUFactorize() == 0
        for axis in range(3):
            dM = np.zeros((G.TotalBFs, off[1]), dtype=M.np_dtype, order="F")
            for s in (1, 2):
                g = G.AssembleBEMMatrixBlockGradient(0, s, omega, real=dt == F64, components=(axis,))[axis]
                dM[off[s]:off[s + 1]] = g.T
            want = M.TraceMInvdM(dM, int(off[1]))
            assert M.TraceMInvDisplacement(G, omega, axis) == want


def test_trace_of_a_displacement_takes_its_own_geometry_only():
    """The blocks come from the matrix's geometry: another one (fewer regions,
    other meshes) is refused."""
    from gbem import RWGGeometry, mesh
    from gbem.api import Material
    V, P = mesh.icosphere(0)
    def geo(shift, m=None):
        return RWGGeometry([{"V": V, "P": P, "material": m}, {"V": V + [0.0, 0.0, shift], "P": P, "material": m}])
    G = geo(4.0, Material(2.0))
    M = G.AssembleBEMMatrix(1.0)
    assert M.LUFactorize() == 0
    t = M.TraceMInvDisplacement(G, 1.0)
    assert M.TraceMInvDisplacement(geo(4.0, Material(2.0)), 1.0) == t
    for other in (geo(4.0), geo(5.0, Material(2.0)), RWGGeometry([{"V": V, "P": P, "material": Material(2.0)}])):
        with pytest.raises(ValueError):
            M.TraceMInvDisplacement(other, 1.0)
