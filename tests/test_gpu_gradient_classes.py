"""The gradient of every angular class: a random symmetric density on water (no SCF, so
nothing cancels) against central differences of the energy expression from the GPU's own
integrals, with and without Schwarz screening."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WATER = np.array([[0.0, -0.0758, 0.02], [0.8668, 0.6014, 0.0], [-0.7, 0.65, 0.31]])


def _molecule(xyz, basis):
    from mmd.molecule import Molecule
    rows = "\n".join(f"{s} {x:.14f} {y:.14f} {z:.14f}" for s, (x, y, z) in zip("OHH", xyz))
    return Molecule("\n0 1\n" + rows + "\n", basis)


def _energy(xyz, basis, P, W):
    mol = _molecule(xyz, basis)
    mol.build(direct=False)
    T = mol.TwoE
    return (2 * np.sum(P * mol.Core) - 2 * np.sum(W * mol.S) + 2 * np.einsum("ij,kl,ijkl", P, P, T)
            - np.einsum("ik,jl,ijkl", P, P, T) + mol.nuc_energy)


@pytest.mark.parametrize("basis", ["sto-3g", "6-31gss", "6-31ppgss", "cc-pvdz"])
def test_gradient_of_a_random_density(basis):
    from mmd.molecule import ANGSTROM
    mol = _molecule(WATER, basis)
    N = mol.nbasis
    rng = np.random.default_rng(N)
    P, F = (0.2 * (A + A.T) for A in rng.standard_normal((2, N, N)))
    mol.P, mol.F, mol.is_converged = P, F, True
    W = P @ F @ P
    full = mol.forces(qtol=0.0)
    # skipped quartets are below 1e-16 each; up to N^4/8 of them, weights below 1
    assert np.abs(mol.forces() - full).max() < 1e-16 * N ** 4
    # central differences: truncation h^2/6 E''' (third derivatives of core terms reach ~1e3 in
    # these units, E ~ 1e2) and rounding 1e-16 E N / h: 1e-4 bohr leaves a few 1e-6
    h = 1e-4
    for atom, d in ((0, 0), (0, 2), (1, 1), (2, 0)):
        step = np.zeros((3, 3))
        step[atom, d] = h * ANGSTROM
        fd = -(_energy(WATER + step, basis, P, W) - _energy(WATER - step, basis, P, W)) / (2 * h)
        assert abs(full[atom, d] - fd) < 1e-5 * max(1.0, abs(fd))
