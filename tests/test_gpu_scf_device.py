"""The RHF iteration's device steps (Fock rows, gradients and DIIS sums over lists
of up to 16 slots a launch) against the oracle's RHF: subspaces of one, of a
full list, and of more than one list."""
import pytest

from mpqc_gb300 import RHF, molecules
from oracle import molecule as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,basis", [(1, "6-31G"), (2, "cc-pVDZ")])
@pytest.mark.parametrize("n_diis", [1, 4, 16, 20])
def test_rhf_energy_for_every_subspace(n, basis, n_diis):
    sym, xyz = molecules.water_cluster(n, seed=5)
    mol = M.Molecule(list(sym), molecules.to_bohr(xyz))
    S, H, G = M.ao_integrals_c(mol, basis)
    ref = M.rhf(S, H, G, mol.n_electrons() // 2, mol.nuclear_repulsion())
    with RHF(sym, xyz, basis, threshold=1e-10, max_iter=400, n_diis=n_diis) as scf:
        e = scf.run()
    # both converged to 1e-10
    assert abs(e - ref.energy) < 1e-9
