"""Small FP64 products and the one-launch Newton-Schulz iterations, through the
accelerated form that uses them (orbital alignment of the incremental K,
re-orthonormalisation of the refined orbitals), on either side of the largest
occupied dimension that fits one CTA (84) and at the smallest ones.

Tolerance: the accelerated form ends with an FP64 Fock build on a density whose
error enters the energy in second order; both forms stop at |dE| < 1e-9, so
they agree to 1e-8 Eh."""
import pytest

import geometry
import tinyscf
from conftest import BAS, DFBAS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nocc", [(0, 5), (1, 4), (4, 17), (20, 81), (21, 85)])
def test_accelerated_form_matches_plain(tmp_path, n, nocc):
    path = str(tmp_path / "m.xyz")
    geometry.write_xyz(path, geometry.alkane(n) if n else geometry.water())
    energies = []
    for accelerated in (False, True):
        e = tinyscf.TinySCF(BAS, DFBAS, path, 60)
        assert e.s.n_occ == nocc
        e.setup(guess=tinyscf.GUESS_LEARNED if accelerated else None)
        if accelerated:
            e.set_k_precision(tinyscf.K_MIXED)
            e.set_density_solver(tinyscf.DENSITY_REFINE)
        e.s.ene_tol = 1e-9
        e.do_SCF()
        energies.append(e.energy)
        if accelerated:
            assert e.counters()[4] > 0     # refinement steps ran
        e.free()
    assert abs(energies[0] - energies[1]) < 1e-8, energies
