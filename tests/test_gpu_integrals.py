"""The integral kernels on shells that cc-pVDZ does not have: s shells with 49
primitive pairs (the Schwarz kernel's lanes take them in two rounds),
contracted p and d shells (its smaller lane groups with several rounds),
contracted auxiliary shells, two to five centres, with every class launched
side by side with the others, against the CPU oracle.

Tolerances: a sum of at most 49 * 50 / 2 primitive quartets of size up to
~30, each rounded at 1e-16 relative, amplified by horizontal recursions over
distances up to 6 Bohr (6^4 / 2^4 at these exponents): 1e-10. The screening
values are relative to their largest. B B^T sees the metric's inverse (its
condition number stays below 1e6 here): 1e-8."""
import numpy as np
import pytest

import oracle
import tinyscf

pytestmark = pytest.mark.gpu

ORB = """!
****
H     0
S   7   1.00
   120.0   0.002
    31.0   0.015
     9.1   0.07
     3.3   0.2
     1.3   0.4
     0.5   0.4
     0.2   0.1
P   3   1.00
     3.1   0.1
     0.9   0.5
     0.3   0.6
D   2   1.00
     1.4   0.4
     0.5   0.7
****
"""
AUX = """!
****
H     0
S   3   1.00
    22.0   0.2
     6.0   0.6
     1.9   0.5
S   1   1.00
     0.6   1.0
P   2   1.00
     2.4   0.5
     0.8   0.6
D   2   1.00
     2.1   0.4
     0.9   0.7
F   2   1.00
     1.9   0.6
     0.8   0.5
****
"""
CENTRES = [(0.0, 0.0, 0.0), (0.9, 0.2, -0.3), (-0.5, 1.4, 0.6), (2.6, -1.1, 0.4), (0.3, 0.5, 2.9)]


@pytest.mark.parametrize("natoms", [2, 3, 5])
def test_contracted_shells_against_oracle(tmp_path, natoms):
    bas, aux, mol = tmp_path / "orb.gbs", tmp_path / "aux.gbs", tmp_path / "m.xyz"
    bas.write_text(ORB)
    aux.write_text(AUX)
    charge = natoms % 2
    mol.write_text("%d\n%d\n" % (natoms, charge) + "".join("H %.6f %.6f %.6f\n" % c for c in CENTRES[:natoms]))
    e = tinyscf.TinySCF(str(bas), str(aux), str(mol), 10)
    e.setup()
    o = oracle.OracleSCF(str(bas), str(aux), str(mol), 10)
    o.setup()
    n, nsh = e.s.nbasfuncs, e.s.nshells
    assert np.abs(e.mat("S_mat") - o.S).max() < 1e-12
    assert np.abs(e.mat("Hcore_mat") - o.H).max() < 1e-10
    sp = e._mat("sp_scrval", (nsh * nsh,))
    bf = e._mat("bf_pair_scrval", (n * n,))
    df = e._mat("df_sp_scrval", (e.s.df_nshells,))
    assert np.abs(sp - o.sp_scrval).max() < 1e-10 * o.sp_scrval.max()
    assert np.abs(bf - o.bf_pair_scrval).max() < 1e-10 * o.bf_pair_scrval.max()
    assert np.abs(df - o.df_sp_scrval).max() < 1e-12 * o.df_sp_scrval.max()
    mask, _, _ = e.csr()
    assert (mask == o.bf_pair_mask).all()
    B = e.df_tensor()
    assert np.abs(B @ B.T - o.df_tensor @ o.df_tensor.T).max() < 1e-8
    e.free()
