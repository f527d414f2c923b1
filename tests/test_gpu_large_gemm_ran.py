"""The DF tensor's product runs on the TMA-fed 168 x 96 tiles where operands and
columns lie on 16-byte units, and not where a slice of the aux index starts at an
odd column or has an odd width."""
import pytest

import tinyscf
from conftest import BAS, DFBAS, xyz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi,bulk", [(0, 0, True), (2, 4, True), (0, 64, True), (0, 1, False), (1, 1, False),
                                        (1, 0, False)])
def test_which_product_runs(lo, hi, bulk):
    e = tinyscf.TinySCF(BAS, DFBAS, xyz("c10h22"), 60)
    if lo or hi:
        e.set_aux_slice(lo, e.s.df_nbf - hi)
    e.compute_Hcore_Ovlp_mat()
    e.compute_sq_Schwarz_scrvals()
    e.prepare_sparsity()
    e.get_initial_guess()
    before = tinyscf.gemm_bulk_count()
    e.build_DF_tensor()
    assert (tinyscf.gemm_bulk_count() > before) == bulk
    e.free()
