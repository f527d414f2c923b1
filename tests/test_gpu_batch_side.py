"""The molecules of a batch whose K builds, refinements and eigensolves run side
by side: the same arithmetic as a batch of each molecule alone, so the same
energies, densities and iteration counts bit for bit."""
import numpy as np
import pytest

import geometry
import tinyscf
from conftest import BAS, DFBAS, xyz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed, refine", [(True, True), (True, False), (False, True), (False, False)])
def test_side_by_side_matches_each_alone(tmp_path, mixed, refine):
    # more molecules than side streams, several of one size and several sizes; every third one
    # has the other density solver
    paths = [xyz("water"), xyz("water"), xyz("c10h22")]
    for seed in range(8):
        p = str(tmp_path / ("w%d.xyz" % seed))
        geometry.write_xyz(p, geometry.water_cluster(seed, nmax=5))
        paths.append(p)

    def solve(picked):
        engines = []
        for k in picked:
            e = tinyscf.TinySCF(BAS, DFBAS, paths[k], 60)
            e.setup(guess=tinyscf.GUESS_LEARNED)
            if mixed:
                e.set_k_precision(tinyscf.K_MIXED)
            if refine != (k % 3 == 2):
                e.set_density_solver(tinyscf.DENSITY_REFINE)
            engines.append(e)
        b = tinyscf.TinySCFBatch(engines)
        b.do_SCF()
        out = [(e.energy, e.s.iter, e.mat("D_mat").copy()) for e in engines]
        b.free()
        for e in engines:
            e.free()
        return out

    alone = [solve([k])[0] for k in range(len(paths))]
    together = solve(list(range(len(paths))))
    for (E, it, D), (E1, it1, D1) in zip(together, alone):
        assert it == it1
        assert E == E1
        assert np.array_equal(D, D1)
