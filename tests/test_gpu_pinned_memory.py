"""The engines' page-locked host memory: at most 256 MB a process, pageable
memory beyond (the same results), and given back by trim_memory once no engine
holds it."""
import gc

import numpy as np
import pytest

import geometry
import tinyscf
from conftest import BAS, DFBAS, xyz

pytestmark = pytest.mark.gpu
LIMIT = 256 << 20


def test_trim_gives_idle_blocks_back():
    gc.collect()
    tinyscf.trim_memory()
    held, idle = tinyscf.pinned_memory()
    e = tinyscf.TinySCF(BAS, DFBAS, xyz("c10h22"), 30)
    e.setup()
    e.set_graph(True)
    e.do_SCF()
    assert tinyscf.pinned_memory()[0] > held
    tinyscf.trim_memory()                       # nothing of a live handle is touched
    first = e.energy
    e.reset_scf()
    e.do_SCF()
    assert e.energy == first
    e.free()
    assert tinyscf.pinned_memory()[0] == held
    assert tinyscf.pinned_memory()[1] > 0
    tinyscf.trim_memory()
    assert tinyscf.pinned_memory()[0] == held
    if held == 0:
        assert tinyscf.pinned_memory()[1] == 0


def test_handles_beyond_the_limit(tmp_path):
    path = str(tmp_path / "c40.xyz")
    geometry.write_xyz(path, geometry.alkane(40))
    gc.collect()
    tinyscf.trim_memory()
    es, held = [], []
    for _ in range(5):                          # 80 MB and more of mirrors each
        es.append(tinyscf.TinySCF(BAS, DFBAS, path, 30))
        es[-1].compute_Hcore_Ovlp_mat()
        held.append(tinyscf.pinned_memory()[0])
        assert sum(tinyscf.pinned_memory()) <= LIMIT + (1 << 20)
    assert held[-1] - held[-2] < held[0]        # the last handle no longer fits
    rng = np.random.default_rng(0)
    n, o = es[0].s.nbasfuncs, es[0].s.n_occ
    F = rng.normal(size=(n, n))
    F = F + F.T
    out = []
    for e in (es[0], es[-1]):
        e.set_fock(F, orthogonal=True)
        e.build_DenMat()
        out.append([e.mat(m) for m in ("S_mat", "X_mat", "Hcore_mat", "D_mat")])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    for e in es:
        e.free()
    tinyscf.trim_memory()
    assert tinyscf.pinned_memory()[1] <= 1 << 20
