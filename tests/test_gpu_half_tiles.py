"""The exchange half-transform's tiles fitted to the occupied dimension: at the
edges of each warp layout (one, two or three rows of warps, more than one tile)
and of its blocks of 8, 16 and 24 occupied orbitals, both aux widths, against the
64 x 64 tile kernel on the same density. (An odd number of auxiliary functions
takes the copies of k_halftransform_pipe: test_gpu_tune.py's HCN.)

Every output is one chain of multiply-adds over the same k in all of these
kernels, so T is the same bit for bit; K = T T^T then runs on the same kernel
for both (autotuner off), and must be equal."""
import os
import subprocess
import sys

import numpy as np
import pytest

import geometry
from conftest import BAS, DFBAS, PKG

pytestmark = pytest.mark.gpu

_RUN = r"""
import sys
import numpy as np
import tinyscf
e = tinyscf.TinySCF(sys.argv[1], sys.argv[2], sys.argv[3], 5)
e.setup()
n, o = e.s.nbasfuncs, e.s.n_occ
C = np.random.default_rng(3).normal(size=(n, o)) / n ** 0.5
e.set_density(C @ C.T, C)
e.build_FockMat()
np.save(sys.argv[4], e.mat("K_mat"))
e.free()
"""


def atoms(name):
    kind, n = name[0], int(name[1:])
    return geometry.alkane(n) if kind == "c" else geometry.water_cluster(11, n, n)


# o = 5, 17, 55, 57 (c14), 65 (w13), 85 (c21), 89 (c22), 125 (c31), 129 (c32), 169 (c42: two parts of 85)
@pytest.mark.parametrize("name", ["w1", "c4", "w11", "c14", "w13", "c21", "c22", "c31", "c32", "c42"])
def test_fitted_tiles_equal_square_tiles(tmp_path, name):
    xyz = str(tmp_path / "m.xyz")
    geometry.write_xyz(xyz, atoms(name))
    got = {}
    for variant in "034":
        out = str(tmp_path / ("k%s.npy" % variant))
        env = dict(os.environ, TINYSCF_KHALF=variant, TINYSCF_OZAKI="0", PYTHONPATH=PKG)
        tune = tmp_path / "tune.txt"            # the other choices of the first run are the others' too
        env["TINYSCF_TUNE_FILE"] = str(tune)
        subprocess.run([sys.executable, "-c", _RUN, BAS, DFBAS, xyz, out], env=env, check=True, timeout=300)
        got[variant] = np.load(out)
    assert np.array_equal(got["0"], got["3"])
    assert np.array_equal(got["0"], got["4"])
