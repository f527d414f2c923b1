"""The accelerated solve gives the same bits in every process: which tile runs a
product is timed only among tiles that sum in the same order, and the order is
chosen by rules. (Tiles that tie used to be picked by a coin toss from process to
process, and the accelerated form turns another rounding of X or of a refinement
product into 1e-9 of its density.) Fresh processes with empty tuner tables."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_RUN = r"""
import sys
import numpy as np
import geometry
import tinyscf
from conftest import BAS, DFBAS
out = []
for n in (13, 20, 23, 37, 40):
    geometry.write_xyz(sys.argv[1] + ".xyz", geometry.alkane(n))
    e = tinyscf.TinySCF(BAS, DFBAS, sys.argv[1] + ".xyz", 100)
    e.s.ene_tol = 1e-8
    e.setup(guess=tinyscf.GUESS_LEARNED)
    out.append(e.mat("X_mat").ravel())
    e.set_k_precision(tinyscf.K_MIXED)
    e.set_density_solver(tinyscf.DENSITY_REFINE)
    e.set_graph(True)
    e.reset_scf()
    e.do_SCF()
    out.append(e.mat("D_mat").ravel())
    e.free()
np.save(sys.argv[1], np.concatenate(out))
"""


def test_same_bits_in_fresh_processes(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([here, os.path.join(os.path.dirname(here), "yatscf-df_b200"),
                                                        os.environ.get("PYTHONPATH", "")]))
    env.pop("TINYSCF_TUNE_FILE", None)
    out = []
    for k in range(4):
        path = str(tmp_path / ("p%d.npy" % k))
        res = subprocess.run([sys.executable, "-c", _RUN, path], env=env, capture_output=True, text=True, timeout=600)
        assert res.returncode == 0, res.stderr[-2000:]
        out.append(np.load(path))
    for x in out[1:]:
        assert np.array_equal(out[0], x), np.abs(out[0] - x).max()
