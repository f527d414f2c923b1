"""The large FP64 product (DF tensor) on the 168 x 96 tiles behind a producer
warp: every output is the same chain of multiply-adds over k as on the 64 x 64
FP64 tensor-core tile, so the two agree bit for bit, with ragged last tiles and
K chunks, column slices of the operand, and the slices that are not aligned for
16-byte copies (which stay on the 128 x 128 tile)."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_RUN = r"""
import sys
import numpy as np
import tinyscf
from conftest import BAS, DFBAS, xyz
out = []
for lo, hi in ((0, 0), (2, 4), (0, 1), (1, 1), (0, 64)):
    e = tinyscf.TinySCF(BAS, DFBAS, xyz("c10h22"), 60)
    if lo or hi:
        e.set_aux_slice(lo, e.s.df_nbf - hi)
    e.setup()
    out.append(e.df_tensor().ravel())
    e.free()
np.save(sys.argv[1], np.concatenate(out))
"""


def test_bulk_tiles_match_the_small_tile(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([here, os.path.join(os.path.dirname(here), "yatscf-df_b200"),
                                                        os.environ.get("PYTHONPATH", "")]))
    keys, out = [], {}
    for variant in (None, 3, 4):
        tune = tmp_path / ("tune%s.txt" % variant)
        tune.write_text("".join("%s %d 0.0\n" % (k, variant) for k in keys))
        res = subprocess.run([sys.executable, "-c", _RUN, str(tmp_path / "B.npy")],
                             env=dict(env, TINYSCF_TUNE_FILE=str(tune)), capture_output=True, text=True, timeout=600)
        assert res.returncode == 0, res.stderr[-2000:]
        if variant is None:
            keys = [line.split()[0] for line in tune.read_text().splitlines() if line.startswith("dgemm:")]
            assert len(keys) >= 5
        out[variant] = np.load(tmp_path / "B.npy")
    assert np.array_equal(out[3], out[4])
