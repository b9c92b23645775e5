"""The two element passes of a 3D solve with a streamed basis, and the basis ring at two chunks a block.

At m = 40 a block's 42 vectors of 700 unknowns take 235 KB, more than its shared memory, so both meshes
stream their basis: 700 unknowns a block are one chunk, 3260 two.  CFDV_ELEM_RING=0 takes the element
matrices by direct loads and puts the basis ring behind the other arrays; each row sums in the same
order as with the element ring, so whole solves agree bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from test_gpu_streamed_basis import test_streamed_solve_repeats_bit_for_bit as repeats

pytestmark = pytest.mark.gpu

_CHILD = r"""
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
from cfdv_b200 import gpu as G, meshgen as mg
out = {}
for shape in ((34, 30, 18), (60, 50, 30)):
    case = mg.duct(*shape)
    case.nodes[:, 3] *= 1.0 + 1e-3 * np.random.default_rng(1).standard_normal(case.n_nodes)
    with G.FDVSolver(case) as s:
        s.load_node_records()
        s.form(s.cfl(0.5), G.PREC_MIXED)
        for prec in (G.PREC_FP64, G.PREC_MIXED):
            for precond in (False, True):
                r = s.gmres(mode=G.GMRES_CORRECT, m=40, restarts=30, rtol=1e-8, precision=prec, precond=precond)
                k = f"{shape[0]}_{prec}_{int(precond)}"
                out[k], out[k + "_est"] = s.du(), r["est"]
np.savez(sys.argv[2], **out)
"""


def test_element_ring_matches_direct_pass_bitwise(tmp_path):
    res = {}
    for ring in ("1", "0"):
        out = str(tmp_path / f"ring{ring}.npz")
        subprocess.run([sys.executable, "-c", _CHILD, ROOT, out], check=True, timeout=600,
                       env=dict(os.environ, CFDV_ELEM_RING=ring))
        res[ring] = dict(np.load(out))
    assert len(res["1"]) == 16 and res["1"].keys() == res["0"].keys()
    for k in res["1"]:
        assert res["1"][k].any(), k
        np.testing.assert_array_equal(res["1"][k], res["0"][k], err_msg=k)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_two_chunks_repeat_bit_for_bit(precision):
    repeats((60, 50, 30), True, precision)
