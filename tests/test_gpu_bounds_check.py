"""GPU: the checked build (lib/libtblite_b200_check.so, index guards that skip
and record any global-memory access outside its structure's own slice; no
trap) runs the singlepoint paths in a fresh process -- plain and mixed forms,
the whole-loop graph, d shells, gradients, the nspin = 2 read-out, the
batched generalized eigensolver -- and records no violation; its results
equal the normal build's (1e-10)."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from tblite_b200 import capi, geometry as g

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CHILD = r"""
import json, sys
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[2])
import numpy as np
from tblite_b200 import capi
capi.load_library(capi.LIB_CHECK_PATH)
import run_cases
out = run_cases.run()
out["violations"] = list(capi.bounds_violations())
out["checked"] = int(capi.load_library().tb_bounds_check_build())
print("RESULT " + json.dumps(out))
"""


def test_checked_build_runs_clean_and_agrees():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    here = os.path.dirname(os.path.abspath(__file__))
    p = subprocess.run([sys.executable, "-c", _CHILD, os.path.join(ROOT, "tblite-cuda_b200"),
                        os.path.join(here, "golden")], capture_output=True, text=True, timeout=900)
    assert p.returncode == 0, p.stderr[-3000:]
    line = [s for s in p.stdout.splitlines() if s.startswith("RESULT ")]
    assert line, p.stdout[-2000:] + p.stderr[-2000:]
    got = json.loads(line[-1][len("RESULT "):])
    assert got["checked"] == 1
    assert got["violations"][0] == 0, got["violations"]
    sys.path.insert(0, os.path.join(here, "golden"))
    import run_cases
    ref = run_cases.run()  # the normal build, this process
    for k, v in ref.items():
        np.testing.assert_allclose(np.asarray(got[k], float), np.asarray(v, float), atol=1e-10, err_msg=k)


_LARGER = r"""
import json, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from tblite_b200 import capi, geometry as g
capi.load_library(sys.argv[2])
calc = capi.Calculator()
rng = np.random.default_rng(77)
mols = [g.alkane(n, rng) for n in (11, 37, 38, 75, 120)]  # 68, 224, 230, 452, 722 AOs, each on a cluster
out = [calc.singlepoint_batch([m], solver=1)[0]["energy"] for m in mols]
fill = g.water_clusters(420, seed=5, nmin=4, nmax=30) + [g.alkane(74, rng)]  # one CTA each, two per SM
out += [r["energy"] for r in calc.singlepoint_batch(fill, solver=1)]
out += [r["energy"] for r in calc.singlepoint_batch(fill[:40], solver=1, precision=1)]
for n in (2, 16, 17, 33, 63, 64, 65, 97, 193, 300, 449, 610):
    a = rng.standard_normal((n, n))
    b = 0.1 * rng.standard_normal((n, n))
    st, res = capi.sygvd_batch([0.5 * (a + a.T)], [np.eye(n) + b @ b.T / n])
    out += [float(st)] + res[0][0].tolist()
print("RESULT " + json.dumps({"out": out, "violations": list(capi.bounds_violations()),
                              "checked": int(capi.load_library().tb_bounds_check_build())}))
"""


def test_checked_build_over_the_eigensolvers_shapes():
    # every walk shape, merges on clusters and on one CTA, leaves at two depths, the
    # factorisation with whole and partial blocks
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    got = []
    for lib in (capi.LIB_CHECK_PATH, capi.LIB_PATH):
        p = subprocess.run([sys.executable, "-c", _LARGER, os.path.join(ROOT, "tblite-cuda_b200"), lib],
                           capture_output=True, text=True, timeout=900)
        assert p.returncode == 0, p.stderr[-3000:]
        got.append(json.loads([s for s in p.stdout.splitlines() if s.startswith("RESULT ")][-1][len("RESULT "):]))
    assert [r["checked"] for r in got] == [1, 0]
    assert got[0]["violations"][0] == 0, got[0]["violations"]
    np.testing.assert_allclose(got[0]["out"], got[1]["out"], atol=1e-10, rtol=0)
