"""An engine on a host without pinned memory to give: it works by copies.  The
allocation is refused by a stand-in for the runtime's call in a child process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

REFUSE = """
int cudaHostAlloc(void **p, unsigned long n, unsigned f) { (void)n; (void)f; *p = 0; return 2; }   /* cudaErrorMemoryAllocation */
"""
USE = """
import sys
import numpy as np
from surfactant_enhanced_spreading_gb300 import config_preset as C, engine as E
s = C.config_droplet(200, 2, cells=(8, 8, 8), seed=5)
eng = E.Engine(s, E.MIXED)
E.mybox_start(eng)
eng.run(99101, 12)
np.savez(sys.argv[1], *eng.state(), eng.forces(), np.array([eng.temperature(), eng.eta]))
"""


def test_results_do_not_need_it(tmp_path):
    import numpy as np
    src, lib, use = tmp_path / "refuse.c", tmp_path / "refuse.so", tmp_path / "use.py"
    src.write_text(REFUSE)
    use.write_text(USE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = []
    for name, preload in (("with", ""), ("without", str(lib))):
        f = tmp_path / (name + ".npz")
        env = dict(os.environ, PYTHONPATH=root)
        if preload:
            env["LD_PRELOAD"] = preload
        r = subprocess.run([sys.executable, str(use), str(f)], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        out.append(np.load(f))
    for k in out[0].files:
        assert np.array_equal(out[0][k], out[1][k])
