"""Results outlive their context: they are read and freed after it, and the
process goes on building and copying."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys
sys.path[:0] = [sys.argv[1] + "/gpu-svo_b200"]
import numpy as np
import svo_b200
from svo_b200 import meshgen

main, ctx = svo_b200.Context(0), svo_b200.Context(0)
v, f = meshgen.jittered_icosphere(4, np.random.default_rng(2))
left = [ctx.build(v, f, res, svo_b200.FLAG_DEDUP) for res in (100, 128, 150)]
want = [r.edges() for r in left]
keys = [r.dedup(1) for r in left]
ctx.close()
for r, w, k in zip(left, want, keys):
    assert r.edges().tobytes() == w.tobytes() and np.array_equal(r.dedup(1), k)
for r in left:
    r.close()
for res in (64, 150):
    g = main.build(v, f, res)
    g.write_voxels(sys.argv[2])
    assert res != 150 or g.edges().tobytes() == want[2].tobytes()
again = svo_b200.Context(0)
assert again.build(v, f, 128).edges().tobytes() == want[1].tobytes()
print("done")
"""


def test_results_after_their_context(svo_mod, tmp_path):
    p = subprocess.run([sys.executable, "-c", PROGRAM, ROOT, str(tmp_path / "voxels.obj")], capture_output=True, text=True,
                       timeout=300, env=dict(os.environ))
    assert p.returncode == 0 and p.stdout.strip().endswith("done"), (p.returncode, p.stderr[-2000:])
