"""The FP64 products without tensor cores (RB_GEMM_ENGINE=dfma, read once a process; run on a GPU): a factor
large enough for the 128 x 64 tile, whose stages take 48 KB beside the descriptor, against the default
engine's."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = """
import sys
sys.path[:0] = [r"{root}", r"{root}/tests"]
import numpy as np
from robinsolver_b200 import workloads as W
from helpers import gpu_rhs, gpu_tree
wl = W.make_workload(2, nrhs=2)
T, op, opts = gpu_tree(wl)
T.factor(wl.L, op, opts)
T.solve(gpu_rhs(wl.rhs))
np.save(r"{out}", np.stack([T.solution_array(r) for r in range(2)]))
T.set_timing(2)
T.clear_stage_times()
T.factor_samples(op.k(T.sample_points(0)))
print(" ".join(sorted(set(e[0] for e in T.stage_times()))))
T.close()
"""


def _run(tmp_path, name, env):
    out = tmp_path / (name + ".npy")
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT, out=out)], env=dict(os.environ, **env), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    import numpy as np
    return np.load(out), r.stdout.split()


def test_dfma_engine_factors_and_solves(tmp_path):
    import numpy as np
    dfma, names = _run(tmp_path, "dfma", {"RB_GEMM_ENGINE": "dfma"})
    tensor, _ = _run(tmp_path, "tensor", {})
    assert "zgemm_dfma" in names
    assert np.abs(dfma - tensor).max() < 1e-10 * np.abs(tensor).max()      # both FP64, about 4 of 16 digits lost
