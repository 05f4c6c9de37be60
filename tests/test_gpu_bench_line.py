"""The end-to-end record of the bench line says whether the field that it ends with is finite: the Kerr-only beam of
cyl_kerr_64 collapses within its 100 steps (test_gpu_parity.py, test_kerr_collapse_long_run), silica stays finite."""
import json
import pathlib
import subprocess
import sys

import pytest

from test_gpu_adjoint import cuda_ready  # noqa: F401 (the fixture builds the extension)

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("workload,finite", [("cyl_kerr_64", False), ("cyl_silica_512", True)])
def test_end_to_end_finite_flag(workload, finite):
    out = subprocess.run([sys.executable, "bench.py", "--workload", workload, "--steps", "2", "--warmup", "3",
                          "--no-cpu-baseline", "--no-fp32", "--adjoint-steps", "0"], cwd=ROOT, check=True,
                         capture_output=True, text=True).stdout
    line = json.loads(out.strip().splitlines()[-1])
    assert line["e2e"]["finite"] is finite
