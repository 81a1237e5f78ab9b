"""MZB_PHASE_TIMING=1 prints the phase times of a CG solve whichever kernel serves it: the
resident one (32^3, 30^3, Poisson-Boltzmann) and the streaming one (144^3)."""
import os
import re
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import numpy as np
from maze_poisson_b200 import library_path
from maze_poisson_b200.c_api import CAPI
lib = CAPI(library_path())
lib.solver_initialize()
b = np.random.default_rng(1).standard_normal(({n},) * 3)
b -= b.mean()
x, one = np.empty_like(b), np.ones_like(b)
if {pb}:
    lib.mzb_conj_grad_pb(b, 0 * b, x, 1e-3, {n}, one, one, one, one)
else:
    lib.mzb_conj_grad(b, 0 * b, x, 1e-3, {n}, 0)
"""


@pytest.mark.parametrize("n,pb", [(32, 0), (30, 0), (32, 1), (144, 0)])
def test_phase_times(product_path, n, pb):
    out = subprocess.run([sys.executable, "-c", SCRIPT.format(n=n, pb=pb)], cwd=ROOT, capture_output=True, text=True,
                         timeout=300, env=dict(os.environ, MZB_PHASE_TIMING="1"))
    assert out.returncode == 0, out.stderr
    lines = [x for x in out.stderr.splitlines() if x.startswith("[cg phases us]")]
    assert len(lines) == 1, out.stderr
    phases = re.findall(r"A ([\d.]+) redA ([\d.]+) B ([\d.]+) redB ([\d.]+)", lines[0])
    assert len(phases) == 5
    assert all(0 < float(t) < 1e3 for p in phases for t in p), lines[0]
