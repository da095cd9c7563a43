"""The tcgen05 convolutions give the mma.sync kernels' outputs bit for bit, in both orders of summation: a whole network's
bf16 roundings follow from the order, and trained weights and stored results with them.  The two sides run in
processes of their own, since MCXG_DN_MMA_SYNC is read once; over the shapes of the kernels' own tests, masked and
with bias and ReLU."""

from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from .test_gpu_conv_roll import CASES as ROLL
from .test_gpu_conv_stream import CASES as STREAM

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

SIDE = r"""
import ast, sys
import numpy as np
import torch
from mcx_gb300._lib import lib

out = {}
for i, (n, d, h, w, cin, cout) in enumerate(ast.literal_eval(sys.argv[1])):
    g = torch.Generator(device="cuda").manual_seed(i)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    vox = n * d * h * w
    x, wt, b, m = rnd(vox, cin).bfloat16(), (rnd(cout, 27, cin) * (2 / 27 / cin) ** 0.5).bfloat16(), rnd(cout) * 0.1, rnd(vox, cout).bfloat16()
    for masked in (False, True):
        y = torch.empty(vox, cout, dtype=torch.bfloat16, device="cuda")
        st = torch.cuda.current_stream().cuda_stream
        rc = lib.mcxg_dn_conv_fwd(x.data_ptr(), wt.data_ptr(), None if masked else b.data_ptr(), m.data_ptr() if masked else None, y.data_ptr(),
                                  n, d, h, w, cin, cout, 27, 0 if masked else 1, st)
        assert rc == 0 and lib.mcxg_dn_check(st) == 0, lib.mcxg_dn_last_error()
        out["%d%d" % (i, masked)] = y.view(torch.int16).cpu().numpy()
np.savez(sys.argv[2], **out)
"""


def test_outputs_of_the_mma_sync_kernels(built, tmp_path):
    cases = [*ROLL, *STREAM]
    files = []
    for sync in ("0", "1"):
        f = tmp_path / f"sync{sync}.npz"
        env = dict(os.environ, MCXG_DN_MMA_SYNC=sync, PYTHONPATH=str(ROOT))
        p = subprocess.run([sys.executable, "-c", SIDE, repr(cases), str(f)], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
        assert p.returncode == 0, p.stderr[-2000:]
        files.append(np.load(f))
    for i, case in enumerate(cases):
        for masked in (0, 1):
            a, b = (f[f"{i}{masked}"] for f in files)
            assert np.array_equal(a, b), (case, masked, int((a != b).sum()))
