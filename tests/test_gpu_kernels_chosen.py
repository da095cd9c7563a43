"""Which kernel a call runs: the tests that compare a kernel with the general one mean something only if their two sides run
different kernels.  The launches of a call by name, from the profiler: over the decks of the plain-path kernel's forward
and replay tests and the shapes of the convolution and weight-gradient tests."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from .test_gpu_conv_roll import CASES as ROLL
from .test_gpu_conv_stream import CASES as STREAM
from .test_gpu_lean import DECKS
from .test_gpu_lean_replay import DECKS as REPLAYS
from .test_gpu_wgrad import CASES as WGRAD

pytestmark = pytest.mark.gpu


def _launched(call):
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return " ".join(e.name for e in p.events())


@pytest.fixture(scope="module")
def launched(built):
    x = torch.zeros(1000, device="cuda")
    for _ in range(3):                      # the first trace of a process may miss its kernels
        seen = _launched(lambda: x.add_(1))
    if "kernel" not in seen:
        pytest.skip("no kernel tracing here")
    return _launched


@pytest.mark.parametrize("name", DECKS)
def test_plain_path(engine, launched, name):
    a = launched(lambda: engine.run(DECKS[name]()))
    b = launched(lambda: engine.run(dict(DECKS[name](), gscatter=15_000_000)))
    assert "lean_kernel<" in a and "transport_kernel<" not in a
    assert "transport_kernel<" in b and "lean_kernel<" not in b


@pytest.mark.parametrize("name", REPLAYS)
def test_replay(engine, launched, name):
    deck, extra = REPLAYS[name]
    cfg = deck()
    rec = engine.run(dict(cfg, issaveseed=1))
    cfg = dict(cfg, seed=np.asfortranarray(rec["seeds"]), detphotons=np.asfortranarray(rec["detp"]), outputtype="jacobian", isnormalized=0)
    cfg.update(extra)
    a, b = launched(lambda: engine.run(dict(cfg))), launched(lambda: engine.run(dict(cfg, gscatter=15_000_000)))
    assert "lean_kernel<" in a and "transport_kernel<" not in a
    assert "transport_kernel<" in b and "lean_kernel<" not in b


def _operands(case):
    n, d, h, w, cin, cout = case
    z = lambda c: torch.zeros(n * d * h * w * c, dtype=torch.bfloat16, device="cuda")  # noqa: E731
    return z(cin), z(cout), torch.zeros(cout * 27 * cin, dtype=torch.bfloat16, device="cuda"), torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("case", ROLL + STREAM, ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d" % c[4:])
def test_convolution(engine, launched, case):
    from mcx_gb300._lib import lib

    cin, cout = case[4:]
    x, y, w, st = _operands(case)
    names = launched(lambda: lib.mcxg_dn_conv_fwd(x.data_ptr(), w.data_ptr(), None, None, y.data_ptr(), *case, 27, 0, st))
    wide = cout % 64 == 0 or (cout % 32 == 0 and cout > 96)         # tap by tap: its weights have to fit
    want = "conv3_roll_kernel<"
    if wide and cin > 144:
        want = "conv3_stream_kernel" if cout % 64 == 0 and cin <= 288 else "conv_fwd_kernel<"
    assert want in names, names


@pytest.mark.parametrize("case", WGRAD, ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d" % c[4:])
def test_weight_gradient(engine, launched, case):
    from mcx_gb300._lib import lib

    n, d, h, w, cin, cout = case
    x, dy, _, st = _operands(case)
    dw = torch.zeros(cout * 27 * cin, device="cuda")
    names = launched(lambda: lib.mcxg_dn_conv_wgrad(dy.data_ptr(), x.data_ptr(), dw.data_ptr(), *case, 27, st))
    new = n * d * h * w * cin >= 1 << 19
    assert ("conv3_wgrad_kernel<" in names) == new and ("conv_wgrad_kernel<" in names) == (not new), names
