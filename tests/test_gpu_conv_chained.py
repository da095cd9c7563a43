"""A data gradient launched straight behind the convolution whose output is its mask, and so started before that one has
ended: the same bits as with the device waited for in between, whatever the mask's buffer held before.  One layer for
each kernel and order of summation: slice by slice, tap by tap, streamed weights."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


@pytest.mark.parametrize("case", [(1, 64, 64, 64, 16, 16, 16), (2, 30, 30, 30, 16, 32, 32), (1, 32, 32, 32, 32, 64, 64), (1, 16, 16, 16, 64, 64, 192)],
                         ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d-%d" % c[4:])
def test_mask_written_by_the_kernel_ahead(engine, case):
    from mcx_gb300._lib import lib

    n, d, h, w, cin, cmid, cout = case          # x (cin) -> mask (cmid); dy (cout) -> dx (cmid), masked
    vox = n * d * h * w
    g = torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF)  # noqa: E731
    xs = [rnd(vox * cin) for _ in range(6)]
    wf, wb, dy = rnd(cmid, 27, cin), rnd(cmid, 27, cout), rnd(vox * cout)
    bias = torch.randn(cmid, generator=g, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    mask = torch.zeros(vox * cmid, dtype=BF, device="cuda")

    def passes(wait):
        out = []
        for x in xs:
            dx = torch.empty(vox * cmid, dtype=BF, device="cuda")
            torch.cuda.synchronize()
            assert lib.mcxg_dn_conv_fwd(x.data_ptr(), wf.data_ptr(), bias.data_ptr(), None, mask.data_ptr(), n, d, h, w, cin, cmid, 27, 1, st) == 0
            if wait:
                torch.cuda.synchronize()
            assert lib.mcxg_dn_conv_fwd(dy.data_ptr(), wb.data_ptr(), None, mask.data_ptr(), dx.data_ptr(), n, d, h, w, cout, cmid, 27, 0, st) == 0
            out.append(dx)
        assert lib.mcxg_dn_check(st) == 0, lib.mcxg_dn_last_error()
        return out

    ref = passes(True)
    assert not torch.equal(ref[0], ref[1])
    for a, b in zip(passes(False), ref):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
