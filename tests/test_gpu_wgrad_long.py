"""The weight gradient's longest sums: so many tiles a CTA that an accumulator in tensor memory adds thousands of K steps,
of operands with a mean, so that the sums grow all the way.  Against float64: an FP32 sum of s steps is off by at most s
roundings (2^-23, where the tensor cores truncate) of the sum of the terms' absolute values; a step's 16 products and the
additions over runs and planes count as 256 more."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


@pytest.mark.parametrize("case,steps", [((4, 128, 128, 128, 48, 16), 4096), ((2, 96, 96, 96, 192, 64), 5536)],
                         ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d" % c[4:] if isinstance(c, tuple) else str(c))
def test_long_sums(engine, case, steps):
    from mcx_gb300._lib import lib

    n, d, h, w, cin, cout = case
    g = torch.Generator(device="cuda").manual_seed(11)
    x = (torch.randn(n, d, h, w, cin, generator=g, device="cuda") + 0.5).clamp_(min=0).to(BF)
    dy = (torch.randn(n, d, h, w, cout, generator=g, device="cuda") + 0.25).to(BF)
    dw = torch.zeros(cout, 27, cin, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert lib.mcxg_dn_conv_wgrad(dy.data_ptr(), x.data_ptr(), dw.data_ptr(), *case, 27, st) == 0, lib.mcxg_dn_last_error()
    assert lib.mcxg_dn_check(st) == 0, lib.mcxg_dn_last_error()
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    ref, size = torch.zeros(cout, 27, cin, dtype=torch.float64, device="cuda"), torch.zeros(cout, 27, cin, dtype=torch.float64, device="cuda")
    for t in range(27):
        for v in range(n):
            xs = xp[v, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + w].reshape(-1, cin).double()
            g64 = dy[v].reshape(-1, cout).double().T
            ref[:, t] += g64 @ xs
            size[:, t] += g64.abs() @ xs.abs()
    assert (ref.abs() > 0.1 * size).all()
    err = ((dw.double() - ref).abs() / size).max().item()
    print("error over the sum of absolute values: %.3g" % err)
    assert err <= (steps + 256) * 2.0 ** -23
