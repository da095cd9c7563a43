"""A convolution of more planes times channel blocks than 32 bits count (69 GB of output): the general kernel takes it, as it
takes what the rolling one refuses otherwise.  Its first and last volumes against the same volumes in a call of their own,
within one bf16 rounding plus 1e-3 of the largest output, as the kernels' own tests have it."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def test_more_planes_than_32_bits_count(engine):
    from mcx_gb300._lib import lib

    if torch.cuda.mem_get_info()[0] < 120 << 30:
        pytest.skip("needs 120 GB")
    d, cin, cout = 1023, 16, 80                     # blocks of 16 outputs: five a plane
    n = 2 ** 31 // (5 * d) + 1
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(n, d * cin, generator=g, dtype=BF, device="cuda")
    w = torch.randn(cout, 27, cin, generator=g, device="cuda").to(BF)
    y = torch.empty(n, d * cout, dtype=BF, device="cuda")
    st = torch.cuda.current_stream().cuda_stream

    def conv(x, y):
        assert lib.mcxg_dn_conv_fwd(x.data_ptr(), w.data_ptr(), None, None, y.data_ptr(), x.shape[0], d, 1, 1, cin, cout, 27, 0, st) == 0, \
            lib.mcxg_dn_last_error()
        assert lib.mcxg_dn_check(st) == 0, lib.mcxg_dn_last_error()

    conv(x, y)
    for part in (slice(0, 64), slice(n - 64, n)):
        ref = torch.empty(64, d * cout, dtype=BF, device="cuda")
        conv(x[part].contiguous(), ref)
        err = (y[part].float() - ref.float()).abs()
        assert (err <= ref.float().abs() * 2.0 ** -8 + 1e-3 * ref.float().abs().max()).all()
    del x, y
    torch.cuda.empty_cache()
