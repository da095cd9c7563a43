"""The 3x3x3 convolution with streamed weights (conv3_stream.cuh) where its index arithmetic can go wrong: the fewest and the
most input channels it takes and one step either way, channel counts that leave a part of a weight buffer, one voxel, one past
a tile in y and x, several channel blocks, more tiles than CTAs, outputs aligned to 16 bytes only.  Against the fp32 CPU
convolution on the same bf16 operands, within one bf16 rounding (2^-8) plus 1e-3 of the largest output for the fp32
summation order."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import denoise_ref as R

pytestmark = pytest.mark.gpu

BF = torch.bfloat16

CASES = [
    # nvol, d, h, w, cin, cout
    (1, 2, 3, 4, 144, 64),          # the widest input whose weights stay
    (1, 1, 1, 1, 160, 64),
    (2, 9, 17, 9, 176, 128),
    (3, 20, 33, 17, 192, 64),
    (1, 2, 5, 20, 272, 192),
    (1, 3, 16, 8, 288, 64),
    (1, 3, 5, 5, 304, 64),          # the general kernel
    (1, 3, 5, 5, 192, 160),         # no whole blocks of 64 outputs: the general kernel
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d" % c[4:])
@pytest.mark.parametrize("masked", [False, True])
def test_streamed_convolution(engine, case, masked):
    from mcx_gb300._lib import lib

    n, d, h, w, cin, cout = case
    vox = n * d * h * w
    rng = np.random.default_rng(sum(case) + masked)
    x = R.bf16(rng.standard_normal((vox, cin)))
    wt = R.bf16(rng.standard_normal((cout, 27, cin)) * R.he_std(cin))
    b = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    mask = R.bf16(rng.standard_normal((vox, cout)))
    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda().to(t).contiguous()  # noqa: E731
    X, W, B, M = dev(x, BF), dev(wt, BF), dev(b, torch.float32), dev(mask, BF)
    buf = torch.full((vox * cout + 24,), 7.0, dtype=BF, device="cuda")
    off = 8 if masked else 16
    st = torch.cuda.current_stream().cuda_stream
    rc = lib.mcxg_dn_conv_fwd(X.data_ptr(), W.data_ptr(), None if masked else B.data_ptr(), M.data_ptr() if masked else None,
                              buf.data_ptr() + 2 * off, n, d, h, w, cin, cout, 27, 0 if masked else 1, st)
    assert rc == 0, lib.mcxg_dn_last_error()
    assert lib.mcxg_dn_check(st) == 0, lib.mcxg_dn_last_error()
    got = buf.float().cpu().numpy()
    assert (got[:off] == 7).all() and (got[off + vox * cout:] == 7).all()
    xt = torch.from_numpy(x.reshape(n, d, h, w, cin)).permute(0, 4, 1, 2, 3)
    ref = R.conv(xt, torch.from_numpy(wt), None if masked else torch.from_numpy(b), relu=not masked)
    ref = ref.permute(0, 2, 3, 4, 1).reshape(vox, cout).numpy().astype(np.float64)
    if masked:
        ref = ref * (mask > 0)
    err = np.abs(got[off:off + vox * cout].reshape(vox, cout) - ref)
    assert (err <= np.abs(ref) * 2.0 ** -8 + 1e-3 * (np.abs(ref).max() + 1e-30)).all(), float(err.max())
