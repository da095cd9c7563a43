"""The rolling-plane 3x3x3 convolution (conv3_roll.cuh) at the sizes where its index arithmetic can go wrong:
grids of one voxel, one plane, one short of and one past a tile; columns whose accumulator ring wraps; odd and even
runs; runs that cross columns, volumes and channel blocks; weights that stay and weights that cycle; outputs aligned
to 16 bytes only.  Against the fp32 CPU convolution on the same bf16 operands, within one bf16 rounding (2^-8) plus
1e-3 of the largest output for the fp32 summation order."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import denoise_ref as R

pytestmark = pytest.mark.gpu

BF = torch.bfloat16

CASES = [
    # nvol, d, h, w, cin, cout
    (1, 1, 1, 1, 16, 16),
    (1, 2, 17, 9, 16, 16),          # one past a tile in y and x
    (2, 3, 15, 7, 32, 16),          # one short
    (1, 70, 5, 3, 16, 16),          # a column longer than the ring of 32 planes, few CTAs' worth of columns
    (3, 61, 20, 17, 16, 16),        # runs that cross columns and volumes
    (1, 33, 9, 40, 48, 16),         # several slices: pieces no longer than the ring
    (1, 23, 18, 10, 16, 48),        # the ring of 10
    (2, 9, 33, 8, 32, 96),          # two blocks of 48 channels
    (1, 19, 16, 24, 96, 32),
    (1, 40, 16, 8, 16, 64),         # the ring of 8
    (4, 11, 17, 9, 64, 64),         # weights cycling through two buffers
    (1, 5, 8, 8, 192, 64),
    (1, 3, 6, 5, 64, 192),
    (2, 8, 8, 8, 128, 128),
    (1, 7, 16, 8, 208, 80),         # more slices than stay resident, a width of five 16-channel blocks
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d" % c[4:])
@pytest.mark.parametrize("masked", [False, True])
def test_rolling_convolution(engine, case, masked):
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
    # the output 16 bytes into its buffer, so aligned to 16 and not to 32, between guard values
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
