"""The tcgen05 weight gradient (conv3_wgrad.cuh) and the chunked bias gradient where their index arithmetic can go
wrong: grids one past a tile in every direction; groups of accumulators that end inside a slice, span two, and are the
last and short; fewer tiles than CTAs; a gradient aligned to 4 bytes only, added to what it held; and two grids below
the line where it takes over.
Against float64 sums of the same bf16 operands: 1e-4 of the largest gradient, as for the general kernel."""

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
    (1, 3, 18, 9, 32, 64),
    (2, 25, 49, 17, 16, 16),
    (1, 33, 40, 50, 16, 16),
    (1, 9, 33, 41, 48, 16),
    (3, 9, 17, 15, 80, 16),
    (1, 37, 33, 27, 16, 32),
    (2, 7, 16, 25, 96, 32),
    (1, 31, 18, 30, 32, 64),
    (2, 7, 9, 22, 192, 64),
    (1, 33, 32, 32, 16, 128),
    (1, 17, 16, 16, 128, 128),
    (1, 9, 17, 17, 208, 128),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d" % c[4:])
def test_weight_and_bias_gradient(engine, case):
    from mcx_gb300._lib import lib

    n, d, h, w, cin, cout = case
    vox = n * d * h * w
    rng = np.random.default_rng(sum(case))
    x = R.bf16(rng.standard_normal((vox, cin)))
    dy = R.bf16(rng.standard_normal((vox, cout)))
    X, DY = (torch.from_numpy(a).cuda().to(BF).contiguous() for a in (x, dy))
    off = 1 + case[0] % 2 * 3                 # 4 or 16 bytes into the buffer
    buf = torch.full((cout * 27 * cin + 8,), 0.5, device="cuda")
    db = torch.full((cout + 2,), 0.25, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    rc = lib.mcxg_dn_conv_wgrad(DY.data_ptr(), X.data_ptr(), buf.data_ptr() + 4 * off, n, d, h, w, cin, cout, 27, st)
    assert rc == 0, lib.mcxg_dn_last_error()
    assert lib.mcxg_dn_bias_grad(DY.data_ptr(), db.data_ptr() + 4, vox, cout, st) == 0
    assert lib.mcxg_dn_check(st) == 0, lib.mcxg_dn_last_error()
    x5 = np.pad(x.astype(np.float64).reshape(n, d, h, w, cin), ((0, 0), (1, 1), (1, 1), (1, 1), (0, 0)))
    dyT = dy.astype(np.float64).T
    ref = np.stack([dyT @ x5[:, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + w].reshape(vox, cin)
                    for t in range(27)], 1).reshape(-1) + 0.5
    got = buf.cpu().numpy()
    assert (got[:off] == 0.5).all() and (got[off + ref.size:] == 0.5).all()
    assert np.abs(got[off:off + ref.size] - ref).max() <= 1e-4 * np.abs(ref).max()
    b = db.cpu().numpy()
    assert b[0] == b[-1] == 0.25
    rb = dyT.sum(1) + 0.25
    assert np.abs(b[1:-1] - rb).max() <= 1e-4 * max(1.0, np.abs(rb).max())


@pytest.mark.parametrize("case", [(1, 33, 33, 31, 16, 16), (1, 35, 33, 30, 16, 32), (1, 9, 31, 31, 64, 64), (1, 17, 17, 15, 128, 128)],
                         ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d" % c[4:])
def test_infinities_stay_with_their_voxels(engine, case):
    """A tile's padding outside the volume meets voxels inside it: an infinity or a NaN at the volume's faces reaches the taps
    that pair it with a voxel of the volume, as in the sum over the volume, and no other."""
    from mcx_gb300._lib import lib

    n, d, h, w, cin, cout = case
    vox = n * d * h * w
    rng = np.random.default_rng(sum(case))
    x = R.bf16(rng.standard_normal((vox, cin)))
    dy = R.bf16(np.abs(rng.standard_normal((vox, cout))) + 0.1)
    x5 = x.reshape(n, d, h, w, cin)
    x5[0, -1, 3, 4, 1], x5[0, 2, -1, 5, 2], x5[0, 4, 5, -1, cin - 1] = np.inf, np.nan, -np.inf
    X, DY = (torch.from_numpy(a).cuda().to(BF).contiguous() for a in (x, dy))
    dw = torch.zeros(cout * 27 * cin, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert lib.mcxg_dn_conv_wgrad(DY.data_ptr(), X.data_ptr(), dw.data_ptr(), n, d, h, w, cin, cout, 27, st) == 0
    assert lib.mcxg_dn_check(st) == 0, lib.mcxg_dn_last_error()
    xp = np.pad(x.astype(np.float64).reshape(n, d, h, w, cin), ((0, 0), (1, 1), (1, 1), (1, 1), (0, 0)))
    dyT = dy.astype(np.float64).T
    with np.errstate(invalid="ignore"):
        ref = np.stack([dyT @ xp[:, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + w].reshape(vox, cin)
                        for t in range(27)], 1).reshape(-1)
    got = dw.cpu().numpy()
    assert (np.isnan(got) == np.isnan(ref)).all()
    assert (got[np.isinf(ref)] == ref[np.isinf(ref)]).all()
    ok = np.isfinite(ref)
    assert ok.any() and not ok.all()
    assert np.abs(got[ok] - ref[ok]).max() <= 1e-4 * np.abs(ref[ok]).max()
