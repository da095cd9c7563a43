"""The weight gradient over a volume that is not a multiple of its tiles, where it meets infinities and NaN: the runs of
tiles that hold one are summed by another body (wgrad_within in conv3_wgrad.cuh).  Values against float64 sums, 1e-4 of
the largest finite gradient as for the finite operands; every output width; groups inside a slice, over two, last and
short; several volumes and runs; infinities on faces, edges and inside, of X and of dY, and X without a finite value.
And the time of such a call: at most 20 finite ones (the copies of a tile, which nothing overlaps, at about a fifth
of the finite kernel's rate, and 4 for the spread of times)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import denoise_ref as R

pytestmark = pytest.mark.gpu

BF = torch.bfloat16

CASES = [
    # nvol, d, h, w, cin, cout
    (2, 25, 49, 17, 16, 16),
    (1, 33, 32, 32, 48, 16),        # ragged in z only
    (3, 16, 17, 32, 80, 16),        # in y only
    (1, 37, 33, 27, 16, 32),
    (2, 8, 16, 41, 96, 32),         # in x only
    (1, 31, 18, 30, 32, 64),
    (2, 7, 9, 22, 192, 64),
    (1, 33, 33, 32, 16, 128),
    (1, 9, 17, 17, 208, 128),
]


def _run(lib, X, DY, case):
    n, d, h, w, cin, cout = case
    dw = torch.zeros(cout * 27 * cin, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert lib.mcxg_dn_conv_wgrad(DY.data_ptr(), X.data_ptr(), dw.data_ptr(), n, d, h, w, cin, cout, 27, st) == 0, lib.mcxg_dn_last_error()
    assert lib.mcxg_dn_check(st) == 0, lib.mcxg_dn_last_error()
    return dw.cpu().numpy()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d" % c[4:])
@pytest.mark.parametrize("where", ["faces", "scattered", "gradient", "everywhere"])
def test_nonfinite_values_reach_the_taps_of_their_pairs(engine, case, where):
    from mcx_gb300._lib import lib

    n, d, h, w, cin, cout = case
    vox = n * d * h * w
    rng = np.random.default_rng(sum(case))
    x5 = R.bf16(rng.standard_normal((vox, cin))).reshape(n, d, h, w, cin)
    dy5 = R.bf16(np.abs(rng.standard_normal((vox, cout))) + 0.1).reshape(n, d, h, w, cout)
    if where == "faces":
        x5[0, -1, 3, 4, 1], x5[0, 2, -1, 5, 2], x5[-1, 4, 5, -1, cin - 1] = np.inf, np.nan, -np.inf
        x5[-1, -1, -1, 7, 5], x5[0, 0, 0, 0, 7] = np.inf, np.inf
    elif where == "scattered":
        for c in range(0, cin, 3):
            x5[rng.integers(n), rng.integers(d), rng.integers(h), rng.integers(w), c] = (np.inf, -np.inf, np.nan)[c % 3]
    elif where == "gradient":
        dy5[0, -1, 3, 4, 0], dy5[-1, 2, -1, -1, cout - 1], x5[0, -1, 2, 2, 3] = np.inf, np.nan, np.inf
    else:
        x5[:] = np.nan
    X, DY = (torch.from_numpy(np.ascontiguousarray(a)).cuda().to(BF).reshape(-1) for a in (x5, dy5))
    got = _run(lib, X, DY, case)
    g3 = got.reshape(cout, 27, cin)
    if where == "everywhere":
        assert np.isnan(g3).all()
        return
    if where == "gradient":
        # every pair of a voxel of dY that is not finite, zeros of the padding among them; X's infinity where it is paired
        fin = np.ones((cout, 27, cin), bool)
        fin[0], fin[cout - 1] = False, False
        for t in range(27):
            z, y, x = d - 1 - (t // 9 - 1), 2 - (t // 3 % 3 - 1), 2 - (t % 3 - 1)
            if 0 <= z < d and 0 <= y < h and 0 <= x < w:
                fin[:, t, 3] = False
        assert (np.isfinite(g3) == fin).all()
        return
    # the finite products by matrix, the others one by one
    bad = ~np.isfinite(x5)
    xp = np.pad(np.where(bad, 0.0, x5).astype(np.float64), ((0, 0), (1, 1), (1, 1), (1, 1), (0, 0)))
    dyT = dy5.reshape(vox, cout).astype(np.float64).T
    ref = np.stack([dyT @ xp[:, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + w].reshape(vox, cin) for t in range(27)], 1)
    for vn, vz, vy, vx, c in np.argwhere(bad):
        for t in range(27):
            z, y, x = vz - (t // 9 - 1), vy - (t // 3 % 3 - 1), vx - (t % 3 - 1)
            if 0 <= z < d and 0 <= y < h and 0 <= x < w:
                ref[:, t, c] += dy5[vn, z, y, x].astype(np.float64) * float(x5[vn, vz, vy, vx, c])
    ok = np.isfinite(ref)
    assert ok.any() and not ok.all()
    assert (np.isnan(g3) == np.isnan(ref)).all()
    assert (g3[np.isinf(ref)] == ref[np.isinf(ref)]).all()
    assert np.abs(g3[ok] - ref[ok]).max() <= 1e-4 * np.abs(ref[ok]).max()


@pytest.mark.parametrize("case", [(2, 65, 65, 65, 16, 16), (4, 33, 33, 33, 96, 32), (4, 17, 17, 17, 128, 128)],
                         ids=lambda c: "x".join(map(str, c[:4])) + " %d-%d" % c[4:])
def test_time_of_a_nonfinite_call(engine, case):
    from mcx_gb300._lib import lib

    n, d, h, w, cin, cout = case
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn(n, d, h, w, cin, generator=g, device="cuda").to(BF)
    DY = torch.randn(n, d, h, w, cout, generator=g, device="cuda").to(BF)

    def best():
        us = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            dw = torch.zeros(cout * 27 * cin, device="cuda")
            torch.cuda.synchronize()
            a.record()
            lib.mcxg_dn_conv_wgrad(DY.data_ptr(), X.data_ptr(), dw.data_ptr(), n, d, h, w, cin, cout, 27, torch.cuda.current_stream().cuda_stream)
            b.record()
            torch.cuda.synchronize()
            us.append(a.elapsed_time(b) * 1e3)
        return min(us)

    finite = best()
    X[0, -1, 3, 4, 1] = float("inf")
    one = best()
    X[:] = float("nan")
    every = best()
    assert max(one, every) <= 20 * finite, (finite, one, every)
