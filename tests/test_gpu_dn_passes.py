"""The denoiser's feature pass and upsampling concatenation at sizes where their tiles and index arithmetic end: rows
shorter than a thread's four voxels, one voxel past a tile in every direction, both tile widths, an output aligned to
16 bytes only, channel counts of one chunk and none; infinities and NaN among the fluence."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import denoise_ref as R

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _st():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("dims", [(1, 1, 1, 1), (2, 3, 2, 5), (1, 5, 17, 33), (1, 4, 16, 32), (2, 9, 9, 65), (1, 1, 8, 64),
                                  (1, 7, 20, 100)], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("offset", [0, 8])
def test_pack(engine, dims, offset):
    from mcx_gb300._lib import lib

    n, d, h, w = dims
    vox, nprop = d * h * w, 4
    rng = np.random.default_rng(sum(dims))
    flux = ((10.0 ** rng.uniform(-9, 0, (n, vox))) * (rng.random((n, vox)) < 0.8)).astype(np.float32)
    labels = rng.integers(0, nprop + 2, (n, vox)).astype(np.uint8)
    props = rng.uniform(0.01, 0.9, (n, nprop, 4)).astype(np.float32)
    props[:, 0] = [0, 0, 1, 1]
    lp = rng.uniform(4, 7, n).astype(np.float32)
    F, L, P, LP = (torch.from_numpy(a).cuda() for a in (flux, labels, props, lp))
    x0 = torch.full((n * vox * 16 + 16,), 7.0, dtype=BF, device="cuda")
    xres = torch.full((n * vox + 1,), 7.0, device="cuda")

    def run():
        rc = lib.mcxg_dn_pack(F.data_ptr(), L.data_ptr(), P.data_ptr(), LP.data_ptr(), x0.data_ptr() + 2 * offset,
                              xres.data_ptr(), n, d, h, w, nprop, _st())
        assert rc == 0, lib.mcxg_dn_last_error()
        assert (x0[:offset] == 7).all() and (x0[offset + n * vox * 16:] == 7).all() and xres[-1] == 7
        return (x0[offset:offset + n * vox * 16].float().cpu().numpy().reshape(n, vox, 16),
                xres[:-1].cpu().numpy().reshape(n, vox))

    got, res = run()
    rx, rl = R.features(flux, labels, props, lp, (d, h, w))
    np.testing.assert_allclose(res, rl, rtol=1e-5, atol=1e-4)
    ref = R.bf16(rx)
    assert (np.abs(got - ref) <= np.abs(ref) * 2.0 ** -7 + 1e-3).all()
    # a NaN counts as an empty neighbour without the empty flag, an infinity reaches its own windows only
    F[0, 0], F[-1, -1] = float("nan"), float("inf")
    odd, ores = run()
    zero = flux.copy()
    zero[0, 0] = 0
    zero[-1, -1] = np.inf
    assert np.isposinf(ores[-1, -1]) and odd[0, 0, 3] == (1.0 if np.isposinf(flux[0, 0]) else 0.0)
    z, y, x = np.meshgrid(np.arange(d), np.arange(h), np.arange(w), indexing="ij")
    near = (np.maximum(np.maximum(d - 1 - z, h - 1 - y), w - 1 - x) <= 1).reshape(-1)
    assert (np.isposinf(ores[-1]) == near).all()


@pytest.mark.parametrize("case", [(1, 2, 2, 2, 8, 8), (2, 4, 6, 10, 16, 8), (1, 2, 6, 34, 0, 8), (1, 4, 2, 14, 24, 0),
                                  (3, 6, 10, 22, 128, 64), (1, 8, 64, 64, 32, 16)], ids=lambda c: "-".join(map(str, c)))
def test_upcat(engine, case):
    from mcx_gb300._lib import lib

    n, d, h, w, c1, c2 = case
    rng = np.random.default_rng(sum(case))
    low = rng.integers(-30000, 30000, (n, d // 2, h // 2, w // 2, c1)).astype(np.int16)
    skip = rng.integers(-30000, 30000, (n, d, h, w, c2)).astype(np.int16)
    guard = np.full(64, 77, np.int16)
    L = torch.from_numpy(np.r_[low.reshape(-1), guard]).cuda()
    S = torch.from_numpy(np.r_[skip.reshape(-1), guard]).cuda()
    cat = torch.full((n * d * h * w * (c1 + c2) + 64,), 77, dtype=torch.int16, device="cuda")
    assert lib.mcxg_dn_upcat(L.data_ptr(), S.data_ptr(), cat.data_ptr(), n, d, h, w, c1, c2, _st()) == 0
    up = low.repeat(2, 1).repeat(2, 2).repeat(2, 3)
    got = cat.cpu().numpy()
    assert np.array_equal(got[:-64].reshape(n, d, h, w, c1 + c2), np.concatenate([up, skip], -1))
    assert (got[-64:] == 77).all()
