"""Chunks whose node box leaves room for one or two scatter tiles, whose warps then
divide the grid values between them or take turns: boxes on both sides of every
limit (four, two and one tile: with the reaction 438, 877 and 1,331 nodes, without
768 and 1,331; with many box records, where the tiles have less room and chunks are
cut into parts, 234, 468 and 937, without 410 and 820), from three particles a chunk
up, runs of one base node on both sides of 2.5 particles, many particles in one cell
of a wide box, stencils that leave the grid, and bins gone stale.  Compared with the
CPU oracle like the other chunk shapes, under the same tolerances."""

import sys

import numpy as np
import pytest

from tests import test_gpu_mpm_chunks as chunks

pytestmark = pytest.mark.gpu

BINS = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)


def _bins_of(ext, per_bin, rng, run=1):
    """All 64 bins (with few box records too many to be cut into parts) with per_bin particles each, `run` of them in a cell, whose stencils
    span ext nodes per axis."""
    lo, hi = 0.01, np.array(ext) - 2 - 0.03
    x = rng.uniform(0.0, 1.0, (64, -(-per_bin // run), 3)) * (hi - lo) + lo
    x[:, 0], x[:, 1] = lo, hi  # both ends of the range in every bin
    x = np.repeat(x, run, 1)[:, :per_bin]
    x = np.floor(x) + np.clip(x - np.floor(x) + (rng.uniform(-0.2, 0.2, x.shape) if run > 1 else 0), 0.01, 0.97)
    return np.clip((0.51 + x + 8.0 * BINS[:, None]).reshape(-1, 3), 1.0, 31.0)


def _cloud(kind, rng):
    if kind == "one_cell_of_a_wide_box":  # 60 particles with one stencil and 35 over the bin
        x = _bins_of((9, 9, 10), 95, rng).reshape(64, 95, 3)
        x[:, 35:] = x[:, 35:36].round() + rng.uniform(0.01, 0.9, (64, 60, 3)) - 0.49
        return np.clip(x.reshape(-1, 3), 1.0, 31.0), (27, 1000), 95
    if kind == "parts":  # one chunk, cut into parts of 25 particles
        return 8.51 + rng.uniform(0, 7.9, (100, 3)), (100, 1000), 100
    if kind == "leaving_the_grid":  # the bin at the upper corner, clamped at 1 - dx
        return np.minimum(24.51 + rng.uniform(0, 7.5, (90, 3)), 31.0), (100, 900), 90
    ext, per_bin, run = kind
    nodes = int(np.prod(ext))
    return _bins_of(ext, per_bin, rng, run), (nodes if RECORDS == "few" else 27, nodes), per_bin


FRESH = [((5, 7, 8), 64, 1), ((6, 8, 9), 64, 1), ((7, 7, 9), 3, 1), ((6, 9, 10), 31, 2), ((8, 8, 9), 33, 1),
         ((8, 8, 9), 90, 3), ((8, 9, 10), 94, 2), ((8, 10, 10), 93, 3), ((9, 9, 10), 3, 1), ((9, 10, 10), 95, 2),
         ((10, 10, 10), 95, 1), ((10, 10, 10), 95, 3)]
STALE = [((9, 10, 11), 95, 1), ((10, 10, 11), 60, 2), ((10, 11, 11), 95, 1), ((11, 11, 11), 90, 3), ((11, 11, 12), 64, 1)]
RECORDS = "few"


@pytest.fixture(params=["few", "many"])
def records(request, monkeypatch):
    """Box records for the chunks only, or (as large clouds have) for every CTA of the device."""
    from mpm_lbm_b200 import mpm

    if request.param == "many":
        monkeypatch.setattr(mpm, "FSI_BIN_CHUNK", 1)
    monkeypatch.setattr(sys.modules[__name__], "RECORDS", request.param)
    monkeypatch.setattr(chunks, "_cloud", _cloud)


@pytest.mark.parametrize("kind", FRESH + ["one_cell_of_a_wide_box", "parts", "leaving_the_grid"], ids=str)
@pytest.mark.parametrize("react", [False, True])
def test_wide_boxes_match_oracle(kind, react, records):
    chunks.test_chunk_shapes_match_oracle(kind, react)


@pytest.mark.parametrize("kind", STALE, ids=str)
@pytest.mark.parametrize("react", [False, True])
def test_stale_bins_match_oracle(kind, react, records, monkeypatch):
    import torch

    from mpm_lbm_b200.mpm import MPMSolid3D

    rebin = MPMSolid3D.rebin

    def from_the_centres(self):  # the particles of a bin have drifted out of it since the binning
        x = self.t_x.clone()
        centre = torch.tensor(((8.0 * BINS + 4.51) * chunks.DX).T, dtype=torch.float32, device=x.device)
        self.t_x.copy_(centre.repeat_interleave(kind[1], 1))
        rebin(self)
        self.t_x.copy_(x)

    monkeypatch.setattr(MPMSolid3D, "rebin", from_the_centres)
    chunks.test_chunk_shapes_match_oracle(kind, react)


@pytest.mark.parametrize("per_bin", [1, 3, 7, 40])
def test_old_boxes_are_zeroed(per_bin):
    """Few and many CTAs without a chunk: the boxes of a buffer are zero when its turn comes again (a node that is not
    keeps twice its mass)."""
    from mpm_lbm_b200.config import MPMConfig
    from mpm_lbm_b200.mpm import MPMSolid3D

    rng = np.random.default_rng(3)
    x = (_bins_of((9, 10, 10), per_bin, rng) if per_bin > 1 else 4.0 + 8.0 * BINS + rng.uniform(0, 3, (64, 3))) * chunks.DX
    vol = np.full(len(x), chunks.DX ** 3, np.float32)
    out = []
    for binned in (True, False):
        s = MPMSolid3D(MPMConfig(n_grid=chunks.G, dx=chunks.DX, dt=1e-4, young_modulus=100.0, p_rho=1.1), len(x))
        s.init_from_numpy(x.astype(np.float32), vol, vol)
        if binned:
            s.substeps_binned(7)
        else:
            for _ in range(7):
                s.substep()
        out.append((s.grid_m.to_numpy(), s.x.to_numpy()))
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=0, atol=2e-5 * out[1][0].max())
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=0, atol=1e-6)
