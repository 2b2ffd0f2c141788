"""The fused field's table kernels against the float64 hash-grid oracle, evaluation by
evaluation: taps inside the centre's grid cell, in a neighbouring one and several cells away,
ragged tile ends, level counts that do not divide a warp, every feature width."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import oracle.hashgrid as hg
from neuralangelo_gb300 import _lib
from neuralangelo_gb300.encoding import GridLayout
from neuralangelo_gb300.fused import FieldArgs

DEV = "cuda"
# (F, taps, levels, active, eps in cells of the finest active level, samples)
CASES = [(8, 6, 16, 8, 0.25, 200), (8, 6, 16, 16, 0.25, 37), (8, 4, 16, 7, 0.3, 51), (8, 4, 16, 8, 1.7, 25),
         (4, 6, 8, 8, 0.9, 19), (4, 4, 8, 5, 0.25, 1), (2, 6, 6, 3, 3.0, 77), (2, 4, 6, 6, 0.0, 26), (8, 6, 16, 1, 0.4, 18)]


class Field:
    """Arguments of the table kernels of one seeded field, and its evaluation points (float32)."""

    def __init__(self, F, taps, levels, active, eps_cells, n, table=True):
        g = torch.Generator().manual_seed(F * 1000 + taps * 100 + active * 10 + n)
        self.lay = lay = GridLayout(levels, F, 14, 16, 1.4)
        self.ora = hg.level_layout(levels, F, 14, 16, 1.4)
        self.F, self.active, self.taps, self.n = F, active, taps, n
        self.eps = np.float32(eps_cells * 4.0 / float(lay.scale[active - 1]))
        self.K0 = max(16, (active * F + 15) // 16 * 16)
        self.evals, self.spt = (7, 18) if taps == 6 else (5, 25)
        self.tiles = (n + self.spt - 1) // self.spt
        self.rows = self.tiles * self.spt * self.evals
        c = torch.randn(3, 3, generator=g)
        d = torch.randn(3, 3, generator=g)
        d = d / d.norm(dim=1, keepdim=True)
        ray = torch.randint(0, 3, (n,), generator=g).sort().values
        t = torch.rand(n, generator=g) * 0.5
        self.table = (torch.randn(lay.n_params, generator=g) * 0.1).half()
        x = (c[ray] * 0.5 + d[ray] * t[:, None]).numpy().astype(np.float32)   # float32 multiply, then add
        if taps == 6:
            off = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
        else:
            off = [(0, 0, 0), (1, -1, -1), (-1, -1, 1), (-1, 1, -1), (1, 1, 1)]
        self.points = np.stack([x + np.array(o, np.float32) * self.eps for o in off])   # [evals, n, 3]
        self.unit = (self.points + np.float32(2)) * np.float32(0.25)
        self.keep = dict(center=c * 0.5, dir=d, ray=ray.int(), t=t, table=self.table)
        self.keep = {k: v.to(DEV).contiguous() for k, v in self.keep.items()}
        self.keep["w"] = torch.zeros(1024, 256, device=DEV)
        a = self.a = FieldArgs()
        a.Ns, a.S = n, 0
        a.sample_ray = self.keep["ray"].data_ptr()
        a.center, a.ray_unit, a.dists = (self.keep[k].data_ptr() for k in ("center", "dir", "t"))
        a.grid, a.active, a.K0, a.taps = lay.struct, active, self.K0, taps
        a.table = self.keep["table"].data_ptr()
        for k in ("w0e", "w0b", "w0x", "b0", "whead", "bhead"):
            setattr(a, k, self.keep["w"].data_ptr())
        a.eps = float(self.eps)

    def row_of(self, e):
        s = np.arange(self.n)
        return s // self.spt * (self.spt * self.evals) + e * self.spt + s % self.spt

    def call(self, name):
        _lib.call(name, ctypes.byref(self.a), _lib.stream_ptr(torch.device(DEV)))
        torch.cuda.synchronize()


@pytest.mark.parametrize("case", CASES)
def test_gather_rows_match_the_oracle_at_every_evaluation(case):
    f = Field(*case)
    KX, K0, AF = 2 * f.K0 + 16, f.K0, f.active * f.F
    x0 = torch.full((f.rows, KX), float("nan"), device=DEV, dtype=torch.float16)
    f.a.x0ext = x0.data_ptr()
    f.call("gbsdf_field_encode")
    got = x0.double().cpu().numpy()
    assert np.isfinite(got).all()                         # every column of every row is written
    table = f.table.double().numpy()
    live = np.zeros(f.rows, bool)
    for e in range(f.evals):
        r = f.row_of(e)
        live[r] = True
        want = hg.encode(f.unit[e], table, f.ora, f.active)[:, :AF]
        pair = got[r, :AF] + got[r, K0 + 16:K0 + 16 + AF]
        # eight float32 products and sums of values below max |table|, then a fp16 residual
        scale = float(np.abs(table).max())
        np.testing.assert_allclose(pair, want, rtol=0, atol=scale * (8 * 2 * 2.0 ** -24 + 2.0 ** -22))
        tail = got[r, K0:K0 + 16]
        np.testing.assert_allclose(tail[:, :3] + tail[:, 4:7], f.points[e], rtol=2.0 ** -20, atol=2.0 ** -22)
        assert (tail[:, 3] == 1).all() and (tail[:, 7] == 1).all() and (tail[:, 11:] == 0).all()
        np.testing.assert_array_equal(tail[:, 8:11], tail[:, :3])
    assert (got[~live] == 0).all()                        # samples past the end
    assert (got[:, AF:K0] == 0).all() and (got[:, K0 + 16 + AF:] == 0).all()
