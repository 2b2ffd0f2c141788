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


SMS = 152
# (F, levels, active, points): one point, a tile's edges, one to six tiles per resident CTA, a
# level count whose columns need padding
POINTS = [(8, 16, 16, 1), (8, 16, 5, 127), (8, 16, 8, 128), (4, 8, 3, 129), (8, 16, 16, 128 * SMS + 1),
          (2, 6, 6, 128 * SMS * 2 + 77), (8, 16, 7, 128 * SMS * 5 + 3)]


@pytest.mark.parametrize("lattice", [False, True])
@pytest.mark.parametrize("case", POINTS)
def test_sdf_points_match_float64_at_tile_edges(case, lattice):
    F, levels, active, n = case
    f = Field(F, 6, levels, active, 0.25, 20)
    g = torch.Generator().manual_seed(n)
    if lattice:
        nz = min(n, 13)
        ny = max(1, min(n // nz, 11))
        dims = (max(1, n // (nz * ny)), ny, nz)
        ax = [torch.rand(k, generator=g) * 2 - 1 for k in dims]
        pts = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    else:
        pts = torch.rand(n, 3, generator=g) * 2 - 1
    K0, AF, H = f.K0, f.active * F, 256
    w0e = torch.zeros(H, K0, dtype=torch.float16)
    w0e[:, :AF] = (torch.randn(H, AF, generator=g) * 0.1).half()
    w0x, b0 = torch.randn(H, 3, generator=g) * 0.1, torch.randn(H, generator=g) * 0.05
    wh, bh = torch.randn(H, generator=g) * 0.1, torch.randn(1, generator=g)
    dev = dict(w0e=w0e, w0x=w0x, b0=b0, whead=wh, bhead=bh)
    f.keep.update({k: v.to(DEV).contiguous() for k, v in dev.items()})
    for k in dev:
        setattr(f.a, k, f.keep[k].data_ptr())
    f.a.beta = 100.0
    out = torch.full((len(pts),), float("nan"), device=DEV)
    err = torch.zeros(1, device=DEV, dtype=torch.int32)
    f.a.err = err.data_ptr()
    null = [None] * 4
    if lattice:
        axd = [a.to(DEV) for a in ax]
        where = [None] + [ctypes.c_void_p(a.data_ptr()) for a in axd]
        shape = dims
    else:
        pd = pts.to(DEV)
        where, shape = [ctypes.c_void_p(pd.data_ptr())] + null[1:], (0, 0, 0)
    _lib.call("gbsdf_sdf_points", ctypes.byref(f.a), len(pts), *where, *shape, ctypes.c_float(-1.0),
              ctypes.c_void_p(out.data_ptr()), _lib.stream_ptr(torch.device(DEV)))
    torch.cuda.synchronize()
    assert err.item() == 0
    pick = np.unique(np.concatenate([np.arange(min(len(pts), 300)), np.arange(max(0, len(pts) - 300), len(pts)),
                                     torch.randint(0, len(pts), (400,), generator=g).numpy()]))
    p32 = pts.numpy()[pick]
    enc = hg.encode((p32 + np.float32(2)) * np.float32(0.25), f.table.double().numpy(), f.ora, f.active)[:, :AF]
    W, X, B = w0e[:, :AF].double().numpy(), w0x.double().numpy(), b0.double().numpy()
    z = enc @ W.T + p32.astype(np.float64) @ X.T + B
    h = np.logaddexp(0.0, 100.0 * z) / 100.0
    a = np.abs(wh.double().numpy())
    want = -(h @ wh.double().numpy() + bh.double().item())
    # pre-activation: K0 + 8 float32 roundings of its terms; softplus: 1e-5 relative, 2e-8
    # absolute; head: 256 roundings of its terms
    dz = (K0 + 8) * 2.0 ** -22 * (np.abs(enc) @ np.abs(W).T + np.abs(p32) @ np.abs(X).T + np.abs(B))
    bound = (dz + 1e-5 * h + 2e-8 + 256 * 2.0 ** -24 * h) @ a + 2.0 ** -22
    assert (np.abs(out.double().cpu().numpy()[pick] - want) <= bound).all()
    assert torch.isfinite(out).all()


# (taps, active levels of 8 features, appearance columns, samples): K0 = 96..128, where two tiles
# share a CTA; one tile, two, an odd number, more than two per CTA, a ragged last one
FORWARD = [(6, 16, 16, 1), (6, 16, 16, 36), (6, 12, 25, 50), (4, 16, 16, 60), (4, 16, 25, 26), (6, 14, 0, 18 * SMS * 3 + 5),
           (4, 13, 16, 25 * SMS * 5 + 1)]


@pytest.mark.parametrize("case", FORWARD)
def test_forward_with_two_tiles_per_cta_equals_one(case):
    """fwd_ctas = 1 keeps one tile in flight; the outputs do not depend on it, bit for bit."""
    taps, active, app, n = case
    f = Field(8, taps, 16, active, 0.25, n)
    g = torch.Generator().manual_seed(n)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    f.a.beta, f.a.two_eps, f.a.eps2, f.a.outside_val = 100.0, 2 * f.a.eps, f.a.eps ** 2, 1000.0
    ldxc = 256 + (22 + app + 1 + 15) // 16 * 16
    dev = dict(w0b=(r(256, f.K0 + 16) * 0.1).half(), whead=r(256) * 0.1, bhead=r(1), app_table=r(4, max(app, 1)),
               app_idx=torch.tensor([2, 0, 3], dtype=torch.int32), outside=torch.tensor([0, 1, 0], dtype=torch.uint8))
    f.keep.update({k: v.to(DEV) for k, v in dev.items()})
    for k in dev:
        setattr(f.a, k, f.keep[k].data_ptr())
    f.a.app_dim, f.a.ldxc, f.a.ld_h0c = app, ldxc, 256
    x0 = torch.zeros(f.rows, 2 * f.K0 + 16, device=DEV, dtype=torch.float16)
    err = torch.zeros(1, device=DEV, dtype=torch.int32)
    f.a.x0ext, f.a.err = x0.data_ptr(), err.data_ptr()
    f.call("gbsdf_field_encode")
    got = []
    for ctas in (1, 2):
        h = lambda w: torch.full((n, w), -7.0, device=DEV, dtype=torch.float16)  # noqa: E731
        o = dict(sdf=torch.full((n,), -7.0, device=DEV), grad=torch.full((n, 3), -7.0, device=DEV),
                 hess=torch.full((n, 3), -7.0, device=DEV), h0c=h(256), h0c_lo=h(256), xc=h(ldxc), xc_lo=h(ldxc))
        for k, v in o.items():
            setattr(f.a, k, v.data_ptr())
        f.a.fwd_ctas = ctas
        f.call("gbsdf_field_mlp_fwd")
        got.append(o)
    assert err.item() == 0
    for k in got[0]:
        assert torch.equal(got[0][k], got[1][k]), k
    assert bool((got[1]["xc"][:, :256] == -7).all()) and bool((got[1]["sdf"] != -7).all())


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("case", CASES)
def test_scatter_matches_the_oracle_sum_over_evaluations(case, fixed):
    f = Field(*case)
    g = torch.Generator().manual_seed(9)
    d_enc = torch.randn(f.rows, f.K0, generator=g)
    scale = 0.37
    f.keep["d_enc"] = d_enc.to(DEV)
    f.keep["out"] = out = torch.zeros(f.lay.n_params, device=DEV)
    f.a.d_enc, f.a.d_table, f.a.d_table_scale = f.keep["d_enc"].data_ptr(), out.data_ptr(), scale
    if fixed:
        f.keep["fix"] = torch.zeros(f.lay.n_params, device=DEV, dtype=torch.int64)
        f.a.d_table_fix = f.keep["fix"].data_ptr()
    want = np.zeros((f.lay.n_entries, f.F))
    mag = np.zeros((f.lay.n_entries, f.F))
    for e in range(f.evals):
        d = np.zeros((f.n, f.lay.n_levels * f.F))
        d[:, :f.active * f.F] = d_enc.numpy()[f.row_of(e), :f.active * f.F]
        want += hg.encode_backward(f.unit[e], d, f.ora, f.active)
        mag += hg.encode_backward(f.unit[e], np.abs(d), f.ora, f.active)
    s32 = float(np.float32(scale))
    for cpt in (0, 2, 4, 8):
        out.zero_()
        f.a.scatter_cpt = cpt
        f.call("gbsdf_field_scatter")
        got = out.double().cpu().numpy().reshape(-1, f.F)
        # float32 weights (four roundings) and products, sums in any order of at most
        # evals * samples terms; 2^-48 steps of the fixed-point form
        bound = mag * s32 * (f.evals * f.n + 8) * 2.0 ** -24 + 8 * f.evals * f.n * 2.0 ** -48
        assert (np.abs(got - want * s32) <= bound).all()
        assert (got[mag == 0] == 0).all()


def test_scatter_keeps_a_non_finite_gradient_to_its_own_corners():
    f = Field(8, 6, 16, 8, 0.9, 40)
    f.keep["d_enc"] = d_enc = torch.ones(f.rows, f.K0, device=DEV)
    bad = f.row_of(3)[7]
    d_enc[bad] = float("inf")
    f.keep["out"] = out = torch.zeros(f.lay.n_params, device=DEV)
    f.keep["flag"] = flag = torch.zeros(1, device=DEV)
    f.a.d_enc, f.a.d_table, f.a.d_table_scale = d_enc.data_ptr(), out.data_ptr(), 1.0
    f.a.found_inf = flag.data_ptr()
    f.call("gbsdf_field_scatter")
    reach = hg.all_indices(f.unit[3][7:8], f.ora, f.active).reshape(-1)
    hit = ~np.isfinite(out.cpu().numpy().reshape(-1, 8)).all(axis=1)
    assert flag.item() == 1 and set(np.flatnonzero(hit)) == set(reach.tolist())
