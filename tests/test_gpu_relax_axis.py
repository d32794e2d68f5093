"""The relaxations with a lane for each axis of a stroke against the one-lane kernels: the same
operations on the same operands, so the same results bit for bit (no tolerance).  Stroke counts
around a warp's ten (eight) strokes and a CTA's, one stroke, periodic wraps in every direction,
both algorithms, every probe start, no iterations allowed, outputs left out."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (34, 29, 41)
CELL = np.diag([6.8, 5.8, 8.2])


def _grid(seed=0):
    import torch

    from ppafm_gb300 import device as D

    rng = np.random.default_rng(seed)
    k = [rng.integers(-2, 3, 3) for _ in range(6)]
    x = np.stack(np.meshgrid(*[np.arange(m) / m for m in N], indexing="ij"), -1) * 2 * np.pi
    F = np.zeros(N + (4,), np.float32)
    for v in k:
        F += rng.normal(0, 0.06, 4) * np.sin(x @ v + rng.uniform(0, 6))[..., None]
    return D.DeviceFF(N, CELL, FE=torch.from_numpy(F.reshape(-1)).cuda())


def _prm(maxIters=120):
    from ppafm_gb300 import device as D

    return D.relax_params(maxIters=maxIters, dt=0.5, kRadial=-20.0 / 16.0, kSpring=(-0.0156, -0.0156, 0.0))


def _with_tps(tps, fn):
    from ppafm_gb300._lib import check, lib

    check(lib().ppgpu_set_relax_tps(tps))
    try:
        return fn()
    finally:
        check(lib().ppgpu_set_relax_tps(0))


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (3, 3, 12), (2, 5, 20), (1, 11, 15), (8, 5, 14), (41, 1, 13), (37, 23, 17)])
@pytest.mark.parametrize("maxIters", [0, 1, 120])
def test_axis_scan_matches_one_lane(gpulib, nx, ny, nz, maxIters):
    from ppafm_gb300 import device as D

    ff = _grid(nx + nz)
    rng = np.random.default_rng(ny)
    xs, ys = rng.uniform(-9, 15, nx), rng.uniform(-9, 15, ny)
    zs = np.linspace(11.0, 2.0, nz)
    W = np.linspace(-1, 1, 11) if nz >= 11 else None

    def run():
        return D.relax_scan(ff, _prm(maxIters), xs, ys, zs, pos_offset=(0.3, -0.2, 1.0), df_weights=W, want_iters=True)

    a, b = _with_tps(1, run), _with_tps(0, run)
    assert sorted(a) == sorted(b)
    for k in a:
        assert a[k].equal(b[k]), k


@pytest.mark.parametrize("r0", [(-0.1, 0.1, 4.0), (0.1, -0.1, 4.0)])
def test_axis_scan_over_the_whole_cell(gpulib, r0):
    """A rest position beside the tip, and strokes in every x cell, the last ones too."""
    from ppafm_gb300 import device as D

    ff = _grid(5)
    xs, ys = np.arange(N[0]) * 0.2 + 0.05, np.arange(N[1]) * 0.2 + 0.07
    zs = np.linspace(11.0, 9.0, 12)
    prm = D.relax_params(maxIters=120, dt=0.5, kRadial=-20.0 / 16.0, kSpring=(-0.0156, -0.0156, 0.0), rPP0=r0)

    def run():
        return D.relax_scan(ff, prm, xs, ys, zs, want_iters=True)

    a, b = _with_tps(1, run), _with_tps(0, run)
    for k in a:
        assert a[k].equal(b[k]), k


@pytest.mark.parametrize("probeStart", [-1, 0, 1])
@pytest.mark.parametrize("relaxAlg", [0, 1])
@pytest.mark.parametrize("nstroke", [1, 10, 11, 40, 203])
def test_axis_strokes_match_one_lane(gpulib, probeStart, relaxAlg, nstroke):
    from ppafm_gb300 import device as D

    ff = _grid(3)
    rng = np.random.default_rng(nstroke)
    tips = np.cumsum(rng.uniform(-0.15, 0.1, (nstroke, 9, 3)), axis=1) + rng.uniform(-8, 14, (nstroke, 1, 3))

    def run():
        return D.relax_strokes(ff, _prm(), tips, probeStart=probeStart, relaxAlg=relaxAlg, iters=True)

    for x, y in zip(_with_tps(1, run), _with_tps(0, run)):
        assert x.equal(y)


@pytest.mark.parametrize("npix,nz", [(1, 1), (8, 12), (9, 15), (33, 14), (1000, 11)])
def test_afm_axis_matches_one_lane(gpulib, npix, nz):
    """The AFMulator kernels choose by the number of strokes, which do not depend on each other: the
    first npix of 41000 by the one-lane kernel, then alone by the other."""
    import torch

    from ppafm_gb300._lib import AFM_NPARAM, check, dptr, iptr, lib, stream_handle, tptr

    ff = _grid(9)
    rng = np.random.default_rng(nz)
    many = 41000
    pts = torch.tensor(np.column_stack([rng.uniform(-9, 15, (many, 2)), rng.uniform(3, 12, many), np.zeros(many)]).astype(np.float32)).cuda()
    prm = np.zeros(AFM_NPARAM)
    c, s = np.cos(0.2), np.sin(0.2)  # a tilted tip
    prm[0:2], prm[4:8], prm[8:12] = (0.5, 0.1), np.array([0.25, 0.25, 0.0, 30.0]) / -16.0217662, (0.1, 0.0, -2.998, 3.0)
    prm[12:24] = [c, 0, -s, 0, 0, 1, 0, 0, s, 0, c, -0.1]
    prm[24] = 0.01
    inv = np.ascontiguousarray(np.linalg.inv(CELL).T)
    nw = min(10, nz)
    W = np.linspace(-1, 1, nw)

    def run(m):
        o = [torch.full((m, nz, 4), 9.0, device="cuda"), torch.full((m, nz, 4), 9.0, device="cuda"), torch.zeros((m, nz), dtype=torch.int32, device="cuda"), torch.full((m, nz - nw + 1), 9.0, device="cuda")]
        n = torch.zeros(1, dtype=torch.int64, device="cuda")
        check(lib().ppgpu_relax_afm(tptr(ff.FE), iptr(np.array(N, np.int32)), dptr(inv), dptr(prm), m, tptr(pts), nz, tptr(o[0]), tptr(o[1]), tptr(o[2]), nw, dptr(W), tptr(o[3]), tptr(n), stream_handle()))
        return o, int(n.item())

    one, _ = run(many)
    axis, total = run(npix)
    for x, y in zip(one, axis):
        assert x[:npix].equal(y)
    it = one[2][:npix]
    assert int((it.clamp(max=127) + 1).sum()) == total


TILTED = np.array([[6.8, 0, 0], [0.9, 5.8, 0], [0.4, -0.5, 8.2]])


@pytest.mark.parametrize("spline", [False, True])
@pytest.mark.parametrize("cell", [CELL, TILTED], ids=["diagonal", "tilted"])
def test_large_scans_match_small_ones(gpulib, cell, spline):
    """More strokes than keep the corners of their cell (77 824): the same bits as scans of a part of
    them, one lane a stroke as well."""
    import torch

    from ppafm_gb300 import device as D

    ff = D.DeviceFF(N, cell, FE=_grid(4).FE)
    rng = np.random.default_rng(8)
    xs, ys, zs = rng.uniform(-9, 15, 260), rng.uniform(-9, 15, 301), np.linspace(11.0, 10.0, 4)
    x = np.linspace(2, 6, 31)
    with D.tip_spline((x, np.column_stack([-1.25 * (x - 4.0), np.full(31, -1.25)])) if spline else None):

        def run(part):
            return D.relax_scan(ff, _prm(60), part, ys, zs, df_weights=np.array([1.0, -2.0]), want_iters=True)

        whole = run(xs)
        parts = [_with_tps(1, lambda p=p: {k: v.clone() for k, v in run(p).items()}) for p in (xs[:130], xs[130:])]
    for k in whole:
        assert whole[k].equal(torch.cat([p[k] for p in parts])), k


def test_large_afm_scans_match_small_ones(gpulib):
    """The AFMulator's relaxation beyond 116 736 strokes against a part of them."""
    import torch

    from ppafm_gb300._lib import AFM_NPARAM, check, dptr, iptr, lib, stream_handle, tptr

    ff = _grid(9)
    rng = np.random.default_rng(12)
    many, some, nz = 117001, 60000, 3
    pts = torch.tensor(np.column_stack([rng.uniform(-9, 15, (many, 2)), rng.uniform(3, 12, many), np.zeros(many)]).astype(np.float32)).cuda()
    prm = np.zeros(AFM_NPARAM)
    prm[0:2], prm[4:8], prm[8:12] = (0.5, 0.1), np.array([0.25, 0.25, 0.0, 30.0]) / -16.0217662, (0.1, 0.0, -2.998, 3.0)
    prm[12:24] = [1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, -0.1]
    inv = np.ascontiguousarray(np.linalg.inv(CELL).T)
    W = np.array([1.0, -2.0])

    def run(m):
        o = [torch.full((m, nz, 4), 9.0, device="cuda"), torch.full((m, nz, 4), 9.0, device="cuda"), torch.zeros((m, nz), dtype=torch.int32, device="cuda"), torch.full((m, nz - 1), 9.0, device="cuda")]
        check(lib().ppgpu_relax_afm(tptr(ff.FE), iptr(np.array(N, np.int32)), dptr(inv), dptr(prm), m, tptr(pts), nz, tptr(o[0]), tptr(o[1]), tptr(o[2]), 2, dptr(W), tptr(o[3]), None, stream_handle()))
        return o

    for x, y in zip(run(many), run(some)):
        assert x[:some].equal(y)
