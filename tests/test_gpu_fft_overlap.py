"""The density-overlap force field in one round trip of the transforms against the calls it stands
for (density_power, potential2forces, poisson, potential2forces), on even, odd and prime sizes, with
and without the Pauli exponent, the negative-density fix and the electrostatic part.

Tolerance: float64 plans differ by the step-by-step form's float32 grids between the transforms
(rho^B and V, 2^-24 of their maxima) and the stored float32: 1e-6 of the field's maximum; float32
transforms leave ~1e-6 of the field's maximum at every point on either side (the FFT tests' figure):
5e-6.  Skewed cells keep the step-by-step form."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _densities(n, seed):
    import torch

    rng = np.random.default_rng(seed)
    x = np.meshgrid(*[np.arange(m) / m for m in n], indexing="ij")
    out = []
    for kind in range(3):
        r = np.zeros(n)
        for _ in range(5):
            c, s = rng.uniform(0, 1, 3), rng.uniform(0.06, 0.12)
            if kind == 2:
                c = np.zeros(3)
            d2 = sum((v - a - np.round(v - a)) ** 2 for v, a in zip(x, c))
            r += rng.uniform(0.5, 2.0) * (rng.choice([-1, 1]) if kind == 1 else 1) * np.exp(-d2 / (2 * s * s))
        r += 1e-3 * rng.normal(size=n)  # some negative values in the tails
        out.append(torch.tensor((r - (r.mean() if kind == 1 else 0)).astype(np.float32)).cuda())
    return out


@pytest.mark.parametrize("n", [(32, 32, 32), (27, 40, 35), (31, 24, 33), (16, 54, 1), (48, 20, 90)])
@pytest.mark.parametrize("B,fix,charge", [(1.0, True, True), (1.2, True, True), (1.0, False, True), (1.0, True, False)])
@pytest.mark.parametrize("f64", [False, True])
def test_overlap_forces_match_the_steps(gpulib, n, B, fix, charge, f64):
    import torch

    from ppafm_gb300.fieldFFT import FFTGrid

    rho_s, rho_q, rho_t = _densities(n, sum(n))
    if B != 1.0 and not fix:
        rho_s.abs_(), rho_t.abs_()
    lvec = np.array([[0, 0, 0], [0.3 * n[0], 0, 0], [0, 0.25 * n[1], 0], [0, 0, 0.28 * n[2]]])
    g = FFTGrid(n, f64=f64)
    ws, wt = (g.density_power(t.clone(), B, fix) for t in (rho_s, rho_t))
    ref = g.potential2forces(ws, wt, lvec, scale=12.0, with_E=True)
    if charge:
        g.potential2forces(g.poisson(rho_q, lvec), rho_t, lvec, FE=ref, scale=-0.01, with_E=True, accumulate=True)
    keep = [t.clone() for t in (rho_s, rho_q, rho_t)]
    FE = torch.full((g.N * 4,), float("nan"), device="cuda")
    g.overlap_forces(rho_s, rho_t, rho_q if charge else None, lvec, FE, B=B, fix_negative=fix, scale_p=12.0, scale_e=-0.01)
    assert all(a.equal(b) for a, b in zip(keep, (rho_s, rho_q, rho_t)))
    a, b = FE.view(-1, 4).double(), ref.view(-1, 4).double()
    tol = (1e-6 if f64 else 5e-6) * b.abs().max(dim=0).values.clamp_min(1e-30)
    tol[:3] = tol[:3].max()
    assert bool(((a - b).abs() <= tol).all()), ((a - b).abs().max(dim=0).values / tol).tolist()


def test_pipeline_forms_agree(gpulib):
    """build_ff in one round trip, then step by step (densities that need converting), and the
    potential as the step-by-step form leaves it."""
    from ppafm_gb300 import HighLevel, workloads

    pl = HighLevel.DensityOverlapPipeline.from_workload(workloads.density_overlap(seed=1, scale=0.2))
    assert pl._one_round_trip()
    a = pl.build_ff().FE.clone()
    Va = pl.V.clone()
    pl.rho_s = pl.rho_s.double()
    assert not pl._one_round_trip()
    b = pl.build_ff().FE
    m = b.view(-1, 4).abs().max(dim=0).values
    m[:3] = m[:3].max()
    assert bool(((a - b).view(-1, 4).abs() <= 5e-6 * m).all())
    assert pl.V.equal(Va)


def test_overlap_forces_rejects_skewed_cells(gpulib):
    import torch

    from ppafm_gb300._lib import PPGPUError
    from ppafm_gb300.fieldFFT import FFTGrid

    g = FFTGrid((8, 8, 8))
    r = g.empty().fill_(1.0)
    FE = torch.empty(g.N * 4, device="cuda")
    with pytest.raises(PPGPUError, match="orthogonal"):
        g.overlap_forces(r, r, None, np.array([[4.0, 0, 0], [0.5, 4, 0], [0, 0, 4]]), FE)


@pytest.mark.parametrize("f64", [False, True])
def test_potential_is_that_of_the_last_build(gpulib, f64):
    """V, one buffer for the pipeline's life, holds the potential that the last build_ff used: bit for
    bit poisson's, whatever happened to the densities since, on any stream, captured or not."""
    import torch

    from ppafm_gb300 import HighLevel, workloads

    pl = HighLevel.DensityOverlapPipeline.from_workload(workloads.density_overlap(seed=2, scale=0.15), f64=f64)
    assert pl._one_round_trip() and pl.Q != 0.0
    V = pl.V
    pl.build_ff()
    first = V.clone()
    assert first.equal(pl.fft.poisson(pl.rho_q, pl.lvec))
    keep = [t.clone() for t in (pl.rho_s, pl.rho_q, pl.rho_t)]
    pl.set_densities(keep[0], 2.0 * keep[1].roll(3, 0), keep[2])
    assert pl.V is V and V.equal(first)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    pl.build_ff(stream=s)
    torch.cuda.current_stream().wait_stream(s)
    second = V.clone()
    assert second.equal(pl.fft.poisson(pl.rho_q, pl.lvec)) and not second.equal(first)
    pl.set_densities(*keep)
    torch.cuda.synchronize()
    out = torch.zeros_like(V)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        pl.build_ff()
        out.copy_(pl.V)
    g.replay()
    torch.cuda.synchronize()
    assert out.equal(first) and V.equal(first)
    pl.V = torch.zeros_like(V)  # another buffer of the caller's
    pl.build_ff()
    assert pl.V.equal(first)


def test_step_by_step_form_allocates_nothing(gpulib):
    """A skewed cell's build_ff, the first one too and on a stream of its own, works in the pipeline's
    buffers: memory taken from the current stream's pool there could still be in use."""
    import torch

    from ppafm_gb300 import HighLevel, workloads

    w = workloads.density_overlap(seed=3, scale=0.12)
    lvec = np.array(w["lvec"], dtype=np.float64)
    lvec[2, 0] += 0.2 * lvec[1, 0]
    pl = HighLevel.DensityOverlapPipeline.from_workload(dict(w, lvec=lvec))
    assert not pl._one_round_trip()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    before = torch.cuda.memory_allocated()
    pl.build_ff(stream=s)
    assert torch.cuda.memory_allocated() == before
    s.synchronize()
    assert bool(torch.isfinite(pl.ff.FE).all())
