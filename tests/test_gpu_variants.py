"""Launch variants of the FFT passes (B200).

Every (row, column) launch-variant pair of an operator gives the same apply
up to the rounding of its transform shape: a variant change re-tiles the
half spectrum for the column tile width it implies, and with it the
free-space Kh and the periodic multiplier table, and switches the row
passes between their fixed-stride and general tile forms.  The autotuner
leaves the apply unchanged the same way.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _apply(op, x):
    y = torch.empty_like(x)
    op.matvec_(x, y)
    torch.cuda.synchronize()
    return y.double().cpu().numpy()


@pytest.mark.parametrize("backend", ["fft", "periodic"])
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 2e-6)])
@pytest.mark.parametrize("Ns", [256, 1024])
def test_every_variant_pair_gives_the_same_apply(backend, dtype, tol, Ns):
    import aspher_b200 as asb
    op = asb.Operator(backend, Ns)
    rv0, cv0, _ = op.variants(dtype)
    g = torch.Generator(device="cuda")
    g.manual_seed(Ns)
    x = torch.randn(Ns * Ns, dtype=dtype, device="cuda", generator=g)
    y0 = _apply(op, x)
    n0 = np.linalg.norm(y0)
    widths = set()
    for rv in range(4):
        for cv in range(4):
            op.set_variants(rv, cv, dtype)
            assert op.variants(dtype)[:2] == (rv, cv)
            widths.add(op.variants(dtype)[2])
            y = _apply(op, x)
            assert np.linalg.norm(y - y0) <= tol * n0, (rv, cv)
    # the sweep crossed column tile widths (so the tables were re-tiled)
    assert len(widths) > 1
    op.set_variants(rv0, cv0, dtype)
    assert np.array_equal(_apply(op, x), y0)


@pytest.mark.parametrize("backend", ["fft", "periodic"])
def test_autotune_keeps_the_apply(backend):
    import aspher_b200 as asb
    Ns = 512
    op = asb.Operator(backend, Ns)
    x = torch.randn(Ns * Ns, dtype=torch.float32, device="cuda")
    y0 = _apply(op, x)
    rv, cv, ms = op.autotune(torch.float32, reps=2)
    assert 0 <= rv < 4 and 0 <= cv < 4 and ms > 0.0
    assert op.variants(torch.float32)[:2] == (rv, cv)
    y = _apply(op, x)
    assert np.linalg.norm(y - y0) <= 2e-6 * np.linalg.norm(y0)


def test_long_rows_of_the_wide_variant():
    """Row variant 3 from 1024 points per row on: 512-thread CTAs, two FP64 rows
    of 2048 points each.  Same apply, and at periodic 4096 the default for its
    time (0.96-0.983 of variant 2's, the default before)."""
    import aspher_b200 as asb
    op = asb.Operator("periodic", 4096)
    x = torch.randn(4096 * 4096, dtype=torch.float64, device="cuda")
    rv, cv, _ = op.variants(torch.float64)

    def ms(row):
        op.set_variants(row, cv, torch.float64)
        y = torch.empty_like(x)
        best = float("inf")
        for _ in range(6):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(20):
                op.matvec_(x, y)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best, y
    (t, y), (t2, y2) = ms(rv), ms(2)
    assert float((y - y2).norm()) <= 1e-13 * float(y2.norm())
    assert t <= 0.995 * t2, (t, t2)


@pytest.mark.parametrize("backend", ["fft", "periodic"])
def test_variants_reach_the_embedded_apply(backend):
    """A grid of 300 on the 512-sided pipeline: row variants with other points
    per thread round differently, within the tolerance of the default's apply."""
    import aspher_b200 as asb
    op = asb.Operator(backend, 300)
    cv = op.variants(torch.float64)[1]
    x = torch.randn(300 * 300, dtype=torch.float64, device="cuda")
    ys = []
    for rv in range(4):
        op.set_variants(rv, cv, torch.float64)
        ys.append(op.matvec_(x, torch.empty_like(x)))
        assert float((ys[-1] - ys[0]).norm()) <= 1e-13 * float(ys[0].norm())
    assert not torch.equal(ys[0], ys[2])  # 16 and 8 points per thread


@pytest.mark.parametrize("backend,Ns,dtype,tol", [
    ("fft", 768, torch.float64, 1e-8), ("periodic", 600, torch.float64, 1e-8),
    ("fft", 256, torch.float64, 1e-8), ("periodic", 512, torch.float64, 1e-8),
    ("fft", 256, torch.float32, 1e-3), ("periodic", 512, torch.float32, 1e-3)])
def test_variants_reach_the_passes_of_a_solve(backend, Ns, dtype, tol):
    """The row passes that carry evaluate(), the direction update and the line
    sums take the row variant: their CTAs reduce in other groups, so ten
    iterations end in other bits of the same pressure (in FP32 the sums are
    rounded to the field's 24 bits and only other points per thread show: sides
    of 3 2^k have 24 in both shapes).  Every pair of variants gives that
    pressure.  FP32 bound: applies that differ by 4e-6 (2e-6 each, the applies'
    own bound) in ten steps, times at most 25 for the preconditioned operator's
    condition: 1e-3."""
    import aspher_b200 as asb
    op = asb.Operator(backend, Ns)
    g = torch.from_numpy(asb.self_affine_gap(Ns, hurst=0.8, rms=0.002, k_lo=1.5, k_hi=Ns / 8,
                                             seed=6)).cuda().to(dtype)

    def pressure(rv, cv):
        op.set_variants(rv, cv, dtype)
        r = asb.solve_device(op, g, 0.02, tol=1e-12, max_iter=10, precond="fourier", dtype=dtype,
                             light=True)
        return r.pressure_device
    p0 = pressure(0, 1)
    assert not torch.equal(pressure(2, 1), p0)
    for rv in range(4):
        for cv in range(4):
            assert float((pressure(rv, cv) - p0).norm()) <= tol * float(p0.norm()), (rv, cv)
