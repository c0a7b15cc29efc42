"""The neuron passes add a spike's term to a potential in binary32 arithmetic (add_term,
csrc/nc_device.cuh) where a rounding test proves the result, and in binary64 elsewhere.
The same operations in numpy: wherever the test passes, the sum equals the reference's
`float += double` (src/NeuCor.cpp:695) bit for bit."""
import numpy as np
import pytest

F = np.float32


def term(x, e):
    return (x.astype(np.float64) * 0.9943) * e


def add_term(p, x, e):
    """(sum, proved), binary32 operation by operation; a product less its own rounding and the
    bounds' products are exact enough in binary64 to stand for fused multiply-adds."""
    k = 0.9943 * e
    hi = F(k)
    lo = F(k - np.float64(hi))
    th = x * hi
    tl = (x.astype(np.float64) * np.float64(hi) - th).astype(F) + x * lo
    s = p + th
    bb = s - p
    err = (p - (s - bb)) + (th - bb)
    r = err + tl
    base = (np.abs(th).astype(np.float64) * 2.0 ** -43 + 2.0 ** -120).astype(F)
    base = (np.abs(s).astype(np.float64) * 2.0 ** -50 + base).astype(F)
    d = (np.abs(r).astype(np.float64) * 2.0 ** -21 + base).astype(F)
    a = s + (r + d)
    return a, a == s + (r - d)


def cases(kind, n, dt, rng):
    c52 = F(np.float64(F(0.2)) * 52.0)
    e = np.exp(0.3702 * dt)
    if kind == "ordinary":
        return rng.uniform(-90, 40, n).astype(F), F(dt) * (c52 * rng.uniform(-1, 1, n).astype(F))
    if kind == "cancel":  # sums near zero
        x = F(dt) * (c52 * rng.random(n).astype(F))
        p = -(term(x, e).astype(F))
        return (p.view(np.int32) + rng.integers(-4, 5, n).astype(np.int32)).view(F), x
    if kind == "ties":    # few-bit sums and terms far below the sum
        return rng.integers(-100, 100, n).astype(F), np.ldexp(1.0 + rng.random(n), -rng.integers(0, 40, n)).astype(F)
    return (rng.integers(0, 2 ** 32, n, dtype=np.uint32).view(F), rng.integers(0, 2 ** 32, n, dtype=np.uint32).view(F))


@pytest.mark.parametrize("dt", [0.02, 0.25, 1.0, 4.0])
@pytest.mark.parametrize("kind", ["ordinary", "cancel", "ties", "any bits"])
def test_proved_sums_are_the_reference_sums(kind, dt):
    rng = np.random.default_rng(3)
    p, x = cases(kind, 400000, dt, rng)
    with np.errstate(all="ignore"):
        a, proved = add_term(p, x, np.exp(0.3702 * dt))
        exact = (p.astype(np.float64) + term(x, np.exp(0.3702 * dt))).astype(F)
    assert np.array_equal(a[proved].view(np.uint32), exact[proved].view(np.uint32))
    if kind == "ordinary":
        assert (~proved).mean() < 1e-4  # the exact form is a rare one


def test_an_absent_term_changes_nothing():
    p = np.concatenate([np.linspace(-90, 40, 9999).astype(F), np.array([np.inf, -1e-38, 1e30], F)])
    with np.errstate(all="ignore"):
        a, proved = add_term(p, np.full(len(p), -0.0, F), np.exp(0.3702))
    assert np.array_equal(a[proved].view(np.uint32), p[proved].view(np.uint32))
