"""The connect kernel tests a bound of the alignment cut before the cut itself: the bound, in the kernel's FP32
operations, must pass every triple that the cut passes (are_aligned of k_ca.cu), also where both sides round,
vanish, overflow or are not numbers, and hardly any other."""
import numpy as np
import pytest

F = np.float32
PTMIN = F(0.899999976158)
THETA = {True: F(0.00200000009499), False: F(0.00300000002608)}


def cut(r1, z1, ri, zi, ro, zo, theta):
    rd, dz = np.abs(r1 - ro), z1 - zo
    d13 = rd * rd + dz * dz
    t = np.abs((z1 * (ri - ro) + zi * (ro - r1)) + zo * (r1 - ri))
    return t * (PTMIN * np.sqrt(d13)) <= (theta * d13) * rd


def bound(r1, z1, ri, zi, ro, zo, theta):
    k = F(float(theta) ** 2 / 0.899999976158 ** 2 * (1 + 1e-5))

    def fma(a, b, c):
        return (a.astype(np.float64) * np.float64(b) + c).astype(F)

    u = ro - r1
    t = (z1 * (ri - ro) + zi * u) + zo * (r1 - ri)
    dz, u2 = z1 - zo, u * u
    lim = fma(u2 * fma(dz, dz.astype(np.float64), u2), k, 1e-30)
    return ~(t * t > lim)


@pytest.mark.parametrize("barrel", [True, False])
@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e-18, 1e12, 1e19])
def test_bound_passes_what_the_cut_passes(barrel, scale):
    rng = np.random.default_rng(5)
    n, theta = 400_000, THETA[barrel]
    r1, z1 = rng.uniform(2, 12, n), rng.uniform(-50, 50, n)
    ri, ro = r1 + rng.uniform(0, 8, n), r1 + rng.uniform(0, 16, n)
    slope = rng.uniform(-5, 5, n)
    zi = z1 + slope * (ri - r1)
    rd, dz = np.abs(ro - r1), slope * (ro - r1)
    # zo off the line by about the cut's limit (a few rounding errors to either side), or by anything
    off = float(theta) / float(PTMIN) * np.hypot(rd, dz) * rd / np.maximum(np.abs(ri - r1), 1e-3)
    near = rng.integers(0, 3, n)
    off *= np.where(near == 0, 1 + rng.normal(0, 1e-6, n), np.where(near == 1, rng.uniform(0, 3, n), 0.0))
    zo = z1 + dz + off * rng.choice([-1, 1], n)
    a = [(v * scale).astype(F) for v in (r1, z1, ri, zi, ro, zo)]
    a[4][:1000] = a[0][:1000]  # equal radii, equal points, and values that are no numbers
    a[5][:500] = a[1][:500]
    for k, v in enumerate((np.inf, -np.inf, np.nan)):
        a[k][1000 + 100 * k:1100 + 100 * k] = v
    with np.errstate(all="ignore"):
        c, b = cut(*a, theta), bound(*a, theta)
    assert not (c & ~b).any()
    if scale == 1.0:
        assert c.sum() > n // 4 and (b & ~c).sum() < n // 4  # only triples at the limit pass the bound alone
        far = near == 2
        assert (b[far] == c[far]).mean() > 0.999
