"""Tracks at the edges of the fits' formulas."""
import numpy as np

B_FIELD = 0.0114256972711507
RADII = (2.9, 6.8, 10.9, 16.0, 20.0, 24.0, 28.0, 32.0)


def _errors(hits):
    """Covariances of 10 um along r-phi and 20 um along z."""
    r = np.hypot(hits[:, 0], hits[:, 1])
    s, c = hits[:, 1] / r, hits[:, 0] / r
    ge = np.zeros((len(hits), 6), np.float32)
    ge[:, 0], ge[:, 1], ge[:, 2] = 1e-6 * s * s, -1e-6 * s * c, 1e-6 * c * c
    ge[:, 5] = 4e-6
    return ge


def flat_tracks(count: int = 6, seed: int = 1):
    """Helices across the beam whose first and last hit have the same z, or nearly so: [(hits, ge)], 3, 4 and 8 hits,
    both charges, measured with the errors of the covariances."""
    rng = np.random.default_rng(seed)
    out = []
    for n in (3, 4, 8):
        for dz in (0.0, 1e-9, -1e-9, 1e-300, 1e-4):
            for k in range(count):
                r, sign = np.array(RADII[:n]), (1, -1)[k % 2]
                radius = rng.uniform(60, 900)
                a = 2 * np.arcsin(r / (2 * radius))
                x, y = radius * np.sin(a), sign * radius * (1 - np.cos(a))
                y = y + rng.normal(0, 1e-3, n)
                phi = rng.uniform(-np.pi, np.pi)
                z = rng.uniform(-20, 20) + rng.normal(0, 2e-3, n)
                z[-1] = z[0] + dz
                hits = np.stack([x * np.cos(phi) - y * np.sin(phi), x * np.sin(phi) + y * np.cos(phi), z], 1)
                out.append((hits, _errors(hits)))
    return out


def straight_tracks(count: int = 8, seed: int = 2):
    """Collinear hits, whose circle has no centre: [(hits, ge)], 3, 4 and 8 hits, along directions in which the
    products of the chords' components are equal but not representable."""
    rng = np.random.default_rng(seed)
    out = []
    for n in (3, 4, 8):
        for dx, dy in ((1, 1), (1, -1), (1, 0.25), (-0.5, 1), (-1, -4), (1, 0), (0, -1)):
            for _ in range(count):
                s = np.array(RADII[:n]) + rng.uniform(0, 0.1, n)
                hits = np.stack([dx * s, dy * s, 1.0 + 0.3 * s], 1)
                out.append((hits, _errors(hits)))
    return out


def centred_tracks(count: int = 12, seed: int = 3):
    """Hits on circles about the beam line, whose impact parameter is the radius: [(hits, ge, radius)], 3, 4 and 8 hits."""
    rng = np.random.default_rng(seed)
    out = []
    for n in (3, 4, 8):
        for r in (2.9, 6.8, 7.0, 10.0):
            for _ in range(count):
                a = np.sort(rng.uniform(0, 2, n))
                z = rng.uniform(-5, 5) + rng.uniform(-1, 1) * r * a + rng.normal(0, 2e-3, n)
                hits = np.stack([r * np.cos(a), r * np.sin(a), z], 1)
                out.append((hits, _errors(hits), r))
    return out


def rounded_straight_tracks(count: int = 400, seed: int = 4):
    """Straight tracks in any direction: collinear up to the rounding of their hits, which decides whether the fast
    fit's circle has a radius of 1e16 cm or none."""
    rng = np.random.default_rng(seed)
    out = []
    for t in range(count):
        hits = np.outer(RADII[:(3, 4, 8)[t % 3]], rng.normal(size=3))
        out.append((hits, _errors(hits)))
    return out
