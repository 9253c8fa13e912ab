"""GPU tests of the step's small-mesh paths.

Deposit tiles have fewer rows where a mesh would give too few of them, both
fixed-point forms of the binary64 deposit are launched on meshes up to 128^3 (the
device picks), the bucket scan runs in one block up to four tiles of 4096 counts and
in two kernels above, and the densest bucket is found by the scan. One KDK step of
each size against the oracle: binary64 positions to 1e-12 of a cell, forces to 1e-12
of the largest; the FP32 form's forces to 1e-4 of the largest (its bar) and what
the deposit's weights cut off (B bits of each fraction, the most up to 16 for which
8 c 2^(3B) < 2^63, c the densest bucket of the states deposited; cutting shifts mass by
up to 2^-B of a cell on three axes, and the force changes by at most twice the largest
within a cell: 9e-5 at 16 bits), its
positions to what that error of the opening kick drifts, the FP32 rounding of the
momenta and two units of the fixed-point coordinates, and the force after the drift
also to what that shift of the particle and of its sources changes.
"""
import numpy as np
import pytest

import hyowon_b200 as hb

pytestmark = pytest.mark.gpu


def state(n, L, clustered, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(0, L, (3, n))
    if clustered:      # one dense knot: more than 63 sources in a bucket
        k = n // 3
        p[:, :k] = np.mod(0.999 * L + rng.normal(0, 0.01 * L, (3, k)), L)
    return p, rng.normal(0, 1.0, (3, n))


def fraction_bits(N, n, L, states):
    """B of the densest bucket (2^shift consecutive cells, some eight particles)."""
    shift = 0
    while (N ** 3 >> (shift + 1)) * 8 >= n and N ** 3 >> (shift + 1):
        shift += 1
    densest = 0
    for p in states:
        i, j, k = (np.minimum((np.mod(c, L) / L * N).astype(np.int64), N - 1) for c in p)
        densest = max(densest, int(np.bincount((((i * N) + j) * N + k) >> shift).max()))
    bits = 16
    while 8 * densest << 3 * bits > 2 ** 63 - 1:
        bits -= 1
    return bits


# buckets + 1 = 4097 at (64, 32768), 16385 (five tiles) at (128, 100000), 5 at (12, 40)
@pytest.mark.parametrize("clustered", [False, True])
@pytest.mark.parametrize("N,n", [(12, 40), (16, 5000), (31, 3000), (32, 4096), (33, 7), (48, 20000),
                                 (64, 32768), (64, 262144), (100, 50000), (128, 100000)])
def test_one_step_against_the_oracle(oracle, N, n, clustered):
    L, m = 100.0, 2.5
    (x, y, z), (px, py, pz) = state(n, L, clustered, N + n)
    K1, D, K2 = 0.01, 0.02, 0.015
    ref = dict(x=x.copy(), y=y.copy(), z=z.copy(), px=px.copy(), py=py.copy(), pz=pz.copy())
    ref["ax"], ref["ay"], ref["az"] = oracle.pm_forces(L, N, x, y, z, uniform_mass=m)
    scale0 = max(float(np.max(np.abs(ref[a]))) for a in ("ax", "ay", "az"))
    drift = oracle.kdk_step(L, N, ref, K1, D, K2, uniform_mass=m)
    scale = max(float(np.max(np.abs(ref[a]))) for a in ("ax", "ay", "az"))
    bits = fraction_bits(N, n, L, [(x, y, z), (ref["x"], ref["y"], ref["z"])])
    for precision, tol in (("fp64", 1e-12), ("fp32", 1e-4 + 6.0 * 2.0 ** -bits)):
        with hb.PMSolver(hb.MeshGeometry(L, N), hb.PMForceMethod.pure_pm(False), precision) as s:
            s.upload(x, y, z, px, py, pz, uniform_mass=m)
            md = s.kdk_step(K1, D, K2)
            got = s.download()
        cell = L / N
        p_max = max(float(np.max(np.abs(p))) for p in (px, py, pz)) + K1 * scale0
        bound = 1e-12 * cell if precision == "fp64" else \
            D * (K1 * tol * scale0 + 2e-7 * p_max) + 2 * L / 2 ** 32
        for a in "xyz":
            d = np.abs((got[a] - ref[a] + L / 2) % L - L / 2)
            assert d.max() <= bound
        err = max(float(np.max(np.abs(got["a" + a] - ref["a" + a]))) for a in "xyz")
        assert err <= tol * scale + 4.0 * scale * bound / cell
        assert abs(md - drift) <= (1e-13 if precision == "fp64" else 1e-5) * drift
