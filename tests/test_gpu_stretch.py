"""The SVD-free fixed-corotated stress (slosh_b200/csrc/stretch.cuh) on both
sides of its range, against the FP64 oracle.

As in test_gpu_svd.py, particles at rest carry chosen deformation gradients,
so that one substep applies the model to F alone: F' is read back from the
records, the Kirchhoff stress from C = -tau V0 (4 / h^2) dt.
The families put the strain at rounding size, small, moderate, just inside and
just outside the range's edge (|X|_F = 1/2 in 3D, X^2 = I / 8 in 2D, b = F F^T
= (1 + m)(I + X)), and well outside, under a random rotation.

Tolerance.  F is FP32, so b is known to a few ulps of its entries: the stress
carries an error of that size times the stiffness, 2e-6 (lambda + 2 mu) +
1e-5 max |tau| and F' 1e-6 + 1e-5 max |F'| (the bounds of test_gpu_svd.py,
which cover the SVD side).
"""
import numpy as np
import pytest

from oracle import oracle as O
from slosh_b200.pipeline import MpmData, MpmPipeline, ParticleModel, SimulationParams, make_particles

pytestmark = pytest.mark.gpu

H = 1.0 / 64.0
DT = 2.0e-5


def _rotation(rng, dim):
    q, r = np.linalg.qr(rng.normal(size=(dim, dim)))
    q = q * np.sign(np.diag(r))[None, :]
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    return q


def _deformations(rng, dim, per):
    """F = U sqrt(b) V^T with b = (1 + m)(I + X), |X|_F = size."""
    edge = 0.5
    out = []
    for size, vol in ((1e-7, 1e-7), (1e-4, 1e-5), (1e-2, -1e-2), (0.2, 0.1), (0.99 * edge, -0.2), (1.01 * edge, 0.2),
                      (0.7, -0.3)):
        for _ in range(per):
            x = rng.normal(size=dim)
            x -= x.mean()
            x *= size / np.linalg.norm(x)
            x *= min(1.0, 0.95 / max(-x.min(), 1e-30))  # b stays positive
            m = vol * rng.uniform(0.5, 1.5)
            s = np.sqrt((1.0 + m) * (1.0 + x))
            out.append(_rotation(rng, dim) @ np.diag(s) @ _rotation(rng, dim).T)
    for _ in range(per):  # no rotation
        out.append(np.eye(dim) + 1e-3 * np.diag(rng.normal(size=dim)))
    return np.asarray(out, np.float32)


@pytest.mark.parametrize("dim", [2, 3])
def test_stretch_update_against_fp64_oracle(cuda_lib, dim):
    rng = np.random.default_rng(7 + dim)
    model = ParticleModel.elastic(1.0e5, 0.3)
    fs = _deformations(rng, dim, 40)
    n = len(fs)
    side = int(np.ceil(n ** (1 / 3)))
    idx = np.arange(n)
    pts = 0.25 + H * np.stack([idx % side, (idx // side) % side, idx // (side * side)], axis=1) + 0.5 * H
    if dim == 2:
        pts = 0.25 + H * np.stack([idx % 32, idx // 32], axis=1) + 0.5 * H
    recs = make_particles(pts, H / 4, 1000.0, model, dim=dim)
    for r in range(dim):
        for c in range(dim):
            recs["def_grad"][:, c * 3 + r] = fs[:, r, c]
    params = SimulationParams((0.0,) * dim, DT)
    data = MpmData(params, recs, [], cell_width=H, grid_capacity=1 << 12, dim=dim)
    MpmPipeline().launch_step(data, 1)
    got = data.download_particles()
    data.close()
    orc = O.Oracle(dim, H, 1 << 12, double=True)
    orc.set_params(params.gravity, DT)
    orc.set_particles(recs)
    orc.step(1)
    ref = orc.get_particles()

    coef = float(recs["init_volume"][0]) * 4.0 / (H * H) * DT
    lam, mu = model.data[0], model.data[1]
    assert np.array_equal(got["enabled"], ref["enabled"])
    tau, tau64 = got["affine"] / coef, ref["affine"] / coef
    per = n // 8
    for k in range(8):
        sel = slice(k * per, (k + 1) * per)
        et = np.abs(tau[sel] - tau64[sel]).max()
        bt = 2e-6 * (lam + 2.0 * mu) + 1e-5 * np.abs(tau64[sel]).max()
        ef = np.abs(got["def_grad"][sel] - ref["def_grad"][sel]).max()
        bf = 1e-6 + 1e-5 * np.abs(ref["def_grad"][sel]).max()
        print(f"family {k}: tau err {et:.3e} (bound {bt:.3e}), F' err {ef:.3e} (bound {bf:.3e})")
        assert et <= bt and ef <= bf, k
