"""The adjoint at ordinary wavelengths against the package's own bar: the vector-Jacobian product of
a random cotangent within 1e-4 of the largest gradient of torch's FP64 autograd of the closed form.
Facets of one to fifty phase radians, near the origin and 60 and 200 um from it, over grids around
the 32 lanes."""
import numpy as np
import pytest
import torch

import abt_b200
from oracle import adjoint_ref as AR
from tests.helpers import outbeams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lam", [0.532, 3.0])
@pytest.mark.parametrize("offset", [0.0, 60.0, 200.0])
@pytest.mark.parametrize("size", [1.0, 10.0, 50.0])
@pytest.mark.parametrize("nt,nphi", [(7, 9), (33, 31)])
def test_vjp(ctx, lam, offset, size, nt, nphi):
    rng = np.random.default_rng(nt + int(size))
    k = 2 * abt_b200.PI_REF / lam
    n = 6
    tri = (rng.normal(size=(n, 3, 3)) + 3.0 * rng.normal(size=(n, 1, 3))) * (0.5 * size / k)
    verts = tri.reshape(-1, 3) + offset / np.sqrt(3.0) * np.array([1.0, -1.0, 1.0])
    faces = np.arange(1, 3 * n + 1).reshape(n, 3)
    geo = abt_b200.make_geometry(verts, faces.tolist())
    beam = outbeams(n, rng, n)
    beam["fi"] = np.arange(1, n + 1)
    th = np.linspace(15.0, 165.0, nt) * abt_b200.PI_REF / 180.0
    ph = (0.3 + np.arange(nphi) * 360.0 / nphi) * abt_b200.PI_REF / 180.0
    G = rng.normal(size=(nphi, nt, 2, 2)) + 1j * rng.normal(size=(nphi, nt, 2, 2))
    X = np.stack(abt_b200.make_far_field_bins(th, ph), -1)
    common = np.exp(1j * k * np.linalg.norm(X, axis=-1))[:, :, None, None]
    gv, gb, _ = ctx.diff_adjoint(beam, None, geo, th, ph, lam, G * common, np.zeros_like(G))
    V = torch.from_numpy(verts.copy()).requires_grad_(True)
    z = torch.from_numpy(beam["ampl"][:, 0::2] + 1j * beam["ampl"][:, 1::2]).requires_grad_(True)
    a = torch.stack([torch.stack([z[:, 0], z[:, 2]], 1), torch.stack([z[:, 1], z[:, 3]], 1)], 1)
    S = AR.forward(V, faces - 1, beam["fi"] - 1, a, beam["prop_out"], beam["vk7"], [], None, [], [],
                   th, ph, lam).reshape(nt, nphi, 2, 2).permute(1, 0, 2, 3)
    (torch.from_numpy(G).conj() * S).real.sum().backward()
    want = V.grad.numpy()
    assert np.max(np.abs(gv - want)) <= 1e-4 * np.max(np.abs(want))
    wa = torch.view_as_real(z.grad).reshape(n, 8).numpy()
    assert np.max(np.abs(gb - wa)) <= 1e-4 * np.max(np.abs(wa))
