"""The adjoint's far-field phase, in fixed point and (1e-5 um: k |c| = 7e6 rad) beyond its
range, over grids around the 32 lanes: the vector-Jacobian product of a random cotangent
against torch's FP64 autograd of the closed form, within 2e-3 of the largest gradient (the
adjoint's bar; at 1e-5 um the FP64 phase k |X| itself is good to 1e-4)."""
import numpy as np
import pytest
import torch

import abt_b200
from oracle import adjoint_ref as AR
from tests.helpers import outbeams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lam", [0.532, 1e-5])
@pytest.mark.parametrize("nt,nphi", [(7, 9), (16, 16), (33, 31)])
def test_random_cotangent(ctx, lam, nt, nphi):
    rng = np.random.default_rng(nt)
    k = 2 * abt_b200.PI_REF / lam
    n = 5
    # facets of a few radians across, near one another far from the origin
    tri = rng.normal(size=(n, 3, 3)) * (2.0 / k) + rng.normal(size=(n, 1, 3)) * (20.0 / k)
    verts = tri.reshape(-1, 3) + np.array([7.0, -5.5, 6.1])
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
    assert np.max(np.abs(gv - want)) <= 2e-3 * np.max(np.abs(want))
    wa = torch.view_as_real(z.grad).reshape(n, 8).numpy()
    assert np.max(np.abs(gb - wa)) <= 2e-3 * np.max(np.abs(wa))
