"""A 3-D right-hand side is as accurate for a flow along z as for the same flow turned to lie along x.

Diagonal products enter the divergence by their own wavenumber only, so what rounding does to the square
of a large velocity does not reach modes that do not vary along it: the large u_z^2 of a jet along z, or
of one of two crossing shear layers, has no part in the smaller components' equations.  Any other form
of the products (a multiple of the identity taken off them, say) is the same in exact arithmetic only.
Each flow's error against the oracle may be 1.5 times that of the turned flow, four times in FP64, where
the oracle's own rounding is as large: the two are the same computation with the axes exchanged, whose
errors are of one size but not the same.  FP32 right-hand sides also stay within 1e-5 or twice the oracle's
single-precision evaluation.
"""

import numpy as np
import pytest
import torch

import azeban_b200 as az
from oracle import euler_oracle as ora
from tests.gpu_helpers import VISC_CFGS, random_field_hat, rel_l2, to_dev, to_host

pytestmark = pytest.mark.gpu


def _jet(N, a):
    """u_z(x, y) of amplitude 1 and an in-plane flow of amplitude a, both invariant along z."""
    flat = ora.fft_backward(random_field_hat(2, N, seed=60 + N, slope=1.0), N)
    along = np.random.default_rng(61 + N).standard_normal((N, N))
    k = np.hypot(ora.signed_index(N)[:, None], np.arange(N // 2 + 1)[None, :])
    along = np.fft.irfft2(np.fft.rfft2(along) / (1.0 + k), s=(N, N))
    u = np.stack([a * flat[0] / np.abs(flat).max(), a * flat[1] / np.abs(flat).max(), along / np.abs(along).max()])
    return np.repeat(u[..., None], N, axis=3)


def _crossing(N, a):
    """Two shear layers that cross: u_x(z) of amplitude a and u_z(x) of amplitude 1."""
    x = np.arange(N) / N
    layer = np.where(x <= 0.5, np.tanh((x - 0.25) / 0.05), np.tanh((0.75 - x) / 0.05))
    u = np.zeros((3, N, N, N))
    u[0] = a * layer[None, None, :]
    u[2] = np.roll(layer, N // 7)[:, None, None]
    return u


def _turned(u):
    """The same flow with z, x, y in the places of x, y, z."""
    return np.stack([np.transpose(u[c], (2, 0, 1)) for c in (2, 0, 1)])


FLOWS = [(_jet, 0.3), (_jet, 0.03), (_jet, 0.01), (_crossing, 0.1), (_crossing, 0.01)]
CASES = [(N, M, flow, a) for N, M in ((32, 48), (42, 64), (64, 96)) for flow, a in FLOWS] + [(20, 384, _jet, 0.03)]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("N,M,flow,a", CASES)
def test_flow_along_z_like_along_x(N, M, flow, a, prec):
    og, g = ora.Grid(3, N, M), az.Grid(3, N, M)
    oeq = ora.IncompressibleEuler(og, ora.make_viscosity(VISC_CFGS["none"], og))
    eq = az.IncompressibleEuler(g, az.make_viscosity(VISC_CFGS["none"], g), prec)
    err = []
    for u in (flow(N, a), _turned(flow(N, a))):
        d_u = to_dev(ora.leray(ora.fft_forward(u)), prec)
        u_hat = to_host(d_u)  # as the solver has it
        d_out = torch.empty_like(d_u)
        eq.dudt(d_out, d_u)
        ref = oeq.dudt(u_hat)
        err.append(rel_l2(to_host(d_out), ref))
        if prec == "f32":
            assert err[-1] <= max(1e-5, 2.0 * rel_l2(oeq.dudt_single(u_hat), ref)), err
        else:
            assert err[-1] <= 1e-12, err
    assert err[0] <= (4.0 if prec == "f64" else 1.5) * err[1], err
