"""Parity of every tuned variant of the right-hand side with the CPU oracle, and of layouts and sizes
that take other paths through the passes.

A variant is a radix plan (0 std, 1 wide): of the last pass of 3-D solves (kind 2) and, at a padded length
of 384, of their column passes (kind 0).  The tuning table picks one per (precision, length, kind); these
tests pin each one against the oracle, so a table entry can never select a kernel whose results differ.
The other passes have one form per length.  Tolerances as in test_gpu_euler.py.
"""

import ctypes as ct

import numpy as np
import pytest
import torch

import azeban_b200 as az
from azeban_b200 import _lib
from oracle import euler_oracle as ora
from tests.gpu_helpers import VISC_CFGS, random_field_hat, rel_l2, to_dev, to_host

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "f32": 1e-5}


class _Variants:
    """Sets the tuning table entries of one (precision, length) for 3-D solves
    and restores the previous ones on exit."""

    def __init__(self, prec, L, cols, epi):
        self.p = 0 if prec == "f64" else 1
        self.L = L
        self.want = {0: cols, 2: epi}

    def __enter__(self):
        self.saved = {}
        for kind, v in self.want.items():
            old = ct.c_int()
            _lib.check(_lib.lib.az_tune_get(self.p, self.L, kind, ct.byref(old)))
            self.saved[kind] = old.value
            _lib.check(_lib.lib.az_tune_set(self.p, self.L, kind, v))
        return self

    def __exit__(self, *exc):
        for kind, v in self.saved.items():
            _lib.check(_lib.lib.az_tune_set(self.p, self.L, kind, v))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("N,M,cols,epi", [(16, 24, 0, 0), (16, 24, 0, 1), (32, 48, 0, 0), (32, 48, 0, 1), (34, 64, 0, 0),
                                          (34, 64, 0, 1), (64, 96, 0, 0), (64, 96, 0, 1), (24, 384, 0, 0),
                                          (24, 384, 1, 1), (256, 384, 1, 0)])
def test_dudt_every_variant(prec, N, M, cols, epi):
    """Both plans of the 3-D last pass, and at M = 384 of the column passes, in both forms of the padding
    (a right-hand side with M >= 2 N + 2 does not depend on M, so the oracle takes a smaller one)."""
    og, g = ora.Grid(3, N, min(M, 2 * N + 16) if M > 128 and N < 128 else M), az.Grid(3, N, M)
    oeq = ora.IncompressibleEuler(og, ora.make_viscosity(VISC_CFGS["smooth"], og))
    u_hat = random_field_hat(3, N, seed=330 + N)
    ref = oeq.dudt(u_hat)
    with _Variants(prec, M, cols, epi):
        eq = az.IncompressibleEuler(g, az.make_viscosity(VISC_CFGS["smooth"], g), prec)
        d_u = to_dev(u_hat, prec)
        d_out = torch.empty_like(d_u)
        eq.dudt(d_out, d_u, 0.0, 0.0, 0.2)
        got = to_host(d_out)
        dt = eq.dt(0.2)
    assert rel_l2(got, ref) <= TOL[prec]
    if og.N_phys_pad == M:  # the largest velocity is that of the padded grid's points
        rel_dt = 1e-13 if prec == "f64" else 1e-6
        assert abs(dt - oeq.dt(0.2)) <= rel_dt * oeq.dt(0.2)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dim,N,M", [(2, 32, 48), (2, 64, 96), (2, 128, 192), (2, 256, 384), (3, 16, 24),
                                     (3, 32, 48), (3, 64, 96), (3, 34, 384), (2, 34, 768)])
def test_dudt_product_pass_sizes(prec, dim, N, M):
    """The product pass (k_zfused in 3-D at M = 384, else k_zline) under the 3/2 rule and under heavy
    padding (M = 384 and 768 with few retained rows), with the step size from its maximum."""
    og = ora.Grid(dim, N, M)
    g = az.Grid(dim, N, M)
    oeq = ora.IncompressibleEuler(og, ora.make_viscosity(VISC_CFGS["smooth"], og))
    u_hat = random_field_hat(dim, N, seed=900 + 10 * dim + N)
    ref = oeq.dudt(u_hat)
    eq = az.IncompressibleEuler(g, az.make_viscosity(VISC_CFGS["smooth"], g), prec)
    d_u = to_dev(u_hat, prec)
    d_out = torch.empty_like(d_u)
    eq.dudt(d_out, d_u, 0.0, 0.0, 0.2)
    got = to_host(d_out)
    dt = eq.dt(0.2)
    assert rel_l2(got, ref) <= TOL[prec]
    rel_dt = 1e-13 if prec == "f64" else 1e-6
    assert abs(dt - oeq.dt(0.2)) <= rel_dt * oeq.dt(0.2)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dim,N,M,B", [(2, 32, 48, 7), (3, 16, 24, 3), (3, 20, 384, 2)])
def test_batch_members_match_single(prec, dim, N, M, B):
    """Each member of a batch equals the same solve alone, bit for bit, over a
    short simulate_until.  Members have different amplitudes, so they finish at
    different steps and the skip flags are exercised."""
    g = az.Grid(dim, N, M)
    v = az.make_viscosity(VISC_CFGS["smooth"], g)
    fields = [random_field_hat(dim, N, seed=900 + b) * (1.0 + 0.5 * b) for b in range(B)]
    eqB = az.IncompressibleEuler(g, v, prec, batch=B)
    simB = az.Simulation(g, 0.2, az.SSP_RK3(eqB), to_dev(np.stack(fields), prec))
    simB.simulate_until(0.02)
    outB = to_host(simB.u())
    _, nB, _ = simB.state()
    for b in range(B):
        eq1 = az.IncompressibleEuler(g, v, prec)
        sim1 = az.Simulation(g, 0.2, az.SSP_RK3(eq1), to_dev(fields[b], prec))
        sim1.simulate_until(0.02)
        assert sim1.state()[1][0] == nB[b]
        np.testing.assert_array_equal(to_host(sim1.u()), outB[b])


@pytest.mark.parametrize("mask", [0, 5, 10, 15])
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dim,N", [(2, 64), (3, 16), (3, 32)])
def test_dudt_every_row_padding(mask, prec, dim, N, monkeypatch):
    """The intermediates' rows may be padded to whole 128-byte lines
    (AZ_PAD_MASK bits: A1, A2, B1, B2); every combination gives the oracle's
    right-hand side, including the grouped column paths of the inverse x pass
    and the epilogue."""
    monkeypatch.setenv("AZ_PAD_MASK", str(mask))
    og = ora.Grid(dim, N)
    g = az.Grid(dim, N)
    oeq = ora.IncompressibleEuler(og, ora.make_viscosity(VISC_CFGS["smooth"], og))
    u_hat = random_field_hat(dim, N, seed=500 + N)
    ref = oeq.dudt(u_hat)
    eq = az.IncompressibleEuler(g, az.make_viscosity(VISC_CFGS["smooth"], g), prec)
    d_u = to_dev(u_hat, prec)
    d_out = torch.empty_like(d_u)
    eq.dudt(d_out, d_u)
    assert rel_l2(to_host(d_out), ref) <= TOL[prec]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dim,N,M", [(3, 34, 384), (2, 34, 768)])
def test_dudt_heavy_padding(prec, dim, N, M):
    """Heavy padding (M far above 3N/2): narrow epilogue tiles of a few mode
    columns, a partial last tile (N = 34 gives odd tile counts), and zero rows
    filling most of every padded line."""
    og = ora.Grid(dim, N, M)
    g = az.Grid(dim, N, M)
    oeq = ora.IncompressibleEuler(og, ora.make_viscosity(VISC_CFGS["smooth"], og))
    u_hat = random_field_hat(dim, N, seed=700 + 10 * dim + N)
    ref = oeq.dudt(u_hat)
    eq = az.IncompressibleEuler(g, az.make_viscosity(VISC_CFGS["smooth"], g), prec)
    d_u = to_dev(u_hat, prec)
    d_out = torch.empty_like(d_u)
    eq.dudt(d_out, d_u, 0.0, 0.0, 0.2)
    assert rel_l2(to_host(d_out), ref) <= TOL[prec]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("epi", [0, 1])
@pytest.mark.parametrize("N,M", [(16, 768), (16, 1536)])
def test_long_line_last_pass_variants(prec, N, M, epi):
    """Both plans of the 3-D last pass at the longest lines, where its tiles
    are a few modes, against the oracle on a small padded grid."""
    og, g = ora.Grid(3, N, 36), az.Grid(3, N, M)
    oeq = ora.IncompressibleEuler(og, ora.make_viscosity(VISC_CFGS["smooth"], og))
    u_hat = random_field_hat(3, N, seed=903 + N)
    with _Variants(prec, M, 0, epi):
        eq = az.IncompressibleEuler(g, az.make_viscosity(VISC_CFGS["smooth"], g), prec)
        d_u = to_dev(u_hat, prec)
        d_out = torch.empty_like(d_u)
        eq.dudt(d_out, d_u, 0.0, 0.0, 0.2)
    assert rel_l2(to_host(d_out), oeq.dudt(u_hat)) <= TOL[prec]
