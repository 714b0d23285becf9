"""The marching-warps RK4 iteration (launch shape 12): strips store 56 columns
(two points per lane), row segments end anywhere.  Against the stage kernels
(shape 2), bit for bit, and in the fused multiply-add arithmetic against the
tile kernels (shape 4)."""
import ctypes
import itertools

import numpy as np
import pytest

import bench as B
import phoenix_b200 as pb
from phoenix_b200 import _lib as L

pytestmark = pytest.mark.gpu

# columns around one and two strips (56, 112), the smallest grid, odd FP64
# widths; rows of one short segment and of several
SIZES = [(8, 8), (10, 9), (54, 37), (56, 12), (58, 140), (112, 35), (114, 301), (250, 97)]
ODD = [(9, 8), (55, 41), (57, 33), (113, 150)]


def run(n_c, n_r, dtype, px, py, shape, monkeypatch, res=True, pump=True, pot=True, temporal=False, fma=False, iters=5,
        plant=()):
    monkeypatch.setenv("PHX_STAGE_SHAPE", str(shape))
    rng = np.random.default_rng([n_c, n_r])
    T = pb.Temporal
    sp = pb.SystemParameters(N_c=n_c, N_r=n_r, L_x=0.3 * n_c, L_y=0.2 * n_r, **B.PHYS, periodic_boundary_x=px,
                             periodic_boundary_y=py, dtype=dtype, dt=0.01, t_max=1e12, fft_every=1e12, use_reservoir=res,
                             pump_temporal=[T("cos", 0.02, 0.05, 40.0) if temporal else T()] if pump and res else [],
                             potential_temporal=[T("gauss", 0.02, 0.05, 1.0) if temporal else T()] if pot else [], fma=fma)
    psi0 = rng.standard_normal((n_r, n_c)) + 1j * rng.standard_normal((n_r, n_c))
    for row, col, value in plant:
        psi0[row, col] = value
    with pb.Solver(sp) as s:
        s.set_field("psi_plus", psi0)
        if res:
            s.set_field("n_plus", rng.random((n_r, n_c)))
            if pump:
                s.set_field("pump_plus", 2.0 * rng.random((n_r, n_c)), 0)
        if pot:
            s.set_field("potential_plus", 0.3 * rng.standard_normal((n_r, n_c)), 0)
        info = s.run(iters)
        assert info.launch_shape == shape
        return [s.get_field("psi_plus")] + ([s.get_field("n_plus")] if res else [])


@pytest.mark.parametrize("px,py", list(itertools.product([True, False], repeat=2)))
@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_edges_of_strips_and_segments(require_gpu, monkeypatch, dtype, px, py):
    for n_c, n_r in SIZES + (ODD if dtype == "f64" else []):
        want = run(n_c, n_r, dtype, px, py, 2, monkeypatch)
        for a, b in zip(run(n_c, n_r, dtype, px, py, 12, monkeypatch), want):
            np.testing.assert_array_equal(a, b, err_msg=f"{n_c} x {n_r}")


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("res,pump,pot,temporal", [(False, False, False, False), (False, False, True, False),
                                                   (True, False, False, False), (True, True, False, False),
                                                   (True, False, True, False), (True, True, False, True),
                                                   (True, True, True, True), (False, False, True, True)])
def test_inputs_and_envelopes(require_gpu, monkeypatch, dtype, res, pump, pot, temporal):
    a = run(114, 70, dtype, True, False, 12, monkeypatch, res, pump, pot, temporal)
    b = run(114, 70, dtype, True, False, 2, monkeypatch, res, pump, pot, temporal)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


# without a potential nothing is multiplied by one: an infinite psi gives what the
# tile kernels (shape 4) make of it
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("temporal,pot", [(True, False), (False, False), (True, True)])
def test_infinite_psi(require_gpu, monkeypatch, dtype, temporal, pot):
    inf = ((10, 20, complex(np.inf, 1.0)), (50, 70, complex(0.0, -np.inf)))
    a = run(114, 70, dtype, True, False, 12, monkeypatch, True, True, pot, temporal, iters=1, plant=inf)
    b = run(114, 70, dtype, True, False, 4, monkeypatch, True, True, pot, temporal, iters=1, plant=inf)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("res,pot,temporal", [(True, True, False), (True, False, False), (True, True, True), (False, True, False)])
def test_fma_arithmetic(require_gpu, monkeypatch, res, pot, temporal):
    a = run(114, 70, "f32", True, True, 12, monkeypatch, res, True, pot, temporal, fma=True)
    b = run(114, 70, "f32", True, True, 4, monkeypatch, res, True, pot, temporal, fma=True)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


def general(n_c, n_r, dtype, px, py, monkeypatch, staged, tetm=False, pumps=1, pot=1, pulse=0, dw=0.0, iters=4, march=None,
            cell=1.0, plant=()):
    """march: PHX_GENERAL_MARCH (by default the rule between the marching and the tile
    kernels); plant: (field, row, column, value) set in the first group of the inputs."""
    monkeypatch.setenv("PHX_TETM_FUSED", "0" if staged else "1")
    monkeypatch.setenv("PHX_GENERAL_FUSED", "0" if staged else "1")
    if march is None:
        monkeypatch.delenv("PHX_GENERAL_MARCH", raising=False)
    else:
        monkeypatch.setenv("PHX_GENERAL_MARCH", march)
    T = pb.Temporal
    rng = np.random.default_rng([n_c, n_r, 3])
    sp = pb.SystemParameters(N_c=n_c, N_r=n_r, L_x=0.3 * n_c * cell, L_y=0.2 * n_r * cell, h_bar_s=0.6582, m_eff=0.5, gamma_c=0.2,
                             gamma_r=0.3, g_c=0.05, g_r=0.08, R=0.04, g_pm=-0.01, delta_LT=0.3, use_twin_mode=tetm,
                             periodic_boundary_x=px, periodic_boundary_y=py, dtype=dtype, dt=0.002 * cell ** 2, t_max=1e12,
                             fft_every=1e12, pump_temporal=[T(), T("cos", 0.004, 0.01, 200.0)][:pumps],
                             potential_temporal=[T("gauss", 0.004, 0.01, 1.0)] * pot,
                             pulse_temporal=[T("iexp", 0.004, 0.01, 50.0)] * pulse, stochastic_amplitude=dw, random_seed=11)
    comps = ("plus", "minus") if tetm else ("plus",)
    with pb.Solver(sp) as s:
        for c in comps:
            z = lambda: rng.standard_normal((n_r, n_c)) + 1j * rng.standard_normal((n_r, n_c))  # noqa: E731
            f = {("psi_", 0): z(), ("n_", 0): rng.random((n_r, n_c))}
            f.update({("pump_", g): 3.0 * rng.random((n_r, n_c)) for g in range(pumps)})
            f.update({("potential_", g): 0.3 * rng.standard_normal((n_r, n_c)) for g in range(pot)})
            f.update({("pulse_", g): z() for g in range(pulse)})
            for name, row, col, value in plant:
                if (name, 0) in f:
                    f[name, 0][row, col] = value
            for (name, g), v in f.items():
                s.set_field(name + c, v, g)
        info = s.run(iters)
        assert staged == (info.kernel_launches >= 4 * iters)
        return [s.get_field(f + c) for c in comps for f in ("psi_", "n_")]


# what a step's template parameters select, on grids around one and two strips;
# the scalar model without any of them is the plain iteration above
INPUTS = [(1, 1, 0, 0.02), (1, 0, 0, 0.02), (1, 1, 1, 0.0), (1, 0, 1, 0.02), (2, 1, 1, 0.0), (2, 0, 0, 0.02)]


@pytest.mark.parametrize("tetm,dtype,pumps,pot,pulse,dw",
                         [(False, d) + i for d in ("f32", "f64") for i in INPUTS] +
                         [(True, d) + i for d in ("f32", "f64") for i in INPUTS + [(1, 1, 0, 0.0)]])
def test_general_and_spinor_iterations(require_gpu, monkeypatch, tetm, dtype, pumps, pot, pulse, dw):
    sizes = [(8, 8, True, True), (56, 13, True, False), (114, 61, False, True), (114, 2461, True, True)]
    if dtype == "f64":  # odd widths: periodic images (with walls in x there are none)
        sizes += [(57, 49, False, False), (57, 33, True, True), (113, 40, True, False), (9, 8, True, True)]
    # the marching kernel whatever the grid, an error where it has no variant: FP64
    # spinors and spinors with two pump groups run the tile kernel
    march = "0" if tetm and (dtype == "f64" or pumps > 1) else "1"
    for n_c, n_r, px, py in sizes:
        want = general(n_c, n_r, dtype, px, py, monkeypatch, True, tetm, pumps, pot, pulse, dw)
        got = general(n_c, n_r, dtype, px, py, monkeypatch, False, tetm, pumps, pot, pulse, dw, march=march)
        for x, y in zip(got, want):
            np.testing.assert_array_equal(x, y, err_msg=f"{n_c} x {n_r}")


def test_forced_marching_kernel_refuses_what_it_has_no_variant_for(require_gpu, monkeypatch):
    with pytest.raises(pb.PhxError, match="PHX_GENERAL_MARCH"):
        general(56, 13, "f32", True, True, monkeypatch, False, pot=1, pulse=2, march="1")


# a run that diverges, from any input and from operations that overflow (|psi|^2,
# R n / dV): not finite where the stage kernels are not, the same values elsewhere
@pytest.mark.parametrize("tetm,dtype,pumps,pot,pulse,dw", [(False, "f32", 1, 1, 1, 0.02), (False, "f32", 2, 0, 0, 0.0),
                                                           (False, "f32", 1, 1, 1, 0.0), (True, "f32", 1, 1, 0, 0.02),
                                                           (True, "f32", 1, 1, 0, 0.0), (False, "f64", 1, 1, 0, 0.02),
                                                           (False, "f64", 2, 1, 1, 0.0)])
def test_values_that_are_not_finite(require_gpu, monkeypatch, tetm, dtype, pumps, pot, pulse, dw):
    inf, huge, big = float("inf"), 1e25 if dtype == "f32" else 1e160, 1e37 if dtype == "f32" else 1e307
    plant = [("psi_", 0, 0, inf), ("psi_", 20, 30, complex(0.5, -inf)), ("psi_", 20, 60, complex(inf, inf)),
             ("psi_", 20, 90, huge * (1 - 1j)), ("psi_", 40, 30, complex(float("nan"), 1.0)), ("n_", 40, 60, inf),
             ("n_", 40, 90, big), ("pump_", 60, 30, inf), ("potential_", 60, 60, inf), ("potential_", 60, 90, -inf)]
    for iters in (1, 2):
        args = (114, 80, dtype, True, False, monkeypatch)
        kind = dict(tetm=tetm, pumps=pumps, pot=pot, pulse=pulse, dw=dw, iters=iters, cell=0.1, plant=plant)
        want = general(*args, True, **kind)
        got = general(*args, False, march="1", **kind)
        assert all(np.isfinite(v).any() and not np.isfinite(v).all() for v in want)
        for x, y in zip(got, want):
            np.testing.assert_array_equal(np.isfinite(x), np.isfinite(y))
            np.testing.assert_array_equal(x[np.isfinite(x)], y[np.isfinite(y)])


# the rule between the marching and the tile kernels, on grids of either side: one
# tile, narrow and long, one round of tiles and several
@pytest.mark.parametrize("tetm,dtype,pot,pulse,dw", [(False, "f32", 1, 1, 0.0), (False, "f32", 0, 0, 0.02),
                                                     (True, "f32", 1, 0, 0.0), (True, "f32", 1, 1, 0.02),
                                                     (False, "f64", 0, 1, 0.0), (False, "f64", 1, 0, 0.02)])
def test_general_iterations_as_dispatched(require_gpu, monkeypatch, tetm, dtype, pot, pulse, dw):
    for n_c, n_r in [(8, 8), (24, 700), (64, 1000), (500, 444), (768, 770)]:
        want = general(n_c, n_r, dtype, True, False, monkeypatch, True, tetm, 1, pot, pulse, dw, iters=2)
        got = general(n_c, n_r, dtype, True, False, monkeypatch, False, tetm, 1, pot, pulse, dw, iters=2)
        for x, y in zip(got, want):
            np.testing.assert_array_equal(x, y, err_msg=f"{n_c} x {n_r}")


# the adjoint's vector-Jacobian kernels: strips of 56 columns, wrapping (even
# widths) and with periodic images (odd ones), and the tiles of small FP64 grids,
# against the four-launch form.
# FP64: the two differ in the order of a few sums, 1e-12 as in the adjoint's own
# tests; FP32: 5 iterations of some 100 rounded operations a stage, 2e-5.
@pytest.mark.parametrize("sweep", ["march", "tiles"])
@pytest.mark.parametrize("n_c,n_r,dtype,tol", [(8, 8, "f64", 1e-12), (57, 33, "f64", 1e-12), (56, 41, "f64", 1e-12),
                                               (113, 70, "f64", 1e-12), (114, 75, "f32", 2e-5), (58, 9, "f32", 2e-5)])
def test_adjoint_sweep(require_gpu, monkeypatch, n_c, n_r, dtype, tol, sweep):
    import torch

    monkeypatch.setenv("PHX_ADJOINT_SWEEP", sweep)
    rng = np.random.default_rng([n_c, n_r, 5])
    ct, rt = (torch.complex64, torch.float32) if dtype == "f32" else (torch.complex128, torch.float64)
    z = lambda: torch.tensor(rng.standard_normal((n_r, n_c)) + 1j * rng.standard_normal((n_r, n_c))).to(ct).cuda()  # noqa: E731
    r = lambda: torch.tensor(rng.random((n_r, n_c))).to(rt).cuda()  # noqa: E731
    psi0, n0, pump, pot, d_psi, d_n = z(), r(), r(), r(), z(), r()
    got = {}
    for stages in ("1", "0"):
        monkeypatch.setenv("PHX_ADJOINT_STAGES", stages)
        sp = pb.SystemParameters(N_c=n_c, N_r=n_r, L_x=0.3 * n_c, L_y=0.3 * n_r, **B.PHYS, periodic_boundary_x=True,
                                 periodic_boundary_y=True, dtype=dtype, dt=0.01, t_max=1e12, fft_every=1e12,
                                 pump_temporal=[pb.Temporal()], potential_temporal=[pb.Temporal()])
        with pb.Solver(sp) as s:
            s.set_field_tensor("pump_plus", pump)
            s.set_field_tensor("potential_plus", pot)
            s.set_field_tensor("psi_plus", psi0)
            s.set_field_tensor("n_plus", n0)
            s.adjoint_forward(5, 2)
            got[stages] = s.adjoint_backward(d_psi, d_n, want_potential=True)
    for a, b in zip(got["0"], got["1"]):
        assert float((a - b).norm() / b.norm()) <= tol


# What the backward rests on: stage values stored by the recompute (the marching
# warps' storing variant in shape 12, tiles in 4, TMA tiles in 10), from checkpoints
# that the marching iterations left without periodic images, for the sweep that needs
# none and the one that does; a second run on the same handle, and iterations before
# the first.  Odd FP64 widths keep their images everywhere.  Tolerances as above, FP32
# for 7 iterations instead of 5.
@pytest.mark.parametrize("shape", [12, 4, 10])
@pytest.mark.parametrize("n_c,n_r,dtype,res,sweep",
                         [(n_c, n_r, "f64", res, sweep) for sweep in ("march", "tiles")
                          for n_c, n_r, res in [(56, 41, True), (57, 33, True), (113, 70, False), (9, 8, True)]] +
                         [(58, 41, "f32", True, "march"), (114, 75, "f32", False, "march")])
def test_adjoint_recompute(require_gpu, monkeypatch, n_c, n_r, dtype, res, sweep, shape):
    import torch

    monkeypatch.setenv("PHX_STAGE_SHAPE", str(shape))
    monkeypatch.setenv("PHX_ADJOINT_SWEEP", sweep)
    rng = np.random.default_rng([n_c, n_r, 6])
    ct, rt = (torch.complex64, torch.float32) if dtype == "f32" else (torch.complex128, torch.float64)
    z = lambda: torch.tensor(rng.standard_normal((n_r, n_c)) + 1j * rng.standard_normal((n_r, n_c))).to(ct).cuda()  # noqa: E731
    r = lambda: torch.tensor(rng.random((n_r, n_c))).to(rt).cuda()  # noqa: E731
    psi0, n0, pump, pot, d_psi, d_n = z(), r(), r(), r(), z(), r()
    got = {}
    for stages in ("1", "0"):
        monkeypatch.setenv("PHX_ADJOINT_STAGES", stages)
        sp = pb.SystemParameters(N_c=n_c, N_r=n_r, L_x=0.3 * n_c, L_y=0.3 * n_r, **B.PHYS, periodic_boundary_x=True,
                                 periodic_boundary_y=True, dtype=dtype, dt=0.01, t_max=1e12, fft_every=1e12,
                                 use_reservoir=res, pump_temporal=[pb.Temporal()] if res else [],
                                 potential_temporal=[pb.Temporal()])
        with pb.Solver(sp) as s:
            s.set_field_tensor("potential_plus", pot)
            s.set_field_tensor("psi_plus", psi0)
            if res:
                s.set_field_tensor("pump_plus", pump)
                s.set_field_tensor("n_plus", n0)
            s.run(3)
            got[stages] = []
            for _ in range(2):
                s.adjoint_forward(7, 2)
                got[stages] += [g for g in s.adjoint_backward(d_psi, d_n if res else None, want_pump=res,
                                                              want_potential=True) if g is not None]
            got[stages].append(s.get_field_tensor("psi_plus"))
            assert s.run(1).launch_shape == shape
    tol = 2.8e-5 if dtype == "f32" else 1e-12
    assert len(got["0"]) == len(got["1"]) == (9 if res else 5)
    assert torch.equal(got["0"][-1], got["1"][-1])  # the forward run does not depend on any of this
    for a, b in zip(got["0"], got["1"]):
        assert float((a - b).norm() / b.norm()) <= tol


# complex envelopes hand an iteration to the stage kernels, which read the periodic
# images that the marching iterations before it left out; and back again
@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_stage_kernels_take_over_from_marching_iterations(require_gpu, monkeypatch, dtype):
    n_c, n_r, dt = 58, 33, 0.01
    t = (ctypes.c_double * 6)(0.0, 3.5 * dt, 3.6 * dt, 6.5 * dt, 6.6 * dt, 20 * dt)
    re = (ctypes.c_double * 6)(1.0, 1.0, 0.8, 0.8, 1.0, 1.0)
    im = (ctypes.c_double * 6)(0.0, 0.0, 0.5, 0.5, 0.0, 0.0)
    out = {}
    for shape in (12, 2):
        monkeypatch.setenv("PHX_STAGE_SHAPE", str(shape))
        rng = np.random.default_rng(7)
        sp = pb.SystemParameters(N_c=n_c, N_r=n_r, L_x=0.3 * n_c, L_y=0.2 * n_r, **B.PHYS, periodic_boundary_x=True,
                                 periodic_boundary_y=True, dtype=dtype, dt=dt, t_max=1e12, fft_every=1e12,
                                 pump_temporal=[pb.Temporal()], potential_temporal=[pb.Temporal()])
        with pb.Solver(sp) as s:
            L.check(s._lib.phx_set_temporal_table(s._h, L.ENVELOPE["potential"], 0, t, re, im, ctypes.c_int64(6)), s._h)
            s.set_field("psi_plus", rng.standard_normal((n_r, n_c)) + 1j * rng.standard_normal((n_r, n_c)))
            s.set_field("n_plus", rng.random((n_r, n_c)))
            s.set_field("pump_plus", 2.0 * rng.random((n_r, n_c)))
            s.set_field("potential_plus", 0.3 * rng.standard_normal((n_r, n_c)))
            launches = [s.run(1).kernel_launches for _ in range(10)]
            assert shape == 2 or (min(launches) == 1 and max(launches) >= 4 and launches[-1] == 1)
            out[shape] = [s.get_field("psi_plus"), s.get_field("n_plus")]
    for a, b in zip(out[12], out[2]):
        np.testing.assert_array_equal(a, b)
