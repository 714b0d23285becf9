"""Device memory of a handle: the planes that its kind of run needs and no more,
so that the largest grids which fit stay those that fitted."""
import pytest

import phoenix_b200 as pb

pytestmark = pytest.mark.gpu

N_C, N_R = 2048, 1536
# ring of 8 on each side, rows padded to 32 points
PLANE = -(-(N_C + 16) // 32) * 32 * (N_R + 16)
NOISE = dict(stochastic_amplitude=1e-3)
# Planes of psi (two reals a point) and n, and of the inputs (pump, potential: one real;
# pulse: two).  State, two stage planes and an accumulator; the plain scalar
# iteration also has a second state plane.  SSFM: state and stage planes and the
# table of factors.
INPUTS = 1 + 1 + 2
KINDS = {
    "scalar": (dict(), 5 * 3 + INPUTS),
    "scalar_noise": (NOISE, 4 * 3 + INPUTS),
    "spinor": (dict(use_twin_mode=True), 2 * (4 * 3 + INPUTS)),
    "spinor_noise": (dict(use_twin_mode=True, **NOISE), 2 * (4 * 3 + INPUTS)),
    "ssfm": (dict(iterator="SSFM"), 3 * 3 + INPUTS + 2),
}


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("kind", list(KINDS))
def test_planes_of_a_handle(require_gpu, kind, dtype):
    import torch

    more, reals = KINDS[kind]

    def run(n_c, n_r):
        s = pb.Solver(pb.SystemParameters(N_c=n_c, N_r=n_r, L_x=100.0, L_y=100.0, periodic_boundary_x=True,
                                          periodic_boundary_y=True, dtype=dtype, dt=1e-3, t_max=1e12, fft_every=1e12,
                                          pump_temporal=[pb.Temporal()], potential_temporal=[pb.Temporal()], **more))
        s.run(2)
        torch.cuda.synchronize()
        return s

    run(64, 48).close()  # what the library itself loads once
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    with run(N_C, N_R):
        used = before - torch.cuda.mem_get_info()[0]
    # cuFFT's workspace (one copy) and the small buffers
    slack = (32 << 20) + (PLANE * 2 * (4 if dtype == "f32" else 8) if kind == "ssfm" else 0)
    assert used <= reals * PLANE * (4 if dtype == "f32" else 8) + slack
