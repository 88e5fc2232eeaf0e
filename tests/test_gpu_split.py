"""The split-stage substep kernel against the plain kernel
at the sizes where its tiles, chunks and queues have their edges: one tile and
one cell more or less, chunks of a few planes, rows of the packed FP32 tile that
lie outside the mesh.  Both evaluate the same equations with their sums in
another order.

Tolerances: per step a field changes by at most dt |rate|, and the two sums of a
rate differ by at most a few hundred roundings (the terms of the stencils and of
the equations) of its largest term.  With dt |term| <= 0.05 max|f| here and
2 steps of 3 substeps, FP64 stays within 6 * 0.05 * 300 * 1.1e-16 < 1e-14 of
max|f|; FP32 rates within 6 * 0.05 * 300 * 6e-8 < 6e-6."""
import numpy as np
import pytest

from astaroth_b200 import capi
from astaroth_b200.device import CONFIG_PARAMS, Device, make_info, seeded_mesh

pytestmark = pytest.mark.gpu

AMP = dict(amp_scalar=1e-2, sigma_uu=3e-2, sigma_aa=3e-3)
SIZES = [(33, 4, 3), (35, 9, 7), (63, 8, 12), (125, 13, 9), (32, 4, 3), (32, 8, 8), (34, 7, 5), (62, 9, 4), (66, 16, 11), (96, 12, 37), (150, 13, 17)]


def run(n, precision, kernel, **params):
    info = make_info(n, precision=precision, **dict(CONFIG_PARAMS, **params))
    info.int_params[capi.IntParam.AC_debug_plain_kernel] = kernel
    f = seeded_mesh(info, 17, **AMP)
    with Device(info) as d:
        d.load_mesh(f)
        for _ in range(2):
            d.integrate_step(1e-3)
        d.synchronize()
        return d.store_mesh()[:, 3:-3, 3:-3, 3:-3].copy(), d.timestep_maxima(), d.timestep()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_split_kernel_equals_plain(n, precision):
    a, ma, _ = run(n, precision, 1)
    b, mb, _ = run(n, precision, 3)
    scale = np.abs(a).reshape(8, -1).max(axis=1)
    err = np.abs(a - b).reshape(8, -1).max(axis=1) / scale
    assert err.max() <= (1e-14 if precision == 0 else 6e-6), err
    np.testing.assert_allclose(ma, mb, rtol=1e-13 if precision == 0 else 6e-6)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(65, 6, 5), (34, 7, 5), (66, 16, 11), (150, 13, 17)])
def test_split_kernel_equals_plain_with_upwinding(n, precision):
    a, ma, _ = run(n, precision, 1, upwind=1)
    b, mb, _ = run(n, precision, 3, upwind=1)
    err = np.abs(a - b).reshape(8, -1).max(axis=1) / np.abs(a).reshape(8, -1).max(axis=1)
    assert err.max() <= (1e-14 if precision == 0 else 6e-6), err
    np.testing.assert_allclose(ma, mb, rtol=1e-13 if precision == 0 else 6e-6)


@pytest.mark.parametrize("n", [(40, 12, 19), (41, 12, 19)])
def test_z_boxes_of_any_size_give_the_same_bits(n):
    """Chunks start and end anywhere: the planes of a substep solved in uneven z boxes."""
    info = make_info(n, **CONFIG_PARAMS)
    info.int_params[capi.IntParam.AC_debug_plain_kernel] = 3
    f = seeded_mesh(info, 5, **AMP)
    out = []
    for cuts in ((0, 19), (0, 1, 3, 4, 11, 19), (0, 6, 13, 19)):
        with Device(info) as d:
            d.load_mesh(f)
            for s in range(3):
                d.periodic_boundconds()
                for z0, z1 in zip(cuts, cuts[1:]):
                    assert d.lib.acDeviceIntegrateSubstep(
                        d.handle, 0, s, capi.Volume(3, 3, 3 + z0),
                        capi.Volume(3 + n[0], 3 + n[1], 3 + z1), 1e-3) == 0
                d.swap_buffers()
            d.synchronize()
            out.append((d.store_mesh(), d.timestep_maxima()))
    for o, m in out[1:]:
        assert np.array_equal(o, out[0][0]) and m == out[0][1]


@pytest.mark.parametrize("precision,n", [(0, (37, 7, 40)), (0, (38, 7, 40)), (1, (38, 11, 40))])
def test_ragged_tiles_give_the_same_bits_every_time(precision, n):
    """Tiles that reach past the mesh in x and y, where the threads of a warp part at
    the loads, copies and stores of cells that the mesh does not have and have to be
    together again at the tensor-memory accesses that follow: planes by TMA and (odd
    nx) by the threads, with and without a previous state."""
    first, _, _ = run(n, precision, 3)
    for _ in range(10):
        again, _, _ = run(n, precision, 3)
        assert np.array_equal(again, first)


def test_fp32_laplacian_of_a_constant():
    """The FP32 coefficients of the Laplacians cancel on a constant as well as FP32 allows.

    A slow large-scale entropy profile about 1 under strong conduction, FP32-compensated
    against FP64: a rounding of a cell's Laplacian has either sign, so that over the mesh
    only what the coefficients leave of s itself is seen.  FP32 leaves at most half an ulp
    of the centre, 3 * 49/18 / ds^2 = 848 at 64^3 (half an ulp: 3.05e-5), times s <= 1.25;
    a rate is K exp(-lnrho) gamma/cp of it, with exp(-lnrho) <= 1.01 here.  Beside that,
    the mean of 64^3 roundings in 30 substeps: 8 roundings of up to 6e-8 * 848 each,
    / sqrt(64^3), is below 1e-6."""
    n, steps, dt, K = 64, 10, 5e-4, 0.05
    out = []
    for precision in (0, 1):
        info = make_info(n, precision=precision, **dict(CONFIG_PARAMS, K_heatcond=K))
        f = np.zeros_like(seeded_mesh(info, 1))
        x = (np.arange(n + 6) - 3) * (2 * np.pi / n)
        f[7] = 1.0 + 0.25 * np.sin(x)[None, None, :] * np.cos(x)[None, :, None] * np.cos(x)[:, None, None]
        with Device(info) as d:
            d.load_mesh(f)
            for _ in range(steps):
                d.integrate_step(dt)
            d.synchronize()
            out.append(d.store_mesh()[:, 3:-3, 3:-3, 3:-3].copy())
    drift = float((out[1][7] - out[0][7]).mean())
    rate = K * 1.01 * CONFIG_PARAMS["gamma"] / CONFIG_PARAMS["cp_sound"]
    assert abs(drift) <= steps * dt * rate * (3.05e-5 * 1.25 + 1e-6), drift


@pytest.mark.parametrize("n,upwind,split", [((33, 33, 33), 0, False), ((255, 12, 3), 0, False),
                                            ((49, 49, 49), 0, False), ((49, 49, 49), 1, True),
                                            ((35, 40, 100), 0, True), ((101, 64, 51), 0, True)])
def test_automatic_choice_for_odd_nx(n, upwind, split):
    """FP64 meshes with nx odd take the faster of the plain kernel (small meshes) and the
    split-stage kernel, in whole steps, calls of the loop and z boxes alike."""
    auto, _, _ = run(n, 0, 0, upwind=upwind)
    assert np.array_equal(auto, run(n, 0, 3 if split else 1, upwind=upwind)[0])
    assert not np.array_equal(auto, run(n, 0, 1 if split else 3, upwind=upwind)[0])
    info = make_info(n, **dict(CONFIG_PARAMS, upwind=upwind))
    with Device(info) as d:
        d.load_mesh(seeded_mesh(info, 17, **AMP))
        for _ in range(2):
            for s in range(3):
                d.periodic_boundconds()
                for z0, z1 in ((0, 2), (2, n[2])):
                    assert d.lib.acDeviceIntegrateSubstep(
                        d.handle, 0, s, capi.Volume(3, 3, 3 + z0),
                        capi.Volume(3 + n[0], 3 + n[1], 3 + z1), 1e-3) == 0
                d.swap_buffers()
        d.synchronize()
        assert np.array_equal(auto, d.store_mesh()[:, 3:-3, 3:-3, 3:-3])
