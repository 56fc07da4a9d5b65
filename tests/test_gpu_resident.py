"""The resident scheme (grid on chip for every time step) against the FP64
solve, over the sizes where its split changes: one cluster with narrow and
wide rows, one or more tile columns, odd sizes, mailboxes between CTAs, tall
and flat grids. Its error may be at most twice that of one TMA launch per
step: both round about the same number of products and sums per point and
step, independently. (A fixed bound between the two would not do: traces
that the wave has not reached hold only its leading tail, 30 decades down,
where either is 1e-5 off.) Where luck makes the other's error small, an
error of 1e-6, the rounding of a hundred FP32 steps, passes as well."""
import numpy as np
import pytest

import psvwave_gb300 as psv

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def model(nx, nz, nt=120, npb=6, seed=0, shots=1, precision="fp32", near=False,
          column=False):
    nxi, nzi = nx - 2 * npb, nz - 2 * npb
    rng = np.random.default_rng(seed + 1000 * nx + nz)
    # Two sources of a shot at the same point: several terms per cell. Two
    # receivers share a cell.
    xs = [int(rng.integers(1, nxi - 1)) for _ in range(shots)]
    zs = [int(rng.integers(1, nzi - 1)) for _ in range(shots)]
    rx = [int(v) for v in rng.integers(0, nxi, 9)]
    rz = [int(v) for v in rng.integers(0, nzi, 9)]
    if near:  # where the wave of 120 steps arrives
        rx = [min(max(xs[0] + int(v), 0), nxi - 1) for v in rng.integers(-8, 9, 9)]
        rz = [min(max(zs[0] + int(v), 0), nzi - 1) for v in rng.integers(-8, 9, 9)]
    if column:
        rx, rz = [xs[0]] * 99, [int(v) for v in rng.permutation(nzi)[:99]]
    p = dict(nt=nt, nx_inner=nxi, nz_inner=nzi, nx_inner_boundary=1, nz_inner_boundary=1,
             dx=1.249, dz=1.3, dt=2.5e-4, np_boundary=npb, np_factor=0.05, scalar_rho=1500.0,
             scalar_vp=2000.0, scalar_vs=800.0, npx=1, npz=1, peak_frequency=90.0,
             source_timeshift=0.0, delay_cycles_per_shot=0, n_sources=2 * shots,
             ix_sources=[x for x in xs for _ in range(2)],
             iz_sources=[z for z in zs for _ in range(2)], moment_angles=[30.0, 75.0] * shots,
             which_source_to_fire_in_which_shot=[[2 * s, 2 * s + 1] for s in range(shots)],
             nr=len(rx) + 1,
             ix_receivers=rx + rx[:1], iz_receivers=rz + rz[:1], snapshot_interval=10)
    m = psv.fdModel.from_parameters(p, precision=precision)
    v = 1.0 + 0.1 * rng.random((3, nx, nz))
    m.set_parameter_fields(2000.0 * v[0], 800.0 * v[1], 1500.0 * v[2])
    return m


SIZES = [(20, 16), (17, 23), (68, 57), (64, 64), (64, 66), (250, 151), (129, 152), (130, 153),
         (96, 305), (31, 700), (400, 300), (401, 257), (611, 129), (700, 515)]


@pytest.mark.parametrize("nx,nz", SIZES)
def test_resident_forward_and_adjoint_are_as_accurate_as_per_step_launches(nx, nz):
    out = []
    for variant in ("two_kernel", "fused_tma", None):
        m = model(nx, nz, precision="fp64" if variant == "two_kernel" else "fp32")
        if variant == "fused_tma":
            m.kernel_variant = variant
        m.forward_simulate(0, True)
        fields = m.get_wavefields()
        m.calculate_l2_misfit()
        m.calculate_l2_adjoint_sources()
        m.reset_kernels()
        m.adjoint_simulate(0)
        out.append(m.get_synthetic_data() + fields + m.get_snapshots() + m.get_lame_kernels() +
                   m.get_wavefields())
    for exact, per_step, resident in zip(*out):
        if np.abs(exact).max() < 1e-36:
            continue  # traces ahead of the wave, below FP32's normal range
        assert rel(resident, exact) <= max(2 * rel(per_step, exact), 1e-6)


@pytest.mark.parametrize("nx,nz", [(68, 57), (250, 151), (400, 300)])
def test_resident_batch_equals_single_runs_bit_for_bit(nx, nz):
    # Whatever team a batch layout gives a member, the arithmetic is the same.
    models = [model(nx, nz, seed=s) for s in range(3)] + [model(nx + 31, nz - 7, seed=9)]
    ref = []
    for m in models:
        m.kernel_variant = "fused_cluster"
        m.forward_simulate(0, False)
        ref.append(m.get_synthetic_data())
        m.set_synthetic_data(*[np.zeros_like(a) for a in ref[-1]])
    b = psv.Batch()
    for m in models:
        b.add(m, 0)
    b.cluster = True
    for mask in (None, [True, False, True, True], None):
        b.set_active(mask)
        for _ in range(3):  # eager, graph capture, graph replay
            b.forward()
        for k, (m, r) in enumerate(zip(models, ref)):
            if mask is None or mask[k]:
                for a, c in zip(m.get_synthetic_data(), r):
                    assert np.array_equal(a, c)


def test_resident_run_in_pieces_equals_one_run(tmp_path, monkeypatch):
    # output_wavefields runs the loop in pieces of one and nine steps, each
    # starting from the fields the last one left.
    monkeypatch.chdir(tmp_path)
    for nx, nz in ((68, 57), (400, 300)):
        a, b = model(nx, nz, nt=60), model(nx, nz, nt=60)
        a.forward_simulate(0, False)
        b.forward_simulate(0, False, output_wavefields=True)
        for x, y in zip(a.get_synthetic_data() + a.get_wavefields(),
                        b.get_synthetic_data() + b.get_wavefields()):
            assert np.array_equal(x, y)


def test_resident_multi_shot_gradient_equals_serial_calls():
    a, b = model(260, 340, shots=2), model(260, 340, shots=2)
    for m in (a, b):
        m.set_observed_data(*[0.5 * np.ones_like(x) for x in m.get_observed_data()])
    a.run_model(False, True)
    for s in range(2):
        b.forward_simulate(s, True)
    b.calculate_l2_misfit()
    b.calculate_l2_adjoint_sources()
    b.reset_kernels()
    for s in range(2):
        b.adjoint_simulate(s)
    b.map_kernels_to_velocity()
    assert a.misfit == b.misfit
    assert np.array_equal(a.get_gradient_vector(), b.get_gradient_vector())


# One to four rows a thread, uneven tiles, the largest that fits and the first
# that does not.
SIZES_F64 = [(20, 16), (17, 23), (64, 66), (250, 151), (96, 305), (31, 700), (400, 300),
             (401, 430), (520, 600)]


@pytest.mark.parametrize("nx,nz", SIZES_F64)
def test_resident_fp64_equals_two_kernel_steps_bit_for_bit(nx, nz, tmp_path, monkeypatch):
    monkeypatch.chdir(tmp_path)
    out = []
    for variant in ("two_kernel", None, "pieces"):
        m = model(nx, nz, nt=70, precision="fp64")
        if variant == "two_kernel":
            m.kernel_variant = variant
        # Twice: eagerly and captured.
        for _ in range(2):
            m.forward_simulate(0, True, output_wavefields=variant == "pieces")
        assert m.kernel_variant == "two_kernel"
        fields = m.get_wavefields()
        m.calculate_l2_misfit()
        m.calculate_l2_adjoint_sources()
        m.reset_kernels()
        for _ in range(2):
            m.adjoint_simulate(0)
        out.append(m.get_synthetic_data() + fields + m.get_snapshots() + m.get_lame_kernels() +
                   m.get_wavefields())
    for steps, resident, pieces in zip(*out):
        assert np.array_equal(resident, steps) and np.array_equal(pieces, steps)


@pytest.mark.parametrize("nx,nz,shots", [(20, 16, 1), (17, 23, 3), (68, 57, 1), (64, 66, 2),
                                         (250, 151, 1), (250, 151, 5), (31, 700, 1),
                                         (400, 300, 1), (400, 300, 3), (401, 257, 2),
                                         (700, 515, 1), (900, 700, 1)])
def test_resident_exact_gradient_is_as_accurate_as_per_step_launches(nx, nz, shots):
    # Clusters and mailboxes, shots on shares of the device and one after the
    # other, one and several segments, a grid that only the forward steps hold.
    # Same criterion as above; sums in float-float pairs add nothing to it.
    out = []
    for variant, ck in (("fp64", 50), ("fused_tma", 50), (None, 50), (None, 0), (None, 7)):
        m = model(nx, nz, shots=shots, near=True, precision="fp64" if variant == "fp64" else "fp32")
        if variant == "fused_tma":
            m.kernel_variant = variant
        m.set_observed_data(*[np.zeros_like(a) for a in m.get_observed_data()])
        for _ in range(3 if variant is None else 1):  # eager, graph capture, graph replay
            misfit, g = m.exact_gradient(ck)
        out.append([np.array([misfit])] + list(g))
    for exact, per_step, resident, whole, sevenths in zip(*out):
        assert rel(resident, exact) <= max(2 * rel(per_step, exact), 1e-6)
        assert np.array_equal(resident, whole) and np.array_equal(resident, sevenths)


def test_resident_many_terms_in_one_tile():
    # A column of receivers, more than a helper warp has threads, whose adjoint
    # sources and their points fall into one tile.
    out = []
    for variant in ("fp64", "fused_tma", None):
        m = model(250, 151, precision="fp64" if variant == "fp64" else "fp32", column=True)
        if variant == "fused_tma":
            m.kernel_variant = variant
        m.set_observed_data(*[np.zeros_like(a) for a in m.get_observed_data()])
        m.run_model(False, True)
        out.append([m.get_gradient_vector()] + list(m.exact_gradient(50)[1]) +
                   list(m.get_lame_kernels()))
    for exact, per_step, resident in zip(*out):
        assert rel(resident, exact) <= max(2 * rel(per_step, exact), 1e-6)
